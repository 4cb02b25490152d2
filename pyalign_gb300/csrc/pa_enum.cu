// The first k optimal alignments of every pair of an all-optimal result, enumerated on the
// device (sm_103a).
//
// The reference yields all optimal alignments of a pair one at a time from a depth-first
// search over the traceback lists (TracebackIterators<true>::Iterator::next,
// solver.h:1647-1716): a LIFO stack of (u, v, path length) entries, seeded with the one
// optimum of Global/Semiglobal or, for local alignment, every cell equal to a strictly
// positive optimum pushed in reverse scan order (solver.h:2060-2091); popping an entry
// truncates the path to its length and appends its point; a point with both coordinates
// >= 0 that continues (local: its value is not 0) pushes its traceback list in stored order
// -- the zero candidate, the diagonal, then the P list (the rows where the vertical gap was
// opened, scanned up its column while the gap extends) and the Q list (solver.h:1328-1369,
// 2995-3016), or one terminal entry when the list is empty -- and any other point ends a
// path, which is yielded unless de-duplication (remove_dup) has already yielded the same
// compressed path (CompressedPath, solver.h:730-760).
//
// enum_kernel runs exactly that search, one warp per pair, over the all-optimal masks the
// DP wrote (pa_dp.cuh layout: stripe q, step s, lane k, one uint4 of 8 rows of 16-bit cells).
// The control flow is warp-uniform: every lane follows the same search, lane 0 alone reads
// and writes the stack and the path (so it always sees its own writes), and the lanes
// cooperate where the work is wide -- a 64-row x 64-column window of mask cells loaded into
// shared memory (one uint4 per lane and row block; the search walks up and left, so a
// diagonal path reloads it every 64 steps), and at each yielded path the compression, the
// map (s_to_t or t_to_s, the reference's build_alignment from the compressed points,
// solver.h:940-1086) and the de-duplication test, 32 path points per lane step.  The last
// entry a point pushes is the next one popped, so it stays in registers and only the others
// are written to the stack.  Most cells of a path have the diagonal as their only entry: from
// every cell the lanes test the 32 cells up its diagonal at once (one ballot), and a run of such
// cells is appended to the path in one step; only the cells that branch go through the search, and
// the openings of a gap are looked for 32 cells at a time as well.
// What bounds it then is round trips: one per window and, per yielded path, those of reading the
// path back, 256 points in flight together.  A yield differs from the one before it only past
// the point where the search turned, mostly near the path's end: with the pair's current map in
// shared memory (pairs of up to ENUM_SMEM_MAP) only that part of map and hash is worked out.  The
// stack's lower 256 entries lie there too.  16 pairs of 2000..3000 x 3000..5000, the first 101
// alignments of each: 9.66 -> 2.14 ms.  Local seeds come from enum_seed_kernel (every cell with the
// seed bit, one block per pair), sorted on the host in the order the reference's stack
// pops them: increasing row, then increasing column.
//
// De-duplication: the compressed points of a path decrease strictly in both coordinates,
// so two compressed paths are equal exactly when their maps are.  Each yielded map carries
// a 64-bit order-free hash and its point count; a new path is compared in full with every
// earlier yield of equal hash and count, so the test is exact.
//
// Bounded memory: the stack of a pair has a fixed capacity; a pair that would exceed it
// stops, flags ENUM_OVERFLOW and is enumerated again from the start with a larger stack by
// the host.  The seed lists are sized the same way (the scan counts every seed).
#include "pa_dp.cuh"
#include "pa_enum.h"

namespace pa {

// every cell of a pair with the local seed bit (256), in any order
__global__ void __launch_bounds__(256) enum_seed_kernel(SeedScanParams p) {
	for (int w = blockIdx.x; w < p.nwork; w += gridDim.x) {
		const int L = p.work[w];
		const int ls = p.len_s[L], lt = p.len_t[L];
		if (ls == 0 || lt == 0) continue;
		const int G = p.G, rpp = G * R, lg = __ffs(G) - 1;  // G is a power of two
		const int64_t S = int64_t(lt) + G - 1, per = S * G;
		const int npass = (ls + rpp - 1) / rpp;
		const uint4 *m = p.masks + p.mask_off[L];
		int2 *out = p.seeds + p.seed_off[L];
		const int cap = p.seed_cap[L];
		for (int q = 0; q < npass; q++)
		for (int64_t e = threadIdx.x; e < per; e += blockDim.x) {
			const int k = int(e & (G - 1));
			const int64_t s = e >> lg;
			const int64_t j = s - k;
			const int i0 = q * rpp + k * R;
			if (j < 0 || j >= lt || i0 >= ls) continue;
			const uint4 c = m[int64_t(q) * per + e];
			const uint32_t wv[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
			for (int r = 0; r < R; r++) {
				if (i0 + r >= ls) break;
				if ((wv[r >> 1] >> (16 * (r & 1))) & 256u) {
					const int x = atomicAdd(&p.seed_n[L], 1);
					if (x < cap) out[x] = make_int2(i0 + r, int(j));
				}
			}
		}
	}
}

constexpr int WIN_B = 8;    // row blocks (of 8 rows) and columns of a warp's window: the searches of
constexpr int WIN_C = 64;   // neighbouring yields differ near the path's end and mostly stay inside
constexpr int SMEM_STACK = 256;  // entries of the stack kept in shared memory

struct Window {
	int gb0, j0;  // row blocks [gb0, gb0 + WIN_B), columns [j0, j0 + WIN_C)
};

// the warp's shared window loaded from row block w.gb0 and column w.j0 on.  Not inlined: the search
// of a single warp waits for instructions as for everything else, so its code is kept small.
__device__ __noinline__ void enum_load(uint4 (*win)[WIN_C], Window w, const uint4 *m, int64_t S, int lg, int ls, int lt,
                                       int lane) {
	__syncwarp();  // every lane is done with the old window
	uint4 x[WIN_B][2];  // every load in flight together
#pragma unroll
	for (int r = 0; r < WIN_B; r++) {
		const int g = w.gb0 + r, q = g >> lg, sb = g & ((1 << lg) - 1);  // G = 2^lg
#pragma unroll
		for (int h = 0; h < 2; h++) {
			const int jj = w.j0 + lane + 32 * h;
			if (jj < lt && g * R < ls) x[r][h] = m[((int64_t(q) * S + jj + sb) << lg) + sb];
		}
	}
#pragma unroll
	for (int r = 0; r < WIN_B; r++)
#pragma unroll
		for (int h = 0; h < 2; h++)
			if (w.j0 + lane + 32 * h < lt && (w.gb0 + r) * R < ls) win[r][lane + 32 * h] = x[r][h];
	__syncwarp();
}

// the window moved so that it holds cell (i, j) (warp-uniform)
__device__ __forceinline__ void enum_place(uint4 (*win)[WIN_C], Window &w, const uint4 *m, int64_t S, int lg, int ls,
                                           int lt, int i, int j, int lane) {
	const int gb = i >> 3;
	if (gb >= w.gb0 && gb < w.gb0 + WIN_B && j >= w.j0 && j < w.j0 + WIN_C) return;
	w.gb0 = max(0, gb - (WIN_B - 1));
	w.j0 = max(0, j - (WIN_C - 1));
	enum_load(win, w, m, S, lg, ls, lt, lane);
}

// this lane's cell (i, j) where the window holds it -- it lies up and left of a cell that the
// window holds -- and `in` says so
__device__ __forceinline__ uint32_t enum_look(uint4 (*win)[WIN_C], const Window &w, int i, int j, bool &in) {
	in = i >= 0 && j >= 0 && (i >> 3) >= w.gb0 && j >= w.j0;
	if (!in) return 0u;
	const uint32_t *e = reinterpret_cast<const uint32_t *>(&win[(i >> 3) - w.gb0][j - w.j0]);
	return (e[(i & 7) >> 1] >> (16 * (i & 1))) & 0xffffu;
}

__device__ __forceinline__ unsigned long long enum_mix(int u, int v) {
	// splitmix64 finaliser of the point: an order-free sum of these hashes a point set
	unsigned long long x = (static_cast<unsigned long long>(static_cast<uint32_t>(u)) << 32) | static_cast<uint32_t>(v);
	x += 0x9e3779b97f4a7c15ull;
	x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
	x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
	return x ^ (x >> 31);
}

// SM: the pair's current map is kept in shared memory (p.smem_map entries).  A block of one warp.
template <bool SM>
__global__ void __launch_bounds__(32) enum_kernel(EnumParams p) {
	__shared__ uint4 win[WIN_B][WIN_C];
	__shared__ int4 top[SMEM_STACK];  // stack entries 0 .. SMEM_STACK - 1 (the others in p.stack)
	extern __shared__ int32_t smap[];
	const int lane = threadIdx.x & 31;
	const int wi = blockIdx.x;
	const int L = p.work[wi];
	const int ls = p.len_s[L], lt = p.len_t[L];
	const int m = min(ls, lt);
	const bool s_side = ls <= lt;  // the map is s_to_t, else t_to_s
	const int64_t S = int64_t(lt) + p.G - 1;
	const uint4 *mk = p.masks + p.mask_off[L];
	int4 *stk = p.stack + p.stack_off[L];
	const int cap = p.stack_cap[L];
	int2 *path = p.path + p.path_off[L];
	int32_t *maps = p.maps + p.map_off[L];
	unsigned long long *hash = p.hash + int64_t(L) * p.k;
	int32_t *npts = p.npts + int64_t(L) * p.k;
	const int plen_cap = ls + lt + 2;
	Window w{-WIN_B, -WIN_C};
	const int lg = __ffs(p.G) - 1;

	int count = 0, sp = 0, si = 0, status = 0;
	const int nseed = p.local ? p.seed_n[L] : 0;
	const int2 *seeds = p.local ? p.seeds + p.seed_off[L] : nullptr;
	bool have = false;
	int eu = 0, ev = 0, epl = 0;
	if (p.resume) {
		const EnumState from = p.state[L];
		have = from.have;
		eu = from.u;
		ev = from.v;
		epl = from.path_len;
		sp = from.sp;
		si = from.si;
		count = from.count;
		for (int x = lane; x < min(sp, SMEM_STACK); x += 32) top[x] = stk[x];
		__syncwarp();
	} else if (!p.local && p.has[L]) {
		eu = p.seed[2 * L];
		ev = p.seed[2 * L + 1];
		have = true;
	}
	// De-duplication makes the search as long as the pair has paths, however few alignments they
	// spell (30 letters against 30 others without gap costs: 10^17 paths, one alignment), so a launch
	// stops after p.cycles and the host launches it again, or not.
	const long long begun = clock64();
	bool paused = false;
	// path points 0 .. low - 1 are those of the last complete path; its hash and point count
	int low = 0, n = 0;
	unsigned long long h = 0;
	if (SM)
		for (int x = lane; x < m; x += 32) smap[x] = -1;
	while (count < p.k) {
		if (!have) {
			if (sp > 0) {
				int4 t = make_int4(0, 0, 0, 0);
				sp--;
				if (sp < SMEM_STACK) {
					__syncwarp();  // lane 0's write of it
					t = top[sp];
				} else if (lane == 0) {
					t = stk[sp];
				}
				eu = __shfl_sync(0xffffffffu, t.x, 0);
				ev = __shfl_sync(0xffffffffu, t.y, 0);
				epl = __shfl_sync(0xffffffffu, t.z, 0);
			} else if (si < nseed) {
				const int2 s = seeds[si++];
				eu = s.x;
				ev = s.y;
				epl = 0;
			} else {
				break;  // exhausted
			}
		}
		have = false;
		low = min(low, epl);
		int plen = epl;
		if (plen >= plen_cap) {  // cannot happen: every step lowers u + v
			status = ENUM_BAD_PATH;
			break;
		}
		bool cont = eu >= 0 && ev >= 0;
		uint32_t c = 0;
		if (cont) {
			enum_place(win, w, mk, S, lg, ls, lt, eu, ev, lane);
			// lane k: cell (eu - k, ev - k), while it lies in the window and its list is the diagonal
			const int i = eu - lane, j = ev - lane;
			bool in;
			c = enum_look(win, w, i, j, in);
			const uint32_t b = __ballot_sync(0xffffffffu, in && (c & 15u) == 2u);
			c = __shfl_sync(0xffffffffu, c, 0);
			const int run = min(b == 0xffffffffu ? 32 : __ffs(int(~b)) - 1, plen_cap - plen);
			if (run > 0) {
				__syncwarp();  // and may overwrite points of an earlier path
				if (lane < run) path[plen + lane] = make_int2(i, j);
				__syncwarp();  // a later path may overwrite these points from other lanes
				eu -= run;
				ev -= run;
				epl = plen + run;
				have = true;
				continue;
			}
			if (p.local && (c & 1u)) cont = false;
		}
		if (lane == 0) path[plen] = make_int2(eu, ev);
		plen++;
		if (cont) {
			// the list in push order; every entry but the last goes to the stack, the last is
			// popped next and stays in registers
			int nu = ENUM_NO_TB, nv = ENUM_NO_TB;
			bool pend = false;
			bool over = false;
			auto add = [&](int u, int v) {
				if (pend) {
					if (sp >= cap) over = true;
					else {
						if (lane == 0) (sp < SMEM_STACK ? top[sp] : stk[sp]) = make_int4(nu, nv, plen, 0);
						sp++;
					}
				}
				nu = u;
				nv = v;
				pend = true;
			};
			// the cells up the column (left along the row) where a gap that ends here may have been
			// opened: from (eu, ev) on while the cell's extend bit is set, 32 cells a look
			auto gap_list = [&](bool up, uint32_t open_bit, uint32_t extend_bit, int k) {
				const int u0 = eu, v0 = ev;
				for (;;) {
					enum_place(win, w, mk, S, lg, ls, lt, up ? k : u0, up ? v0 : k, lane);
					bool in;
					const uint32_t x = enum_look(win, w, up ? k - lane : u0, up ? v0 : k - lane, in);
					const uint32_t go = __ballot_sync(0xffffffffu, in && (x & extend_bit) && k - lane > 0);
					const uint32_t seen = __ballot_sync(0xffffffffu, in);
					const int n = go == 0xffffffffu ? 32 : __ffs(int(~go)) - 1;  // cells the gap goes on from
					const bool ends = n < 32 && ((seen >> n) & 1u);              // it ends at cell n, in the window
					const uint32_t upto = n + ends >= 32 ? 0xffffffffu : (1u << (n + ends)) - 1u;
					uint32_t opens = __ballot_sync(0xffffffffu, (x & open_bit) != 0) & upto;
					for (; opens; opens &= opens - 1) {
						const int m = k - (__ffs(int(opens)) - 1) - 1;
						add(up ? m : u0, up ? v0 : m);
					}
					if (ends) break;
					k -= n;
				}
			};
			// both gaps' first 16 cells in one look: lanes 0-15 up the column, 16-31 left along the row
			uint32_t go2 = 0, open2 = 0, seen2 = 0;
			if (p.affine && (c & 12u)) {
				const int k = lane & 15;
				const bool up = lane < 16;
				bool in;
				const uint32_t x = enum_look(win, w, up ? eu - k : eu, up ? ev : ev - k, in);
				go2 = __ballot_sync(0xffffffffu, in && (x & (up ? 32u : 128u)) && (up ? eu : ev) - k > 0);
				open2 = __ballot_sync(0xffffffffu, (x & (up ? 16u : 64u)) != 0);
				seen2 = __ballot_sync(0xffffffffu, in);
			}
			auto near_list = [&](bool up) {
				const uint32_t go = (up ? go2 : go2 >> 16) & 0xffffu, seen = up ? seen2 : seen2 >> 16;
				const int n = __ffs(int(~go)) - 1;  // at most 16
				const bool ends = n < 16 && ((seen >> n) & 1u);
				uint32_t opens = (up ? open2 : open2 >> 16) & ((1u << (n + ends)) - 1u);
				for (; opens; opens &= opens - 1) {
					const int m = __ffs(int(opens));
					add(up ? eu - m : eu, up ? ev : ev - m);
				}
				if (!ends) gap_list(up, up ? 16u : 64u, up ? 32u : 128u, (up ? eu : ev) - n);
			};
			if (c & 1u) add(ENUM_NO_TB, ENUM_NO_TB);
			if (c & 2u) add(eu - 1, ev - 1);
			if (c & 4u) {
				if (p.affine) {
					near_list(true);
				} else {
					add(eu - 1, ev);
				}
			}
			if (c & 8u) {
				if (p.affine) {
					near_list(false);
				} else {
					add(eu, ev - 1);
				}
			}
			if (over) {
				status = ENUM_OVERFLOW;
				break;
			}
			eu = nu;
			ev = nv;
			epl = plen;
			have = true;
			continue;
		}

		// ---- a complete path: path[0, plen).  Its map, hash and point count.  With the map in
		// shared memory only what differs from the last complete path is worked out: the points
		// from low - 1 on, whose map entries are those at or below that point's coordinate (a path
		// falls in both coordinates, and strictly at each aligned cell before it)
		__syncwarp();  // the path's writes are visible to the warp
		int32_t *mp = maps + int64_t(count) * m;
		unsigned long long dh = 0;  // this lane's change of the hash and the count
		int dn = 0;
		int first = 0;
		if (SM) {
			int bound = m - 1;
			if (low > 0) {
				const int2 a = path[low - 1];
				bound = min(bound, s_side ? a.x : a.y);
				first = low - 1;
			}
			for (int x = lane; x <= bound; x += 32) {
				const int y = smap[x];
				if (y >= 0) {
					dh -= s_side ? enum_mix(x, y) : enum_mix(y, x);
					dn--;
					smap[x] = -1;
				}
			}
			__syncwarp();
		} else {
			for (int x = lane; x < m; x += 32) mp[x] = -1;
			h = 0;
			n = 0;
			__syncwarp();
		}
		for (int t0 = first; t0 + 1 < plen; t0 += 32 * 8) {
			// lane l holds points t0 + 32 x + l; a point's successor comes from the next lane
			int2 a[8];
#pragma unroll
			for (int x = 0; x < 8; x++) {
				const int t = t0 + 32 * x + lane;
				a[x] = t < plen ? path[t] : make_int2(0, 0);
			}
			const int2 past = t0 + 256 < plen ? path[t0 + 256] : make_int2(0, 0);
#pragma unroll
			for (int x = 0; x < 8; x++) {
				int bx = __shfl_down_sync(0xffffffffu, a[x].x, 1), by = __shfl_down_sync(0xffffffffu, a[x].y, 1);
				const int fx = x < 7 ? __shfl_sync(0xffffffffu, a[x < 7 ? x + 1 : 7].x, 0) : past.x;
				const int fy = x < 7 ? __shfl_sync(0xffffffffu, a[x < 7 ? x + 1 : 7].y, 0) : past.y;
				if (lane == 31) {
					bx = fx;
					by = fy;
				}
				if (t0 + 32 * x + lane + 1 < plen && bx != a[x].x && by != a[x].y && a[x].x >= 0 && a[x].y >= 0) {
					int32_t *const to = SM ? smap : mp;
					if (s_side) to[a[x].x] = a[x].y;
					else to[a[x].y] = a[x].x;
					dh += enum_mix(a[x].x, a[x].y);
					dn++;
				}
			}
		}
		low = plen;
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) {
			dh += __shfl_xor_sync(0xffffffffu, dh, o);
			dn += __shfl_xor_sync(0xffffffffu, dn, o);
		}
		h += dh;
		n += dn;
		__syncwarp();  // the map is complete
		bool dup = false;
		if (p.remove_dup) {
			for (int r0 = 0; r0 < count && !dup; r0 += 32) {
				// 32 earlier yields at a time; those of equal hash and count are compared in full
				const int rl = r0 + lane;
				uint32_t like = __ballot_sync(0xffffffffu, rl < count && hash[rl] == h && npts[rl] == n);
				for (; like && !dup; like &= like - 1) {
					const int32_t *mr = maps + int64_t(r0 + __ffs(int(like)) - 1) * m;
					bool same = true;
					for (int x = lane; x < m; x += 32) same &= mr[x] == (SM ? smap[x] : mp[x]);
					dup = __all_sync(0xffffffffu, same);
				}
			}
		}
		if (dup) {  // (between two yields lie |s| + |t| + 2 entries at most)
			paused = __shfl_sync(0xffffffffu, clock64() - begun, 0) > p.cycles;
			if (paused) break;
			continue;
		}
		if (SM) {
#pragma unroll 8
			for (int x = lane; x < m; x += 32) mp[x] = smap[x];
		}
		if (lane == 0) {
			hash[count] = h;
			npts[count] = n;
		}
		__syncwarp();  // the other lanes read them at the next yield
		if (p.paths) {
			int2 *po = p.paths + p.paths_off[L] + int64_t(count) * plen_cap;
			for (int t = lane; t < plen; t += 32) po[t] = path[t];
			if (lane == 0) p.path_len[int64_t(L) * p.k + count] = plen;
			__syncwarp();  // the path may be overwritten
		}
		count++;
	}
	// the slots past the last result hold no data of an earlier, abandoned search: -1 maps,
	// empty walks
	for (int64_t x = int64_t(count) * m + lane; x < int64_t(p.k) * m; x += 32) maps[x] = -1;
	if (p.paths)
		for (int j = count + lane; j < p.k; j += 32) p.path_len[int64_t(L) * p.k + j] = 0;
	if (paused) {
		__syncwarp();  // lane 0's writes
		for (int x = lane; x < min(sp, SMEM_STACK); x += 32) stk[x] = top[x];
	}
	if (lane == 0) {
		p.count[L] = count;
		p.status[L] = paused ? ENUM_PAUSED : status;
		p.state[L] = EnumState{have, eu, ev, epl, sp, si, count};
	}
}

cudaError_t enum_seed_scan(const SeedScanParams &p, int grid, cudaStream_t st) {
	enum_seed_kernel<<<grid, 256, 0, st>>>(p);
	return cudaGetLastError();
}

cudaError_t enum_solve(const EnumParams &p, cudaStream_t st) {
	if (p.nwork <= 0) return cudaSuccess;
	if (p.smem_map > 0) {
		const int bytes = p.smem_map * 4;
		if (bytes > 32 * 1024)  // beside 12 KB of static shared memory
			if (cudaError_t e = cudaFuncSetAttribute(enum_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
			                                         ENUM_SMEM_MAP * 4))
				return e;
		enum_kernel<true><<<p.nwork, 32, bytes, st>>>(p);
	} else {
		enum_kernel<false><<<p.nwork, 32, 0, st>>>(p);
	}
	return cudaGetLastError();
}

}  // namespace pa
