// Co-optimal traceback path counts over the all-optimal masks (sm_103a).
//
// The reference enumerates every optimal alignment with a depth-first search over the
// traceback lists (TracebackIterators<true>::Iterator::next, solver.h:1647-1716): from each
// seed it follows every entry of a cell's list -- the zero candidate of local alignment, the
// diagonal, and for affine gaps the P/Q lists, which hold the cells where a vertical or
// horizontal gap was opened (solver.h:2995-3016) -- until a point with a negative coordinate
// or (local) a value that is not strictly positive.  Without de-duplication every leaf of
// that search is one result, so the number of results is a sum over the traceback graph:
//
//   N(u, v)  = 1                                    u < 0, v < 0, or local with D(u, v) = 0
//            = max(1, [zero] + [diag] N(u-1, v-1) + [P] Pc(u, v) + [Q] Qc(u, v))   otherwise
//   Pc(u, v) = [P open] N(u-1, v) + [P extend, u > 0] Pc(u-1, v)     (linear gaps: N(u-1, v))
//   Qc(u, v) = [Q open] N(u, v-1) + [Q extend, v > 0] Qc(u, v-1)     (linear gaps: N(u, v-1))
//
// (an empty list pushes one terminal entry, hence the max), and the count of a pair is N
// summed over its seeds: every cell equal to a strictly positive optimum for local
// alignment, the one seed of Global/Semiglobal otherwise.  N depends only on cells above
// and to the left, so it runs in the DP's own wavefront order, over the DP's own mask layout
// (pa_dp.cuh: per pair, stripe q, step s, lane k one uint4 holding 8 rows of 16-bit cells):
// a group of G lanes per pair, lane k owning 8 rows of each G * 8-row stripe, column
// s - k in step s; (N, Pc) of a lane's last row reach the next lane by a shuffle, the last
// lane's row crosses to the next stripe through a double-buffered boundary row in global
// memory, and (N, Qc) of each row stay in registers along the row.  Counts are uint64,
// exact below 2^64 and saturating at 2^64 - 1.
//
// Few long pairs (masks written with G = 32 or 16): path_count_chain_kernel gives every 256-row
// (128-row) stripe of every pair to its own warp, like the DP's stripe-chained mode -- tickets numbered
// stripe-major (stripe q of the pair at rank w is ticket level_start[q] + w), the warp of
// stripe q reading the boundary row of stripe q - 1 while that stripe's warp still writes
// it, behind a progress counter published every 32 columns (bounded waits: past the limit
// the kernel flags ST_TIMEOUT and finishes).  Each ticket writes its own partial count (the
// seeds inside its stripe); the host adds a pair's partials.
//
// Global and Semiglobal have one seed, and few cells lie on a co-optimal path from it: a band some
// cells wide along one path of the whole matrix.  path_count_band_kernel counts forward from the
// seed over anti-diagonals of that band alone -- how many partial paths reach a cell, in the cell
// itself, inside its vertical and inside its horizontal list -- and adds up those that end.  Both
// orders count the same paths, and saturating sums of counts are the saturated count.  A block per
// pair, a row per thread: one dependent cell per step instead of eight, O(|s| + |t|) steps instead
// of O(|s| |t|) cells, and where the band is one cell wide 32 diagonal steps at once.  A step is
// bound by its chain (a barrier, a shuffle, four saturating sums), about 490 cycles.  Two things
// are left to the kernels above, the pair being flagged: a band too wide for the block, and a list
// whose entries all come to nothing (an extension past the border; such a cell counts once, which
// a forward sum cannot see).  Two warps a pair where there are more pairs than SMs (their band up
// to 53 rows), eight (up to 245) for few pairs and those that two were too narrow for.  One pair of
// 512 x 512: 0.60 -> 0.26 ms; 16 of 2048 x 2048: 2.66 -> 1.1 ms; 1000 of 64 x 64: 151 -> 74 us, of
// 256 x 256: 449 -> 250 us, or 435 when one of them needs the second launch; 16 of 2000..3000 x
// 3000..5000 with 20 letters: 5.98 -> 0.9 ms.
#include <climits>
#include "pa_dp.cuh"

namespace pa {

struct CountParams {
	int32_t npairs;
	int32_t G;                 // group width of the DP launch that wrote the masks
	int32_t local, affine;
	const int32_t *len_s, *len_t;
	const int64_t *mask_off;   // per pair, in uint4 units
	const uint4 *masks;
	const int32_t *seed;       // (i, j) per pair: the single seed of Global/Semiglobal
	unsigned long long *counts;
	unsigned long long *scratch;  // per group slot: 2 buffers x (N, Pc) x max |t|
	int64_t scratch_stride;       // uint64 per slot (per pair in the chained kernel)
	int32_t *work_counter;
	// stripe-chained kernel
	int32_t ntickets, nlevels;
	const int32_t *level_start;   // nlevels + 1 ticket offsets
	const int32_t *order;         // pairs by stripe count, most first
	int32_t *progress;            // per ticket: columns of its boundary row written
	int32_t *status;              // ST_TIMEOUT
	unsigned long long *partial;  // per ticket: the count of the seeds in its stripe
};

__device__ __forceinline__ unsigned long long sat_add(unsigned long long a, unsigned long long b) {
	const unsigned long long c = a + b;
	return c < a ? ~0ull : c;
}

__device__ __forceinline__ unsigned long long shfl_up64(unsigned long long x, int G) {
	const uint32_t lo = __shfl_up_sync(0xffffffffu, uint32_t(x), 1, G);
	const uint32_t hi = __shfl_up_sync(0xffffffffu, uint32_t(x >> 32), 1, G);
	return (unsigned long long)(hi) << 32 | lo;
}

// One lane's R rows in column j: N, Pc from the row above (uN, uP) and the diagonal dN,
// N and Qc of each row to the left (Nl, Ql, updated in place); the seed counts of its cells
// add into acc.  Returns (N, Pc) of the last row in uN, uP.
__device__ __forceinline__ void count_rows(const CountParams &p, const uint32_t (&ws)[4], int row0, int j, int ls,
                                           int si, int sj, unsigned long long dN, unsigned long long &uN,
                                           unsigned long long &uP, unsigned long long (&Nl)[R],
                                           unsigned long long (&Ql)[R], unsigned long long &acc) {
#pragma unroll
	for (int r = 0; r < R; r++) {
		const int i = row0 + r;
		const uint32_t c = (ws[r >> 1] >> (16 * (r & 1))) & 0xffffu;
		const unsigned long long lN = Nl[r], lQ = Ql[r];
		unsigned long long Pc, Qc;
		if (p.affine) {
			Pc = sat_add((c & 16u) ? uN : 0ull, ((c & 32u) && i > 0) ? uP : 0ull);
			Qc = sat_add((c & 64u) ? lN : 0ull, ((c & 128u) && j > 0) ? lQ : 0ull);
		} else {
			Pc = uN;
			Qc = lN;
		}
		unsigned long long N;
		if (p.local && (c & 1u)) {
			N = 1ull;  // D = 0: the search stops here
		} else {
			unsigned long long t = (c & 1u) ? 1ull : 0ull;
			t = sat_add(t, (c & 2u) ? dN : 0ull);
			t = sat_add(t, (c & 4u) ? Pc : 0ull);
			t = sat_add(t, (c & 8u) ? Qc : 0ull);
			N = t ? t : 1ull;
		}
		if (i < ls) {
			if (p.local ? (c & 256u) != 0 : (i == si && j == sj)) acc = sat_add(acc, N);
		}
		dN = lN;  // N(i, j - 1) is the diagonal of row i + 1
		Nl[r] = N;
		Ql[r] = Qc;
		uN = N;
		uP = Pc;
	}
}

__global__ void __launch_bounds__(BLOCK) path_count_kernel(CountParams p) {
	const int G = p.G;
	const int lane = threadIdx.x & 31;
	const int sub = lane % G, grp = lane / G, gpw = 32 / G;
	const int warp_global = int((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5);
	const int slot = warp_global * gpw + grp;
	const int rpp = G * R;
	const int64_t half = p.scratch_stride / 2;
	for (;;) {
		int base = 0;
		if (lane == 0) base = atomicAdd(p.work_counter, gpw);
		base = __shfl_sync(0xffffffffu, base, 0);
		if (base >= p.npairs) break;
		const int pair = base + grp;
		const bool have = pair < p.npairs;
		const int ls = have ? p.len_s[pair] : 0, lt = have ? p.len_t[pair] : 0;
		const int npass = (ls == 0 || lt == 0) ? 0 : (ls + rpp - 1) / rpp;
		const int nsteps = npass ? lt + G - 1 : 0;
		int wpass = npass, wsteps = nsteps;
		for (int o = 16; o > 0; o >>= 1) {
			wpass = max(wpass, __shfl_xor_sync(0xffffffffu, wpass, o));
			wsteps = max(wsteps, __shfl_xor_sync(0xffffffffu, wsteps, o));
		}
		const int si = (have && !p.local) ? p.seed[2 * pair] : -1;
		const int sj = (have && !p.local) ? p.seed[2 * pair + 1] : -1;
		const uint4 *M = p.masks + (have ? p.mask_off[pair] : 0);
		const int64_t S = int64_t(lt) + G - 1;
		unsigned long long acc = 0;
		unsigned long long *slot_rows = p.scratch + int64_t(slot) * p.scratch_stride;
		for (int q = 0; q < wpass; q++) {
			const bool pass_active = q < npass;
			const int row0 = q * rpp + sub * R;
			const unsigned long long *bin = slot_rows + (q & 1) * half;
			unsigned long long *bout = slot_rows + ((q + 1) & 1) * half;
			const bool write_boundary = sub == G - 1 && q + 1 < npass;
			unsigned long long Nl[R], Ql[R];
#pragma unroll
			for (int r = 0; r < R; r++) {
				Nl[r] = 1ull;  // N(i, -1): a leaf
				Ql[r] = 0ull;  // no Q list at column -1
			}
			unsigned long long outN = 1ull, outP = 0ull;  // this lane's last row, previous column
			unsigned long long prev_up = 1ull;            // N(row0 - 1, j - 1); column -1 is a leaf
			// the mask words of the next four steps and (lane 0) the boundary row of the next two
			// columns, loaded ahead: one pair's steps are a chain of dependent cells, so a load
			// used in its own step would cost a memory round trip per step
			const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
			auto load = [&](int st) -> uint4 {
				const int jj = st - sub;
				return (pass_active && jj >= 0 && jj < lt) ? __ldg(M + (int64_t(q) * S + st) * G + sub) : zero4;
			};
			auto load_row = [&](int col) -> ulonglong2 {
				if (sub != 0 || !pass_active || col >= lt) return make_ulonglong2(1ull, 0ull);
				if (q == 0) return make_ulonglong2(1ull, 0ull);  // N(-1, j): a leaf; no P list above
				return make_ulonglong2(bin[2 * col], bin[2 * col + 1]);
			};
			uint4 w0 = load(0), w1 = load(1), w2 = load(2), w3 = load(3);
			ulonglong2 b0 = load_row(0), b1 = load_row(1);
			for (int s = 0; s < wsteps; s++) {
				const uint4 w = w0;
				w0 = w1;
				w1 = w2;
				w2 = w3;
				w3 = load(s + 4);
				const ulonglong2 bcur = b0;  // lane 0: (N, Pc) above row 0 in column s
				b0 = b1;
				b1 = load_row(s + 2);
				const int j = s - sub;
				unsigned long long upN = shfl_up64(outN, G);
				unsigned long long upP = shfl_up64(outP, G);
				const bool act = pass_active && j >= 0 && j < lt;
				if (act) {
					if (sub == 0) {
						upN = bcur.x;
						upP = bcur.y;
					}
					const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
					unsigned long long uN = upN, uP = upP;
					count_rows(p, ws, row0, j, ls, si, sj, prev_up, uN, uP, Nl, Ql, acc);
					outN = uN;
					outP = uP;
					if (write_boundary) {
						bout[2 * j] = outN;
						bout[2 * j + 1] = outP;
					}
				}
				prev_up = upN;
			}
			__syncwarp();
		}
		// the group's sum
		for (int o = 1; o < G; o <<= 1) {
			const uint32_t lo = __shfl_xor_sync(0xffffffffu, uint32_t(acc), o, G);
			const uint32_t hi = __shfl_xor_sync(0xffffffffu, uint32_t(acc >> 32), o, G);
			acc = sat_add(acc, (unsigned long long)(hi) << 32 | lo);
		}
		if (have && sub == 0) p.counts[pair] = acc;
	}
}

// G: the width of the masks' groups, 32 or (stripes of 128 rows) 16, then half of the lanes idle
template <int G>
__global__ void __launch_bounds__(BLOCK) path_count_chain_kernel(CountParams p) {
	constexpr int rpp = G * R;
	const int lane = threadIdx.x & 31;
	const int sub = lane;
	for (;;) {
		int t = 0;
		if (lane == 0) t = atomicAdd(p.work_counter, 1);
		t = __shfl_sync(0xffffffffu, t, 0);
		if (t >= p.ntickets) break;
		int q = 0;
		while (q + 1 < p.nlevels && p.level_start[q + 1] <= t) q++;
		const int w = t - p.level_start[q];
		const int pair = p.order[w];
		const int prod = q > 0 ? p.level_start[q - 1] + w : -1;  // the stripe above: an earlier ticket
		const int ls = p.len_s[pair], lt = p.len_t[pair];
		const int npass = (ls == 0 || lt == 0) ? 0 : (ls + rpp - 1) / rpp;
		const int si = p.local ? -1 : p.seed[2 * pair], sj = p.local ? -1 : p.seed[2 * pair + 1];
		const uint4 *M = p.masks + p.mask_off[pair];
		const int64_t S = int64_t(lt) + G - 1;
		unsigned long long acc = 0;
		const bool pass_active = q < npass;
		unsigned long long *rows = p.scratch + int64_t(pair) * p.scratch_stride;
		const unsigned long long *bin = rows + (q & 1) * (p.scratch_stride / 2);
		unsigned long long *bout = rows + ((q + 1) & 1) * (p.scratch_stride / 2);
		const bool write_boundary = sub == G - 1 && q + 1 < npass;
		const int32_t *prog_in = q > 0 ? p.progress + prod : nullptr;
		int32_t avail = 0;  // lane 0: columns of bin known to be written
		const int row0 = q * rpp + sub * R;
		unsigned long long Nl[R], Ql[R];
#pragma unroll
		for (int r = 0; r < R; r++) {
			Nl[r] = 1ull;
			Ql[r] = 0ull;
		}
		unsigned long long outN = 1ull, outP = 0ull, prev_up = 1ull;
		const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
		auto load = [&](int st) -> uint4 {
			const int jj = st - sub;
			return (pass_active && sub < G && jj >= 0 && jj < lt) ? __ldg(M + (int64_t(q) * S + st) * G + sub) : zero4;
		};
		// lane 0: the boundary row of column col, once the stripe above has published it
		auto load_row = [&](int col) -> ulonglong2 {
			if (sub != 0 || !pass_active || col >= lt || q == 0) return make_ulonglong2(1ull, 0ull);
			if (avail < col + 1) avail = wait_progress(prog_in, col + 1, p.status);
			return make_ulonglong2(__ldcg(bin + 2 * col), __ldcg(bin + 2 * col + 1));
		};
		uint4 w0 = load(0), w1 = load(1), w2 = load(2), w3 = load(3);
		ulonglong2 b0 = load_row(0), b1 = load_row(1);
		int pub_next = PUB_CHUNK;
		const int nsteps = pass_active ? lt + G - 1 : 0;
		for (int s = 0; s < nsteps; s++) {
			const uint4 wcur = w0;
			w0 = w1;
			w1 = w2;
			w2 = w3;
			w3 = load(s + 4);
			const ulonglong2 bcur = b0;
			b0 = b1;
			b1 = load_row(s + 2);
			const int j = s - sub;
			unsigned long long upN = shfl_up64(outN, G);
			unsigned long long upP = shfl_up64(outP, G);
			if (sub < G && j >= 0 && j < lt) {
				if (sub == 0) {
					upN = bcur.x;
					upP = bcur.y;
				}
				const uint32_t ws[4] = {wcur.x, wcur.y, wcur.z, wcur.w};
				unsigned long long uN = upN, uP = upP;
				count_rows(p, ws, row0, j, ls, si, sj, prev_up, uN, uP, Nl, Ql, acc);
				outN = uN;
				outP = uP;
				if (write_boundary) {
					bout[2 * j] = outN;
					bout[2 * j + 1] = outP;
					if (j + 1 == pub_next && j + 1 < lt) {  // columns < j + 1 are written
						st_release(p.progress + t, j + 1);
						pub_next += PUB_CHUNK;
					}
				}
			}
			prev_up = upN;
		}
		if (write_boundary) st_release(p.progress + t, lt);  // every column
		for (int o = 1; o < G; o <<= 1) {
			const uint32_t lo = __shfl_xor_sync(0xffffffffu, uint32_t(acc), o);
			const uint32_t hi = __shfl_xor_sync(0xffffffffu, uint32_t(acc >> 32), o);
			acc = sat_add(acc, (unsigned long long)(hi) << 32 | lo);
		}
		if (lane == 0) p.partial[t] = acc;
	}
}

struct BandParams {
	int32_t npairs;
	const int32_t *work;       // the pairs to count
	int32_t G;
	int32_t affine;
	const int32_t *len_s, *len_t;
	const int64_t *mask_off;
	const uint4 *masks;
	const int32_t *seed;
	unsigned long long *counts;
	int32_t *left;             // per pair: 0 = counted, 1 = the band is too wide, 2 = a list came to nothing
};

// NW warps: 32 NW consecutive rows.  The band's extent is looked at every BAND_STEP anti-diagonals;
// the window of masks is then loaded anew if the next ones may leave it: the least of 64 x 64,
// 128 x 128 ... 32 NW x 32 NW cells that leaves the band room.
constexpr int BAND_STEP = 8;  // even

template <int NW>
__global__ void __launch_bounds__(32 * NW) path_count_band_kernel(BandParams p) {
	constexpr int W = 32 * NW;
	typedef unsigned long long U;
	extern __shared__ uint4 win[];  // W / R row blocks x W columns at most
	__shared__ U xg[2][NW], xp[2][NW], val;
	__shared__ uint32_t s2[NW], s1[NW], so[NW];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	const int pair = p.work[blockIdx.x];
	const int ls = p.len_s[pair], lt = p.len_t[pair];
	const int64_t S = int64_t(lt) + p.G - 1;
	const uint4 *M = p.masks + p.mask_off[pair];
	const bool affine = p.affine;
	// row u lives in lane u mod 32 of warp (u / 32) mod NW.  What the cells of the last two
	// anti-diagonals pass on: their diagonal (dg1: the last one's, dg2: the one before), and of the
	// last one the openings and extensions of the vertical list (to row u - 1) and of the
	// horizontal one (to row u).  The seed arrives like a diagonal from one row and column further
	U dg1 = 0, dg2 = 0, po = 0, pe = 0, qo = 0, qe = 0, ended = 0;
	bool lost = false, dead = false;
	const int si = p.seed[2 * pair], sj = p.seed[2 * pair + 1];
	int hi = si + 1, d = si >= 0 && sj >= 0 ? si + sj : -1;  // the band's largest row; the anti-diagonal
	int wb = 8, wc = 64, gb0 = -wb, j0 = -wc;  // the window: row blocks [gb0, gb0 + wb), columns [j0, j0 + wc)
	int par = 0;
	// masks for rows [r0, r1] and columns [c0, c1], r1 and c1 inside the pair; false: too many.  Every
	// thread calls it alike
	auto ensure = [&](int r0, int r1, int c0, int c1) {
		r0 = max(r0, 0);
		c0 = max(c0, 0);
		if ((r0 >> 3) >= gb0 && (r1 >> 3) < gb0 + wb && c0 >= j0 && c1 < j0 + wc) return true;
		wc = 64;
		while (wc < W && wc < 2 * max(r1 - r0, c1 - c0)) wc *= 2;
		wb = wc / R;
		gb0 = max(0, (r1 >> 3) - (wb - 1));
		j0 = max(0, c1 - (wc - 1));
		if ((r0 >> 3) < gb0 || c0 < j0) return false;
		__syncthreads();  // every warp is done with the old window
		// a row block per warp and turn, 64 columns at a time
		for (int r = w; r < wb; r += NW) {
			const int gb = gb0 + r, q = gb / p.G, sb = gb - q * p.G;
			if (gb * R >= ls) break;
			const uint4 *from = M + (int64_t(q) * S + sb) * p.G + sb;
			for (int h = lane; h < wc; h += 64) {
				const bool in0 = j0 + h < lt, in1 = j0 + h + 32 < lt;
				uint4 x0, x1;
				if (in0) x0 = from[int64_t(j0 + h) * p.G];
				if (in1) x1 = from[int64_t(j0 + h + 32) * p.G];
				if (in0) win[r * wc + h] = x0;
				if (in1) win[r * wc + h + 32] = x1;
			}
		}
		__syncthreads();
		return true;
	};
	auto cell = [&](int u, int v) {
		const uint32_t *e = reinterpret_cast<const uint32_t *>(win + (((u >> 3) - gb0) & (wb - 1)) * wc + ((v - j0) & (wc - 1)));
		return e[(u & 7) >> 1] >> (16 * (u & 1));
	};
	auto row_of = [&]() { return hi - ((hi - int(threadIdx.x)) & (W - 1)); };  // this thread's, in (hi - W, hi]
	if (row_of() == hi) dg2 = 1;
	while (d >= 0) {
		// where the band is: what the next anti-diagonals receive
		const uint32_t b2 = __ballot_sync(0xffffffffu, dg2 != 0), b1 = __ballot_sync(0xffffffffu, dg1 != 0);
		const uint32_t bo = __ballot_sync(0xffffffffu, (po | pe | qo | qe) != 0);
		if (lane == 0) {
			s2[w] = b2;
			s1[w] = b1;
			so[w] = bo;
		}
		if (dg1 | dg2) val = dg1 | dg2;  // read only if there is just one
		__syncthreads();
		int top = INT_MIN, low = INT_MAX, many = 0, now = 0;
		if (lane < NW) {
			// the rows of warp `lane`: block b, and of the largest block only those up to hi, the others
			// being W rows below
			const int tb = hi >> 5, b = tb - ((tb - lane) & (NW - 1));
			const uint32_t x2 = s2[lane], x1 = s1[lane], xo = so[lane], x = x2 | x1 | xo;
			const uint32_t cut = b == tb && (hi & 31) != 31 ? (2u << (hi & 31)) - 1u : 0xffffffffu;
			const uint32_t in = x & cut, out = x & ~cut;
			if (in) {
				top = 32 * b + 31 - __clz(int(in));
				low = 32 * b + __ffs(int(in)) - 1;
			}
			if (out) {
				top = max(top, 32 * b - W + 31 - __clz(int(out)));
				low = min(low, 32 * b - W + __ffs(int(out)) - 1);
			}
			many = __popc(x2) + __popc(x1) + 2 * __popc(xo);
			now = x2 != 0;
		}
		top = __reduce_max_sync(0xffffffffu, top);
		low = __reduce_min_sync(0xffffffffu, low);
		many = __reduce_add_sync(0xffffffffu, many);
		now = __reduce_or_sync(0xffffffffu, now);
		if (many == 0) break;
		// rows below hi - W would share the threads of the largest ones
		hi = top;
		if (low - BAND_STEP - 2 <= hi - W) {
			lost = true;
			break;
		}
		if (many == 1) {
			// one path set on a diagonal and nothing else under way: runs of cells whose only entry is
			// the diagonal are passed 32 at a time, by every warp alike
			const U f = val;
			if (!now) d--;
			int u = hi - 1, run = 32;
			while (run > 0) {
				if (u < 0 || d - u < 0) break;
				ensure(u, u, d - u, d - u);
				const int i = u - lane, j = d - u - lane;
				const bool simple = i >= 0 && j >= 0 && (i >> 3) >= gb0 && j >= j0 && (cell(i, j) & 15u) == 2u;
				const uint32_t b = __ballot_sync(0xffffffffu, simple);
				run = b == 0xffffffffu ? 32 : __ffs(int(~b)) - 1;
				u -= run;
				d -= 2 * run;
			}
			if (u < 0 || d - u < 0) {
				if (threadIdx.x == 0) ended = sat_add(ended, f);
				break;
			}
			hi = u + 1;
			low = hi;
			dg1 = 0;
			dg2 = row_of() == hi ? f : 0ull;
		}
		if (!ensure(low - BAND_STEP, min(hi, ls - 1), d - BAND_STEP + 1 - hi, min(d - low + 1, lt - 1))) {
			lost = true;
			break;
		}
		const int above = (w + 1) & (NW - 1);
		if (many > 1 && (s2[w] | s1[w] | so[w] | s2[above] | s1[above] | so[above]) == 0) {
			// nothing in this warp's rows, nor in the next warp's, that could reach them
			if (lane == 0) xg[0][w] = xg[1][w] = xp[0][w] = xp[1][w] = 0;
			for (int step = 0; step < BAND_STEP; step++) __syncthreads();
			d -= BAND_STEP;
			continue;
		}
		// A thread without partial paths reads some cell of the window and passes on zeros: no thread
		// branches.  Cells with partial paths are inside the pair: paths that leave it end
		const int u = row_of();
		uint32_t next = cell(u, d - u);
#pragma unroll
		for (int step = 0; step < BAND_STEP; step++) {
			const int v = d - u;
			const U g = sat_add(dg2, po);
			if (lane == 0) {
				xg[par][w] = g;
				if (affine) xp[par][w] = pe;
			}
			const uint32_t c = next;
			next = cell(u, v - 1);
			__syncthreads();
			U f = (U)(__shfl_down_sync(0xffffffffu, uint32_t(g >> 32), 1)) << 32 | __shfl_down_sync(0xffffffffu, uint32_t(g), 1);
			U P = 0;
			if (affine)
				P = (U)(__shfl_down_sync(0xffffffffu, uint32_t(pe >> 32), 1)) << 32 | __shfl_down_sync(0xffffffffu, uint32_t(pe), 1);
			if (lane == 31) {
				f = xg[par][above];
				if (affine) P = xp[par][above];
			}
			f = sat_add(f, qo);
			const U x = sat_add(P, (c & 4u) ? f : 0ull), y = sat_add(qe, (c & 8u) ? f : 0ull);
			const U zero = (c & 15u) == 0u || (c & 1u) ? f : 0ull;  // no entry, or the zero candidate
			const U diag = (c & 2u) ? f : 0ull;
			const bool oP = !affine || (c & 16u), eP = affine && (c & 32u) && u > 0;
			const bool oQ = !affine || (c & 64u), eQ = affine && (c & 128u) && v > 0;
			dead = dead || (x && !oP && !eP) || (y && !oQ && !eQ);
			const U ox = oP ? x : 0ull, oy = oQ ? y : 0ull;
			dg2 = dg1;
			dg1 = diag;
			po = ox;
			qo = oy;
			pe = eP ? x : 0ull;
			qe = eQ ? y : 0ull;
			ended = sat_add(ended, zero);
			if (__any_sync(0xffffffffu, u == 0 || v == 0) && (u == 0 || v == 0)) {  // what leaves the pair ends
				ended = sat_add(ended, diag);
				dg1 = 0;
				if (u == 0) {
					ended = sat_add(ended, ox);
					po = 0;
				}
				if (v == 0) {
					ended = sat_add(ended, oy);
					qo = 0;
				}
			}
			par ^= 1;
			d--;
		}
	}
	for (int o = 16; o > 0; o >>= 1) {
		const uint32_t a = __shfl_xor_sync(0xffffffffu, uint32_t(ended), o), b = __shfl_xor_sync(0xffffffffu, uint32_t(ended >> 32), o);
		ended = sat_add(ended, (U)(b) << 32 | a);
	}
	dead = __any_sync(0xffffffffu, dead);
	__syncthreads();
	if (lane == 0) {
		xg[0][w] = ended;
		so[w] = dead;
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		for (int k = 1; k < NW; k++) {
			ended = sat_add(ended, xg[0][k]);
			dead = dead || so[k];
		}
		p.counts[pair] = ended;
		p.left[pair] = dead ? 2 : lost ? 1 : 0;
	}
}

cudaError_t launch_path_count(const CountParams &p, int grid, cudaStream_t st) {
	if (p.ntickets > 0 && p.G == 16) path_count_chain_kernel<16><<<grid, BLOCK, 0, st>>>(p);
	else if (p.ntickets > 0) path_count_chain_kernel<32><<<grid, BLOCK, 0, st>>>(p);
	else path_count_kernel<<<grid, BLOCK, 0, st>>>(p);
	return cudaGetLastError();
}

}  // namespace pa

// host-side declaration for pa_host.cu
namespace pa {
cudaError_t path_count_band(int32_t npairs, const int32_t *work, int32_t G, int32_t affine, const int32_t *len_s,
                            const int32_t *len_t, const int64_t *mask_off, const void *masks, const int32_t *seed,
                            unsigned long long *counts, int32_t *left, bool wide, cudaStream_t st) {
	if (npairs == 0) return cudaSuccess;
	BandParams p{npairs, work, G, affine, len_s, len_t, mask_off, static_cast<const uint4 *>(masks), seed, counts, left};
	const int bytes = wide ? 256 * 256 * 2 : 64 * 64 * 2;
	if (wide) {
		if (cudaError_t e = cudaFuncSetAttribute(path_count_band_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes))
			return e;
		path_count_band_kernel<8><<<npairs, 256, bytes, st>>>(p);
	} else {
		path_count_band_kernel<2><<<npairs, 64, bytes, st>>>(p);
	}
	return cudaGetLastError();
}
cudaError_t path_count_solve(int32_t npairs, int32_t G, int32_t local, int32_t affine, const int32_t *len_s,
                             const int32_t *len_t, const int64_t *mask_off, const void *masks, const int32_t *seed,
                             unsigned long long *counts, unsigned long long *scratch, int64_t scratch_stride,
                             int32_t *work_counter, int grid, cudaStream_t st, int32_t ntickets,
                             int32_t nlevels, const int32_t *level_start, const int32_t *order, int32_t *progress,
                             int32_t *status, unsigned long long *partial) {
	CountParams p{};
	p.ntickets = ntickets;
	p.nlevels = nlevels;
	p.level_start = level_start;
	p.order = order;
	p.progress = progress;
	p.status = status;
	p.partial = partial;
	p.npairs = npairs;
	p.G = G;
	p.local = local;
	p.affine = affine;
	p.len_s = len_s;
	p.len_t = len_t;
	p.mask_off = mask_off;
	p.masks = static_cast<const uint4 *>(masks);
	p.seed = seed;
	p.counts = counts;
	p.scratch = scratch;
	p.scratch_stride = scratch_stride;
	p.work_counter = work_counter;
	return launch_path_count(p, grid, st);
}
}  // namespace pa
