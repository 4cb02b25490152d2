// General gap cost solve (GeneralGapCostSolver, solver.h:3056-3184) in 32 x 32 tiles: scores
// and one alignment per pair, where the caller needs no cell matrices (pa_wsb.cu writes those).
//
// D(u, v) is the best of its head candidates -- (local zero), the diagonal -- and of the
// vertical gaps D(k, v) - w_s(u - k), k = -1..u-1, and the horizontal gaps
// D(u, k) - w_t(v - k), k = -1..v-1.  Only the maximum is needed to go on: which candidate won
// matters for the cells of the recovered path alone, a few hundred of a pair's 10^5, and the
// walk finds it there by scanning again (the first candidate in the reference's order that
// equals D).  So the sweep keeps no positions, and a maximum may be taken in any order.
//
// For the rows of one earlier tile the vertical candidates of a tile are a max-plus product of
// a Toeplitz matrix w_s(u - k) with that tile's D, and likewise horizontally with the
// transposed D: every value read serves 8 rows or 4 columns from registers, and a step to the
// next k needs one new gap cost because the window of costs slides.  A candidate costs half a
// packed add and half a three-way max instead of two loads, an add, a compare and two selects.
//
// A CTA of 4 warps solves one tile, taken from a list ordered by tile anti-diagonal (a tile
// waits only on tiles earlier in the list, which running CTAs hold).  Its warps take 8 of every
// 32 rows (columns) each, so the four follow the finished tiles above and to the left together,
// over counters of finished tiles per tile column and tile row; their partial maxima meet in
// shared memory.  Inside the tile one warp runs a skewed wavefront, lane v on column v at row
// step - v: vertical candidates are pushed into 32 registers that shift down a row per step,
// horizontal ones are pulled from the rows in shared memory, whose pitch (66 floats, 65 odd)
// keeps the lanes' skewed reads in distinct banks.
//
// 64 pairs of 300 x 300 (1.73 G candidates, local, log gap): the sweep 3.97 -> 0.35 ms, the walk
// 0.18 -> 0.12 ms, the whole call 4.3 -> 0.57 ms.  What bounds it now: the chain of 19 tile
// anti-diagonals, about 12 us each when alone (2 x 8 phases of a tile, its load and store round
// trips), and between them the issue slots of the max-plus products.
#include <climits>
#include <cmath>
#include <cstddef>
#include "pa_dp.cuh"
#include "pa_wsb.h"

namespace pa {

namespace {

constexpr int T = WSB_TILE;
constexpr int XP = 2 * T + 1;      // floats per row of the skewed tile: T guards, T cells, odd
constexpr int AP = T + 2;          // pitch of the tile's scan maxima and similarities
constexpr int NS = 8;              // steps of the tile's wavefront per phase
constexpr int XR = 2 + NS;         // rows before step 0: the halo's steps -2 and -1, guards

__device__ __forceinline__ float max3(float a, float b, float c) {
	float d;
	asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
	return d;
}

// both halves of a + b in one packed add (each rounded as an ordinary float32 add)
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
	float2 d;
	asm("{.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 z, x, y;\n\t"
	    "mov.b64 {%0, %1}, z;}"
	    : "=f"(d.x), "=f"(d.y)
	    : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
	return d;
}

// order-preserving key of a float that is not NaN, with -0 and +0 equal
__device__ __forceinline__ uint32_t order_key(float f) {
	const uint32_t b = __float_as_uint(f == 0.0f ? 0.0f : f);
	return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// similarity of cell (u, v), normalised (multiplied by the direction's sign)
__device__ __forceinline__ float similarity(const WsbTileParams &p, int pair, int u, int v) {
	if (p.sub_kind == SUB_DENSE)
		return p.dense[int64_t(pair) + int64_t(u) * p.dense_si + int64_t(v) * p.dense_sj] * p.sign;
	const uint32_t x = p.a[int64_t(pair) * p.a_stride + u], y = p.b[int64_t(pair) * p.b_stride + v];
	if (p.sub_kind == SUB_BINARY) return (x == y ? p.eq : p.ne) * p.sign;
	if (x >= uint32_t(p.table_rows) || y >= uint32_t(p.table_cols)) {
		atomicOr(p.status, ST_BAD_CODE);
		return 0.0f;
	}
	return p.table[size_t(x) * size_t(p.table_cols) + y] * p.sign;
}

// waits until a counter of finished tiles reaches `need` (lane 0 polls, bounded)
__device__ __forceinline__ void wait_tiles(const int32_t *counter, int need, int &have, int lane, int32_t *status) {
	if (have >= need) return;
	int got = 0;
	if (lane == 0) got = wait_progress(counter, need, status);
	have = __shfl_sync(0xffffffffu, got, 0);
	__syncwarp();  // the other lanes read after lane 0's acquire
}

struct Smem {
	float part[4][T][T];     // the warps' partial scan maxima (first: written 16 bytes at a time)
	// the tile in wavefront order: X[XR + s][T + v] = D(u0 + s - v, v0 + v), the halo above
	// (row -1, at s = v - 1) and to the left (column -1, at s = u - 1) included; -inf elsewhere
	float X[XR + 2 * T - 1][XP];
	float A[T][AP];          // the tile's scan maxima over the cells outside it
	float S[T][AP];          // similarities
	float M[NS][T];          // a phase's scan maxima over everything before the phase
	int32_t ticket;
};

__global__ void __launch_bounds__(128, 4) wsb_tile_kernel(WsbTileParams p) {
	extern __shared__ __align__(16) unsigned char wsb_tile_smem[];
	static_assert(offsetof(Smem, part) % 16 == 0, "16-byte stores");
	Smem &sm = *reinterpret_cast<Smem *>(wsb_tile_smem);
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int tx = lane & 7, ty = lane >> 3;  // a thread's 8 x 4 cells: rows 8 ty + r, columns 4 tx + c
	for (int x = tid; x < (XR + 2 * T - 1) * XP; x += 128) (&sm.X[0][0])[x] = -INFINITY;
	for (;;) {
		if (tid == 0) sm.ticket = atomicAdd(p.work_counter, 1);
		__syncthreads();
		const int ticket = sm.ticket;
		if (ticket >= p.ntiles) return;
		const int2 tk = p.tiles[ticket];
		const int pair = tk.x, I = tk.y >> 16, J = tk.y & 0xffff;
		const int ls = p.len_s[pair], lt = p.len_t[pair];
		const int NI = (ls + T - 1) / T, NJ = (lt + T - 1) / T;
		const int64_t ld = int64_t(NJ) * T, ldt = int64_t(NI) * T;
		float *D = p.vals + p.vals_off[pair];      // D(u, v) at u * ld + v, in whole tiles
		float *DT = p.vals_t + p.vals_off[pair];   // the same transposed, v * ldt + u
		int32_t *rows_done = p.progress + p.prog_off[pair];  // tiles finished per tile row,
		int32_t *cols_done = rows_done + NI;                 // and per tile column
		const int u0 = I * T, v0 = J * T;

		// similarities of the tile's cells (cells past the lengths: never used)
		for (int x = tid; x < T * T; x += 128) {
			const int u = u0 + (x >> 5), v = v0 + (x & 31);
			sm.S[x >> 5][x & 31] = (u < ls && v < lt) ? similarity(p, pair, u, v) : 0.0f;
		}

		// ---- scan candidates from the finished tiles of this column and this row
		float2 acc[8][2];
#pragma unroll
		for (int r = 0; r < 8; r++) acc[r][0] = acc[r][1] = make_float2(-INFINITY, -INFINITY);
		int have_v = 0, have_h = 0;
		for (int K = 0; K < max(I, J); K++) {
			if (K < I) {
				wait_tiles(cols_done + J, K + 1, have_v, lane, p.status);
				const float *src = D + int64_t(K * T + warp * 8) * ld + v0 + 4 * tx;
				const float *g = p.ngap_s + ((I - K) * T + 8 * ty - 8 * warp);  // g[r - k]
				float4 x[8];
#pragma unroll
				for (int k = 0; k < 8; k++) x[k] = __ldcg(reinterpret_cast<const float4 *>(src + k * ld));
				float w[15];
#pragma unroll
				for (int k = 0; k < 15; k++) w[k] = __ldg(g + k - 7);
#pragma unroll
				for (int k = 0; k < 8; k += 2)
#pragma unroll
					for (int r = 0; r < 8; r++) {
						const float wa = w[7 + r - k], wb = w[6 + r - k];
						const float2 a0 = add2(make_float2(x[k].x, x[k].y), make_float2(wa, wa));
						const float2 a1 = add2(make_float2(x[k].z, x[k].w), make_float2(wa, wa));
						const float2 b0 = add2(make_float2(x[k + 1].x, x[k + 1].y), make_float2(wb, wb));
						const float2 b1 = add2(make_float2(x[k + 1].z, x[k + 1].w), make_float2(wb, wb));
						acc[r][0].x = max3(acc[r][0].x, a0.x, b0.x);
						acc[r][0].y = max3(acc[r][0].y, a0.y, b0.y);
						acc[r][1].x = max3(acc[r][1].x, a1.x, b1.x);
						acc[r][1].y = max3(acc[r][1].y, a1.y, b1.y);
					}
			}
			if (K < J) {
				wait_tiles(rows_done + I, K + 1, have_h, lane, p.status);
				const float *src = DT + int64_t(K * T + warp * 8) * ldt + u0 + 8 * ty;
				const float *g = p.ngap_t + ((J - K) * T + 4 * tx - 8 * warp);  // g[c - k]
				float w[11];
#pragma unroll
				for (int k = 0; k < 11; k++) w[k] = __ldg(g + k - 7);
#pragma unroll
				for (int kh = 0; kh < 8; kh += 4) {
					float4 x[4][2];
#pragma unroll
					for (int k = 0; k < 4; k++) {
						x[k][0] = __ldcg(reinterpret_cast<const float4 *>(src + (kh + k) * ldt));
						x[k][1] = __ldcg(reinterpret_cast<const float4 *>(src + (kh + k) * ldt + 4));
					}
#pragma unroll
					for (int k = 0; k < 4; k += 2)
#pragma unroll
						for (int r = 0; r < 8; r++) {
							const float4 xa4 = x[k][r >> 2], xb4 = x[k + 1][r >> 2];
							const float xa = (r & 3) == 0 ? xa4.x : (r & 3) == 1 ? xa4.y : (r & 3) == 2 ? xa4.z : xa4.w;
							const float xb = (r & 3) == 0 ? xb4.x : (r & 3) == 1 ? xb4.y : (r & 3) == 2 ? xb4.z : xb4.w;
							const int q = 7 - (kh + k);  // w[q + c]: the cost of column c's gap from row k
							const float2 a0 = add2(make_float2(xa, xa), make_float2(w[q], w[q + 1]));
							const float2 a1 = add2(make_float2(xa, xa), make_float2(w[q + 2], w[q + 3]));
							const float2 b0 = add2(make_float2(xb, xb), make_float2(w[q - 1], w[q]));
							const float2 b1 = add2(make_float2(xb, xb), make_float2(w[q + 1], w[q + 2]));
							acc[r][0].x = max3(acc[r][0].x, a0.x, b0.x);
							acc[r][0].y = max3(acc[r][0].y, a0.y, b0.y);
							acc[r][1].x = max3(acc[r][1].x, a1.x, b1.x);
							acc[r][1].y = max3(acc[r][1].y, a1.y, b1.y);
						}
				}
			}
		}
#pragma unroll
		for (int r = 0; r < 8; r++)
			*reinterpret_cast<float4 *>(&sm.part[warp][8 * ty + r][4 * tx]) =
			    make_float4(acc[r][0].x, acc[r][0].y, acc[r][1].x, acc[r][1].y);
		// the halo: D(u0 - 1, v0 - 1 .. v0 + 31) and D(u0 .. u0 + 31, v0 - 1) (every warp has
		// seen both neighbours finished, unless there is none)
		if (warp == 0) {
			const int v = v0 + lane;
			sm.X[XR - 1 + lane][T + lane] = I > 0 ? __ldcg(D + int64_t(u0 - 1) * ld + v) : p.top_D[min(v, lt - 1) + 1];
			if (lane == 0)
				sm.X[XR - 2][T - 1] = I == 0 ? p.top_D[v0] : J == 0 ? p.left_D[u0] : __ldcg(D + int64_t(u0 - 1) * ld + v0 - 1);
		} else if (warp == 1) {
			const int u = u0 + lane;
			sm.X[XR - 1 + lane][T - 1] = J > 0 ? __ldcg(DT + int64_t(v0 - 1) * ldt + u) : p.left_D[min(u, ls - 1) + 1];
		}
		__syncthreads();
		for (int x = tid; x < T * T; x += 128) {
			const int i = x >> 5, j = x & 31, u = min(u0 + i, ls - 1), v = min(v0 + j, lt - 1);
			// the gaps from the borders: k = -1 above and to the left
			const float m = max3(sm.part[0][i][j], sm.part[1][i][j], fmaxf(sm.part[2][i][j], sm.part[3][i][j]));
			sm.A[i][j] = max3(m, p.top_D[v + 1] + p.ngap_s[u + 1], p.left_D[u + 1] + p.ngap_t[v + 1]);
		}

		// ---- the tile itself: step s is the anti-diagonal of cells (s - v, v), lane v, in
		// phases of NS steps.  A candidate at distance d, up or to the left, comes from step
		// s - d.  First every warp takes two of the phase's steps and the sources before the
		// phase; then one warp runs the phase's steps, each adding the sources of the phase
		// from registers (its own column) and by shuffles (the row's columns to the left).
		float ws[T], wt[T];  // the gap costs of the distances inside a tile
#pragma unroll
		for (int d = 1; d < T; d++) {
			ws[d] = __ldg(p.ngap_s + d);
			wt[d] = __ldg(p.ngap_t + d);
		}
		float best = -INFINITY;
		int best_i = -1;
		const bool vcol = v0 + lane < lt;
		float wl[NS];  // costs of the near columns to the left, -inf where this tile has none
#pragma unroll
		for (int d = 1; d < NS; d++) wl[d] = lane >= d ? wt[d] : -INFINITY;
#pragma unroll 1
		for (int s0 = 0; s0 < 2 * T - 1; s0 += NS) {
			__syncthreads();
			{
				const int i0 = 2 * warp, s = s0 + i0;  // steps s and s + 1
				const float *x = &sm.X[XR + s][T + lane];
				float m0 = sm.A[min(max(s - lane, 0), T - 1)][lane], m1 = sm.A[min(max(s + 1 - lane, 0), T - 1)][lane];
				// sources at step s - e, distance e of step s and e + 1 of step s + 1; a batch of
				// NS sources at a time, its loads in flight together
#pragma unroll
				for (int c = 0; c < T; c += NS) {
					if (s + 1 < c) break;  // warp-uniform: every source lies before the tile
					float up[NS], l0[NS], l1[NS];
#pragma unroll
					for (int q = 0; q < NS; q++) {
						const int e = c + q + 1;
						const bool on = e < T && (c > 0 || e > i0);  // a source before the phase
						up[q] = on ? x[-e * XP] : -INFINITY;
						l0[q] = on ? x[-e * XP - e] : -INFINITY;
						l1[q] = on && e < T - 1 ? x[-e * XP - e - 1] : -INFINITY;
					}
#pragma unroll
					for (int q = 0; q < NS; q++) {
						const int e = c + q + 1;
						if (e < T) m0 = max3(m0, up[q] + ws[e], l0[q] + wt[e]);
						if (e < T - 1) m1 = max3(m1, up[q] + ws[e + 1], l1[q] + wt[e + 1]);
					}
				}
				sm.M[i0][lane] = m0;
				sm.M[i0 + 1][lane] = m1;
			}
			__syncthreads();
			if (warp == 0) {
				// everything the steps read from shared memory, before the first of them: the
				// diagonal comes from there at the tile's edge and in the first two steps
				float m[NS], sv[NS], dv[NS], h[NS];  // h: this lane's values of the phase's steps
#pragma unroll
				for (int k = 0; k < NS; k++) {
					const int s = s0 + k;
					m[k] = sm.M[k][lane];
					sv[k] = sm.S[min(max(s - lane, 0), T - 1)][lane];
					dv[k] = sm.X[XR + s - 2][T + lane - 1];
				}
#pragma unroll
				for (int k = 0; k < NS; k++) {
					const int i = s0 + k - lane;
					const bool act = i >= 0 && i < T;
					if (k >= 2) {
						const float d2 = __shfl_up_sync(0xffffffffu, h[k - 2], 1);
						if (lane > 0 && i > 0) dv[k] = d2;
					}
					const float dg = dv[k] + sv[k];
					float D_ = dg;
					if (p.local == LOC_LOCAL) {
						D_ = 0.0f;
						if (dg > D_) D_ = dg;
					}
					float x = m[k];
#pragma unroll
					for (int d = k; d >= 1; d--) {  // the last step's values last
						const float left = __shfl_up_sync(0xffffffffu, h[k - d], d);
						x = max3(x, h[k - d] + ws[d], left + wl[d]);
					}
					if (x > D_) D_ = x;
					h[k] = act ? D_ : -INFINITY;
					const bool up = act && vcol && u0 + i < ls && D_ >= best;
					best = up ? D_ : best;
					best_i = up ? i : best_i;
				}
#pragma unroll
				for (int k = 0; k < NS; k++)
					if (s0 + k >= lane && s0 + k - lane < T) sm.X[XR + s0 + k][T + lane] = h[k];
			}
		}
		if (warp == 0 && p.local == LOC_LOCAL) {
			// the seed: the largest value, of equal ones the largest row, then column
			unsigned long long key = 0;
			if (best_i >= 0)
				key = (static_cast<unsigned long long>(order_key(best)) << 32) |
				      (uint32_t(u0 + best_i) * uint32_t(lt) + uint32_t(v0 + lane));
			for (int o = 16; o > 0; o >>= 1) {
				const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
				key = other > key ? other : key;
			}
			if (lane == 0 && key) atomicMax(p.best + pair, key);
		}
		__syncthreads();
		// ---- the finished tile, both ways round
#pragma unroll
		for (int q = 0; q < 8; q++) {
			const int x = warp * 8 + q;
			__stcg(D + int64_t(u0 + x) * ld + v0 + lane, sm.X[XR + x + lane][T + lane]);
			__stcg(DT + int64_t(v0 + x) * ldt + u0 + lane, sm.X[XR + x + lane][T + x]);
		}
		__syncthreads();
		if (tid == 0) {
			__threadfence();
			st_release(cols_done + J, I + 1);
			st_release(rows_done + I, J + 1);
		}
	}
}

// Score, seed and (with maps) the alignment of each pair, a warp per pair.  The walk resolves
// 32 diagonal steps per round (lane l tests cell (u - l, v - l)), and finds the gap a cell came
// from by scanning its candidates in the reference's order for the first that equals D.
__global__ void __launch_bounds__(128) wsb_tile_walk_kernel(WsbTileParams p) {
	const int pair = blockIdx.x * 4 + int(threadIdx.x >> 5);
	const int lane = threadIdx.x & 31;
	if (pair >= p.npairs) return;
	const int ls = p.len_s[pair], lt = p.len_t[pair];
	const int NI = (ls + T - 1) / T, NJ = (lt + T - 1) / T;
	const int64_t ld = int64_t(NJ) * T, ldt = int64_t(NI) * T;
	const float *D = p.vals + p.vals_off[pair], *DT = p.vals_t + p.vals_off[pair];
	const bool local = p.local == LOC_LOCAL;
	auto V = [&](int u, int v) { return u < 0 ? p.top_D[v + 1] : v < 0 ? p.left_D[u + 1] : D[int64_t(u) * ld + v]; };

	// seeds (Local 2035-2058, Global 2174-2188, Semiglobal 2266-2294)
	int si = -1, sj = -1, has = 0;
	float best = -INFINITY;
	if (local) {
		const unsigned long long key = p.best[pair];
		if (key) {
			const uint32_t pos = uint32_t(key);
			si = int(pos / uint32_t(lt));
			sj = int(pos % uint32_t(lt));
			best = V(si, sj);
			has = 1;
		}
	} else if (p.local == LOC_GLOBAL) {
		si = ls - 1;
		sj = lt - 1;
		best = V(si, sj);
		has = 1;
	} else {
		// the first strict optimum of the last row (j ascending), then the last column
		int pos = INT_MAX;
		for (int x = lane; x < lt + ls; x += 32) {
			const float val = x < lt ? V(ls - 1, x) : V(x - lt, lt - 1);
			if (val > best) {
				best = val;
				pos = x;
			}
		}
		for (int o = 16; o > 0; o >>= 1) {
			const float ov = __shfl_xor_sync(0xffffffffu, best, o);
			const int op = __shfl_xor_sync(0xffffffffu, pos, o);
			if (ov > best || (ov == best && op < pos)) {
				best = ov;
				pos = op;
			}
		}
		has = best > -INFINITY;
		if (has) {
			si = pos < lt ? ls - 1 : pos - lt;
			sj = pos < lt ? pos : lt - 1;
		}
	}
	if (lane == 0) {
		p.score[pair] = has ? best * p.sign : -INFINITY * p.sign;
		p.seed[2 * pair] = si;
		p.seed[2 * pair + 1] = sj;
		p.has_seed[pair] = has;
	}
	if (!p.maps) return;
	int32_t *map = p.maps + p.map_off[pair];
	for (int k = lane; k < min(ls, lt); k += 32) map[k] = -1;
	__syncwarp();
	if (!has) return;
	int u = si, v = sj;
	while (u >= 0 && v >= 0) {
		const int iu = u - lane, iv = v - lane;
		bool diag = false;
		if (iu >= 0 && iv >= 0) {
			const float d = V(iu, iv), dg = V(iu - 1, iv - 1) + similarity(p, pair, iu, iv);
			// no scan candidate beat the diagonal (a NaN diagonal outside local alignment stays)
			diag = (!local || d > 0.0f) && (d == dg || (!local && isnan(dg)));
		}
		const uint32_t bal = __ballot_sync(0xffffffffu, diag);
		const int run = bal == 0xffffffffu ? 32 : __ffs(int(~bal)) - 1;
		if (run > 0) {
			if (lane < run) {
				if (ls <= lt) map[iu] = iv;
				else map[iv] = iu;
			}
			u -= run;
			v -= run;
			continue;
		}
		const float d = V(u, v);
		if (local && !(d > 0.0f)) break;
		int nu = u, nv = v;
		// both scans 128 positions at a time, every load of a batch in flight: the first hit of
		// the vertical one (k = q - 1), else of the horizontal one
		int kv = INT_MAX, kh = INT_MAX;
		for (int q0 = 0; q0 <= max(u, v) && kv == INT_MAX; q0 += 128) {
			float xv[4], xh[4];
#pragma unroll
			for (int r = 0; r < 4; r++) {
				const int q = q0 + 32 * r + lane;
				xv[r] = q <= u ? (q == 0 ? p.top_D[v + 1] : DT[int64_t(v) * ldt + q - 1]) + p.ngap_s[u + 1 - q] : NAN;
				xh[r] = q <= v ? (q == 0 ? p.left_D[u + 1] : D[int64_t(u) * ld + q - 1]) + p.ngap_t[v + 1 - q] : NAN;
			}
#pragma unroll
			for (int r = 0; r < 4; r++) {
				const uint32_t bv = __ballot_sync(0xffffffffu, xv[r] == d), bh = __ballot_sync(0xffffffffu, xh[r] == d);
				if (bv && kv == INT_MAX) kv = q0 + 32 * r + __ffs(int(bv)) - 2;
				if (bh && kh == INT_MAX) kh = q0 + 32 * r + __ffs(int(bh)) - 2;
			}
		}
		const bool found = kv != INT_MAX || kh != INT_MAX;
		if (kv != INT_MAX) nu = kv;
		else nv = kh;
		if (!found) break;  // a launch that gave up (ST_TIMEOUT): not a value of this kernel
		u = nu;
		v = nv;
	}
}

}  // namespace

cudaError_t launch_wsb_tiles(const WsbTileParams &p, int sm_count, cudaStream_t st) {
	if (p.npairs == 0) return cudaSuccess;
	if (p.ntiles > 0) {
		// the attribute belongs to the device's copy of the kernel; setting it again is cheap
		if (cudaError_t e = cudaFuncSetAttribute(wsb_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                                         int(sizeof(Smem))))
			return e;
		const int grid = p.ntiles < sm_count * 4 ? p.ntiles : sm_count * 4;
		wsb_tile_kernel<<<grid, 128, sizeof(Smem), st>>>(p);
		if (cudaError_t e = cudaGetLastError()) return e;
	}
	wsb_tile_walk_kernel<<<(p.npairs + 3) / 4, 128, 0, st>>>(p);
	return cudaGetLastError();
}

}  // namespace pa
