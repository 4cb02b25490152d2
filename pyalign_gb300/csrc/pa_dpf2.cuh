// Two-column float32 DP kernel (sm_103a).
//
// Same recurrences, tie rules, seeds and float32 operations as dp_kernel (pa_dp.cuh;
// solver.h:2825-2855, 2970-3036, 3213-3251, 1226-1427, 1980-2327) for float scoring without
// all-optimal masks or Solution values, in group mode: results are bit-identical.  A lane updates
// its R = 8 rows in two adjacent columns per step (traceback words in the dp2_kernel layout), so
// a step's shuffles, loads, stores and bookkeeping serve 16 cells.
//
// What bounds it with many pairs is issue and the ALU pipe (compares, selects, maxima: 64 lanes
// a clock and SM; adds run at 128 and integer multiply-adds at 64 on the FMA pipe beside it).  So
// a cell does on the ALU pipe only what must be there -- 8 operations per affine cell, see cell_f
// -- its compares' predicates are the traceback flags, and these enter the step's traceback word
// by predicated multiply-adds of constants, one per flag.  Similarities enter by one fused
// multiply-add with the direction's sign (exact: the product is +-S).  Local seeds: the step's
// largest value is folded by three-way maxima and compared with the lane's best once per step;
// only a step that reaches it looks for the row and column.
//
// SUBF_DENSE: S with stride 1 along s; each lane keeps the next column pairs of its 8 rows in
// flight in a shared-memory ring (16-byte cp.async), laid out so that the lanes of a warp read
// consecutive 16-byte words.  Measured against dp_kernel
// (both with tuned group widths): 4,096 series pairs of 128..1024, DTW, 1.75 -> 0.85 ms; 8,192
// dense pairs of 32..512, global Gotoh, 1.72 -> 0.87 ms; 4,096 of 64..256 423 -> 209 us.  1,024
// dense pairs of 100..400, local, 0.98 -> 0.38 ms: there one warp per pair and the chain of cells
// down its rows bound it (issue 52%, 1.7 warps per scheduler).
#pragma once

#include "pa_dp.cuh"

namespace pa {

enum { SUBF_DENSE = 0, SUBF_SERIES = 1, SUBF_TABLE = 2 };
constexpr int DPF2_RING = 4;  // column pairs in flight per lane (one less than the slots)

// The traceback words of a step before its cells: 8 nibbles (row r at bits 4 (R - 1 - r)) of code
// 2, the diagonal, or for local alignment 3, zero.  Cells subtract from the code and add the
// extend bits.
template <int LOC>
struct WordF {
	static constexpr int32_t value = LOC == LOC_LOCAL ? 0x33333333 : 0x22222222;
};

// One cell of row r: (D, P) from above, the D to the left and its Q, the diagonal D and the
// similarity (sign * S is added to the diagonal); Q is updated in place, the traceback flags go
// into mw (see WordF; the nibble is code | P-extend << 2 | Q-extend << 3).
//
// The tie rule (zero, diagonal, P, Q: a later one wins only when strictly larger) and NaN (a NaN
// never wins a compare, but stays where it comes first) with one maximum less in the chain: the
// gaps' larger value m = max(P, Q), which ignores a NaN beside a number, wins over the head when
// m > head; it is P's when P equals m, else Q's.
template <int GAP, int LOC, int TB, int ROW>
__device__ __forceinline__ void cell_f(const DpParams<float> &p, float S, float sign, float dsave, float old, float &Q,
                                       float uD, float uP, float &D, float &P, int32_t &mw) {
	constexpr int SH = 4 * (R - 1 - ROW);
	constexpr int32_t ONE = -(1 << SH);                           // code - 1
	constexpr int32_t TWO = int32_t(0u - (2u << SH));             // code - 2
	constexpr int32_t PX = int32_t(4u << SH), QX = int32_t(8u << SH);  // extend bits
	constexpr bool tb = TB == TB_ONE;
	float head = GAP == GAP_DTW ? dsave : __fmaf_rn(S, sign, dsave);
	float gs, gt;  // the vertical and the horizontal candidate
	if (GAP == GAP_AFFINE) {
		const float oP = uD + p.c_open_s, eP = uP + p.c_ext_s, oQ = old + p.c_open_t, eQ = Q + p.c_ext_t;
		if (tb) {
			asm("{.reg .pred p, q;\n\t"
			    "setp.gt.f32 p, %4, %3;\n\tselp.f32 %0, %4, %3, p;\n\t"
			    "setp.gt.f32 q, %6, %5;\n\tselp.f32 %1, %6, %5, q;\n\t"
			    "@p mad.lo.s32 %2, %7, %8, %2;\n\t@q mad.lo.s32 %2, %7, %9, %2;}"
			    : "=&f"(gs), "=&f"(gt), "+r"(mw)
			    : "f"(oP), "f"(eP), "f"(oQ), "f"(eQ), "r"(p.one), "n"(PX), "n"(QX));
		} else {
			gs = eP > oP ? eP : oP;
			gt = eQ > oQ ? eQ : oQ;
		}
		P = gs;
		Q = gt;
	} else if (GAP == GAP_LINEAR) {
		gs = uD + p.c_up;
		gt = old + p.c_left;
		P = gs;
	} else {
		gs = uD;
		gt = old;
	}
	if (tb && LOC != LOC_LOCAL) {
		asm("{.reg .pred x, w;\n\t.reg .f32 m;\n\t"
		    "max.f32 m, %3, %4;\n\tsetp.gt.f32 x, m, %2;\n\tselp.f32 %0, m, %2, x;\n\t"
		    "setp.neu.and.f32 w, %3, m, x;\n\t"
		    "@x mad.lo.s32 %1, %5, %6, %1;\n\t@w mad.lo.s32 %1, %5, %6, %1;}"
		    : "=&f"(D), "+r"(mw)
		    : "f"(head), "f"(gs), "f"(gt), "r"(p.one), "n"(ONE));
	} else if (tb) {
		asm("{.reg .pred x, y, w, t;\n\t.reg .f32 m, h;\n\t"
		    "max.f32 m, %3, %4;\n\tmax.f32 h, %2, 0f00000000;\n\t"
		    "setp.gt.f32 x|y, m, h;\n\tselp.f32 %0, m, h, x;\n\t"
		    "setp.neu.and.f32 w, %3, m, x;\n\tsetp.gt.and.f32 t, %2, 0f00000000, y;\n\t"
		    "@x mad.lo.s32 %1, %5, %7, %1;\n\t@w mad.lo.s32 %1, %5, %6, %1;\n\t@t mad.lo.s32 %1, %5, %6, %1;}"
		    : "=&f"(D), "+r"(mw)
		    : "f"(head), "f"(gs), "f"(gt), "r"(p.one), "n"(ONE), "n"(TWO));
	} else {
		if (LOC == LOC_LOCAL) head = fmaxf(head, 0.0f);
		const float m = fmaxf(gs, gt);
		D = m > head ? m : head;
	}
	if (GAP == GAP_DTW) D = __fmaf_rn(S, sign, D);
}

__device__ __forceinline__ float max3f(float a, float b, float c) {
	float d;
	asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
	return d;
}

template <int GAP, int LOC, int TB, int SUB>
__global__ void __launch_bounds__(BLOCK, 4) dpf2_kernel(DpParams<float> p) {
	static_assert(TB != TB_ALL, "all-optimal masks use dp_kernel");
	constexpr bool LOCSEED = LOC == LOC_LOCAL;
	if (!codes_valid(p)) return;

	extern __shared__ __align__(16) unsigned char smem_raw[];
	float *stab = reinterpret_cast<float *>(smem_raw);
	const bool table_in_smem = SUB == SUBF_TABLE && p.table_rows <= MAX_SMEM_TABLE && p.table_cols <= MAX_SMEM_TABLE;
	if (table_in_smem) {
		const int n = p.table_rows * p.table_cols;
		for (int k = threadIdx.x; k < n; k += blockDim.x) stab[k] = p.table[k];
		__syncthreads();
	}
	const float *tab = table_in_smem ? stab : p.table;
	// slot s, word q of this thread: ring[(4 s + q) * BLOCK] (words: column j0 rows 0-3, 4-7, column j1)
	float4 *ring = reinterpret_cast<float4 *>(smem_raw) + threadIdx.x;

	const int G = p.G;
	const int lane = threadIdx.x & 31;
	const int sub = lane % G;
	const int grp = lane / G;
	const int gpw = 32 / G;
	const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const int slot = warp_global * gpw + grp;
	const int64_t half = p.scratch_stride / 2;
	const float NEG = p.neg_inf;
	const int rpp = G * R;
	const float sign = SUB == SUBF_TABLE ? 1.0f : p.dense_sign;  // (tables come normalised)
	float2 *scr = reinterpret_cast<float2 *>(p.scratch) + int64_t(slot) * p.scratch_stride;
	int cursor = -2;

	for (;;) {
		const int2 task = next_task(p.work_counter, p.spread, p.spread_classes, p.spread_size,
		                            (p.npairs + gpw - 1) / gpw, cursor);
		if (task.x < 0) break;
		cursor = task.y;
		const int w = task.x * gpw + grp;
		const int pair = w < p.npairs ? p.order[w] : -1;
		const int ls = pair >= 0 ? p.len_s[pair] : 0;
		const int lt = pair >= 0 ? p.len_t[pair] : 0;
		const bool empty = ls == 0 || lt == 0;
		const int npass = empty ? 0 : (ls + rpp - 1) / rpp;
		const int nsteps_pair = ((lt + 1) >> 1) + G - 1;
		int wpass = npass, wsteps = empty ? 0 : nsteps_pair;
		for (int o = 16; o > 0; o >>= 1) {
			wpass = max(wpass, __shfl_xor_sync(0xffffffffu, wpass, o));
			wsteps = max(wsteps, __shfl_xor_sync(0xffffffffu, wsteps, o));
		}
		const uint32_t *arow = SUB != SUBF_DENSE ? p.a + int64_t(pair < 0 ? 0 : pair) * p.a_stride : nullptr;
		const uint32_t *brow = SUB != SUBF_DENSE ? p.b + int64_t(pair < 0 ? 0 : pair) * p.b_stride : nullptr;
		const float *drow = SUB == SUBF_DENSE ? p.dense + (pair >= 0 ? p.dense_off[pair] : 0) : nullptr;

		float l_best = NEG;
		int l_bi = -1, l_bj = -1;
		float row_best = NEG;
		int row_bj = -1;
		float col_best = NEG;
		int col_bi = -1;
		float glob = NEG;
		bool have_glob = false;

		for (int q = 0; q < wpass; q++) {
			const bool pass_active = q < npass;
			const int row0 = q * rpp + sub * R;
			const int nvalid = ls - row0;
			const float4 *bin = reinterpret_cast<const float4 *>(scr + (q & 1) * half);  // a step's (D, P) pairs
			float4 *bout = reinterpret_cast<float4 *>(scr + ((q + 1) & 1) * half);
			const bool write_boundary = sub == G - 1 && q + 1 < npass;
			// lane 0: (D, P) above the next step's two columns, read one step ahead -- the top
			// border, or what this warp's last lane wrote in the previous pass (rows of the
			// boundary hold an even number of columns: a last odd column's partner is unused)
			float4 bn = make_float4(NEG, NEG, NEG, NEG);
			if (sub == 0 && pass_active) {
				if (q == 0) {
					bn.x = p.top_D[1];
					if (lt > 1) bn.z = p.top_D[2];
				} else {
					bn = bin[0];
				}
			}
			uint32_t qa[R];  // codes of the rows (the series' raw values); the table's row offsets
			float Dl[R], Ql[R];
#pragma unroll
			for (int r = 0; r < R; r++) {
				const int i = row0 + r;
				const bool in = pass_active && i < ls;
				qa[r] = SUB != SUBF_DENSE && in ? arow[i] : 0u;
				if (SUB == SUBF_TABLE) qa[r] *= uint32_t(p.table_cols);
				Dl[r] = in ? p.left_D[i + 1] : NEG;
				Ql[r] = NEG;
			}
			float outD0 = Dl[R - 1], outP0 = NEG, outD1 = Dl[R - 1], outP1 = NEG;
			float prev_up = (pass_active && row0 <= ls) ? p.left_D[row0] : NEG;  // D(row0 - 1, j0 - 1)
			const bool last_row_lane = pass_active && nvalid >= 1 && nvalid <= R;
			const int r_last = nvalid - 1;
			uint32_t tn0 = SUB != SUBF_DENSE && pass_active ? brow[0] : 0u;
			uint32_t tn1 = SUB != SUBF_DENSE && pass_active && lt > 1 ? brow[1] : 0u;
			uint2 *mrow = nullptr;
			if (TB == TB_ONE && pass_active)
				mrow = reinterpret_cast<uint2 *>(p.masks) + p.mask_off[pair] / 2 + int64_t(q) * nsteps_pair * G + sub;

			// dense: column pair jp's words into ring slot jp % DPF2_RING, one commit group per
			// step.  Four rows are read whole: the host admits only layouts whose row count is a
			// multiple of 4, so they exist (cells past |s| are never used)
			const float *dcol = SUB == SUBF_DENSE ? drow + row0 : nullptr;  // column 2 jp of the next fetch
			const bool half0 = pass_active && nvalid > 0, half1 = pass_active && nvalid > 4;
			auto fetch = [&](int jp) {
				if constexpr (SUB == SUBF_DENSE) {
					float4 *dst = ring + (jp & (DPF2_RING - 1)) * 4 * BLOCK;
					const float *src1 = dcol + p.dense_sj;
					const bool c0 = 2 * jp < lt, c1 = 2 * jp + 1 < lt;
					if (c0 && half0) cp_async16(dst, dcol);
					if (c0 && half1) cp_async16(dst + BLOCK, dcol + 4);
					if (c1 && half0) cp_async16(dst + 2 * BLOCK, src1);
					if (c1 && half1) cp_async16(dst + 3 * BLOCK, src1 + 4);
					cp_async_commit();
					dcol = src1 + p.dense_sj;  // called for jp = 0, 1, 2, ...
				}
			};
			if constexpr (SUB == SUBF_DENSE)
				for (int k = 0; k < DPF2_RING - 1; k++) fetch(k);

			for (int s = 0; s < wsteps; s++) {
				const int jp = s - sub, j0 = 2 * jp, j1 = j0 + 1;
				float upD0 = __shfl_up_sync(0xffffffffu, outD0, 1, G);
				float upD1 = __shfl_up_sync(0xffffffffu, outD1, 1, G);
				float upP0 = NEG, upP1 = NEG;
				if (GAP == GAP_AFFINE) {
					upP0 = __shfl_up_sync(0xffffffffu, outP0, 1, G);
					upP1 = __shfl_up_sync(0xffffffffu, outP1, 1, G);
				}
				const bool act = pass_active && jp >= 0 && j0 < lt;
				const bool act1 = act && j1 < lt;
				const uint32_t tc0 = tn0, tc1 = tn1;
				if (SUB != SUBF_DENSE) {
					if (act && j0 + 2 < lt) tn0 = brow[j0 + 2];
					if (act && j0 + 3 < lt) tn1 = brow[j0 + 3];
				}
				if (sub == 0 && act) {
					upD0 = bn.x;
					upP0 = bn.y;
					upD1 = bn.z;
					upP1 = bn.w;
					if (j0 + 2 < lt) {
						if (q == 0) {
							bn.x = p.top_D[j0 + 3];
							if (j0 + 3 < lt) bn.z = p.top_D[j0 + 4];
						} else {
							bn = bin[jp + 1];
						}
					}
				}
				if (act) {
					float S0[R], S1[R];
					if constexpr (SUB == SUBF_DENSE) {
						// this step's group is complete once at most DPF2_RING - 2 newer ones remain;
						// the refill goes to the slot read in the previous step
						cp_async_wait<DPF2_RING - 2>();
						const float4 *src = ring + (jp & (DPF2_RING - 1)) * 4 * BLOCK;
						const float4 a = src[0], b = src[BLOCK], c = src[2 * BLOCK], d = src[3 * BLOCK];
						fetch(jp + DPF2_RING - 1);
						S0[0] = a.x, S0[1] = a.y, S0[2] = a.z, S0[3] = a.w;
						S0[4] = b.x, S0[5] = b.y, S0[6] = b.z, S0[7] = b.w;
						S1[0] = c.x, S1[1] = c.y, S1[2] = c.z, S1[3] = c.w;
						S1[4] = d.x, S1[5] = d.y, S1[6] = d.z, S1[7] = d.w;
					} else if constexpr (SUB == SUBF_SERIES) {
#pragma unroll
						for (int r = 0; r < R; r++) {
							S0[r] = fabsf(__uint_as_float(qa[r]) - __uint_as_float(tc0));
							S1[r] = fabsf(__uint_as_float(qa[r]) - __uint_as_float(tc1));
						}
					} else {
#pragma unroll
						for (int r = 0; r < R; r++) {
							S0[r] = tab[qa[r] + tc0];
							S1[r] = tab[qa[r] + tc1];
						}
					}
					int32_t mw0 = WordF<LOC>::value, mw1 = WordF<LOC>::value;
					float dsave0 = prev_up, dsave1 = upD0;  // D(i-1, j0-1), D(i-1, j0) for row 0
					float uD0 = upD0, uP0 = upP0, uD1 = upD1, uP1 = upP1;
					float c0[R];  // column j0 (Dl: column j1 after the step, past |t| in a last odd column)
					auto row = [&](auto rc) {
						constexpr int r = decltype(rc)::value;
						const float old = Dl[r];
						float Q = Ql[r], D0, P0 = NEG, D1, P1 = NEG;
						cell_f<GAP, LOC, TB, r>(p, S0[r], sign, dsave0, old, Q, uD0, uP0, D0, P0, mw0);
						cell_f<GAP, LOC, TB, r>(p, S1[r], sign, dsave1, D0, Q, uD1, uP1, D1, P1, mw1);
						dsave0 = old;
						dsave1 = D0;
						c0[r] = D0;
						Dl[r] = D1;
						Ql[r] = Q;
						uD0 = D0;
						uP0 = P0;
						uD1 = D1;
						uP1 = P1;
					};
					row(std::integral_constant<int, 0>());
					row(std::integral_constant<int, 1>());
					row(std::integral_constant<int, 2>());
					row(std::integral_constant<int, 3>());
					row(std::integral_constant<int, 4>());
					row(std::integral_constant<int, 5>());
					row(std::integral_constant<int, 6>());
					row(std::integral_constant<int, 7>());
					outD0 = uD0;
					outP0 = uP0;
					outD1 = uD1;
					outP1 = uP1;
					if (write_boundary) bout[jp] = make_float4(outD0, outP0, outD1, outP1);
					if (TB == TB_ONE) *mrow = make_uint2(uint32_t(mw0), uint32_t(mw1));
					if (LOCSEED) {
						float m0, m1;
						if (nvalid >= R) {
							m0 = max3f(max3f(c0[0], c0[1], c0[2]), max3f(c0[3], c0[4], c0[5]), fmaxf(c0[6], c0[7]));
							m1 = max3f(max3f(Dl[0], Dl[1], Dl[2]), max3f(Dl[3], Dl[4], Dl[5]), fmaxf(Dl[6], Dl[7]));
						} else {  // rows past |s| are no seeds
							m0 = m1 = NEG;
#pragma unroll
							for (int r = 0; r < R; r++)
								if (r < nvalid) {
									m0 = fmaxf(m0, c0[r]);
									m1 = fmaxf(m1, Dl[r]);
								}
						}
						if (!act1) m1 = NEG;
						const float m = fmaxf(m0, m1);
						if (TB == TB_NONE) {
							l_best = fmaxf(l_best, m);
						} else if (m >= l_best && m > NEG) {
							// the step's cell of that value with the largest row, then column; it replaces an
							// equal best of a row not below it (solver.h:2048-2056)
							int bi = -1, bj = -1;
#pragma unroll
							for (int r = 0; r < R; r++)
								if (r < nvalid) {
									if (c0[r] == m) bi = r, bj = j0;
									if (act1 && Dl[r] == m) bi = r, bj = j1;
								}
							if (m > l_best || row0 + bi >= l_bi) {
								l_best = m;
								l_bi = row0 + bi;
								l_bj = bj;
							}
						}
					} else {
						const bool odd = j0 == lt - 1, last = odd || j1 == lt - 1;
						if (last_row_lane && q == npass - 1 && (LOC == LOC_SEMI || last)) {
							float x0 = c0[0], x1 = Dl[0];  // the last row's values
#pragma unroll
							for (int r = 1; r < R; r++)
								if (r == r_last) x0 = c0[r], x1 = Dl[r];
							if (LOC == LOC_SEMI) {
								if (x0 > row_best) { row_best = x0; row_bj = j0; }
								if (act1 && x1 > row_best) { row_best = x1; row_bj = j1; }
							} else {
								glob = odd ? x0 : x1;
								have_glob = true;
							}
						}
						if (LOC == LOC_SEMI && last) {
#pragma unroll
							for (int r = 0; r < R; r++) {
								const float x = odd ? c0[r] : Dl[r];
								if (r < nvalid && x > col_best) { col_best = x; col_bi = row0 + r; }
							}
						}
					}
				}
				if (TB == TB_ONE) mrow += G;
				prev_up = upD1;
			}
			__syncwarp();
		}
		finish_pair<float, LOC, TB, false, false>(p, G, sub, pair, ls, lt, empty, npass, 0, -1, 0, NEG, l_best, l_bi,
		                                          l_bj, row_best, row_bj, col_best, col_bi, glob, have_glob);
	}
}

}  // namespace pa
