// Packed 16-bit DP kernel for scores alone, and with one traceback (sm_103a).
//
// Same recurrences and scores as dp_kernel (pa_dp.cuh; solver.h:2825-2855, 2970-3036, 1980-2327)
// for integer scoring whose values provably fit in 16 bits.  As in dp16_kernel (pa_dp16.cuh)
// every 32-bit register holds the same cell of two pairs -- a twin of consecutive pairs of the
// processing order -- and every add and maximum updates both.  Without a traceback there is
// nothing to tag: values are plain signed 16-bit numbers (value + offset, offset 0 for local
// alignment), which quadruples dp16_kernel's range -- 5000 x 10000 residues fit -- and leaves a
// cell four ALU operations (the similarity's byte permute, P, Q and the three-way maximum with
// the zero floor in the same instruction) and three packed adds on the FMA pipe for two pairs.
// The int32 kernels issue about ten for one.
//
// A lane updates 8 rows in two adjacent columns per step.  Similarities are int8: up to 4 letters
// of t as row profiles in registers (SUBS_PROFILE, one byte permute per twin cell picks both
// halves and extends their signs), up to 32 as column profiles in shared memory (SUBS_COLPROF:
// per letter and thread the 8 scores of the thread's rows, one 64-bit load per pair and column,
// then the same permute).  What a step needs to know of its two columns' letters -- the permute
// selectors, or the profiles' offsets -- is worked out once per column, not once per lane: every
// 16 steps each group turns its next 32 columns into words of a ring in shared memory, and a step
// reads its pair of words in one load.
//
// Group mode: a group of G lanes per twin sweeps its stripes of 8 G rows.  Stripe-chained mode
// (CHAIN, G = 32): a warp per 256-row stripe, as in pa_dp.cuh, with the boundary rows moved 32
// columns at a time: the row above arrives by one coalesced load of the warp into shared memory,
// a chunk ahead where it is already there, and this stripe's last row leaves through shared
// memory by one coalesced store and one release per chunk, so that no step waits for L2 and no
// lane runs code of its own.
//
// Cells past a pair's own lengths (the twin computes the larger shape): rows past |s| score -128,
// so a local optimum cannot lie there alone (a gap costs at least 0), and the global and
// semiglobal results are read at the pair's own last row and column; columns past |t| of the
// shorter pair are masked out of the local maximum.  The host's bounds cover the whole rectangle,
// padding rows included.
//
// Measured against the int32 kernels it replaces (DP alone): 32,768 DNA pairs of 100..250 x
// 200..500, local Gotoh, 1.41 -> 0.63-0.66 ms; 256 pairs of 5000 x 10000 residues, semiglobal Gotoh,
// chained, 10.6 -> 5.4 ms.  What bounds it: group mode issue (66%) and the ALU pipe (59%); chained,
// four to five warps per scheduler on 229 instructions a step and the waits of one stripe for the
// one above (issue 53%).
#pragma once

#include "pa_dp16.cuh"

namespace pa {

// With one traceback (TB): value * 4 + tag, the tag's order zero 3 > diagonal 2 > P 1 > Q 0 as in the
// int32 kernels.  P = max(extend, open) is formed with tag 0 for its extension and 1 for its
// opening, Q with 0 and 2 -- among equals the opening wins -- and then P takes its tag 1 and Q its
// tag 0 for the choice of D.  The nibble of a cell, 4 (key - D) + (the opening bits), is dp16_kernel's
// (code in bits 2-3, P-open bit 0, Q-open bit 1), worked out on the FMA pipe: differences of packed
// values and the shift by a nibble are integer multiply-adds, exact in the end although a half may
// borrow on the way.  Four tag values leave a quarter of the range (600 residues at 11 each still
// fit, scores of -32 .. 31), eight ALU operations a twin cell of affine gaps.  Seeds as dp2_kernel's:
// a local optimum's position is looked for only in steps whose maximum reaches the lane's best.
// DNA that fits dp16_kernel's bounds stays there.  4,096 protein pairs of 50..600, global Gotoh, DP
// alone: int32 0.73 -> 0.55 ms (too few pairs to fill the GPU with twins); whole calls, 6,400 of
// 79..479 x 64..645 global linear 0.86 -> 0.61 ms.

enum { SUBS_PROFILE = 0, SUBS_COLPROF = 1 };
constexpr int CHAIN_CHUNK = PUB_CHUNK;  // boundary columns read at a time

__device__ __forceinline__ uint32_t s_add(uint32_t a, uint32_t b) {
	uint32_t d;
	asm("add.s16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
	return d;
}

// One cell of each half; D and P of this cell, Q in place.
template <int GAP, int LOC>
__device__ __forceinline__ void cell_s16(const DpParams<int32_t> &p, uint32_t S, uint32_t dsave, uint32_t old,
                                         uint32_t &Q, uint32_t uD, uint32_t uP, uint32_t &D, uint32_t &P) {
	if (GAP == GAP_AFFINE) {
		P = __viaddmax_s16x2(uP, p.h_ext_s, s_add(uD, p.k_open_s));
		Q = __viaddmax_s16x2(Q, p.h_ext_t, s_add(old, p.k_open_t));
	} else {
		P = s_add(uD, p.k_up);
		Q = s_add(old, p.k_left);
	}
	const uint32_t t = s_add(dsave, S);
	D = LOC == LOC_LOCAL ? __vimax3_s16x2_relu(t, P, Q) : __vimax3_s16x2(t, P, Q);
}

// The same with a traceback: the tagged key, D and P clean but for P's tag 1, Q clean; `open`
// receives a word whose difference to the clean Q is the opening bits.
template <int GAP, int LOC>
__device__ __forceinline__ uint32_t cell_t16(const DpParams<int32_t> &p, uint32_t S, uint32_t dsave, uint32_t old,
                                             uint32_t &Q, uint32_t uD, uint32_t uP, uint32_t &D, uint32_t &P,
                                             uint32_t &open) {
	constexpr uint32_t CLEAN = 0xFFFCFFFCu, ONE = 0x00010001u, ZERO = 0x00030003u;
	if (GAP == GAP_AFFINE) {
		const uint32_t rP = __viaddmax_s16x2(uP, p.h_ext_s, s_add(uD, p.k_open_s));
		const uint32_t rQ = __viaddmax_s16x2(Q, p.h_ext_t, s_add(old, p.k_open_t));
		open = (rP & ONE) | (rQ & ~ONE);
		P = (rP & CLEAN) | ONE;
		Q = rQ & CLEAN;
	} else {
		P = s_add(uD, p.k_up);
		Q = s_add(old, p.k_left);
	}
	const uint32_t key = LOC == LOC_LOCAL ? __viaddmax_s16x2(dsave, S, __vimax3_s16x2(P, Q, ZERO))
	                                      : __vimax3_s16x2(s_add(dsave, S), P, Q);
	D = key & CLEAN;
	return key;
}

// The cell's nibbles behind those of the rows above it, in each half of w.
template <int GAP>
__device__ __forceinline__ void put_nib_t16(const DpParams<int32_t> &p, uint32_t &w, uint32_t key, uint32_t D, uint32_t Q,
                                            uint32_t open) {
	const int32_t below = imad(int32_t(key), p.minus_one, int32_t(D));  // -(the code)
	if (GAP == GAP_AFFINE)
		w = uint32_t(imad(below, p.minus_four, imad(int32_t(Q), p.minus_one, imad(int32_t(w), p.sixteen, int32_t(open)))));
	else
		w = uint32_t(imad(imad(int32_t(w), p.minus_four, below), p.minus_four, 0));
}

// Warps of a block: in stripe-chained mode one, so that the stripes in flight spread evenly over
// the SMs (a stripe cannot outrun the one above it, so the fullest SM sets the pace of all: 2,560
// stripes lie 16 or 17 to an SM; in blocks of four, 16 or 20).
__host__ __device__ constexpr int s16_warps(bool chain) { return chain ? 1 : WARPS; }
// Columns of a letter ring: those of a group's lanes in flight and one chunk, a power of two
__host__ __device__ constexpr int s16_ring(int G) { return G == 32 ? 128 : 64; }
// Shared memory of a block's letter rings and chunk buffers, in bytes.  A ring is padded by the
// columns of its group's lanes, so the groups of a warp read distinct banks.  (With 20 letters the
// column profiles leave 45 KB blocks, five to an SM, room for 4 KB of these: hence 2-byte words
// and one buffer per direction.)
__host__ __device__ constexpr int s16_smem(int G, bool colprof, bool chain) {
	return s16_warps(chain) * ((32 / G) * (s16_ring(G) + 2 * G) * (colprof ? 2 : 4) + (chain ? 2 * CHAIN_CHUNK * 8 : 0));
}

// The most dynamic shared memory a launch asks for: the table, the rings, 32 column profiles
constexpr int S16_SMEM_MOST = MAX_SMEM_TABLE * MAX_COLPROF + s16_smem(1, true, false) + MAX_COLPROF * 32 * WARPS * 16;
static_assert(s16_smem(1, false, false) <= S16_SMEM_MOST && s16_smem(32, true, true) <= S16_SMEM_MOST, "rings");

template <int GAP, int LOC, int SUB, bool CHAIN, bool TB>
__global__ void __launch_bounds__(32 * s16_warps(CHAIN), CHAIN ? (TB ? 16 : 17) : 4) dps16_kernel(DpParams<int32_t> p) {
	constexpr bool LOCAL = LOC == LOC_LOCAL;
	constexpr int32_t NONE = INT32_MIN;
	constexpr int NW = s16_warps(CHAIN), NT = 32 * NW;  // warps and threads of a block
	constexpr int STEPS = CHAIN_CHUNK / 2;  // steps per chunk of 32 columns
	typedef typename std::conditional<SUB == SUBS_PROFILE, uint32_t, uint16_t>::type Word;
	if (!codes_valid(p)) return;

	extern __shared__ __align__(16) unsigned char smem_raw[];
	int8_t *stab = reinterpret_cast<int8_t *>(smem_raw);
	const int cols = p.table_cols;
	for (int k = threadIdx.x; k < p.table_rows * cols; k += blockDim.x) stab[k] = int8_t(p.table[k]);
	__syncthreads();
	const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
	const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const int G = CHAIN ? 32 : p.G;
	const int sub = lane % G, grp = lane / G, gpw = 32 / G;
	// after the table: this warp's chunk buffers (chained), its groups' letter rings, the column
	// profiles (letter c of pair h at colprof[(2 c + h) * NT + thread])
	unsigned char *sm = smem_raw + ((size_t(p.table_rows) * cols + 15) & ~size_t(15));
	uint2 *const chunk = reinterpret_cast<uint2 *>(sm) + wib * (2 * CHAIN_CHUNK);  // of the row above, and out
	uint2 *const outrow = chunk + CHAIN_CHUNK;
	if (CHAIN) sm += NW * 2 * CHAIN_CHUNK * 8;
	const int ring_n = s16_ring(G), ring_mask = ring_n - 1;
	Word *const ring = reinterpret_cast<Word *>(sm) + (wib * gpw + grp) * (ring_n + 2 * G);
	sm += size_t(NW) * gpw * (ring_n + 2 * G) * sizeof(Word);
	unsigned char *const colprof = sm + threadIdx.x * 8;

	const int slot = warp_global * gpw + grp;
	const int64_t half = p.scratch_stride / 2;
	const int ntwins = (p.npairs + 1) >> 1;
	const int rpp = G * R;
	const int32_t off = p.h_off;
	auto pack = [&](int32_t v) { return uint32_t(((TB ? 4 * v : v) + off) & 0xffff) * 0x10001u; };  // a value in both halves
	const uint32_t NEG = p.h_neg, LOW = p.h_low;
	int cursor = -2;

	for (;;) {
		int w = 0, q_lo = 0, prod = -1, base = 0;
		if constexpr (CHAIN) {
			if (lane == 0) base = atomicAdd(p.work_counter, 1);
			base = __shfl_sync(0xffffffffu, base, 0);
			if (base >= p.ntickets) break;
			int lo = 0, hi = p.nlevels - 1;
			while (lo < hi) {
				const int mid = (lo + hi + 1) >> 1;
				if (p.level_start[mid] <= base) lo = mid;
				else hi = mid - 1;
			}
			q_lo = lo;
			w = base - p.level_start[lo];
			if (lo > 0) prod = p.level_start[lo - 1] + w;
		} else {
			const int2 t = next_task(p.work_counter, p.spread, p.spread_classes, p.spread_size,
			                         (ntwins + gpw - 1) / gpw, cursor);
			if (t.x < 0) break;
			cursor = t.y;
			w = t.x * gpw + grp;
		}
		uint2 *scr = reinterpret_cast<uint2 *>(p.scratch) + int64_t(CHAIN ? w : slot) * p.scratch_stride;
		const int pa = w < ntwins ? p.order[2 * w] : -1;
		const int pb = (w < ntwins && 2 * w + 1 < p.npairs) ? p.order[2 * w + 1] : -1;
		const int lsA = pa >= 0 ? p.len_s[pa] : 0, ltA = pa >= 0 ? p.len_t[pa] : 0;
		const int lsB = pb >= 0 ? p.len_s[pb] : 0, ltB = pb >= 0 ? p.len_t[pb] : 0;
		const bool emptyA = lsA == 0 || ltA == 0, emptyB = lsB == 0 || ltB == 0;
		const int npA = emptyA ? 0 : (lsA + rpp - 1) / rpp, npB = emptyB ? 0 : (lsB + rpp - 1) / rpp;
		const int rsA = emptyA ? 0 : lsA, rsB = emptyB ? 0 : lsB;
		const int ctA = emptyA ? 0 : ltA, ctB = emptyB ? 0 : ltB;
		const int ls = max(rsA, rsB), lt = max(ctA, ctB), ctmin = min(ctA, ctB);
		const int npass = max(npA, npB);
		const int nsteps = ((lt + 1) >> 1) + G - 1;
		// (tickets count a pair without columns by its rows: those past the twin's stripes are void)
		if (CHAIN && q_lo > 0 && q_lo >= npass) continue;
		int wpass = npass, wsteps = npass ? nsteps : 0;
		for (int o = 16; o > 0; o >>= 1) {
			wpass = max(wpass, __shfl_xor_sync(0xffffffffu, wpass, o));
			wsteps = max(wsteps, __shfl_xor_sync(0xffffffffu, wsteps, o));
		}
		const uint32_t *arowA = p.a + int64_t(pa < 0 ? 0 : pa) * p.a_stride;
		const uint32_t *arowB = p.a + int64_t(pb < 0 ? 0 : pb) * p.a_stride;
		const uint32_t *browA = p.b + int64_t(pa < 0 ? 0 : pa) * p.b_stride;
		const uint32_t *browB = p.b + int64_t(pb < 0 ? 0 : pb) * p.b_stride;

		uint32_t l_best = 0;                 // local: the lane's best per half (at least 0)
		int32_t resA = NONE, resB = NONE;    // global: the result; semiglobal: the lane's best seed value
		// with a traceback: where the best lies (semiglobal: in the last column; rowA: the last row's)
		int32_t iA = -1, jA = -1, iB = -1, jB = -1, rowA = NONE, rowB = NONE;
		uint32_t reach = 0x00030003u;  // local: a maximum above this reaches the lane's best (and 0)

		const int q_hi = CHAIN ? min(q_lo + 1, npass) : wpass;
		for (int q = q_lo; q < q_hi; q++) {
			const bool pass_active = q < npass;
			const int row0 = q * rpp + sub * R;
			// (rows of the boundary hold an even number of columns, one 16-byte word per step)
			const uint4 *bin = reinterpret_cast<const uint4 *>(scr + (q & 1) * half);
			uint4 *bout = reinterpret_cast<uint4 *>(scr + ((q + 1) & 1) * half);
			const bool write_boundary = sub == G - 1 && q + 1 < npass;
			const int32_t *prog_in = CHAIN && q > 0 ? p.progress + prod : nullptr;
			int avail = 0;

			uint32_t prA[R], prB[R], Dl[R], Ql[R];
#pragma unroll
			for (int r = 0; r < R; r++) {
				const int i = row0 + r;
				const bool vA = pass_active && i < rsA, vB = pass_active && i < rsB;
				prA[r] = prB[r] = 0x80808080u;  // -128: a row past |s|
				const uint32_t ca = vA ? arowA[i] : 0u, cb = vB ? arowB[i] : 0u;
				if (SUB == SUBS_PROFILE) {
					if (vA)
						for (int c = 0; c < cols; c++)
							prA[r] = (prA[r] & ~(0xffu << (8 * c))) | ((uint32_t(stab[ca * cols + c]) & 0xffu) << (8 * c));
					if (vB)
						for (int c = 0; c < cols; c++)
							prB[r] = (prB[r] & ~(0xffu << (8 * c))) | ((uint32_t(stab[cb * cols + c]) & 0xffu) << (8 * c));
				} else {  // the rows' table offsets, for the column profiles below
					prA[r] = vA ? ca * cols : 0xffffffffu;
					prB[r] = vB ? cb * cols : 0xffffffffu;
				}
				Dl[r] = (pass_active && i < ls) ? pack(p.left_D[i + 1]) : LOW;
				Ql[r] = NEG;
			}
			if (SUB == SUBS_COLPROF) {
				for (int c = 0; c < cols; c++) {
					uint2 x = make_uint2(0u, 0u), y = x;
#pragma unroll
					for (int r = 0; r < R; r++) {
						const uint32_t a = prA[r] == 0xffffffffu ? 0x80u : uint32_t(stab[prA[r] + c]) & 0xffu;
						const uint32_t b = prB[r] == 0xffffffffu ? 0x80u : uint32_t(stab[prB[r] + c]) & 0xffu;
						(r < 4 ? x.x : x.y) |= a << (8 * (r & 3));
						(r < 4 ? y.x : y.y) |= b << (8 * (r & 3));
					}
					*reinterpret_cast<uint2 *>(colprof + (2 * c) * (NT * 8)) = x;
					*reinterpret_cast<uint2 *>(colprof + (2 * c + 1) * (NT * 8)) = y;
				}
			}
			uint32_t outD0 = Dl[R - 1], outP0 = NEG, outD1 = Dl[R - 1], outP1 = NEG;
			uint32_t prev_up = (pass_active && row0 <= ls) ? pack(p.left_D[row0]) : LOW;  // D(row0-1, j0-1)
			const int nvA = rsA - row0, nvB = rsB - row0;
			// global and semiglobal: this lane holds the last row of a pair in that pair's last stripe;
			// the steps in which it meets the pairs' last columns
			const bool lastA = pass_active && q == npA - 1 && nvA >= 1 && nvA <= R;
			const bool lastB = pass_active && q == npB - 1 && nvB >= 1 && nvB <= R;
			const int endA = ctA ? ((ctA - 1) >> 1) + sub : -1, endB = ctB ? ((ctB - 1) >> 1) + sub : -1;

			uint32_t *mA = nullptr, *mB = nullptr;  // this lane's traceback words of step 0
			if (TB) {
				uint32_t *m = reinterpret_cast<uint32_t *>(p.masks);
				if (pass_active && q < npA) mA = m + p.mask_off[pa] + (int64_t(q) * (((ltA + 1) >> 1) + G - 1) * G + sub) * 2;
				if (pass_active && q < npB) mB = m + p.mask_off[pb] + (int64_t(q) * (((ltB + 1) >> 1) + G - 1) * G + sub) * 2;
			}
			// semiglobal: a lane of the warp holds a last row in this pass (warp-uniform)
			const bool has_last = LOC == LOC_SEMI && __any_sync(0xffffffffu, lastA || lastB);
			uint32_t rmax[LOC == LOC_SEMI && !TB ? R : 1];
#pragma unroll
			for (int r = 0; r < (LOC == LOC_SEMI && !TB ? R : 1); r++) rmax[r] = 0x80008000u;

			// group mode: (D, P) above the next step's columns, for the group's first lane: the top
			// border, or what this warp's last lane wrote in the previous pass, a step ahead
			uint4 bn = make_uint4(NEG, NEG, NEG, NEG);
			if (!CHAIN && sub == 0 && pass_active) {
				if (q == 0) {
					bn.x = pack(p.top_D[1]);
					if (lt > 1) bn.z = pack(p.top_D[2]);
				} else {
					bn = bin[0];
				}
			}
			// chained: columns [32 c, 32 c + 32) of the row above, one per lane, into `above`; false
			// when they are not there yet (never with `wait`)
			uint2 above = make_uint2(NEG, NEG);
			auto fetch_chunk = [&](int c, bool wait) {
				const int j = c * CHAIN_CHUNK + lane, need = min(lt, (c + 1) * CHAIN_CHUNK);
				if (q == 0) {
					if (j < lt) above.x = pack(p.top_D[j + 1]);
					return true;
				}
				if (avail < need) {
					int v = 0;
					if (lane == 0) {
						v = ld_acquire(prog_in);
						if (v < need && wait) v = wait_progress(prog_in, need, p.status);
					}
					avail = __shfl_sync(0xffffffffu, v, 0);
					__syncwarp();  // the other lanes read after lane 0's acquire
					if (avail < need) return false;
				}
				if (j < lt) above = __ldcg(reinterpret_cast<const uint2 *>(bin) + j);
				return true;
			};
			bool ahead = false;  // `above` holds the next chunk
			// the 32 columns from j on as ring words, by the group's own lanes.  Up to four columns a
			// lane (G of 8 and more) are loaded a chunk ahead, so no step waits for memory.
			constexpr int AHEAD = CHAIN ? 1 : 4;
			uint32_t nA[AHEAD], nB[AHEAD];
			auto load_letters = [&](int j) {
#pragma unroll
				for (int k = 0; k < AHEAD; k++) {
					const int jj = j + sub + k * G;
					const bool in = k * G < CHAIN_CHUNK && jj < lt;
					nA[k] = in ? browA[jj] : 0u;
					nB[k] = in ? browB[jj] : 0u;
				}
			};
			auto put_word = [&](int jj, uint32_t cA, uint32_t cB) {
				if constexpr (SUB == SUBS_PROFILE)  // half A: byte cA of prA, half B: byte cB of prB, signs extended
					ring[jj & ring_mask] = cA * 0x11u + cB * 0x1100u + 0xC480u;
				else  // the two profiles' numbers
					ring[jj & ring_mask] = Word((2 * cA) | ((2 * cB + 1) << 8));
			};
			auto fill_ring = [&](int j) {
#pragma unroll
				for (int k = 0; k < AHEAD; k++)
					if (k * G < CHAIN_CHUNK) put_word(j + sub + k * G, nA[k], nB[k]);
				for (int k = sub + AHEAD * G; k < CHAIN_CHUNK; k += G)
					if (j + k < lt) put_word(j + k, browA[j + k], browB[j + k]);
				load_letters(j + CHAIN_CHUNK);
			};
			if (pass_active) load_letters(0);
			// chained: the finished part of this stripe's last row, columns [j, e), to memory, and
			// its progress
			auto put_row = [&](int j, int e) {
				__syncwarp();
				uint2 *o = reinterpret_cast<uint2 *>(bout);
				if (j + lane < e) __stcg(o + j + lane, outrow[lane]);
				__syncwarp();
				if (lane == 0 && e < lt) st_release(p.progress + base, e);
			};

			for (int s = 0; s < wsteps; s++) {
				const int j0 = 2 * (s - sub), j1 = j0 + 1;
				if ((s & (STEPS - 1)) == 0) {  // warp-uniform
					__syncwarp();  // the lanes are done with what the new words and chunk replace
					if (pass_active && 2 * s < lt) fill_ring(2 * s);
					if (CHAIN && 2 * s < lt) {
						const int c = s / STEPS;
						if (!ahead) fetch_chunk(c, true);
						chunk[lane] = above;
						ahead = (c + 1) * CHAIN_CHUNK < lt && fetch_chunk(c + 1, false);
					}
					__syncwarp();
				}
				uint32_t upD0 = __shfl_up_sync(0xffffffffu, outD0, 1, G);
				uint32_t upD1 = __shfl_up_sync(0xffffffffu, outD1, 1, G);
				uint32_t upP0 = 0u, upP1 = 0u;
				if (GAP == GAP_AFFINE) {
					upP0 = __shfl_up_sync(0xffffffffu, outP0, 1, G);
					upP1 = __shfl_up_sync(0xffffffffu, outP1, 1, G);
				}
				const bool act = pass_active && j0 >= 0 && j0 < lt;
				if (CHAIN) {
					const uint4 b = *reinterpret_cast<const uint4 *>(chunk + ((2 * s) & (CHAIN_CHUNK - 1)));
					if (sub == 0) {
						upD0 = b.x;
						upP0 = b.y;
						upD1 = b.z;
						upP1 = b.w;
					}
				} else if (sub == 0 && act) {
					upD0 = bn.x;
					upP0 = bn.y;
					upD1 = bn.z;
					upP1 = bn.w;
					if (j0 + 2 < lt) {
						if (q == 0) {
							bn.x = pack(p.top_D[j0 + 3]);
							if (j0 + 3 < lt) bn.z = pack(p.top_D[j0 + 4]);
						} else {
							bn = bin[s + 1];
						}
					}
				}
				if (act) {
					uint32_t sel0 = 0, sel1 = 0;
					uint2 xA0, xB0, xA1, xB1;
					if constexpr (SUB == SUBS_PROFILE) {
						const uint2 x = *reinterpret_cast<const uint2 *>(ring + (j0 & ring_mask));
						sel0 = x.x;
						sel1 = x.y;
					} else {
						uint32_t x = *reinterpret_cast<const uint32_t *>(ring + (j0 & ring_mask));
						if (j1 >= lt) x &= 0xffffu;  // (a last odd column's partner has no word)
						xA0 = *reinterpret_cast<const uint2 *>(colprof + (x & 0xffu) * (NT * 8));
						xB0 = *reinterpret_cast<const uint2 *>(colprof + ((x >> 8) & 0xffu) * (NT * 8));
						xA1 = *reinterpret_cast<const uint2 *>(colprof + ((x >> 16) & 0xffu) * (NT * 8));
						xB1 = *reinterpret_cast<const uint2 *>(colprof + (x >> 24) * (NT * 8));
					}
					uint32_t dsave0 = prev_up, dsave1 = upD0;
					uint32_t uD0 = upD0, uP0 = upP0, uD1 = upD1, uP1 = upP1;
					uint32_t c0[R];  // column j0 (Dl: column j1 after the step)
					uint32_t mlo0 = 0, mhi0 = 0, mlo1 = 0, mhi1 = 0;
					auto sub_of = [&](int r, uint32_t sel, uint2 a, uint2 b) {
						if (SUB == SUBS_PROFILE) return uint32_t(prmt(prA[r], prB[r], sel));
						return uint32_t(r < 4 ? prmt(a.x, b.x, uint32_t(r) * 0x1111u + 0xC480u)
						                      : prmt(a.y, b.y, uint32_t(r - 4) * 0x1111u + 0xC480u));
					};
#pragma unroll
					for (int r = 0; r < R; r++) {
						const uint32_t old = Dl[r];
						uint32_t Q = Ql[r], D0, P0, D1, P1;
						if constexpr (TB) {
							uint32_t open = 0;
							uint32_t key = cell_t16<GAP, LOC>(p, sub_of(r, sel0, xA0, xB0), dsave0, old, Q, uD0, uP0, D0, P0, open);
							put_nib_t16<GAP>(p, r < 4 ? mlo0 : mhi0, key, D0, Q, open);
							key = cell_t16<GAP, LOC>(p, sub_of(r, sel1, xA1, xB1), dsave1, D0, Q, uD1, uP1, D1, P1, open);
							put_nib_t16<GAP>(p, r < 4 ? mlo1 : mhi1, key, D1, Q, open);
						} else {
							cell_s16<GAP, LOC>(p, sub_of(r, sel0, xA0, xB0), dsave0, old, Q, uD0, uP0, D0, P0);
							cell_s16<GAP, LOC>(p, sub_of(r, sel1, xA1, xB1), dsave1, D0, Q, uD1, uP1, D1, P1);
						}
						dsave0 = old;
						dsave1 = D0;
						c0[r] = D0;
						Dl[r] = D1;
						Ql[r] = Q;
						uD0 = D0;
						uP0 = P0;
						uD1 = D1;
						uP1 = P1;
					}
					outD0 = uD0;
					outP0 = uP0;
					outD1 = uD1;
					outP1 = uP1;
					if (write_boundary) {
						const uint4 o = make_uint4(outD0, outP0, outD1, outP1);
						if (CHAIN) *reinterpret_cast<uint4 *>(outrow + (j0 & (CHAIN_CHUNK - 1))) = o;
						else bout[s - sub] = o;
					}
					if (TB) {
						// rows 0-3 of each half in mlo, 4-7 in mhi, row r at bits 4 (R - 1 - r) of the word
						if (mA && j0 < ctA)
							reinterpret_cast<uint2 *>(mA)[int64_t(s) * G] =
							    make_uint2(__byte_perm(mhi0, mlo0, 0x5410), __byte_perm(mhi1, mlo1, 0x5410));
						if (mB && j0 < ctB)
							reinterpret_cast<uint2 *>(mB)[int64_t(s) * G] =
							    make_uint2(__byte_perm(mhi0, mlo0, 0x7632), __byte_perm(mhi1, mlo1, 0x7632));
					}
					if (LOCAL) {
						uint32_t m0 = __vimax3_s16x2(c0[0], c0[1], c0[2]), m1 = __vimax3_s16x2(Dl[0], Dl[1], Dl[2]);
						m0 = __vimax3_s16x2(m0, c0[3], c0[4]);
						m1 = __vimax3_s16x2(m1, Dl[3], Dl[4]);
						m0 = __vimax3_s16x2(m0, c0[5], c0[6]);
						m1 = __vimax3_s16x2(m1, Dl[5], Dl[6]);
						m0 = __vmaxs2(m0, c0[7]);
						m1 = __vmaxs2(m1, Dl[7]);
						if (j1 >= ctmin) {  // columns past a pair's |t| (values are at least 0)
							m0 &= colmask16(j0, ctA, ctB);
							m1 &= colmask16(j1, ctA, ctB);
						}
						if (!TB) {
							l_best = __vimax3_s16x2(l_best, m0, m1);
						} else if (__vimax3_s16x2(m0, m1, reach) != reach) {
							// the step's best of a half reaches the lane's: its largest row, then column
							const uint32_t m = __vmaxs2(m0, m1);
							auto look = [&](int sh, int ct, int32_t &best, int32_t &bi, int32_t &bj) {
								const int32_t v = int32_t((m >> sh) & 0xffffu);
								if (v == 0 || v < best) return;
								int at = 0, aj = j0;
#pragma unroll
								for (int r = 0; r < R; r++) {
									const bool x0 = int32_t((c0[r] >> sh) & 0xffffu) == v, x1 = j1 < ct && int32_t((Dl[r] >> sh) & 0xffffu) == v;
									if (x0 || x1) {
										at = r;
										aj = x1 ? j1 : j0;
									}
								}
								if (v > best || row0 + at >= bi) {
									bi = row0 + at;
									bj = aj;
								}
								best = v;
							};
							look(0, ctA, resA, iA, jA);
							look(16, ctB, resB, iB, jB);
							reach = uint32_t(max(resA, 4) - 1) | uint32_t(max(resB, 4) - 1) << 16;
						}
					} else {
						auto lo16 = [](uint32_t x) { return int32_t(int16_t(x & 0xffffu)); };
						auto hi16 = [](uint32_t x) { return int32_t(x) >> 16; };
						if (TB && LOC == LOC_SEMI && has_last) {
							// the first of the largest in the pair's last row, by the lane that holds it
							auto row_of = [&](const uint32_t (&x)[R], int nv) {
								uint32_t v = x[0];
#pragma unroll
								for (int r = 1; r < R; r++)
									if (r == nv - 1) v = x[r];
								return v;
							};
							if (lastA && j0 < ltA) {
								const int32_t x = lo16(row_of(c0, nvA)) - off, y = lo16(row_of(Dl, nvA)) - off;
								if (x > rowA) { rowA = x; jA = j0; }
								if (j1 < ltA && y > rowA) { rowA = y; jA = j1; }
							}
							if (lastB && j0 < ltB) {
								const int32_t x = hi16(row_of(c0, nvB)) - off, y = hi16(row_of(Dl, nvB)) - off;
								if (x > rowB) { rowB = x; jB = j0; }
								if (j1 < ltB && y > rowB) { rowB = y; jB = j1; }
							}
						} else if (!TB && LOC == LOC_SEMI && has_last) {
							// the running maximum of every row over the columns inside each pair's |t|; the last
							// row's is taken after the pass
							if (j1 < ctmin) {
#pragma unroll
								for (int r = 0; r < R; r++) rmax[TB ? 0 : r] = __vimax3_s16x2(rmax[TB ? 0 : r], c0[r], Dl[r]);
							} else {
								const uint32_t m0 = colmask16(j0, ctA, ctB), m1 = colmask16(j1, ctA, ctB);
#pragma unroll
								for (int r = 0; r < R; r++)
									rmax[TB ? 0 : r] = __vimax3_s16x2(rmax[TB ? 0 : r], (c0[r] & m0) | (0x80008000u & ~m0), (Dl[r] & m1) | (0x80008000u & ~m1));
							}
						}
						if (s == endA) {  // the pair's last column
							const bool odd = j0 == ltA - 1;
#pragma unroll
							for (int r = 0; r < R; r++)
								if (LOC == LOC_SEMI ? r < nvA : (lastA && r == nvA - 1)) {
									const int32_t x = lo16(odd ? c0[r] : Dl[r]) - off;
									if (TB && x > resA) iA = row0 + r;
									resA = max(resA, x);
								}
						}
						if (s == endB) {
							const bool odd = j0 == ltB - 1;
#pragma unroll
							for (int r = 0; r < R; r++)
								if (LOC == LOC_SEMI ? r < nvB : (lastB && r == nvB - 1)) {
									const int32_t x = hi16(odd ? c0[r] : Dl[r]) - off;
									if (TB && x > resB) iB = row0 + r;
									resB = max(resB, x);
								}
						}
					}
				}
				prev_up = upD1;
				if (CHAIN && q + 1 < npass) {
					// lane 31 has finished step s - 31: a chunk of its row, or the row's end
					const int done = s - 31 + 1;
					if (done > 0 && ((done & (STEPS - 1)) == 0 || s == wsteps - 1)) {
						const int e = min(2 * done, lt), j = (2 * done - 1) & ~(CHAIN_CHUNK - 1);
						put_row(j, e);
					}
				}
			}
			if (!TB && LOC == LOC_SEMI && has_last) {
#pragma unroll
				for (int r = 0; r < R; r++) {
					if (lastA && r == nvA - 1) resA = max(resA, int32_t(int16_t(rmax[TB ? 0 : r] & 0xffffu)) - off);
					if (lastB && r == nvB - 1) resB = max(resB, (int32_t(rmax[TB ? 0 : r]) >> 16) - off);
				}
			}
			__syncwarp();
		}

		// ---- the twin's results: maxima over the group (global: the one lane that has it)
		if (LOCAL && !TB) {
			resA = emptyA ? NONE : int32_t(l_best & 0xffffu);
			resB = emptyB ? NONE : int32_t(l_best >> 16);
		}
		// with positions: local, the largest row, then column, of the largest; semiglobal, the
		// smallest row of the last column's largest (the last row's is one lane's)
		auto fold = [&](int32_t &v, int32_t &i, int32_t &j, int32_t ov, int32_t oi, int32_t oj) {
			const bool take = LOCAL ? ov > v || (ov == v && (oi > i || (oi == i && oj > j)))
			                        : oi >= 0 && (i < 0 || ov > v || (ov == v && oi < i));
			if (take) {
				v = ov;
				i = oi;
				if (LOCAL) j = oj;
			}
		};
		for (int o = 1; o < G; o <<= 1) {
			const int32_t oA = __shfl_xor_sync(0xffffffffu, resA, o, G), oB = __shfl_xor_sync(0xffffffffu, resB, o, G);
			if (TB && LOC != LOC_GLOBAL) {
				const int32_t oiA = __shfl_xor_sync(0xffffffffu, iA, o, G), ojA = __shfl_xor_sync(0xffffffffu, jA, o, G);
				const int32_t oiB = __shfl_xor_sync(0xffffffffu, iB, o, G), ojB = __shfl_xor_sync(0xffffffffu, jB, o, G);
				fold(resA, iA, jA, oA, oiA, ojA);
				fold(resB, iB, jB, oB, oiB, ojB);
				if (LOC == LOC_SEMI) {
					const int32_t orA = __shfl_xor_sync(0xffffffffu, rowA, o, G), orB = __shfl_xor_sync(0xffffffffu, rowB, o, G);
					if (orA > rowA) { rowA = orA; jA = ojA; }
					if (orB > rowB) { rowB = orB; jB = ojB; }
				}
			} else {
				resA = max(resA, oA);
				resB = max(resB, oB);
			}
		}
		if (CHAIN) {
			// fold in the stripes above, pass the twin's best on (a record per ticket)
			if (q_lo > 0) {
				if (ld_acquire(p.progress + prod) < lt) wait_progress(p.progress + prod, lt, p.status);
				const int4 rc = __ldcg(p.chain + prod);
				if (TB && LOCAL) {  // positions in 16 bits each (the host's bound)
					fold(resA, iA, jA, rc.x, rc.z < 0 ? -1 : rc.z >> 16, rc.z < 0 ? -1 : rc.z & 0xffff);
					fold(resB, iB, jB, rc.y, rc.w < 0 ? -1 : rc.w >> 16, rc.w < 0 ? -1 : rc.w & 0xffff);
				} else if (TB && LOC == LOC_SEMI) {
					fold(resA, iA, jA, rc.x, rc.z, -1);
					fold(resB, iB, jB, rc.y, rc.w, -1);
				} else {
					resA = max(resA, rc.x);
					resB = max(resB, rc.y);
				}
			}
			if (q_lo < npass - 1 && lane == 0) {
				int32_t zA = iA, zB = iB;
				if (LOCAL) {
					zA = iA < 0 ? -1 : iA << 16 | jA;
					zB = iB < 0 ? -1 : iB << 16 | jB;
				}
				p.chain[base] = make_int4(resA, resB, zA, zB);
				st_release(p.progress + base, lt);  // every column (put_row, before a __syncwarp), and the record
			}
		}
		if (sub == 0) {
#pragma unroll
			for (int h = 0; h < 2; h++) {
				const int pair = h ? pb : pa;
				if (pair < 0) continue;
				// chained: written by the ticket of the pair's own last stripe (its first, if it has no
				// cells), which holds its last row's best; the record passed down does not carry that, and
				// the twin's later stripes hold nothing of this pair
				if (CHAIN && q_lo != max((h ? npB : npA) - 1, 0)) continue;
				const int n = h ? lsB : lsA, m = h ? ltB : ltA;
				int32_t v = h ? resB : resA;
				if (n == 0 || m == 0) {
					// no cells: a border cell, or none (finish_pair)
					v = NONE;
					if (LOC == LOC_GLOBAL) v = n == 0 ? p.top_D[m] : p.left_D[n];
					if (LOC == LOC_SEMI) {
						for (int j = 0; j < m; j++) v = max(v, p.top_D[j + 1]);
						for (int i = 0; i < n; i++) v = max(v, p.left_D[i + 1]);
					}
				}
				int32_t si = -1, sj = -1;  // scores alone: no seed
				if (TB && n > 0 && m > 0) {
					const int32_t bi = h ? iB : iA, bj = h ? jB : jA, row = h ? rowB : rowA;
					si = n - 1;
					sj = m - 1;
					if (LOCAL) {
						if (v == NONE) v = 0;  // every cell is 0: the last one
						if (v > 0) {
							si = bi;
							sj = bj;
						}
					}
					if (LOC == LOC_SEMI) {
						if (bj >= 0 && (bi < 0 || !(v > row))) {
							v = row;
							sj = bj;
						} else {
							si = bi;
						}
					}
					v >>= 2;
				} else if (TB) {
					if (LOC == LOC_GLOBAL) {
						si = n - 1;
						sj = m - 1;
					}
					if (LOC == LOC_SEMI) {
						int32_t b = NONE;
						for (int j = 0; j < m; j++)
							if (p.top_D[j + 1] > b) { b = p.top_D[j + 1]; si = n - 1; sj = j; }
						for (int i = 0; i < n; i++)
							if (p.left_D[i + 1] > b) { b = p.left_D[i + 1]; si = i; sj = m - 1; }
					}
				}
				p.score[pair] = v == NONE ? -INFINITY * p.out_sign : float(v) * p.out_sign;
				p.seed[2 * pair] = si;
				p.seed[2 * pair + 1] = sj;
				p.has_seed[pair] = v != NONE;
			}
		}
	}
}

}  // namespace pa
