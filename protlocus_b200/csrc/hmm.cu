/*
 * hmm.cu -- sm_100a kernels of the integer profile DP, mp_hmm_dp_score
 * (hmm.c:252-291): one profile, many regions, one frame-0 codon per row.
 *
 * Every cell of row i depends only on row i-1 (columns j-1 and j), so a row is
 * computed in parallel across the profile: one warp per region, lane t owns
 * HMM_C consecutive columns of a 32*HMM_C-column tile and keeps their M/I/D
 * values of the previous row in registers, updated in place from the last
 * column down.  The value of column j-1 at a lane's first column comes from lane
 * t-1 by __shfl_up_sync, and across tiles from a per-row edge buffer that lane
 * 31 of the previous tile wrote (two buffers by tile parity, so a tile never
 * writes the rows it reads).  The 7 transition scores of a lane's columns
 * are row-invariant and sit in registers for the whole tile; the emissions are
 * staged in shared memory transposed ([residue][column], a zero row for stop
 * and ambiguous codons) so that one 16-byte load gives a lane its 8 columns.
 * Padding columns beyond m carry transitions of -2^28: every state there stays
 * 0 and cannot change the maximum.
 *
 * Two kernels.  k_hmm_pair takes two regions per warp, their states in the two 16-bit
 * halves of every register, for profiles whose values provably fit (pl_hmm_profile_create);
 * k_hmm_dp keeps 32-bit states for the others.
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include "plk.h"

#define FULL 0xffffffffu
#define HMM_C 8                    /* columns per lane */
#define HMM_TILE (32 * HMM_C)      /* columns per tile */
#define HMM_WARPS 8

extern "C" void plk_add_launches(uint64_t n);

/* codon index per row of every region: HMMER column, 20 = no emission (stop or a code > 3) */
__global__ void k_hmm_codons(const uint8_t *__restrict__ nt, const int32_t *__restrict__ off,
		const int32_t *__restrict__ len, const int64_t *__restrict__ row_off, int n,
		const uint8_t *__restrict__ codon_alpha, uint8_t *__restrict__ rows)
{
	for (int q = blockIdx.x; q < n; q += gridDim.x) {
		const int tlen = len[q] / 3;
		const uint8_t *s = nt + off[q];
		uint8_t *o = rows + row_off[q];
		/* the bytes up to the next region (16-aligned) are rows without emission */
		for (int i = tlen + threadIdx.x; i < (tlen + 15) / 16 * 16; i += blockDim.x) o[i] = 20;
		for (int i = threadIdx.x; i < tlen; i += blockDim.x) {
			const int b0 = s[3 * i], b1 = s[3 * i + 1], b2 = s[3 * i + 2];
			o[i] = b0 > 3 || b1 > 3 || b2 > 3 ? 20 : codon_alpha[b0 << 4 | b1 << 2 | b2];
		}
	}
}

template <bool SMEM_EMIT>
__global__ void __launch_bounds__(32 * HMM_WARPS)
k_hmm_dp(const plk_hmm_prof_t P, const uint8_t *__restrict__ rows, const int64_t *__restrict__ row_off,
		const int32_t *__restrict__ len, const int32_t *__restrict__ order, int n, int32_t *counter,
		int4 *__restrict__ edge, int64_t edge_stride, int32_t *__restrict__ score)
{
	extern __shared__ __align__(16) int16_t s_emit[];  /* [21][mpad] when SMEM_EMIT */
	const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
	const int ntile = P.mpad / HMM_TILE;
	if (SMEM_EMIT) {
		const int4 *src = (const int4*)P.emit_t;
		int4 *dst = (int4*)s_emit;
		for (int x = threadIdx.x; x < 21 * P.mpad / 8; x += blockDim.x) dst[x] = src[x];
		__syncthreads();
	}
	const int16_t *emit = SMEM_EMIT ? s_emit : (const int16_t*)P.emit_t;
	if (wib >= P.warps) return;
	int4 *my_edge = edge + (int64_t)(blockIdx.x * P.warps + wib) * 2 * edge_stride;
	for (;;) {
		int idx = 0;
		if (lane == 0) idx = atomicAdd(counter, 1);
		idx = __shfl_sync(FULL, idx, 0);
		if (idx >= n) break;
		const int q = order[idx];
		const int tlen = len[q] / 3;
		const uint8_t *aa = rows + row_off[q];
		int best = 0;
		for (int t = 0; t < ntile; ++t) {
			const int c0 = t * HMM_TILE + lane * HMM_C;     /* column j-1 of the lane's first cell */
			int tr[7][HMM_C];
#pragma unroll
			for (int k = 0; k < 7; ++k) {
				const int4 *p = (const int4*)(P.trans_t + (int64_t)k * P.mpad + c0);
				const int4 a = __ldg(p), b = __ldg(p + 1);
				tr[k][0] = a.x, tr[k][1] = a.y, tr[k][2] = a.z, tr[k][3] = a.w;
				tr[k][4] = b.x, tr[k][5] = b.y, tr[k][6] = b.z, tr[k][7] = b.w;
			}
			int pm[HMM_C], pi[HMM_C], pd[HMM_C];
#pragma unroll
			for (int c = 0; c < HMM_C; ++c) pm[c] = pi[c] = pd[c] = 0;
			int4 nxt = make_int4(0, 0, 0, 0);                 /* edge of row i-1 for lane 0 */
			const int4 *rd = my_edge + (int64_t)((t + 1) & 1) * edge_stride;  /* written by tile t-1 */
			int4 *wr = my_edge + (int64_t)(t & 1) * edge_stride;              /* read by tile t+1 */
			for (int i = 0; i < tlen; ++i) {
				const int a = aa[i];
				const int4 ev = *(const int4*)(emit + (int64_t)a * P.mpad + c0);
				int e[HMM_C];
				e[0] = (int)(int16_t)(ev.x & 0xffff), e[1] = ev.x >> 16;
				e[2] = (int)(int16_t)(ev.y & 0xffff), e[3] = ev.y >> 16;
				e[4] = (int)(int16_t)(ev.z & 0xffff), e[5] = ev.z >> 16;
				e[6] = (int)(int16_t)(ev.w & 0xffff), e[7] = ev.w >> 16;
				/* previous-row values of column j-1 for the lane's first cell */
				int nm = __shfl_up_sync(FULL, pm[HMM_C - 1], 1);
				int ni = __shfl_up_sync(FULL, pi[HMM_C - 1], 1);
				int nd = __shfl_up_sync(FULL, pd[HMM_C - 1], 1);
				if (lane == 0) nm = nxt.x, ni = nxt.y, nd = nxt.z;
				if (lane == 0 && t > 0) nxt = rd[i];  /* row i of the previous tile, used by row i+1 */
#pragma unroll
				for (int c = HMM_C - 1; c >= 0; --c) {
					const int am = c ? pm[c - 1] : nm, ai = c ? pi[c - 1] : ni, ad = c ? pd[c - 1] : nd;
					int from = max(am + tr[0][c], ai + tr[3][c]);
					from = max(from, ad + tr[5][c]);
					const int cm = max(from + e[c], 0);
					const int ci = max(max(pm[c] + tr[1][c], pi[c] + tr[4][c]), 0);
					const int cd = max(max(am + tr[2][c], ad + tr[6][c]), 0);
					best = max(best, max(cm, ci));
					pm[c] = cm, pi[c] = ci, pd[c] = cd;
				}
				if (lane == 31 && t + 1 < ntile) wr[i] = make_int4(pm[HMM_C - 1], pi[HMM_C - 1], pd[HMM_C - 1], 0);
			}
			__syncwarp();  /* the next tile reads this tile's edge */
		}
#pragma unroll
		for (int o = 16; o >= 1; o >>= 1) best = max(best, __shfl_xor_sync(FULL, best, o));
		if (lane == 0) score[q] = best;
	}
}

/* Two regions of one profile per warp in int16x2.
 *
 * The DP is bound by the integer pipe: the 32-bit kernel runs nine add+max steps per cell,
 * and the same nine DPX steps in their 16x2 form (__viaddmax_s16x2: max(a + b, c), one
 * instruction) update the cell of two regions.  Every state is at least 0 (the DP's own
 * clamp) and, with no transition above 0, at most m times the largest emission, so states fit
 * 15 bits; the host clamps transitions and emissions that any path takes below 0 from the
 * largest state (they then still end at the clamp), so no 16-bit sum wraps.  Rows past a
 * region's end carry no emission: the states only fall, and the maximum stays.
 *
 * A lane owns C of the 32 * C columns of a tile, C the least that covers m in ceil(m / 256)
 * tiles: with 8 columns always, 30 % of the cells of profiles of 50-800 columns were padding.
 * The tables keep 8 slots a lane whatever C is (16-byte loads), row indices are read four rows
 * at a time, and the two regions' emissions, 32-bit words with the value in the low half, join
 * by a multiply-add on the FMA pipe (joined by byte permutes the ALU pipe, the bound, carried
 * one instruction more per column).  The maximum is taken over M alone, two columns per step:
 * an I is at most the M it left.
 *
 * Measured, 64 profiles of 50-800 columns against the six frames of 2 Mb (1254
 * regions of 12 kb, eight profiles' launches side by side): 99.6 -> 59 ms; the ALU pipe is 87 %
 * busy with two warps a scheduler (19 passes of ncu on one 659-column profile). */
template <int C, bool SMEM_EMIT>
__global__ void __launch_bounds__(32 * HMM_WARPS, 2)
k_hmm_pair(const plk_hmm_prof_t P, const uint8_t *__restrict__ rows, const int64_t *__restrict__ row_off,
		const int32_t *__restrict__ len, const int32_t *__restrict__ order, int n, int32_t *counter,
		int4 *__restrict__ edge, int64_t edge_stride, int32_t *__restrict__ score)
{
	extern __shared__ __align__(16) uint32_t s_emit2[];  /* [21][mpad] when SMEM_EMIT */
	const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
	const int ntile = P.mpad / HMM_TILE;
	if (SMEM_EMIT) {
		const int4 *src = (const int4*)P.emit_t;
		int4 *dst = (int4*)s_emit2;
		for (int x = threadIdx.x; x < 21 * P.mpad / 4; x += blockDim.x) dst[x] = src[x];
		__syncthreads();
	}
	const uint32_t *emit = SMEM_EMIT ? s_emit2 : (const uint32_t*)P.emit_t;
	if (wib >= P.warps) return;
	int4 *my_edge = edge + (int64_t)(blockIdx.x * P.warps + wib) * 2 * edge_stride;
	for (;;) {
		int idx = 0;
		if (lane == 0) idx = atomicAdd(counter, 1);
		idx = 2 * __shfl_sync(FULL, idx, 0);
		if (idx >= n) break;
		const bool two = idx + 1 < n;
		const int q0 = order[idx], q1 = two ? order[idx + 1] : q0;
		const int n0 = (len[q0] / 3 + 3) / 4, n1 = two ? (len[q1] / 3 + 3) / 4 : 0;  /* groups of four rows */
		const uint32_t *r0 = (const uint32_t*)(rows + row_off[q0]), *r1 = (const uint32_t*)(rows + row_off[q1]);
		const int ng = max(n0, n1);
		unsigned best = 0;
		for (int t = 0; t < ntile; ++t) {
			const int slot = t * HMM_TILE + lane * HMM_C;
			unsigned tr[7][C];
#pragma unroll
			for (int k = 0; k < 7; ++k) {
				const int4 *p = (const int4*)(P.trans_t + (int64_t)k * P.mpad + slot);
				const int4 a = __ldg(p), b = __ldg(p + 1);
				const int v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
				for (int c = 0; c < C; ++c) tr[k][c] = (unsigned)v[c];
			}
			unsigned pm[C], pi[C], pd[C];
#pragma unroll
			for (int c = 0; c < C; ++c) pm[c] = pi[c] = pd[c] = 0;
			int4 nxt = make_int4(0, 0, 0, 0);                 /* edge of row i-1 for lane 0 */
			const int4 *rd = my_edge + (int64_t)((t + 1) & 1) * edge_stride;  /* written by tile t-1 */
			int4 *wr = my_edge + (int64_t)(t & 1) * edge_stride;              /* read by tile t+1 */
			uint32_t u0 = 0 < n0 ? r0[0] : 0x14141414u, u1 = 0 < n1 ? r1[0] : 0x14141414u;
			for (int g = 0; g < ng; ++g) {
				const uint32_t w0 = u0, w1 = u1;
				u0 = g + 1 < n0 ? r0[g + 1] : 0x14141414u, u1 = g + 1 < n1 ? r1[g + 1] : 0x14141414u;
#pragma unroll
				for (int r = 0; r < 4; ++r) {
					const int i = 4 * g + r;
					const uint32_t *e0 = emit + (int)(w0 >> (8 * r) & 0xff) * P.mpad + slot;
					const uint32_t *e1 = emit + (int)(w1 >> (8 * r) & 0xff) * P.mpad + slot;
					unsigned e[8];
#pragma unroll
					for (int c = 0; c < C; c += 4) { /* region 0 in the low half, region 1 in the high one */
						const uint4 a = *(const uint4*)(e0 + c), b = *(const uint4*)(e1 + c);
						e[c] = b.x * P.hi + a.x, e[c + 1] = b.y * P.hi + a.y;
						e[c + 2] = b.z * P.hi + a.z, e[c + 3] = b.w * P.hi + a.w;
					}
					/* previous-row values of column j-1 for the lane's first cell */
					unsigned nm = __shfl_up_sync(FULL, pm[C - 1], 1);
					unsigned ni = __shfl_up_sync(FULL, pi[C - 1], 1);
					unsigned nd = __shfl_up_sync(FULL, pd[C - 1], 1);
					if (lane == 0) nm = (unsigned)nxt.x, ni = (unsigned)nxt.y, nd = (unsigned)nxt.z;
					if (lane == 0 && t > 0) nxt = rd[i];  /* row i of the previous tile, used by row i+1 */
#pragma unroll
					for (int c = C - 1; c >= 0; --c) {
						const unsigned am = c ? pm[c - 1] : nm, ai = c ? pi[c - 1] : ni, ad = c ? pd[c - 1] : nd;
						unsigned from = __viaddmax_s16x2(ad, tr[5][c], 0x80008000u);
						from = __viaddmax_s16x2(ai, tr[3][c], from);
						from = __viaddmax_s16x2(am, tr[0][c], from);
						const unsigned cm = __viaddmax_s16x2(from, e[c], 0u);
						const unsigned ci = __viaddmax_s16x2(pi[c], tr[4][c], __viaddmax_s16x2(pm[c], tr[1][c], 0u));
						const unsigned cd = __viaddmax_s16x2(ad, tr[6][c], __viaddmax_s16x2(am, tr[2][c], 0u));
						if (C % 2 && c == 0) best = __vmaxs2(best, cm);
						else if ((C - 1 - c) % 2) best = __vimax3_s16x2(best, cm, pm[c + 1]);
						pm[c] = cm, pi[c] = ci, pd[c] = cd;
					}
					if (lane == 31 && t + 1 < ntile) wr[i] = make_int4((int)pm[C - 1], (int)pi[C - 1], (int)pd[C - 1], 0);
				}
			}
			__syncwarp();  /* the next tile reads this tile's edge */
		}
		int b0 = (int)(best & 0xffffu), b1 = (int)(best >> 16);
#pragma unroll
		for (int o = 16; o >= 1; o >>= 1) b0 = max(b0, __shfl_xor_sync(FULL, b0, o)), b1 = max(b1, __shfl_xor_sync(FULL, b1, o));
		if (lane == 0) {
			score[q0] = b0;
			if (two) score[q1] = b1;
		}
	}
}

typedef void (*hmm_kernel_t)(const plk_hmm_prof_t, const uint8_t*, const int64_t*, const int32_t*, const int32_t*, int,
		int32_t*, int4*, int64_t, int32_t*);

extern "C" int plk_hmm_smem_bytes(int32_t mpad, int32_t cols)
{
	const int smem = 21 * mpad * (cols ? 4 : 2);
	return smem <= (cols ? PLK_HMM_SMEM_PAIR : PLK_HMM_SMEM_MAX) ? smem : 0;
}

static int hmm_smem(const plk_hmm_prof_t *p) { return plk_hmm_smem_bytes(p->mpad, p->cols); }

/* the kernel of a profile (cols: columns a lane of k_hmm_pair, 0 for 32-bit states) */
static hmm_kernel_t hmm_kernel(const plk_hmm_prof_t *p)
{
	const bool smem = hmm_smem(p) > 0;
	switch (p->cols) {
	case 0: return smem ? k_hmm_dp<true> : k_hmm_dp<false>;
	case 2: return k_hmm_pair<2, true>;  /* up to four columns a lane in a profile of one tile, whose tables fit shared memory, as those of up to 7 do */
	case 3: return k_hmm_pair<3, true>;
	case 4: return k_hmm_pair<4, true>;
	case 5: return k_hmm_pair<5, true>;
	case 6: return k_hmm_pair<6, true>;
	case 7: return k_hmm_pair<7, true>;
	default: return smem ? k_hmm_pair<8, true> : k_hmm_pair<8, false>;
	}
}

extern "C" int plk_hmm_ctas_per_sm(const plk_hmm_prof_t *p)
{
	int n = 0;
	hmm_kernel_t f = hmm_kernel(p);
	cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, PLK_HMM_SMEM_PAIR);
	if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, f, 32 * HMM_WARPS, hmm_smem(p));
	return e == cudaSuccess ? n : -1;
}

extern "C" int plk_hmm_warps_per_cta(void) { return HMM_WARPS; }

extern "C" int plk_hmm_codons(const uint8_t *nt, const int32_t *off, const int32_t *len, const int64_t *row_off,
		int32_t n, const uint8_t *codon_alpha, uint8_t *rows, void *stream)
{
	if (n <= 0) return 0;
	k_hmm_codons<<<n < 4096 ? n : 4096, 128, 0, (cudaStream_t)stream>>>(nt, off, len, row_off, n, codon_alpha, rows);
	plk_add_launches(1);
	return (int)cudaGetLastError();
}

extern "C" int plk_hmm_dp(const plk_hmm_prof_t *p, const uint8_t *rows, const int64_t *row_off, const int32_t *len,
		const int32_t *order, int32_t n, int32_t *counter, void *edge, int64_t edge_stride_rows, int32_t n_ctas,
		int32_t warps, int32_t *score, void *stream)
{
	if (n <= 0) return 0;
	cudaStream_t st = (cudaStream_t)stream;
	cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(int32_t), st);
	if (e != cudaSuccess) return (int)e;
	hmm_kernel_t f = hmm_kernel(p);
	e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, PLK_HMM_SMEM_PAIR);
	if (e != cudaSuccess) return (int)e;
	plk_hmm_prof_t P = *p;
	P.warps = warps;
	f<<<n_ctas, 32 * HMM_WARPS, hmm_smem(p), st>>>(P, rows, row_off, len, order, n, counter, (int4*)edge, edge_stride_rows, score);
	plk_add_launches(1);
	return (int)cudaGetLastError();
}
