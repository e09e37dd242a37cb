/*
 * chain.cu -- the anchor-chaining DP on the device (chain.c:160-208, the fill loop
 * of mp_chain): for every anchor i of a query, the best chain score f[i] ending
 * there, its predecessor p[i] and the peak score v[i] along that chain.
 *
 * Two kernels.  k_chain_score computes comput_sc of every anchor against the 32
 * before it, a lane per pair.  k_chain_fill walks one query per thread, one or four such
 * threads per warp (the host orders queries longest first, so the longest start
 * first).  The loop over predecessors is the reference's,
 * statement for statement: a running best (strictly greater wins, so the nearest j
 * keeps a tie), a skip counter that rises on a non-improving predecessor already
 * marked by this anchor (t[j] == i), falls on an improving one (floored at 0) and
 * ends the loop when it passes max_skip, and a mark t[p[j]] = i after every scored
 * j.  Queries are independent, so thousands of them fill the GPU; within a query
 * the order of comparisons is the reference's and the results are bit-exact.
 * Different queries' loops share neither trip counts nor branches, so 32 of them
 * in a warp ran their paths one after the other and left two warps an SM (8.3 ms
 * for 10,000 queries, 1.2 M anchors); a warp each is bound by issue, and scoring a
 * pair was 80 of its 110 instructions on a single lane: 5.5 ms, with the scores
 * taken from the rows 2.9 + 0.09, the loop's records read four ahead and its branches
 * turned into selects 2.2 + 0.09.
 * Scores (comput_sc, chain.c:112-152) use the reference's float operations one at
 * a time, rounded to nearest as the CPU build rounds them (no fused multiply-add).
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include <limits.h>
#include "plk.h"

extern "C" void plk_add_launches(uint64_t n);

namespace {

constexpr int CHAIN_THREADS = 128;
constexpr int BLOCK_BONUS = 2;  /* MP_BLOCK_BONUS (protlocus.h:47) */

/* log2 approximation of the reference (mppriv.h:143-151), valid for x >= 2: the
 * exponent field minus 128 plus a quadratic in the mantissa scaled to [1, 2); the
 * coefficients are the reference's, so the penalties match it bit for bit */
__device__ __forceinline__ float chain_log2(float x)
{
	uint32_t i = __float_as_uint(x);
	const float e = (float)(int)(((i >> 23) & 255u) - 128u);
	i = (i & ~(255u << 23)) + (127u << 23);
	const float m = __uint_as_float(i);
	float q = __fadd_rn(__fmul_rn(-0.34484843f, m), 2.02466578f);
	q = __fsub_rn(__fmul_rn(q, m), 0.67487759f);
	return __fadd_rn(e, q);
}

/* the score of chaining anchor aj before ai, INT_MIN when they cannot chain */
__device__ __forceinline__ int chain_score(uint64_t ai, uint64_t aj, const plk_chain_args_t &A)
{
	const int32_t dq = (int32_t)ai - (int32_t)aj, dq3 = dq * 3;
	int32_t dr3, dd, sc, dd_signed = 0;
	if (dq <= 0 || dq3 > A.max_dist_x) return INT_MIN;
	if (dq > A.max_dist_y) return INT_MIN;
	if (A.bbit > 0) { /* block resolution: gaps inside one block width count as zero */
		const int32_t bs = 1 << A.bbit;
		dr3 = (int32_t)(((ai >> 32) - (aj >> 32)) << A.bbit);
		if (dq3 >= dr3 - bs && dq3 <= dr3 + bs) dd = dd_signed = 0;
		else if (dq3 < dr3 - bs) dd = dr3 - bs - dq3, dd_signed = -dd;
		else dd = dq3 - (dr3 + bs), dd_signed = dd;
	} else {
		dr3 = (int32_t)((ai >> 32) - (aj >> 32));
		if (dr3 == 0) return INT_MIN;
		dd = dr3 > dq3 ? dr3 - dq3 : dq3 - dr3;
		dd_signed = dq3 - dr3;
	}
	if (dd > A.bw) return INT_MIN;
	if (A.bbit > 0) {
		sc = A.kmer < dq ? A.kmer : dq;
	} else if (A.kmer <= dq && A.kmer * 3 <= dr3) {
		sc = A.kmer;
	} else {
		const int32_t dr = dr3 / 3, rem = dr3 - dr * 3, dg = dr < dq ? dr : dq;
		sc = dg < A.kmer ? dg : A.kmer;
		if (rem != 0) --sc; /* frameshift */
	}
	if (dd > 0) {
		const float lin = __fmul_rn((float)dd, 0.33334f);
		const float lg = dd >= 2 ? __fadd_rn(__fmul_rn(A.coef, __fsub_rn(chain_log2((float)(dd + 1)), 1.0f)), 1.0f)
				: (float)dd;
		if (A.is_spliced && dd_signed < 0) sc -= __float2int_rz(lin < lg ? lin : lg);
		else sc -= __float2int_rz(__fadd_rn(lin, lg));
	}
	if (A.bbit > 0 && (ai >> 32) == (aj >> 32) && dd == 0) sc += BLOCK_BONUS;
	return sc;
}

/* rows[(row0 + i - i0) * 32 + k] = the score of chaining anchor i - 1 - k before anchor i, k < 32, for
 * this launch's anchors: a CTA per query, a warp per anchor */
__global__ void __launch_bounds__(CHAIN_THREADS) k_chain_score(plk_chain_args_t A)
{
	const int q = A.order[blockIdx.x];
	if (q < 0 || q >= A.n_all) return;  /* k_chain_fill reports it */
	const int64_t base = A.off[q];
	const int n = A.n[q], lane = threadIdx.x & 31, end = min(n, A.i1);
	if (base < 0 || n < 0 || base + n > A.n_a) return;
	const uint64_t *__restrict__ a = A.a + base;
	int32_t *row = A.rows + (A.row0[blockIdx.x] << 5);
	for (int i = A.i0 + (threadIdx.x >> 5); i < end; i += CHAIN_THREADS / 32) {
		const int j = i - 1 - lane;
		if (j >= 0) row[((int64_t)(i - A.i0) << 5) + lane] = chain_score(a[i], a[j], A);
	}
}

/* One query per thread: the reference's sequential loop over predecessors, with its
 * early exit, skip counter and marks, so the order of every comparison is the
 * reference's.  Per anchor a record {f, p, t, v}.  Every per-query index is checked against the
 * query's length; a bad one records the site and the query (err[0], err[1]) and the access is
 * skipped.  A batch whose score rows do not fit runs in several launches, every query some
 * anchors further in each (its walk's three values kept between them): launches of fewer
 * queries instead, each waiting for its own longest walk, took 1,100 ms for 400 queries of
 * 100,000 anchors where these take 110. */
__global__ void __launch_bounds__(CHAIN_THREADS) k_chain_fill(plk_chain_args_t A)
{
	if (threadIdx.x & (A.stride - 1)) return;
	const int qi = (blockIdx.x * CHAIN_THREADS + threadIdx.x) / A.stride;
	if (qi >= A.n_q) return;
	const int q = A.order[qi];
	if (q < 0 || q >= A.n_all) { atomicExch(A.err, 1); return; }
	const int64_t base = A.off[q];
	const int n = A.n[q];
	if (base < 0 || n < 0 || base + n > A.n_a) { atomicExch(A.err, 2), atomicExch(A.err + 1, q); return; }
	const uint64_t *__restrict__ a = A.a + base;
	const int32_t *__restrict__ rows = A.rows + (A.row0[qi] << 5);
	const int end = min(n, A.i1);
	int32_t *f = A.f + base, *p = A.p + base, *v = A.v + base;
	int4 *rec = (int4*)A.rec + base;
#define CHK(x, site) ((unsigned)(x) < (unsigned)n ? true : (atomicExch(A.err, (site)), atomicExch(A.err + 1, q), false))
	int st = 0, hi = -1, hf = 0;
	if (A.i0 > 0) {
		const int4 s = ((const int4*)A.state)[q];
		st = s.x, hi = s.y, hf = s.z;
	}
	unsigned long long pairs = 0;
	for (int i = A.i0; i < end; ++i) {
		const uint64_t ai = a[i];
		const int32_t *row = rows + ((int64_t)(i - A.i0) << 5);
		if (i + 2 < end) { /* the next anchors' row and the anchors, on their way from L2 */
			asm volatile("prefetch.global.L1 [%0];" :: "l"(row + 64));
			asm volatile("prefetch.global.L1 [%0];" :: "l"(a + min(i + 16, n - 1)));
		}
		int max_f = A.kmer, max_j = -1, n_skip = 0;
		while (st < i && (((ai >> 32) - (a[st] >> 32)) << A.bbit) > (uint64_t)(int64_t)A.max_dist_x) ++st;
		if (hi >= 0 && hi >= st && CHK(hi, 12)) { /* the best anchor so far, even beyond the skip limit */
			const int s = hf + (i - 1 - hi < 32 ? row[i - 1 - hi] : chain_score(ai, a[hi], A));
			if (s > max_f) max_f = s, max_j = hi;
		} else hf = 0, hi = -1;
		if (i - st > A.max_iter) st = i - A.max_iter;
		int j = i - 1;
		bool more = true;
		/* predecessor j with its record and score (INT_MIN: they cannot chain), as selects: live = the
		 * loop still runs; marked is whether the predecessor of j was marked */
#define CHAIN_STEP(r, sc, live, marked) do { \
			const bool ok = (live) && (sc) != INT_MIN; \
			const int s = (sc) + (r).x; \
			const bool better = ok && s > max_f, skip = ok && !better && (r).z == i; \
			n_skip = better ? max(n_skip - 1, 0) : n_skip + skip; \
			more = more && !(skip && n_skip > A.max_skip); \
			max_f = better ? s : max_f, max_j = better ? j : max_j; \
			marked = ok && more && (r).y >= 0; \
			if (marked && CHK((r).y, 14)) rec[(r).y].z = i; \
		} while (0)
		const int near = st > i - 32 ? st : i - 32;  /* predecessors whose scores are in the row */
		while (more && j >= near) {
			/* j counts down from i - 1 in fours.  The four records are read before any of their marks
			 * is set (read one by one each waited for the mark before it: 2.9 against 2.6 ms); a mark
			 * on a later one of the four goes to its copy too */
			const int4 s4 = *(const int4*)(row + (i - 1 - j));
			const int sc[4] = {s4.x, s4.y, s4.z, s4.w}, j0 = j;
			int4 r[4];
#pragma unroll
			for (int u = 0; u < 4; ++u) r[u] = rec[j0 - u >= 0 ? j0 - u : 0];
#pragma unroll
			for (int u = 0; u < 4; ++u) {
				const bool live = more && j >= near;
				bool marked;
				CHAIN_STEP(r[u], sc[u], live, marked);
#pragma unroll
				for (int x = u + 1; x < 4; ++x) r[x].z = marked && r[u].y == j0 - x ? i : r[x].z;
				j -= live;
			}
		}
		for (; more && j >= st; --j) {
			const int sc = chain_score(ai, a[j], A);
			const int4 r = rec[j];
			bool marked;
			CHAIN_STEP(r, sc, true, marked);
		}
#undef CHAIN_STEP
		pairs += (unsigned)(i - 1 - j);
		int pk = max_f;
		if (max_j >= 0 && CHK(max_j, 16)) pk = max(pk, rec[max_j].w);
		rec[i] = make_int4(max_f, max_j, 0, pk);
		f[i] = max_f, p[i] = max_j, v[i] = pk;
		if (hf < max_f) hf = max_f, hi = i;
	}
#undef CHK
	if (end < n) ((int4*)A.state)[q] = make_int4(st, hi, hf, 0);
	if (A.pairs) atomicAdd(A.pairs, pairs);
}

} /* namespace */

extern "C" int plk_chain_fill(const plk_chain_args_t *a, void *stream)
{
	if (a->n_q <= 0) return 0;
	cudaStream_t st = (cudaStream_t)stream;
	k_chain_score<<<a->n_q, CHAIN_THREADS, 0, st>>>(*a);
	cudaError_t e = cudaGetLastError();
	if (e != cudaSuccess) return (int)e;
	const int per = CHAIN_THREADS / a->stride;
	k_chain_fill<<<(a->n_q + per - 1) / per, CHAIN_THREADS, 0, st>>>(*a);
	plk_add_launches(2);
	return (int)cudaGetLastError();
}
