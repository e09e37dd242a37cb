/*
 * forward.cu -- sm_100a kernel of the profile-HMM recheck score, rc_score
 * (recheck.c:283-440): multihit-local Forward in log space (float), and with
 * null2 the Backward pass, posterior usage and the biased-composition
 * correction (the ByExpectation null2), giving the bit score and the bias.
 *
 * One lane per peptide.  Every DP of rc_score is a chain along the row (D and
 * the exit sum E in the Forward, the B sum and D in the Backward) on top of
 * work that only reads the row before, so a peptide is one lane's in every warp of
 * a CTA, each warp running its part of the reference's loops in the reference's
 * order, and the parallelism is across peptides: a CTA takes up to 32 peptides of
 * one profile (the transition and emission rows it reads are the same for every
 * lane), sorted by length so the lanes run about as many rows.  The M/I loops
 * over a row's columns are software-pipelined (one level of M(k)'s sum is taken
 * with the next column's other), which keeps four logsums in flight per thread.
 *
 * The DP matrices live in a per-group scratch region, interleaved by lane
 * (element e of lane l at e*32 + l), so every access of a warp is one coalesced
 * run: the Forward M/I rows (all rows when some peptide of the group takes
 * null2, else two), the Backward M/I rows, two Forward D rows, and the special
 * states of every row.
 *
 * Keeping every float operation in the reference's order matters: the bias is
 * exp of a sum over all residues of log-odds normalised by the Forward total,
 * so a reordering that moves the total by 1e-4 nats moves the bias by L x 1e-4
 * of itself.  The transcendental steps carry the host's bits too: rc_logsum's
 * expf and log1pf are glibc's algorithms restated, as one function of the difference
 * (glibc_mathf.cuh, equal to the host libm on every float), the length model's logf values come from the
 * host with the peptide record, every float step is written in its rounded form
 * (no contraction into FMA), and the null2 residue sum runs in the reference's
 * order.  Only the final double-precision exp/log/log1p of the bias are the
 * device's own; their results are rounded to float.
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include "plk.h"
#include "glibc_mathf.cuh"

#define RC_NEG (-1e30f)
#define RC_NCODE 21
#define RC_LN2 0.69314718055994531

extern "C" void plk_add_launches(uint64_t n);

enum { T_MM, T_IM, T_DM, T_BM, T_MI, T_II, T_MD, T_DD }; /* recheck.c:74; a row is two float4 */

/* the 2^(j/32) table of expf, copied to shared memory by every CTA of the kernel */
__shared__ uint64_t s_exp2[32];

/* N independent logsums (rc_logsum, recheck.c:260-265) without branches: mn - mx is
 * -|a - b| exactly; past 50 or at -inf the term's value is not used */
template <int N>
__device__ __forceinline__ void lsn(const float (&a)[N], const float (&b)[N], float (&r)[N])
{
	float t[N], l[N];
#pragma unroll
	for (int j = 0; j < N; ++j) t[j] = fabsf(__fsub_rn(a[j], b[j]));
	gl_log1pexp_n<N>(t, l, s_exp2);
#pragma unroll
	for (int j = 0; j < N; ++j) {
		const float mx = a[j] > b[j] ? a[j] : b[j], mn = a[j] > b[j] ? b[j] : a[j];
		r[j] = glm_self(mn <= RC_NEG || t[j] > 50.0f, mx, __fadd_rn(mx, l[j]));
	}
}

__device__ __forceinline__ float ls(float a, float b)
{
	const float x[1] = {a}, y[1] = {b};
	float r[1];
	lsn<1>(x, y, r);
	return r[0];
}

/* a group's region, every array interleaved by lane:
 *   FMI float2 {M, I} [rows][M+1]: rows = lmax+1 when full, else rows i-1 and i at (i & 1)
 *   BMI float2 {M, I} [lmax+1][M+1]: the Backward rows (full groups only)
 *   D   float [2][M+1]: the Forward's two D rows (recheck.c:296), then lum / lui
 *   SP  float [6][lmax+1]: xN, xJ, xC of the Forward, bN, bJ, bC of the Backward (full)
 * Row index t is the group's step: a lane's row i is at t = i + lmax - len, so that the lanes,
 * whose lengths differ, end together and their rows of a Backward step and of a usage sum lie
 * side by side (indexed by i, every lane of a Backward step read another 32 bytes); a lane's
 * rows before its row 0 hold -inf. */
extern "C" int64_t plk_rc_group_floats(int32_t lmax, int32_t M, int32_t full)
{
	const int64_t W = (int64_t)M + 1, rows = full ? (int64_t)lmax + 1 : 2, sp = full ? (int64_t)lmax + 1 : 0;
	return (2 * rows * W + 2 * sp * W + 2 * W + 6 * sp) * 32;
}

struct RcLane {
	float2 *fmi, *bmi;  /* the lane's element 0 of each array */
	float *d, *sp;
	int full, lmax, off;  /* off: steps before the lane's row 1, less one */
};

/* element (row, column k) of a lane's matrix with rows of W columns */
__device__ __forceinline__ size_t rc_ix(int row, int k, int W) { return ((size_t)row * W + k) << 5; }

/* the first half of a profile's transition row's first half: MM, IM */
__device__ __forceinline__ float2 ldt2(const float4 *p) { return __ldg((const float2*)p); }

/* the DP rows stream through L2 only, which keeps L1 for the profile's rows */
__device__ __forceinline__ float2 ldr2(const float2 *p) { return __ldcg(p); }
__device__ __forceinline__ float ldr(const float *p) { return __ldcg(p); }
__device__ __forceinline__ void str2(float2 *p, float2 v) { __stcg(p, v); }
__device__ __forceinline__ void str(float *p, float v) { __stcg(p, v); }

/*
 * The passes run on RC_WARPS warps of a group's CTA, split along their dependences so that a
 * row takes little more than its chain of logsums:
 *   Forward   RC_MI warps: M(k), I(k), columns k = w + 1 modulo RC_MI, from the row above; the D
 *             warp: D(k) = ls(M(k-1) + MD, D(k-1) + DD) along the row; the E warp: ls(M(k), D(k))
 *             and its sum over the columns, then the row's special states, whose xB the M/I
 *             warps need;
 *   Backward  the feed warp: what the chain adds, ready in shared memory; the chain warp: the B
 *             sum over the row below, then D along the row from the last column; RC_MI warps:
 *             M(k), I(k) from the row below and the D they need.
 * What bounds a group: the Backward's three logsums a column, one after another (243 cycles each
 * alone, 730 a column; 860 to 900 measured), while the Forward takes 600 beside it; the usage
 * sums take 50 a column and row.  With M/I and chain on one warp each and the terms of
 * gl_log1pexp_n as two functions a column took 3,100.  4,000 peptides to 600 residues, 96
 * profiles to 800 positions, null2: 765 -> 220 ms, 185 -> 139 without null2; 20,000 peptides,
 * 480 profiles: 1,050 -> 505 ms.  Tried: four M/I warps a pass (they take issue slots from the
 * chains: 10% slower); the chain's own loads a column or eight ahead (1,060 cycles) or through
 * asynchronous copies into rings (1,300: the bookkeeping stands between the steps); unrolled
 * chain loops (35 cycles a column for instruction fetch).
 * Per column, a value crosses between warps through a ring in
 * shared memory whose slots are 64-bit words holding the value and a tag (the pass
 * step t and column count c as t * (M + 2) + c), written and read whole, so the
 * consumer lane waits for its slot to carry the tag and needs no fence; the consumer
 * hands its progress back the same way, and the producer does not overwrite a slot
 * the consumer has not taken.  A look at a tag costs some 100 cycles with its branch and vote, so
 * the D and E warps look at RC_BK columns at once.  Once per row, where a warp reads rows that
 * others wrote to global memory, and once per block of the feed warp, the writer advances a counter
 * after a block fence.  Every wait is bounded
 * by a clock limit: on expiry the CTA's abort flag and the launch's error word are
 * set and every warp leaves its loops (the barriers that follow are still met).
 */
#define RC_MI 2                        /* M/I warps of a pass; divides RC_PB and RC_Q */
/* warps of a CTA; those of one residue modulo 4 share a scheduler: the Backward's chain has the feed
 * warp beside it, the M/I warps of the two passes share two, D and E one */
#define RC_W_D 2
#define RC_W_E 6
#define RC_W_B 3
#define RC_W_F 7
#define RC_WARPS (2 * RC_MI + 4)
#define RC_UW 10                       /* warps of a CTA: those past RC_WARPS wait for the usage sums */
#define RC_Q 32                        /* ring depth, columns */
#define RC_BK 4                        /* columns that the Forward's D and E warps take at a time */
#define RC_CK 4                        /* columns for which an M/I warp of the Forward looks for free slots */
#define RC_PB 16                       /* columns of a block of the Backward's chain */
#define RC_FB 4                        /* blocks that the feed warp may be ahead */
#define RC_SPIN_LIMIT 10000000000LL    /* clock cycles, some seconds: the default limit of a wait */
#define FULL 0xffffffffu

struct RcSync {
	volatile int fe, fd, fm[RC_MI];             /* Forward rows done by the E, D and M/I warps */
	volatile int bp, bm[RC_MI], abort;          /* Backward: row L, rows done by the M/I warps, */
	volatile int bw, bf;                        /* blocks written by the feed warp and taken by the chain warp */
	long long lim;                              /* clock cycles a wait may take */
	volatile unsigned long long m[RC_Q][32];    /* M(i, k) of the Forward's M/I warps, tagged */
	volatile unsigned long long d[RC_Q][32];    /* D(i, k) of the Forward's D warp, tagged */
	volatile unsigned long long dn[RC_Q][32];   /* D(i, k+1) of the Backward's chain warp, tagged */
	volatile unsigned long long fcons[32], bcons[RC_MI][32], bE[32];  /* consumer progress; bE of a Backward row */
	float2 fd2[RC_FB * RC_PB + 1][32];          /* the feed warp's blocks; one column past them for the step that looks ahead */
	float xB[32], tot[32], u[3][32];
};

__device__ __forceinline__ unsigned long long rc_pack(const int tag, const float v)
{
	return ((unsigned long long)(unsigned)tag << 32) | __float_as_uint(v);
}

/* the value of a slot once it carries tag (exactly, or at least tag when ge); false in
 * ok when the wait ran out or the CTA aborted.  nap: the waiter is ahead of the chains and
 * leaves its scheduler to them between looks */
__device__ __forceinline__ float rc_take(RcSync &Y, volatile unsigned long long &slot, const int tag, const bool ge,
		int *err, bool &ok, const bool nap = false)
{
	unsigned long long v = slot;
	if (ge ? (int)(v >> 32) < tag : (int)(v >> 32) != tag) {
		const long long t0 = clock64();
		for (;;) {
			v = slot;
			if (ge ? (int)(v >> 32) >= tag : (int)(v >> 32) == tag) break;
			if (Y.abort) { ok = false; break; }
			if (clock64() - t0 > Y.lim) { Y.abort = 1; atomicExch(err, 1); ok = false; break; }
			if (nap) __nanosleep(100);
		}
	}
	return __uint_as_float((unsigned)v);
}

/* wait until the RC_BK columns of a ring from k on (those up to M) carry their tags */
__device__ __forceinline__ void rc_take_block(RcSync &Y, volatile unsigned long long (*ring)[32], const int k, const int M,
		const int tag0, int *err, bool &ok)
{
	const int lane = threadIdx.x & 31;
	long long t0 = 0;
	for (;;) {
		unsigned long long x[RC_BK];
		bool all = true;
#pragma unroll
		for (int j = 0; j < RC_BK; ++j) x[j] = ring[min(k + j, M) % RC_Q][lane];
#pragma unroll
		for (int j = 0; j < RC_BK; ++j) all &= (int)(x[j] >> 32) == tag0 + min(k + j, M);
		if (all) break;
		if (Y.abort) { ok = false; break; }
		const long long now = clock64();
		if (t0 == 0) t0 = now;
		else if (now - t0 > Y.lim) { Y.abort = 1; atomicExch(err, 1); ok = false; break; }
	}
}

/* the value of a slot that is known to carry its tag */
__device__ __forceinline__ float rc_val(const volatile unsigned long long &slot)
{
	return __uint_as_float((unsigned)slot);
}

/* warp-wide wait until ctr >= target, then a block fence (the rows the other warp wrote
 * before its matching rc_publish are visible); false when it ran out or the CTA aborted */
__device__ __forceinline__ bool rc_wait(RcSync &Y, volatile int &ctr, const int target, int *err)
{
	int ok = 1;
	if ((threadIdx.x & 31) == 0 && ctr < target) {
		const long long t0 = clock64();
		while (ctr < target) {
			if (Y.abort) { ok = 0; break; }
			if (clock64() - t0 > Y.lim) { Y.abort = 1; atomicExch(err, 1); ok = 0; break; }
			__nanosleep(32);
		}
	}
	ok = __shfl_sync(FULL, ok, 0);
	__threadfence_block();
	return ok != 0;
}

/* the chain warp's wait for the feed warp's block seq: as a rule it was seen written when the block
 * before began, and nothing is waited for; ready is the same in all lanes */
__device__ __forceinline__ bool rc_feed_next(RcSync &Y, int &ready, const int seq, int *err)
{
	if (ready <= seq && !rc_wait(Y, Y.bw, seq + 1, err)) return false;
	__threadfence_block();
	ready = __shfl_sync(FULL, Y.bw, 0);
	return true;
}

/* make the warp's writes so far visible to the CTA, then set ctr = v */
__device__ __forceinline__ void rc_publish(volatile int &ctr, const int v)
{
	__syncwarp();
	__threadfence_block();
	if ((threadIdx.x & 31) == 0) ctr = v;
}

/* the same for n counters side by side */
__device__ __forceinline__ bool rc_wait_all(RcSync &Y, volatile int *ctr, const int n, const int target, int *err)
{
	for (int x = 0; x < n; ++x) if (!rc_wait(Y, ctr[x], target, err)) return false;
	return true;
}

#define NEG2 make_float2(RC_NEG, RC_NEG)

/* Forward M/I warp w (recheck.c:305-311), columns k = w + 1, w + 1 + RC_MI, ..: for each row M(k) =
 * ls(ls(M'(k-1) + MM, I'(k-1) + IM), ls(xB' + BM, D'(k-1) + DM)) + e(k) and I(k) = ls(M'(k) + MI,
 * I'(k) + II) from the row above ('); the first level of the warp's next column is taken with
 * the second level of this one.  A lane before its row 1 gets -inf. */
__device__ bool rc_fwd_mi(const RcLane &S, const plk_rc_pep_t &P, const plk_rc_prof_t &R,
		const uint8_t *__restrict__ dsq, const int w, RcSync &Y, int *err)
{
	const int M = R.M, W = M + 1, W2 = M + 2, lane = threadIdx.x & 31;
	const float4 *T4 = (const float4*)R.tsc;
	float xB = P.lmove;
	for (int i = 1; i <= S.lmax; ++i) {
		if (i >= 2) {  /* row i-1: the other M/I warps' columns, the D row, xB */
			if (!rc_wait_all(Y, Y.fm, RC_MI, i - 1, err) || !rc_wait(Y, Y.fd, i - 1, err) || !rc_wait(Y, Y.fe, i - 1, err)) return false;
			xB = Y.xB[lane];
		}
		const bool act = i > S.off;
		const int rp = S.full ? i - 1 : (i - 1) & 1, rc = S.full ? i : i & 1;
		const float2 *pr = S.fmi + rc_ix(rp, 0, W);
		float2 *cr = S.fmi + rc_ix(rc, 0, W);
		const float *dp = S.d + ((i & 1) ? 0 : ((size_t)W << 5));   /* recheck.c:303 */
		const float *mcol = R.msc + (act ? dsq[i - 1 - S.off] : 0);
		if (w == 0) str2(cr, NEG2);
		if (w + 1 <= M) {
			/* pk, t1, ms: column k's row above at k, second half of tsc row k-1, e(k); nu, nk, nd, n0, n1, nms:
			 * all of the warp's next column, loaded two steps ahead (past M, the last one's again) */
			const int k0 = w + 1, k1 = k0 + RC_MI <= M ? k0 + RC_MI : k0;
			const float2 pu = ldr2(pr + ((size_t)(k0 - 1) << 5));
			const float pd = ldr(dp + ((size_t)(k0 - 1) << 5));
			float2 pk = ldr2(pr + ((size_t)k0 << 5));
			float2 nu = ldr2(pr + ((size_t)(k1 - 1) << 5)), nk = ldr2(pr + ((size_t)k1 << 5));
			float nd = ldr(dp + ((size_t)(k1 - 1) << 5));
			const float4 t0 = __ldg(T4 + 2 * (k0 - 1));
			float4 t1 = __ldg(T4 + 2 * (k0 - 1) + 1), n0 = __ldg(T4 + 2 * (k1 - 1)), n1 = __ldg(T4 + 2 * (k1 - 1) + 1);
			float ms = __ldg(mcol + (size_t)(k0 - 1) * RC_NCODE), nms = __ldg(mcol + (size_t)(k1 - 1) * RC_NCODE);
			float a, b;
			int chk = 0;
			{
				const float la[2] = {pu.x + t0.x, xB + t0.w}, lb[2] = {pu.y + t0.y, pd + t0.z};
				float lr[2];
				lsn<2>(la, lb, lr);
				a = lr[0], b = lr[1];
			}
#pragma unroll 1
			for (int k = k0; k <= M; k += RC_MI) {
				const int kq = k + 2 * RC_MI <= M ? k + 2 * RC_MI : k;
				const float2 qu = ldr2(pr + ((size_t)(kq - 1) << 5)), qk = ldr2(pr + ((size_t)kq << 5));
				const float qd = ldr(dp + ((size_t)(kq - 1) << 5));
				const float4 q0 = __ldg(T4 + 2 * (kq - 1)), q1 = __ldg(T4 + 2 * (kq - 1) + 1);
				const float qms = __ldg(mcol + (size_t)(kq - 1) * RC_NCODE);
				if (--chk < 0) {
					/* the slots of the warp's next RC_CK columns are free: the E warp has taken what they
					 * held, and so has the D warp, whose D of those columns the E warp had */
					const int kf = min(k + (RC_CK - 1) * RC_MI, M) - RC_Q;
					bool ok = true;
					if (kf > 0) rc_take(Y, Y.fcons[lane], i * W2 + kf, true, err, ok, true);
					if (!__all_sync(FULL, ok)) return false;
					chk = RC_CK - 1;
				}
				/* M(k)'s second level, I(k), the next column's first level */
				const float la[4] = {a, pk.x + t1.x, nu.x + n0.x, xB + n0.w}, lb[4] = {b, pk.y + t1.y, nu.y + n0.y, nd + n0.z};
				float lr[4];
				lsn<4>(la, lb, lr);
				const float mrk = glm_self(act, lr[0] + ms, RC_NEG);     /* M(k) */
				const float irk = glm_self(act && k < M, lr[1], RC_NEG); /* I(k) */
				a = lr[2], b = lr[3];
				Y.m[k % RC_Q][lane] = rc_pack(i * W2 + k, mrk);
				str2(cr + ((size_t)k << 5), make_float2(mrk, irk));
				pk = nk, t1 = n1, ms = nms, nu = qu, nk = qk, nd = qd, n0 = q0, n1 = q1, nms = qms;
			}
		}
		rc_publish(Y.fm[w], i);
	}
	return true;
}

/* Forward D warp (recheck.c:312-313): D(k) = ls(M(k-1) + MD, D(k-1) + DD) in column order from the
 * M/I warps' M; D(1) = ls(M(0) + 0, D(0) + 0) = -inf exactly, as the reference's D(1) */
__device__ bool rc_fwd_d(const RcLane &S, const plk_rc_prof_t &R, RcSync &Y, int *err)
{
	const int M = R.M, W = M + 1, W2 = M + 2, lane = threadIdx.x & 31;
	const float4 *T4 = (const float4*)R.tsc;
	for (int i = 1; i <= S.lmax; ++i) {
		const bool act = i > S.off;
		float *dr = S.d + ((i & 1) ? ((size_t)W << 5) : 0);
		if (i >= 2) { /* the E warp has emptied the ring of row i-1, and row i-2's D, in the same half,
		               * has been read: the M/I warps are past row i-1 */
			if (!rc_wait(Y, Y.fe, i - 1, err) || !rc_wait_all(Y, Y.fm, RC_MI, i - 1, err)) return false;
		}
		str(dr, RC_NEG);
		float mr1 = RC_NEG, dr1 = RC_NEG, md = 0.0f, dd = 0.0f;
		float4 tr = __ldg(T4 + 1);  /* tsc row k-1 in step k: MD, DD of D(k+1) */
#pragma unroll 1
		for (int k = 1; k <= M; ++k) {
			if (((k - 1) & (RC_BK - 1)) == 0) {
				bool ok = true;
				const int kl = min(k + RC_BK - 1, M);  /* the E warp has taken what the block's slots held */
				if (kl > RC_Q) rc_take(Y, Y.fcons[lane], i * W2 + kl - RC_Q, true, err, ok);
				rc_take_block(Y, Y.m, k, M, i * W2, err, ok);
				if (!__all_sync(FULL, ok)) return false;
			}
			const float m = rc_val(Y.m[k % RC_Q][lane]);
			const float4 tn = __ldg(T4 + 2 * (k < M ? k : k - 1) + 1);
			const float drk = glm_self(act, ls(mr1 + md, dr1 + dd), RC_NEG);  /* tsc row k-2 */
			Y.d[k % RC_Q][lane] = rc_pack(i * W2 + k, drk);
			str(dr + ((size_t)k << 5), drk);
			mr1 = m, dr1 = drk, md = tr.z, dd = tr.w, tr = tn;
		}
		rc_publish(Y.fd, i);
	}
	return true;
}

/* Forward E warp (recheck.c:314-317): E = ls(E, ls(M(k), D(k))) in column order, then xJ, xC, xN and
 * xB of the row; tot = xC(L) + lmove. */
__device__ bool rc_fwd_e(const RcLane &S, const plk_rc_pep_t &P, const plk_rc_prof_t &R, const bool on,
		RcSync &Y, int *err)
{
	const int M = R.M, W2 = M + 2, lane = threadIdx.x & 31;
	const float lmove = P.lmove, lloop = P.lloop, lE = -(float)RC_LN2;
	const size_t sps = (size_t)(S.lmax + 1) << 5;
	float *xNf = S.sp, *xJf = xNf + sps, *xCf = xJf + sps;
	const bool keep = on && P.null2;
	float xN = 0.0f, xB = lmove, xJ = RC_NEG, xC = RC_NEG;
	const size_t o = (size_t)S.off << 5;  /* row 0 */
	if (keep) str(xNf + o, 0.0f), str(xJf + o, RC_NEG), str(xCf + o, RC_NEG);
	for (int i = 1; i <= S.lmax; ++i) {
		float e = RC_NEG, tq = RC_NEG;  /* tq: the term of the column before (ls(-inf, -inf) = -inf at first) */
#pragma unroll 1
		for (int k = 1; k <= M; ++k) {
			if (((k - 1) & (RC_BK - 1)) == 0) {
				bool ok = true;
				rc_take_block(Y, Y.d, k, M, i * W2, err, ok);  /* D after M: M's block is there too */
				rc_take_block(Y, Y.m, k, M, i * W2, err, ok);
				if (!__all_sync(FULL, ok)) return false;
			}
			const float la[2] = {rc_val(Y.m[k % RC_Q][lane]), e}, lb[2] = {rc_val(Y.d[k % RC_Q][lane]), tq};
			if (((k - 1) & (RC_BK - 1)) == RC_BK - 1 || k == M) Y.fcons[lane] = rc_pack(i * W2 + k, 0.0f);
			float lr[2];
			lsn<2>(la, lb, lr);
			tq = lr[0], e = lr[1];
		}
		e = ls(e, tq);
		if (i > S.off) {
			xJ = ls(xJ + lloop, e + lE);
			xC = ls(xC + lloop, e + lE);
			xN = xN + lloop;
			xB = ls(xN + lmove, xJ + lmove);
			if (keep) str(xNf + ((size_t)i << 5), xN), str(xJf + ((size_t)i << 5), xJ), str(xCf + ((size_t)i << 5), xC);
		}
		Y.xB[lane] = xB;
		rc_publish(Y.fe, i);
	}
	Y.tot[lane] = xC + lmove;  /* C->T after the peptide's last row */
	return true;
}

/* Backward feed warp: what the chain warp adds, in the order in which it needs it, RC_PB columns a
 * block: for B M(i+1, k) + t[k-1].BM + e(k, x(i+1)), k from 1 on, then for D(k)
 * {M(i+1, k+1) + e(k+1, x(i+1)) + t[k].DM, t[k-1].DD}, k from M-1 down (past the row's end, its last
 * column again).  The loads of a block are in flight together, and none of them, nor an address, stands
 * between the chain's steps. */
__device__ bool rc_bwd_feed(const RcLane &S, const plk_rc_pep_t &P, const plk_rc_prof_t &R,
		const uint8_t *__restrict__ dsq, const bool n2, RcSync &Y, int *err)
{
	const int M = R.M, W = M + 1, lane = threadIdx.x & 31, L = n2 ? P.len : 1;
	int seq = 0;  /* blocks written */
	for (int t = 0; t + 2 <= S.lmax; ++t) {
		const int i = L - 1 - t;
		const bool act = n2 && i >= 1;
		if (t == 0 ? !rc_wait(Y, Y.bp, 0, err) : !rc_wait_all(Y, Y.bm, RC_MI, t - 1, err)) return false;  /* row i+1's M */
		const float2 *nx = S.bmi + rc_ix(S.lmax - t, 0, W);
		const float *mcol = R.msc + (act ? dsq[i] : 0);  /* residue i+1 */
		for (int c = 0; c < 2 * M - 1; c += RC_PB) { /* M columns of B, M - 1 of D: each from a block's start */
			float2 v[RC_PB];
			if (c < M) {
				float m[RC_PB], b[RC_PB], e[RC_PB];
#pragma unroll
				for (int j = 0; j < RC_PB; ++j) {
					const int k = min(c + 1 + j, M);
					m[j] = ldr2(nx + ((size_t)k << 5)).x, b[j] = __ldg(R.tsc + (size_t)(k - 1) * 8 + T_BM), e[j] = __ldg(mcol + (size_t)(k - 1) * RC_NCODE);
				}
#pragma unroll
				for (int j = 0; j < RC_PB; ++j) v[j] = make_float2(m[j] + b[j] + e[j], 0.0f);
			} else {
				float m[RC_PB], e[RC_PB], d[RC_PB];
#pragma unroll
				for (int j = 0; j < RC_PB; ++j) {
					const int k = max(M - 1 - (c - M) - j, 1);
					m[j] = ldr2(nx + ((size_t)(k + 1) << 5)).x, e[j] = __ldg(mcol + (size_t)k * RC_NCODE);
					d[j] = __ldg(R.tsc + (size_t)k * 8 + T_DM), v[j].y = __ldg(R.tsc + (size_t)(k - 1) * 8 + T_DD);
				}
#pragma unroll
				for (int j = 0; j < RC_PB; ++j) v[j].x = m[j] + e[j] + d[j];
			}
			if (seq >= RC_FB && !rc_wait(Y, Y.bf, seq - RC_FB + 1, err)) return false;  /* the block's place is free */
#pragma unroll
			for (int j = 0; j < RC_PB; ++j) Y.fd2[seq % RC_FB * RC_PB + j][lane] = v[j];
			rc_publish(Y.bw, ++seq);
			if (c < M && c + RC_PB >= M) c = M - RC_PB;  /* D's columns begin a block */
		}
	}
	return true;
}

/* Backward chain warp (recheck.c:323-375 without M and I): row L, then for each row i
 * (step t = L-1-i of the lane's rows) B = the sum over the columns of M(i+1, k) +
 * t[k-1].BM + e(k, x(i+1)) in column order, the special states, and D along the row
 * from the last column, D(k) = ls(M(i+1, k+1) + e(k+1) + DM, ls(D(k+1) + DD, bE)), handing
 * D(k+1) and bE to the M/I warps.  A group's time is this warp's, three logsums a column, so its
 * loops hold little else: with its own loads and their addresses a column took 1,060 to 1,300
 * cycles. */
__device__ bool rc_bwd_chain(const RcLane &S, const plk_rc_pep_t &P, const plk_rc_prof_t &R,
		const bool n2, RcSync &Y, int *err)
{
	const int M = R.M, W = M + 1, W2 = M + 2, lane = threadIdx.x & 31, L = n2 ? P.len : 1;
	const float4 *T4 = (const float4*)R.tsc;
	const float lmove = P.lmove, lloop = P.lloop, lE = -(float)RC_LN2;
	const size_t sps = (size_t)(S.lmax + 1) << 5;
	float *bNg = S.sp + 3 * sps, *bJg = bNg + sps, *bCg = bJg + sps;
	float bC = lmove, bE = bC + lE, bJ = RC_NEG, bN = RC_NEG;
	if (n2) { /* row L: M(M) = D(M) = bE; M(k) = ls(bE, D(k+1) + t[k-1].MD), D(k) = ls(bE, D(k+1) + t[k-1].DD) */
		float2 *rw = S.bmi + rc_ix(S.lmax, 0, W);
		float dn = bE;
		str2(rw + ((size_t)M << 5), make_float2(bE, RC_NEG));
		float4 t1 = __ldg(T4 + 2 * (M >= 2 ? M - 2 : 0) + 1);  /* tsc row k-1 for k = M-1 */
		for (int k = M - 1; k >= 1; --k) {
			const float4 tn = __ldg(T4 + 2 * (k >= 2 ? k - 2 : 0) + 1);
			const float la[2] = {bE, bE}, lb[2] = {dn + t1.z, dn + t1.w};
			float lr[2];
			lsn<2>(la, lb, lr);
			dn = lr[1];
			str2(rw + ((size_t)k << 5), make_float2(lr[0], RC_NEG));
			t1 = tn;
		}
		str2(rw, NEG2);
		const size_t o = (size_t)S.lmax << 5;
		str(bNg + o, bN), str(bJg + o, bJ), str(bCg + o, bC);
	}
	rc_publish(Y.bp, 0);  /* row L */
	int seq = 0, ready = 0;  /* blocks of the feed warp taken; known to be written */
	for (int t = 0; t + 2 <= S.lmax; ++t) {
		const int i = L - 1 - t;
		const bool act = n2 && i >= 1;
		float bB = RC_NEG;
		for (int k = 1; k <= M; k += RC_PB) {
			if (!rc_feed_next(Y, ready, seq, err)) return false;
			const float2 *v = &Y.fd2[seq % RC_FB * RC_PB][lane];
			const int n = min(RC_PB, M + 1 - k);
			float x = v[0].x;
#pragma unroll 1
			for (int j = 0; j < n; ++j) {
				v += 32;
				const float xn = v[0].x;  /* past the block: not used */
				bB = ls(bB, x);
				x = xn;
			}
			__syncwarp();
			++seq;
			if (lane == 0) Y.bf = seq;  /* read and used: the place is free */
		}
		if (act) {
			const float bJn = bJ, bCn = bC, bNn = bN;
			bJ = ls(bJn + lloop, bB + lmove);
			bC = bCn + lloop;
			bE = ls(bJ + lE, bC + lE);
			bN = ls(bNn + lloop, bB + lmove);
			const size_t o = (size_t)(S.lmax - 1 - t) << 5;
			str(bNg + o, bN), str(bJg + o, bJ), str(bCg + o, bC);
		}
		Y.bE[lane] = rc_pack(t * W2, bE);
		/* D along the row, last column first; D(k+1) goes to the ring before D(k) is formed */
		float dn = bE;
		for (int k0 = M - 1; k0 >= 1; k0 -= RC_PB) {
			const int c = M - k0;  /* columns handed over so far, the block's first included */
			if (c > RC_Q) {  /* the M/I warps have taken what the block's slots hold */
				bool ok = true;
#pragma unroll
				for (int j = RC_PB - RC_MI; j < RC_PB; ++j)
					rc_take(Y, Y.bcons[j % RC_MI][lane], t * W2 + c - RC_Q + j, true, err, ok);
				if (!__all_sync(FULL, ok)) return false;
			}
			if (!rc_feed_next(Y, ready, seq, err)) return false;
			const float2 *v = &Y.fd2[seq % RC_FB * RC_PB][lane];
			const int k1 = max(k0 - RC_PB + 1, 1);
			float2 x = v[0];
			int tag = t * W2 + c;
#pragma unroll 1
			for (int k = k0; k >= k1; --k, ++tag) {
				v += 32;
				const float2 xn = v[0];  /* past the block: not used */
				Y.dn[k % RC_Q][lane] = rc_pack(tag, dn);
				dn = ls(x.x, ls(dn + x.y, bE));
				x = xn;
			}
			__syncwarp();
			++seq;
			if (lane == 0) Y.bf = seq;  /* read and used: the place is free */
		}
	}
	return true;
}

/* Backward M/I warp w (recheck.c:362-366), columns k = M - 1 - w, M - 1 - w - RC_MI, ..: for row i,
 * M(k) = ls(ls(mn1 + MM, I(i+1, k) + MI), ls(bE, D(k+1) + MD)) and I(k) = ls(mn1 + IM, I(i+1, k) + II),
 * mn1 = M(i+1, k+1) + e(k+1), from the chain warp's bE and D(k+1). */
__device__ bool rc_bwd_mi(const RcLane &S, const plk_rc_pep_t &P, const plk_rc_prof_t &R,
		const uint8_t *__restrict__ dsq, const bool n2, const int w, RcSync &Y, int *err)
{
	const int M = R.M, W = M + 1, W2 = M + 2, lane = threadIdx.x & 31, L = n2 ? P.len : 1;
	const float4 *T4 = (const float4*)R.tsc;
	for (int t = 0; t + 2 <= S.lmax; ++t) {
		const int i = L - 1 - t;
		const bool act = n2 && i >= 1;
		if (t == 0 ? !rc_wait(Y, Y.bp, 0, err) : !rc_wait_all(Y, Y.bm, RC_MI, t - 1, err)) return false;  /* row i+1 */
		const float2 *nx = S.bmi + rc_ix(S.lmax - t, 0, W);
		float2 *rw = S.bmi + rc_ix(S.lmax - 1 - t, 0, W);
		const float *mcol = R.msc + (act ? dsq[i] : 0);
		/* the row's operands two of the warp's columns ahead; M(k)'s second level with the next
		 * column's first (the one before the warp's first column is a stand-in, not stored) */
		const int kf = max(M - 1 - w, 0), kg = max(kf - RC_MI, 0);
		float up = ldr2(nx + ((size_t)min(kf + 1, M) << 5)).x, nup = ldr2(nx + ((size_t)min(kg + 1, M) << 5)).x;
		float iu = ldr2(nx + ((size_t)kf << 5)).y, niu = ldr2(nx + ((size_t)kg << 5)).y;
		/* tsc row k: MM, IM; row k-1: MI, II, MD; e(k+1) */
		float2 tk = ldt2(T4 + 2 * min(kf, M - 1)), ntk = ldt2(T4 + 2 * kg);
		float4 r1 = __ldg(T4 + 2 * max(kf - 1, 0) + 1), nr1 = __ldg(T4 + 2 * max(kg - 1, 0) + 1);
		float me = __ldg(mcol + (size_t)min(kf, M - 1) * RC_NCODE), nme = __ldg(mcol + (size_t)kg * RC_NCODE);
		float a = RC_NEG, b = RC_NEG, ip = RC_NEG;
		bool ok = true;
		const float bE = rc_take(Y, Y.bE[lane], t * W2, false, err, ok, true);
		if (!__all_sync(FULL, ok)) return false;
		if (act && w == 0) str2(rw + ((size_t)M << 5), make_float2(bE, RC_NEG));
		int k = M - 1 - w;
#pragma unroll 1
		for (; k >= 1; k -= RC_MI) {
			const int c = M - k, kn = max(k - 2 * RC_MI, 0);
			const float2 q = ldr2(nx + ((size_t)kn << 5));
			const float qup = ldr2(nx + ((size_t)(kn + 1) << 5)).x;
			const float2 qtk = ldt2(T4 + 2 * kn);
			const float4 qr1 = __ldg(T4 + 2 * max(kn - 1, 0) + 1);
			const float qme = __ldg(mcol + (size_t)kn * RC_NCODE);
			const float dk1 = rc_take(Y, Y.dn[k % RC_Q][lane], t * W2 + c, false, err, ok);
			if (!__all_sync(FULL, ok)) return false;
			Y.bcons[w][lane] = rc_pack(t * W2 + c, 0.0f);
			const float mn1 = up + me;
			const float la[4] = {mn1 + tk.x, bE, mn1 + tk.y, a}, lb[4] = {iu + r1.x, dk1 + r1.z, iu + r1.y, b};
			float lr[4];
			lsn<4>(la, lb, lr);
			if (act && k + RC_MI < M) str2(rw + ((size_t)(k + RC_MI) << 5), make_float2(lr[3], ip));
			a = lr[0], b = lr[1], ip = lr[2];
			up = nup, iu = niu, nup = qup, niu = q.y;
			tk = ntk, r1 = nr1, me = nme, ntk = qtk, nr1 = qr1, nme = qme;
		}
		if (act && k + RC_MI < M) str2(rw + ((size_t)(k + RC_MI) << 5), make_float2(ls(a, b), ip));
		if (act && w == 0) str2(rw, NEG2);
		rc_publish(Y.bm[w], t);
	}
	return true;
}

/* posterior usage of columns [k_lo, k_hi] in log space, rows in ascending order
 * (recheck.c:382-390), eight columns at a time with the next row's values loaded one
 * row ahead (a block past k_hi repeats column k_hi and is not stored; lui(M) stays
 * -inf); lum / lui go to the D rows */
#define RC_UB 8
__device__ void rc_usage_lane(const RcLane &S, const plk_rc_pep_t &P, const int M, const int k_lo, const int k_hi)
{
	const int W = M + 1;
	float *lum = S.d, *lui = S.d + ((size_t)W << 5);
	for (int k0 = k_lo; k0 <= k_hi; k0 += RC_UB) {
		int kk[RC_UB];
		float um[RC_UB], ui[RC_UB];
		float2 f[RC_UB], g[RC_UB];
#pragma unroll
		for (int j = 0; j < RC_UB; ++j) {
			kk[j] = min(k0 + j, k_hi);
			um[j] = ui[j] = RC_NEG;
			f[j] = ldr2(S.fmi + rc_ix(S.off + 1, kk[j], W)), g[j] = ldr2(S.bmi + rc_ix(S.off + 1, kk[j], W));
		}
		for (int i = 1; i <= S.lmax; ++i) {
			if (i <= S.off) continue;
			const int in = min(i + 1, S.lmax);  /* row L's values again on the last row: not used */
			float2 fn[RC_UB], gn[RC_UB];
#pragma unroll
			for (int j = 0; j < RC_UB; ++j) fn[j] = ldr2(S.fmi + rc_ix(in, kk[j], W)), gn[j] = ldr2(S.bmi + rc_ix(in, kk[j], W));
			float sa[RC_UB], sb[RC_UB];
#pragma unroll
			for (int j = 0; j < RC_UB; ++j) sa[j] = f[j].x + g[j].x, sb[j] = f[j].y + g[j].y;
			lsn<RC_UB>(um, sa, um);
			lsn<RC_UB>(ui, sb, ui);
#pragma unroll
			for (int j = 0; j < RC_UB; ++j) f[j] = fn[j], g[j] = gn[j];
		}
#pragma unroll
		for (int j = 0; j < RC_UB; ++j)
			if (k0 + j <= k_hi) str(lum + ((size_t)(k0 + j) << 5), um[j]), str(lui + ((size_t)(k0 + j) << 5), k0 + j < M ? ui[j] : RC_NEG);
	}
}

/* usage of the special states N, J, C (recheck.c:391-395) */
__device__ void rc_special_usage(const RcLane &S, const plk_rc_pep_t &P, float &uN, float &uJ, float &uC)
{
	const size_t sps = (size_t)(S.lmax + 1) << 5;
	const float *xNf = S.sp, *xJf = xNf + sps, *xCf = xJf + sps, *bNg = xCf + sps, *bJg = bNg + sps, *bCg = bJg + sps;
	const float lloop = P.lloop;
	uN = uJ = uC = RC_NEG;
	for (int i = S.off + 1; i <= S.lmax; ++i) {
		const float ua[3] = {uN, uJ, uC};
		const float ub[3] = {ldr(xNf + ((size_t)(i - 1) << 5)) + ldr(bNg + ((size_t)i << 5)) + lloop,
		                     ldr(xJf + ((size_t)(i - 1) << 5)) + ldr(bJg + ((size_t)i << 5)) + lloop,
		                     ldr(xCf + ((size_t)(i - 1) << 5)) + ldr(bCg + ((size_t)i << 5)) + lloop};
		float ur[3];
		lsn<3>(ua, ub, ur);
		uN = ur[0], uJ = ur[1], uC = ur[2];
	}
}

/* the null2 bias (recheck.c:404-431) from the usage; returns it in nats */
__device__ float rc_null2_bias(const RcLane &S, const plk_rc_pep_t &P, const plk_rc_prof_t &R,
		const uint8_t *__restrict__ dsq, const float tot, const float uN, const float uJ, const float uC)
{
	const int M = R.M, W = M + 1, L = P.len;
	const float *msc = R.msc, logL = P.logL;
	const float *lum = S.d, *lui = S.d + ((size_t)W << 5);
	/* li, then the 20 residues' sums over the columns, each in column order */
	const float xfac = ls(ls(uN, uJ), uC) - tot - logL;
	float li = RC_NEG;
	for (int k = 1; k < M; ++k) li = ls(li, ldr(lui + ((size_t)k << 5)) - tot - logL);
	float v[20];
#pragma unroll
	for (int x = 0; x < 20; ++x) v[x] = ls(xfac, li);
	for (int k = 1; k <= M; ++k) {
		const float u = ldr(lum + ((size_t)k << 5)) - tot - logL;
		const float *mr = msc + (size_t)(k - 1) * RC_NCODE;
#pragma unroll
		for (int x0 = 0; x0 < 20; x0 += 4) {
			const float va[4] = {v[x0], v[x0 + 1], v[x0 + 2], v[x0 + 3]};
			const float vb[4] = {u + __ldg(mr + x0), u + __ldg(mr + x0 + 1), u + __ldg(mr + x0 + 2), u + __ldg(mr + x0 + 3)};
			float vr[4];
			lsn<4>(va, vb, vr);
			v[x0] = vr[0], v[x0 + 1] = vr[1], v[x0 + 2] = vr[2], v[x0 + 3] = vr[3];
		}
	}
	double s_odds = 0.0;
#pragma unroll
	for (int x = 0; x < 20; ++x) s_odds += exp((double)v[x]);
	const float lnodds_X = (float)log(s_odds / 20.0);
	/* the residue sum in the reference's order (recheck.c:427) */
	double n2 = 0.0;
	for (int i = 0; i < L; ++i) {
		const int x = dsq[i];
		float w = lnodds_X;
#pragma unroll
		for (int c = 0; c < 20; ++c) if (x == c) w = v[c];
		n2 = __dadd_rn(n2, (double)w);
	}
	const double a = __dadd_rn(log(1.0 / 256.0), n2);
	return (float)(a > 0.0 ? __dadd_rn(a, log1p(exp(-a))) : log1p(exp(a)));
}

struct RcArgs {
	const plk_rc_prof_t *prof;
	const plk_rc_pep_t *pep;
	const uint8_t *dsq;
	const int32_t *order;
	const plk_rc_grp_t *grp;
	int32_t n_grp;
	float *scratch, *bits, *bias;
	int *err;  /* set when a wait between warps ran out */
	long long spin_limit;
};

/* one CTA per group (the hardware hands the groups, longest first, to the
 * SMs as they free up); lane l of every warp takes the group's l-th peptide.  Then the warps
 * share the columns' usage sums, one takes the special states' too, and warp 0 the
 * bias and the score. */
__global__ void __launch_bounds__(32 * RC_UW, 1) k_rc_lanes(RcArgs A)
{
	__shared__ RcSync Y;
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	if (threadIdx.x < 32) s_exp2[threadIdx.x] = glm_exp2_tab_dev[threadIdx.x];
	if (threadIdx.x == 0) Y.fe = Y.fd = Y.bp = -1, Y.bw = Y.bf = 0, Y.abort = 0, Y.lim = A.spin_limit;
	if (threadIdx.x < RC_MI) Y.fm[threadIdx.x] = Y.bm[threadIdx.x] = -1;
	for (int x = threadIdx.x; x < RC_Q * 32; x += blockDim.x)  /* no slot carries a tag yet */
		Y.m[x >> 5][x & 31] = Y.d[x >> 5][x & 31] = Y.dn[x >> 5][x & 31] = rc_pack(-1, 0.0f);
	if (threadIdx.x < 32) Y.fcons[threadIdx.x] = Y.bE[threadIdx.x] = rc_pack(-1, 0.0f);
	for (int x = threadIdx.x; x < RC_MI * 32; x += blockDim.x) Y.bcons[x >> 5][x & 31] = rc_pack(-1, 0.0f);
	__syncthreads();
	const plk_rc_grp_t G = A.grp[blockIdx.x];
	const bool on = lane < G.count;  /* every thread stays for the barriers and the warp-wide steps */
	const int q = on ? A.order[G.first + lane] : 0;
	const plk_rc_pep_t P = A.pep[q];
	const plk_rc_prof_t R = A.prof[G.prof];
	const int M = R.M;
	const size_t W = (size_t)M + 1, rows = G.full ? (size_t)G.lmax + 1 : 2, brows = G.full ? (size_t)G.lmax + 1 : 0;
	float *base = A.scratch + G.scratch_off;
	RcLane S;
	S.fmi = (float2*)base + lane;
	S.bmi = (float2*)base + ((rows * W) << 5) + lane;
	S.d = base + (((rows + brows) * W) << 6) + lane;
	S.sp = S.d + ((2 * W) << 5);
	S.full = G.full, S.lmax = G.lmax, S.off = on ? G.lmax - P.len : G.lmax;
	const uint8_t *dsq = A.dsq + P.dsq_off;
	const bool n2 = on && P.null2;
	/* step 0 of the Forward: row 0 or a row before it */
	for (int k = w; k <= M; k += RC_UW)
		str2(S.fmi + rc_ix(0, k, M + 1), NEG2), str(S.d + ((size_t)k << 5), RC_NEG);
	__syncthreads();
	if (w == RC_W_D) rc_fwd_d(S, R, Y, A.err);
	else if (w == RC_W_E) rc_fwd_e(S, P, R, on, Y, A.err);
	else if (w == RC_W_B) { if (G.full) rc_bwd_chain(S, P, R, n2, Y, A.err); }
	else if (w == RC_W_F) { if (G.full) rc_bwd_feed(S, P, R, dsq, n2, Y, A.err); }
	else { /* of the other six, the first RC_MI to the Forward, the next to the Backward */
		const int x = w < RC_WARPS ? w - (w > RC_W_D) - (w > RC_W_B) - (w > RC_W_E) - (w > RC_W_F) : 2 * RC_MI;
		if (x < RC_MI) rc_fwd_mi(S, P, R, dsq, x, Y, A.err);
		else if (G.full && x < 2 * RC_MI) rc_bwd_mi(S, P, R, dsq, n2, x - RC_MI, Y, A.err);
	}
	__syncthreads();
	const bool ok = !Y.abort;
	if (G.full && ok) {  /* the same for the whole CTA */
		if (w < RC_UW - 1) {
			if (n2) for (int k = 1 + RC_UB * w; k <= M; k += RC_UB * (RC_UW - 1)) rc_usage_lane(S, P, M, k, min(k + RC_UB - 1, M));
		} else if (n2) {
			float uN, uJ, uC;
			rc_special_usage(S, P, uN, uJ, uC);
			Y.u[0][lane] = uN, Y.u[1][lane] = uJ, Y.u[2][lane] = uC;
		}
	}
	__syncthreads();
	if (w == 0 && on && ok) {
		const float tot = Y.tot[lane];
		const float bias = n2 ? rc_null2_bias(S, P, R, dsq, tot, Y.u[0][lane], Y.u[1][lane], Y.u[2][lane]) : 0.0f;
		/* recheck.c:432-437; null1 = L*logf(p1) + logf(1-p1) comes from the host */
		A.bits[q] = __fdiv_rn(__fsub_rn(__fsub_rn(tot, P.null1), bias), (float)RC_LN2);
		A.bias[q] = __fdiv_rn(bias, (float)RC_LN2);
	}
}

extern "C" int plk_rc_forward(const plk_rc_prof_t *prof, const plk_rc_pep_t *pep, const uint8_t *dsq,
		const int32_t *order, const plk_rc_grp_t *grp, int32_t n_grp, float *scratch, float *bits, float *bias,
		int *err, int64_t spin_limit, void *stream)
{
	if (n_grp <= 0) return 0;
	RcArgs A;
	A.spin_limit = spin_limit > 0 ? spin_limit : RC_SPIN_LIMIT;
	A.prof = prof, A.pep = pep, A.dsq = dsq, A.order = order, A.grp = grp, A.n_grp = n_grp;
	A.scratch = scratch, A.bits = bits, A.bias = bias, A.err = err;
	k_rc_lanes<<<(unsigned)n_grp, 32 * RC_UW, 0, (cudaStream_t)stream>>>(A);
	plk_add_launches(1);
	return (int)cudaGetLastError();
}

__global__ void k_mathf_eval(int fn, uint32_t lo, uint32_t stride, int64_t n, float *out)
{
	if (fn >= 4) {  /* four consecutive arguments per thread */
		for (int64_t i0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4; i0 < n; i0 += (int64_t)gridDim.x * blockDim.x * 4) {
			float x[4], y[4];
#pragma unroll
			for (int j = 0; j < 4; ++j) x[j] = __uint_as_float(lo + (uint32_t)((uint64_t)(i0 + j < n ? i0 + j : i0) * stride));
			if (fn == 6) gl_log1pexp_n<4>(x, y, glm_exp2_tab_dev);
			else
#pragma unroll
				for (int j = 0; j < 4; ++j)
					y[j] = fn == 4 ? gl_expf_rng(x[j]) : fn == 5 ? gl_log1pf_unit(x[j]) : gl_log1pf_unit(gl_expf_rng(-x[j]));
#pragma unroll
			for (int j = 0; j < 4; ++j) if (i0 + j < n) out[i0 + j] = y[j];
		}
		return;
	}
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
		const float x = __uint_as_float(lo + (uint32_t)((uint64_t)i * stride));
		out[i] = fn == 0 ? gl_expf(x) : fn == 1 ? gl_log1pf(x) : fn == 2 ? gl_expf_rng(x) : gl_log1pf_unit(x);
	}
}

extern "C" __attribute__((visibility("default"))) int pl_rc_mathf_eval(int32_t device, int32_t fn, uint32_t lo,
		uint32_t stride, int64_t n, float *out)
{
	float *d = 0;
	if (fn < 0 || fn > 7 || n < 0 || !out) return 0;
	if (n == 0) return 1;
	if (cudaSetDevice(device) != cudaSuccess || cudaMalloc((void**)&d, sizeof(float) * (size_t)n) != cudaSuccess) return 0;
	int64_t grid = (n + 255) / 256;
	if (grid > 148 * 16) grid = 148 * 16;
	k_mathf_eval<<<(unsigned)grid, 256>>>(fn, lo, stride, n, d);
	plk_add_launches(1);
	cudaError_t e = cudaGetLastError();
	if (e == cudaSuccess) e = cudaMemcpy(out, d, sizeof(float) * (size_t)n, cudaMemcpyDeviceToHost);
	cudaFree(d);
	return e == cudaSuccess;
}
