/*
 * gapless.cu -- sm_100a kernel of the gapless X-drop candidate prefilter (the
 * device replacement of ns_gapless_xdrop_batch, nasw-cuda.cu:1151-1295; same
 * scores, bit for bit).
 *
 * One warp per candidate.  For each anchor (at most 32, nasw-cuda.cu:1174):
 *   seed    the residue of every codon end of the block (plus the k-mer's reach) goes
 *           into shared memory once, twelve a lane: three aligned words of the packed
 *           genome hold their 14 bases, and three bases, as they lie in the genome,
 *           index a 4096-entry residue table (one per strand).  A lane then scores
 *           eight neighbouring deltas from 24 staged bytes against the scores of the
 *           k-mer's query residues, copied to a row each.  The best seed is a warp max
 *           over score * 8192 + (8191 - delta), so ties go to the smaller target end as
 *           in the reference's reduction;
 *   extend  left, then right: 32 steps at a time, one per lane, with warp
 *           prefix sums of the step scores and prefix maxima of the running
 *           score; the first step that leaves the sequence or breaks the X-drop
 *           ends the walk, and the best prefix (first step reaching it) is the
 *           reference's left_best / left_len (nasw-cuda.cu:1229-1252).
 * The warp then ranks the segments and sums them greedily with the overlap rule
 * of nasw-cuda.cu:1259-1293, a segment per lane.
 *
 * Bound by instruction issue (base by base with 64-bit bounds, and six scattered
 * query reads per delta, an anchor cost some 3,000 warp instructions).  131,072
 * candidates of 8 anchors, 256-wide blocks: 4.4 -> 1.64 ms.
 *
 * Every index is bounds-checked against the buffer sizes, so malformed
 * candidates read as missing bases / residues instead of faulting.
 */
#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>
#include "plk.h"
#include "../../include/plgpu.h"

#define FULL 0xffffffffu
#define GL_WARPS 8
#define GL_MAX_ANCHORS 32

extern "C" void plk_add_launches(uint64_t n);

struct GlArgs {
	const uint8_t *packed;
	int64_t bases;
	const uint8_t *queries;
	int64_t query_aa;
	const ns_gpu_gapless_candidate_t *cand;
	int32_t n_cand;
	const ns_gpu_gapless_anchor_t *anchors;
	int64_t n_anchors;
	int32_t block_width, kmer, xdrop, asize;
	int32_t *scores;
	unsigned long long *steps;  /* extension steps walked (for throughput accounting) */
};

__device__ __forceinline__ int gl_base(const GlArgs &A, const ns_gpu_gapless_candidate_t &C, int64_t pos)
{ /* nasw-cuda.cu:1151-1160 */
	if (pos < 0 || pos >= C.target_length) return 4;
	const int64_t a = C.target_offset + (C.reverse ? C.target_length - 1 - pos : pos);
	if (a < 0 || a >= A.bases) return 4;
	const int b = (__ldg(A.packed + (a >> 1)) >> ((a & 1) * 4)) & 0xf;
	return C.reverse && b < 4 ? 3 - b : b;
}

__device__ __forceinline__ int gl_aa(const GlArgs &A, const ns_gpu_gapless_candidate_t &C, const uint8_t *codon,
		int64_t end)
{ /* nasw-cuda.cu:1162-1170 */
	const int b0 = gl_base(A, C, end - 2), b1 = gl_base(A, C, end - 1), b2 = gl_base(A, C, end);
	return b0 < 4 && b1 < 4 && b2 < 4 ? codon[b0 << 4 | b1 << 2 | b2] : 20;
}

__device__ __forceinline__ int gl_query(const GlArgs &A, const ns_gpu_gapless_candidate_t &C, int64_t pos)
{
	const int64_t a = C.query_offset + pos;
	return a >= 0 && a < A.query_aa ? __ldg(A.queries + a) : 0;
}

/* bytes of a warp's staged residues: whole rounds of twelve, and the eight-byte reads past the last delta */
__host__ __device__ __forceinline__ int gl_stride(const int block_width, const int kmer)
{
	return (block_width + 3 * (kmer - 1) + 24 + 15) / 16 * 16;
}

/* the 16 packed bits from base a on (a nibble each), a within the genome's bytes */
__device__ __forceinline__ unsigned gl_nibbles(const GlArgs &A, const int64_t a)
{
	const uint8_t *p = A.packed + (a >> 1);
	return ((unsigned)__ldg(p) | (unsigned)__ldg(p + 1) << 8) >> ((int)(a & 1) * 4);
}

struct GlCand {
	ns_gpu_gapless_candidate_t C;
	const uint8_t *q;      /* its query, when all of it lies in the buffer */
	const uint8_t *tab;    /* residue table of its strand */
	int64_t lo, hi;        /* target positions whose codon end lies inside target and genome with the
	                        * bytes that gl_nibbles reads: [lo, hi) */
};

__device__ __forceinline__ int gl_q(const GlArgs &A, const GlCand &G, const int pos)
{
	const int v = G.q ? __ldg(G.q + pos) : gl_query(A, G.C, pos);
	return v < A.asize ? v : A.asize - 1;
}

/* residue of the codon ending at te (any te) */
__device__ __forceinline__ int gl_res(const GlArgs &A, const GlCand &G, const uint8_t *codon, const int64_t te)
{
	if (te >= G.lo && te < G.hi) {
		const int64_t a = G.C.target_offset + (G.C.reverse ? G.C.target_length - 1 - te : te - 2);
		return G.tab[gl_nibbles(A, a) & 0xfffu];
	}
	return min(gl_aa(A, G.C, codon, te), 31);
}

/* One side of the X-drop extension, 32 steps per round.  DIR = -1: left, +1: right.
 * Returns best (>= 0) and sets len (steps up to the first step reaching it). */
template <int DIR>
__device__ __forceinline__ int gl_extend(const GlArgs &A, const GlCand &G, const uint8_t *codon, const int *sm, const int lane,
		const int qend, const int64_t te0, int &len, unsigned &walked)
{
	int carry = 0, best = 0, blen = 0, st = 0;
	const int kmer = A.kmer;
	for (;;) {
		const int step = st + lane + 1;
		int pos;
		int64_t te;
		bool valid;
		if (DIR < 0) {
			pos = qend - kmer - (step - 1);
			te = te0 - (int64_t)(kmer - 1 + step) * 3;
			valid = pos >= 0 && te - 2 >= 0;
		} else {
			pos = qend + step;
			te = te0 + (int64_t)step * 3;
			valid = pos < G.C.query_length && te < G.C.target_length;
		}
		int v = 0;
		if (valid) v = sm[gl_res(A, G, codon, te) * A.asize + gl_q(A, G, pos)];
		int running = v;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const int x = __shfl_up_sync(FULL, running, o);
			if (lane >= o) running += x;
		}
		running += carry;
		const unsigned inval = __ballot_sync(FULL, !valid);
		const int first_invalid = inval ? __ffs(inval) - 1 : 32;
		int rmax = lane < first_invalid ? running : INT_MIN;  /* maximum of the round up to this step */
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const int x = __shfl_up_sync(FULL, rmax, o);
			if (lane >= o) rmax = max(rmax, x);
		}
		const unsigned brk = __ballot_sync(FULL, lane < first_invalid && max(best, rmax) - running > A.xdrop);
		const int first_brk = brk ? __ffs(brk) - 1 : 32;
		const int stop = min(first_invalid, first_brk + 1);  /* steps processed in this round */
		const int m = __shfl_sync(FULL, rmax, stop > 0 ? stop - 1 : 0);
		if (stop > 0 && m > best) { /* strict improvement: the first step reaching it */
			const unsigned at = __ballot_sync(FULL, lane < stop && running == m);
			blen = st + __ffs(at);
			best = m;
		}
		walked += stop;
		if (stop < 32) break;
		carry = __shfl_sync(FULL, running, 31);
		st += 32;
	}
	len = blen;
	return best;
}

/* residues of the window's codon ends base .. base + win - 1 into saa, twelve per lane and round */
__device__ __forceinline__ void gl_stage(const GlArgs &A, const GlCand &G, const uint8_t *codon, uint8_t *saa, const int64_t base,
		const int win, const int lane)
{
	const bool words = ((uintptr_t)A.packed & 3) == 0;
	for (int x0 = 12 * lane; x0 < win; x0 += 384) {
		const int64_t te = base + x0;
		/* their 14 bases from genome position a on, in three words that must lie in the buffer */
		const int64_t a = G.C.target_offset + (G.C.reverse ? G.C.target_length - 1 - (te + 11) : te - 2), w = a >> 3;
		uint32_t o[3];
		if (words && te >= G.lo && te + 11 < G.hi && (w + 3) * 8 <= A.bases) {
			const uint32_t *p = reinterpret_cast<const uint32_t*>(A.packed) + w;
			const uint32_t p0 = __ldg(p), p1 = __ldg(p + 1), p2 = __ldg(p + 2);
			const unsigned sh = (unsigned)(a & 7) * 4;
			const uint32_t v0 = __funnelshift_r(p0, p1, sh), v1 = __funnelshift_r(p1, p2, sh);
			uint32_t t[12];
#pragma unroll
			for (int i = 0; i < 12; ++i) t[i] = G.tab[(i < 8 ? __funnelshift_r(v0, v1, 4 * i) : v1 >> (4 * i - 32)) & 0xfffu];
#pragma unroll
			for (int i = 0; i < 3; ++i) o[i] = t[4 * i] + (t[4 * i + 1] << 8) + (t[4 * i + 2] << 16) + (t[4 * i + 3] << 24);
			if (G.C.reverse) { /* the codon ends run down the genome */
				const uint32_t z = __byte_perm(o[2], 0, 0x0123);
				o[1] = __byte_perm(o[1], 0, 0x0123), o[2] = __byte_perm(o[0], 0, 0x0123), o[0] = z;
			}
		} else {
			o[0] = o[1] = o[2] = 0;
			for (int i = 0; i < 12; ++i) {
				const uint32_t r = (uint32_t)gl_res(A, G, codon, te + i) << (8 * (i & 3));
				if (i < 4) o[0] |= r;
				else if (i < 8) o[1] |= r;
				else o[2] |= r;
			}
		}
		uint32_t *d = reinterpret_cast<uint32_t*>(saa + x0);
		d[0] = o[0], d[1] = o[1], d[2] = o[2];
	}
}

/* K: the k-mer length, compiled in for the mapper's 5, 6 and 7 (0: any length) */
template <int K>
__global__ void __launch_bounds__(32 * GL_WARPS) k_gapless(GlArgs A, const int8_t *__restrict__ mat,
		const uint8_t *__restrict__ codon_g)
{
	extern __shared__ __align__(16) uint8_t gl_smem[];
	__shared__ int sm[32 * 32];
	__shared__ uint8_t codon[64];
	__shared__ uint8_t tab[2][4096];  /* residue of three bases as they lie in the genome, read forward / on the other strand */
	__shared__ int prof[GL_WARPS][K > 0 ? K : 1][32];
	__shared__ int seg[GL_WARPS][3][GL_MAX_ANCHORS];
	const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
	for (int x = threadIdx.x; x < 32 * 32; x += blockDim.x) sm[x] = x < A.asize * A.asize ? mat[x] : 0;
	for (int x = threadIdx.x; x < 64; x += blockDim.x) codon[x] = codon_g[x];
	__syncthreads();
	for (int x = threadIdx.x; x < 4096; x += blockDim.x) {
		const int n0 = x & 15, n1 = x >> 4 & 15, n2 = x >> 8;
		const bool ok = n0 < 4 && n1 < 4 && n2 < 4;
		tab[0][x] = ok ? min((int)codon[n0 << 4 | n1 << 2 | n2], 31) : 20;
		tab[1][x] = ok ? min((int)codon[(3 - n2) << 4 | (3 - n1) << 2 | (3 - n0)], 31) : 20;
	}
	__syncthreads();
	const int kmer = K > 0 ? K : A.kmer;
	const int win = A.block_width + 3 * (kmer - 1);            /* codon ends of one anchor's seed scan */
	uint8_t *saa = gl_smem + (size_t)wib * gl_stride(A.block_width, kmer);
	for (int x = lane; x < gl_stride(A.block_width, kmer); x += 32) saa[x] = 0;  /* bytes past the window stay residue 0 */
	__syncwarp();
	unsigned long long walked_sum = 0;
	for (int ci = blockIdx.x * GL_WARPS + wib; ci < A.n_cand; ci += gridDim.x * GL_WARPS) {
		GlCand G;
		G.C = A.cand[ci];
		const int64_t ql = G.C.query_length;
		G.q = G.C.query_offset >= 0 && G.C.query_offset + ql <= A.query_aa ? A.queries + G.C.query_offset : 0;
		G.tab = tab[G.C.reverse ? 1 : 0];
		{ /* codon ends with all three bases inside the target, and their nibbles' two bytes in the genome */
			const int64_t off = G.C.target_offset, tl = G.C.target_length;
			G.lo = 2, G.hi = tl;
			if (G.C.reverse) { /* bases off + tl - 1 - te .. + 2, the last byte one further */
				G.lo = max(G.lo, off + tl + 3 - A.bases), G.hi = min(G.hi, off + tl);
			} else { /* bases off + te - 2 .. off + te */
				G.lo = max(G.lo, 2 - off), G.hi = min(G.hi, A.bases - off - 2);
			}
		}
		const int na = G.C.anchor_count < GL_MAX_ANCHORS ? G.C.anchor_count : GL_MAX_ANCHORS;
		int n_seg = 0;
		for (int ai = 0; ai < na; ++ai) {
			const int64_t aidx = (int64_t)G.C.anchor_offset + ai;
			if (aidx < 0 || aidx >= A.n_anchors) break;
			const ns_gpu_gapless_anchor_t an = A.anchors[aidx];
			const int qe = an.query_end;
			if (!(qe >= kmer - 1 && qe < G.C.query_length)) continue;
			const int64_t tb = an.target_block;
			gl_stage(A, G, codon, saa, tb - (int64_t)3 * (kmer - 1), win, lane);
			if (K > 0) {
#pragma unroll
				for (int k = 0; k < K; ++k)
					prof[wib][k][lane] = lane < A.asize ? sm[lane * A.asize + gl_q(A, G, qe - K + 1 + k)] : 0;
			}
			__syncwarp();
			/* deltas whose k-mer lies in the target */
			const int64_t dl = (int64_t)(kmer - 1) * 3 + 2 - tb, dh = G.C.target_length - tb;
			const int d_lo = dl > 0 ? (int)min(dl, (int64_t)A.block_width) : 0;
			const int d_hi = dh < A.block_width ? (int)max(dh, (int64_t)0) : A.block_width;
			int key = INT_MIN;  /* score * 8192 + (8191 - delta): scores are below 64 * 128, deltas below 8192 */
			if (K > 0) {
				for (int d0 = 8 * lane; d0 < d_hi; d0 += 256) {
					constexpr int NB = 8 + 3 * (K > 0 ? K - 1 : 0), NW = (NB + 7) / 8 * 2;
					uint32_t w[NW];
#pragma unroll
					for (int i = 0; i < NW; i += 2) {
						const uint2 x = *reinterpret_cast<const uint2*>(saa + d0 + 4 * i);
						w[i] = x.x, w[i + 1] = x.y;
					}
					int r[NB];
#pragma unroll
					for (int i = 0; i < NB; ++i) r[i] = (int)__byte_perm(w[i >> 2], 0, 0x4440 + (i & 3));
#pragma unroll
					for (int j = 0; j < 8; ++j) {
						int sc = 0;
#pragma unroll
						for (int k = 0; k < K; ++k) sc += prof[wib][k][r[j + 3 * k]];
						const int d = d0 + j;
						if (d >= d_lo && d < d_hi) key = max(key, sc * 8192 + 8191 - d);
					}
				}
			} else {
				for (int d = lane; d < d_hi; d += 32) {
					if (d < d_lo) continue;
					int sc = 0;
					for (int k = 0; k < kmer; ++k) sc += sm[saa[d + 3 * k] * A.asize + gl_q(A, G, qe - kmer + 1 + k)];
					key = max(key, sc * 8192 + 8191 - d);
				}
			}
#pragma unroll
			for (int o = 16; o >= 1; o >>= 1) key = max(key, __shfl_xor_sync(FULL, key, o));
			__syncwarp();
			if (key == INT_MIN) continue;  /* no valid target end in the block */
			const int seed = key >> 13;
			const int64_t te = tb + (8191 - (key & 8191));
			int ll, rl;
			unsigned wk = 0;
			const int lb = gl_extend<-1>(A, G, codon, sm, lane, qe, te, ll, wk);
			const int rb = gl_extend<1>(A, G, codon, sm, lane, qe, te, rl, wk);
			walked_sum += wk;
			if (lane == 0) {
				seg[wib][0][n_seg] = seed + lb + rb;
				seg[wib][1][n_seg] = qe - (kmer - 1) - ll;
				seg[wib][2][n_seg] = qe + rl;
			}
			++n_seg;
		}
		__syncwarp();
		{ /* nasw-cuda.cu:1259-1293: stable sort by score, greedy overlap-scaled sum */
			int total = 0;
			const int my = lane < n_seg ? seg[wib][0][lane] : INT_MIN;
			int rank = 0;
			for (int i = 0; i < n_seg; ++i) {
				const int x = __shfl_sync(FULL, my, i);
				rank += x > my || (x == my && i < lane);
			}
			const int b = lane < n_seg ? seg[wib][1][lane] : 0, e = lane < n_seg ? seg[wib][2][lane] : 0;
			__syncwarp();
			if (lane < n_seg) seg[wib][0][rank] = my, seg[wib][1][rank] = b, seg[wib][2][rank] = e;
			__syncwarp();
			const int ss = lane < n_seg ? seg[wib][0][lane] : 0, qs = lane < n_seg ? seg[wib][1][lane] : 0,
					qq = lane < n_seg ? seg[wib][2][lane] : 0;
			unsigned out = 0;  /* segments that earlier ones cover: they take part no more */
			for (int i = 0; i < n_seg; ++i) {
				const int si = __shfl_sync(FULL, ss, i), bi = __shfl_sync(FULL, qs, i), ei = __shfl_sync(FULL, qq, i);
				const int len = ei - bi + 1;
				if (i > 0 && si < A.xdrop) break;
				const int s0 = max(bi, qs), e0 = min(ei, qq);
				int overlap = lane < i && !(out >> lane & 1) && e0 >= s0 ? e0 - s0 + 1 : 0;
				if (__ballot_sync(FULL, overlap > 0)) {
#pragma unroll
					for (int o = 16; o >= 1; o >>= 1) overlap += __shfl_xor_sync(FULL, overlap, o);
				} else overlap = 0;
				if (overlap >= len) { out |= 1u << i; continue; }
				if (overlap > 0) total += (int)((long long)si * (len - overlap) / len);
				else total += si;
			}
			if (lane == 0) A.scores[ci] = n_seg ? total : INT_MIN;
		}
		__syncwarp();
	}
	if (lane == 0 && walked_sum) atomicAdd(A.steps, walked_sum);
}

extern "C" int plk_gapless_smem_bytes(int32_t block_width, int32_t kmer)
{
	return GL_WARPS * gl_stride(block_width, kmer);
}

extern "C" int plk_gapless(const uint8_t *packed, int64_t bases, const uint8_t *queries, int64_t query_aa,
		const void *cand, int32_t n_cand, const void *anchors, int64_t n_anchors, int32_t block_width, int32_t kmer,
		int32_t xdrop, const int8_t *mat_dev, int32_t asize, const uint8_t *codon_dev, int32_t *scores,
		unsigned long long *steps, int32_t n_sm, void *stream)
{
	if (n_cand <= 0) return 0;
	GlArgs A;
	A.packed = packed, A.bases = bases, A.queries = queries, A.query_aa = query_aa;
	A.cand = (const ns_gpu_gapless_candidate_t*)cand, A.n_cand = n_cand;
	A.anchors = (const ns_gpu_gapless_anchor_t*)anchors, A.n_anchors = n_anchors;
	A.block_width = block_width, A.kmer = kmer, A.xdrop = xdrop, A.asize = asize, A.scores = scores, A.steps = steps;
	const int smem = plk_gapless_smem_bytes(block_width, kmer);
	void (*f)(GlArgs, const int8_t*, const uint8_t*) = kmer == 6 ? k_gapless<6> : kmer == 5 ? k_gapless<5> :
			kmer == 7 ? k_gapless<7> : k_gapless<0>;
	cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
	if (e != cudaSuccess) return (int)e;
	int per_sm = 0;
	e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, 32 * GL_WARPS, smem);
	if (e != cudaSuccess) return (int)e;
	int64_t grid = (int64_t)(per_sm > 0 ? per_sm : 1) * n_sm;
	const int64_t need = (n_cand + GL_WARPS - 1) / GL_WARPS;
	if (grid > need) grid = need;
	f<<<(unsigned)grid, 32 * GL_WARPS, smem, (cudaStream_t)stream>>>(A, mat_dev, codon_dev);
	plk_add_launches(1);
	return (int)cudaGetLastError();
}
