/*
 * pffeat.cu -- per-candidate features of the learned prefilter, one CTA per
 * candidate (a protein and the genomic window a chained candidate spans, on the
 * strand the DP would read).
 *
 *  1. the protein's aa 5-mers go into a shared-memory hash table (4096 slots, first
 *     occurrence kept) and its aa 3-mers into 256 composition bins;
 *  2. the window is translated (all three frames: every position is the end of a
 *     codon); each codon end adds its window 3-mer to 256 more bins and looks its
 *     5-mer up in the table: a hit is an anchor (window position, protein position).
 *     The scan is the work (24,000 positions a candidate).  Each warp takes a
 *     contiguous part of the window, a lane 16 consecutive positions of it from one
 *     aligned 16-byte load, and everything between the bases and the two lookups stays
 *     in registers: the codes and residues before a lane's own come from the lane (or
 *     the step) before by shuffles, so the scan has no barrier.  The lookup tables sit
 *     in shared memory (as kernel constants their divergent reads serialised), and a
 *     65,536-bit map of the protein's 5-mers, 0.6 % full for a 420-residue protein,
 *     sends few warps to the hash table.  The first 1024 anchors by position are kept:
 *     when there are more, the warps go over their parts again in order (below);
 *  3. the anchors are sorted by position and chained: the longest chain increasing in
 *     both coordinates whose nucleotide gap is not shorter than 3x the residue gap
 *     minus 60 (frameshift slack).  A lane holds one anchor of a block of 32: the
 *     eight warps take the predecessors before the block among them, then one warp
 *     the block's own, each final anchor broadcast to the later ones (no reduction per
 *     anchor); the chain's sums come by pointer jumping instead of a walk;
 *  4. features: the 512 composition bins (scaled so a uniform composition is 1) and 20
 *     scalars of the anchors and the best chain (counts, coverage, span, frame
 *     changes, the window positions where the protein would start and end); the chain
 *     ends are also returned as integers for window tightening.
 *
 * Measured, 16,384 candidates of 2,048 proteins (393 M positions): the kernel 4.6 -> 1.2 ms
 * (tables and scan in bytes 4.6 -> 2.3, the chain without a reduction per anchor 1.8, no
 * branch per position 1.2); it issues on 65 % of the slots, the rest mostly waits on the
 * barriers around the chain.
 *
 * Feature row layout (bf16, F_DIM = 576 columns): [0,256) protein 3-mer bins,
 * [256,512) window 3-mer bins, [512,532) scalars, [532,576) zero.
 */
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include "plk.h"

extern "C" void plk_add_launches(uint64_t n);

namespace {

constexpr int THREADS = 256;
constexpr int HSLOTS = 4096;
constexpr int MAXA = 1024;
constexpr int F_DIM = PLK_PF_FDIM;
constexpr uint8_t BAD = 255;

struct FeatSmem {
	union {
		struct { int32_t hkey[HSLOTS], hpos[HSLOTS]; };
		struct { /* the chain, once the scan is done */
			int32_t p[MAXA], r[MAXA], f[MAXA], up[2][MAXA], sum[2][MAXA], part[THREADS / 32][32];
		} c;
	};
	int32_t bins[512];
	int64_t akey[MAXA];
	uint32_t map[2048];            /* word hmul(code) >> 21, bit code & 31 of every 5-mer in the table */
	uint8_t nt4[256], aa20[256], codon[64];
	int32_t n_anchor, tot_p, tot_w;
	int32_t part_n[THREADS / 32];  /* anchors of each warp's part of the window */
	int32_t chain[8];
};

__device__ __forceinline__ uint32_t hmul(uint32_t code) { return code * 2654435761u; }
__device__ __forceinline__ uint32_t h5(uint32_t h) { return h >> 20; }                                /* slot: 12 bits */
__device__ __forceinline__ uint32_t h3(uint32_t code) { return ((code * 40503u) >> 8) & 255u; }

/* first protein position of a 5-mer, or -1 */
__device__ __forceinline__ int32_t lookup5(const FeatSmem &S, const uint32_t code)
{
	uint32_t sl = h5(hmul(code));
	for (int t = 0; t < HSLOTS; ++t, sl = (sl + 1) & (HSLOTS - 1)) {
		const int32_t key = S.hkey[sl];
		if (key == 0) break;
		if (key == (int32_t)code + 1) return S.hpos[sl];
	}
	return -1;
}

/* More anchors than places: the window's first MAXA of them, whatever order the scan met them in
 * (the warps raced for the places, and a candidate's features could differ from run to run).  Warp w
 * goes over its positions [lo, hi) again, a position a lane and a step of 32 at a time, and writes its
 * anchors in order from base, the number that the warps before it hold, until the places are full.
 * The residues at p - 3 .. p - 12 come from the lanes of this step and the one before; the first
 * step, before lo, is there for them alone. */
__device__ __noinline__ void first_anchors(FeatSmem &S, const uint8_t *__restrict__ nt, const int32_t nl, const int64_t lo,
		const int64_t hi, int base, const int lane)
{
	uint32_t prev = BAD;
	for (int64_t b = lo - 32; b < hi && base < MAXA; b += 32) {
		const int64_t p = b + lane;
		uint32_t r = BAD;
		if (p >= 2 && p < nl) {
			const uint32_t c0 = S.nt4[nt[p - 2]], c1 = S.nt4[nt[p - 1]], c2 = S.nt4[nt[p]];
			if (!((c0 | c1 | c2) & 0x80)) r = S.codon[c0 << 4 | c1 << 2 | c2];
		}
		uint32_t code = 0;
		bool ok = p >= lo && p < hi;
#pragma unroll
		for (int k = 4; k >= 0; --k) {
			const uint32_t x = __shfl_sync(0xffffffffu, r, (lane - 3 * k) & 31), y = __shfl_sync(0xffffffffu, prev, (lane - 3 * k) & 31),
					v = lane >= 3 * k ? x : y;
			ok = ok && v != BAD;
			code = code * 20u + v;
		}
		const int32_t rp = ok ? lookup5(S, code) : -1;
		const uint32_t hit = __ballot_sync(0xffffffffu, rp >= 0);
		const int at = base + __popc(hit & ((1u << lane) - 1));
		if (rp >= 0 && at < MAXA) S.akey[at] = (p << 20) | (int64_t)rp;
		base += __popc(hit);
		prev = r;
	}
}

/* bit 7 of a word's four bytes, in order */
__device__ __forceinline__ uint32_t high_bits(const uint32_t w) { return (((w >> 7) & 0x01010101u) * 0x10204080u) >> 28; }

__global__ void __launch_bounds__(THREADS) k_pf_features(plk_pf_feat_args_t A)
{
	extern __shared__ __align__(16) uint8_t smem_raw[];
	FeatSmem &S = *reinterpret_cast<FeatSmem *>(smem_raw);
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int64_t q = blockIdx.x;
	if (q >= A.n) return;
	const plk_pf_cand_t C = A.cand[q];
	const int32_t nl = C.nl, al = C.al;
	const uint8_t *nt = A.nt + C.nt_off;
	const uint8_t *aa = A.aa + C.aa_off;
	for (int i = tid; i < 256; i += THREADS) {
		const uint8_t c = A.tabs.nt4[i];
		S.nt4[i] = c > 3 ? 0x80 : c;  /* bit 7: no base */
		S.aa20[i] = A.tabs.aa20[i];
	}
	for (int i = tid; i < 64; i += THREADS) {
		const uint8_t x = A.tabs.codon[i];
		S.codon[i] = x < 20 ? x : BAD;
	}
	for (int i = tid; i < 2048; i += THREADS) S.map[i] = 0;
	for (int i = tid; i < HSLOTS; i += THREADS) S.hkey[i] = 0, S.hpos[i] = 0x7fffffff;
	for (int i = tid; i < 512; i += THREADS) S.bins[i] = 0;
	if (tid == 0) S.n_anchor = 0, S.tot_p = 0, S.tot_w = 0;
	__syncthreads();

	/* 1. protein k-mers */
	int cnt3 = 0;
	for (int p = tid; p < al; p += THREADS) {
		uint8_t r[5];
		bool ok = true;
		const int w = p >= 4 ? 5 : p + 1;
		for (int k = 0; k < w; ++k) {
			const uint8_t x = S.aa20[aa[p - k]];
			r[k] = x < 20 ? x : BAD;
			if (r[k] == BAD) ok = false;
		}
		if (p >= 2 && r[0] != BAD && r[1] != BAD && r[2] != BAD) {
			atomicAdd(&S.bins[h3((uint32_t)r[2] * 400u + r[1] * 20u + r[0])], 1);
			++cnt3;
		}
		if (p >= 4 && ok) {
			const uint32_t code = (((r[4] * 20u + r[3]) * 20u + r[2]) * 20u + r[1]) * 20u + r[0];
			const uint32_t h = hmul(code);
			uint32_t s = h5(h);
			atomicOr(&S.map[h >> 21], 1u << (code & 31));
			for (int t = 0; t < HSLOTS; ++t, s = (s + 1) & (HSLOTS - 1)) {
				const int32_t old = atomicCAS(&S.hkey[s], 0, (int32_t)code + 1);
				if (old == 0 || old == (int32_t)code + 1) { atomicMin(&S.hpos[s], p); break; }
			}
		}
	}
	atomicAdd(&S.tot_p, cnt3);
	__syncthreads();

	/* 2. window scan, in groups of 16 positions P = p + a0 that start at 16-byte boundaries of the
	 * bases.  Warp w takes groups [gb, ge); its first step starts a group early, uncounted, for
	 * the codes and residues that reach into the part */
	int cntw = 0, nh = 0;
	const int a0 = (int)((uintptr_t)nt & 15);
	const int ng = (int)(((int64_t)nl + a0 + 15) / 16), gb = (int)((int64_t)ng * warp / (THREADS / 32)),
			ge = (int)((int64_t)ng * (warp + 1) / (THREADS / 32));
	{
		const uint4 *ntv = reinterpret_cast<const uint4 *>(nt - a0);
		/* of the position group before lane 0's: 2 codes with their marks, 12 residues */
		uint32_t pc = 0x30000000u, p1 = ~0u, p2 = ~0u, p3 = ~0u;
		for (int g0 = gb - 1; gb < ge && g0 < ge; g0 += 32) {
			const int g = g0 + lane;
			const int64_t p0 = 16 * (int64_t)g - a0;  /* the group's first position in the window */
			uint32_t x[4];
			if (p0 >= 0 && p0 + 16 <= nl && g < ge) {
				const uint4 q4 = __ldg(ntv + g);
				x[0] = q4.x, x[1] = q4.y, x[2] = q4.z, x[3] = q4.w;
			}
			/* codes: two bits each, the first position highest; bad: bit k = position k has no base */
			uint32_t cw = 0, bad = 0, any = 0x80;
			if (p0 >= 0 && p0 + 16 <= nl && g < ge) {
				any = 0;
#pragma unroll
				for (int k = 0; k < 16; ++k) {
					const uint32_t t = S.nt4[__byte_perm(x[k >> 2], 0, 0x4440 + (k & 3))];
					cw = cw * 4 + t, any |= t;
				}
			}
			if (any & 0x80) { /* an N, or the window's ends: one position at a time */
				cw = 0;
				for (int k = 0; k < 16; ++k) {
					const int64_t p = p0 + k;
					const uint32_t t = p >= 0 && p < nl && g < ge ? S.nt4[nt[p]] : 0x80u;
					cw = cw * 4 + (t & 3), bad |= (t >> 7) << k;
				}
			}
			/* residues of the 16 codons: the two codes before come from the lane before */
			const uint32_t last = (cw & 15) | (bad >> 14) << 28;
			uint32_t before = __shfl_up_sync(0xffffffffu, last, 1);
			if (lane == 0) before = pc;
			pc = __shfl_sync(0xffffffffu, last, 31);
			const uint32_t bb = bad << 2 | before >> 28, badc = bb | bb >> 1 | bb >> 2;  /* bit k: the codon ending at k */
			uint32_t v[28], o[4];
#pragma unroll
			for (int k = 0; k < 16; ++k) {
				const uint32_t idx = k < 2 ? ((before & 15) << (2 * k + 2) | cw >> (30 - 2 * k)) & 63 : cw >> (30 - 2 * k) & 63;
				v[12 + k] = S.codon[idx];
				o[k >> 2] = k & 3 ? o[k >> 2] + (v[12 + k] << (8 * (k & 3))) : v[12 + k];
			}
			uint32_t rb = high_bits(o[0]) | high_bits(o[1]) << 4 | high_bits(o[2]) << 8 | high_bits(o[3]) << 12;
			rb |= badc & 0xffffu;
			/* the 12 residues before and their marks (a byte with bit 7) */
			const uint32_t m1 = (rb >> 4 & 15) * 0x00204081u & 0x01010101u, m2 = (rb >> 8 & 15) * 0x00204081u & 0x01010101u,
					m3 = (rb >> 12 & 15) * 0x00204081u & 0x01010101u;
			const uint32_t s1 = o[1] | m1 << 7, s2 = o[2] | m2 << 7, s3 = o[3] | m3 << 7;
			uint32_t b1 = __shfl_up_sync(0xffffffffu, s1, 1), b2 = __shfl_up_sync(0xffffffffu, s2, 1),
					b3 = __shfl_up_sync(0xffffffffu, s3, 1);
			if (lane == 0) b1 = p1, b2 = p2, b3 = p3;
			p1 = __shfl_sync(0xffffffffu, s1, 31), p2 = __shfl_sync(0xffffffffu, s2, 31), p3 = __shfl_sync(0xffffffffu, s3, 31);
			const uint32_t m = high_bits(b1) | high_bits(b2) << 4 | high_bits(b3) << 8 | rb << 12;  /* bit i: v[i] is none */
			const uint32_t bad3 = m | m << 3 | m << 6, bad5 = bad3 | m << 9 | m << 12;
			if (g < gb || g >= ge || (bad3 >> 12 & 0xffffu) == 0xffffu) continue;
			cntw += __popc(~bad3 & 0x0ffff000u);
			uint32_t pr[28];
#pragma unroll
			for (int k = 0; k < 12; ++k) v[k] = __byte_perm(k < 4 ? b1 : k < 8 ? b2 : b3, 0, 0x4440 + (k & 3));
#pragma unroll
			for (int i = 3; i < 28; ++i) pr[i] = v[i - 3] * 20u + v[i];
			uint32_t hits = 0;  /* bit i: the map has the 5-mer ending at v[i] */
#pragma unroll
			for (int i = 12; i < 28; ++i) {
				const uint32_t tri = v[i - 6] * 400u + pr[i];
				if (!(bad3 >> i & 1)) atomicAdd(&S.bins[256 + h3(tri)], 1);
				const uint32_t code = pr[i - 9] * 8000u + tri, w = S.map[hmul(code) >> 21];
				hits |= __funnelshift_r(w, w, code - i) & (1u << i);
			}
			hits &= ~bad5;
			while (hits) {  /* few lanes have one: the 5-mer again, from its bytes */
				const int i = __ffs(hits) - 1;
				hits &= hits - 1;
				uint32_t code = 0;
#pragma unroll
				for (int k = 4; k >= 0; --k) {
					const int at = i - 3 * k;  /* byte of b1 b2 b3 o[0] .. o[3] */
					const uint32_t w = at < 4 ? b1 : at < 8 ? b2 : at < 12 ? b3 : at < 16 ? o[0] : at < 20 ? o[1] : at < 24 ? o[2] : o[3];
					code = code * 20u + (w >> (8 * (at & 3)) & 255);
				}
				const int32_t rp = lookup5(S, code);
				if (rp >= 0) {
					const int at = atomicAdd(&S.n_anchor, 1);
					++nh;
					/* both coordinates are k-mer ends */
					if (at < MAXA) S.akey[at] = ((p0 + i - 12) << 20) | (int64_t)rp;
				}
			}
		}
	}
	atomicAdd(&S.tot_w, cntw);
	__syncthreads();

	/* 3. sort the kept anchors by (position, protein position) -- all keys differ -- and chain them */
	const int na_all = S.n_anchor, na = na_all < MAXA ? na_all : MAXA;
	if (na_all > MAXA) {
		for (int o = 16; o >= 1; o >>= 1) nh += __shfl_xor_sync(0xffffffffu, nh, o);
		if (lane == 0) S.part_n[warp] = nh;
		__syncthreads();
		int base = 0;
		for (int w = 0; w < warp; ++w) base += S.part_n[w];
		first_anchors(S, nt, nl, 16 * (int64_t)gb - a0, 16 * (int64_t)ge - a0, base, lane);
		__syncthreads();
	}
	if (na <= THREADS) { /* an anchor per thread: its rank by counting */
		int rank = 0;
		const int64_t key = tid < na ? S.akey[tid] : 0;
		if (tid < na)
			for (int k = 0; k < na; ++k) rank += S.akey[k] < key;
		if (tid < na) S.c.p[rank] = (int32_t)(key >> 20), S.c.r[rank] = (int32_t)(key & 0xFFFFF);
		__syncthreads();
	} else {
		int np2 = 1;
		while (np2 < na) np2 <<= 1;
		for (int i = na + tid; i < np2; i += THREADS) S.akey[i] = INT64_MAX;
		__syncthreads();
		for (int k = 2; k <= np2; k <<= 1)
			for (int j = k >> 1; j > 0; j >>= 1) {
				for (int i = tid; i < np2; i += THREADS) {
					const int l = i ^ j;
					if (l > i) {
						const int64_t a = S.akey[i], b = S.akey[l];
						const bool up = (i & k) == 0;
						if ((a > b) == up) S.akey[i] = b, S.akey[l] = a;
					}
				}
				__syncthreads();
			}
		for (int i = tid; i < na; i += THREADS) S.c.p[i] = (int32_t)(S.akey[i] >> 20), S.c.r[i] = (int32_t)(S.akey[i] & 0xFFFFF);
		__syncthreads();
	}
	for (int b0 = 0; b0 < na; b0 += 32) {
		const int j = b0 + lane;
		const int32_t pj = j < na ? S.c.p[j] : 0, rj = j < na ? S.c.r[j] : 0;  /* lanes past the end take nothing: r >= 4 */
		int32_t best = 0;  /* f * 2048 + k + 1 of the best predecessor: ties to the largest k */
		for (int k = warp; k < b0; k += THREADS / 32) {
			const int32_t pk = S.c.p[k], rk = S.c.r[k];
			if (pk < pj && rk < rj && pj - pk >= 3 * (rj - rk) - 60) best = max(best, S.c.f[k] * 2048 + k + 1);
		}
		S.c.part[warp][lane] = best;
		__syncthreads();
		if (warp == 0) {
			for (int w = 1; w < THREADS / 32; ++w) best = max(best, S.c.part[w][lane]);
			for (int k = 0; k < 32; ++k) {
				const int32_t fk = (__shfl_sync(0xffffffffu, best, k) >> 11) + 1, pk = __shfl_sync(0xffffffffu, pj, k),
						rk = __shfl_sync(0xffffffffu, rj, k);
				if (k < lane && pk < pj && rk < rj && pj - pk >= 3 * (rj - rk) - 60) best = max(best, fk * 2048 + b0 + k + 1);
			}
			if (j < na) {
				const int32_t u = best ? (best & 2047) - 1 : j;  /* a chain's first anchor points at itself */
				S.c.f[j] = (best >> 11) + 1;
				S.c.up[0][j] = u;
				/* its link to the one before: a frame change (high half) and the residues it covers */
				S.c.sum[0][j] = u == j ? 0 : ((pj % 3 != S.c.p[u] % 3) << 16) + min(5, rj - S.c.r[u]);
			}
		}
		__syncthreads();
	}
	int buf = 0;
	for (int d = 1; d < na; d <<= 1, buf ^= 1) { /* sums over the links back to the chain's start */
		for (int j = tid; j < na; j += THREADS) {
			const int u = S.c.up[buf][j];
			S.c.sum[buf ^ 1][j] = S.c.sum[buf][j] + S.c.sum[buf][u];
			S.c.up[buf ^ 1][j] = S.c.up[buf][u];
		}
		__syncthreads();
	}
	if (warp == 0) {
		int32_t top = 0;  /* the first anchor with the largest f */
		for (int j = lane; j < na; j += 32) top = max(top, S.c.f[j] * 2048 + 2047 - j);
#pragma unroll
		for (int o = 16; o >= 1; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
		if (lane == 0) {
			const int jb = 2047 - (top & 2047), first = na ? S.c.up[buf][jb] : 0;
			S.chain[0] = na ? top >> 11 : 0;
			S.chain[1] = na ? S.c.sum[buf][jb] >> 16 : 0;
			S.chain[2] = na ? (S.c.sum[buf][jb] & 0xffff) + 5 : 0;
			S.chain[3] = na ? S.c.p[first] : -1, S.chain[4] = na ? S.c.p[jb] : -1;
			S.chain[5] = na ? S.c.r[first] : -1, S.chain[6] = na ? S.c.r[jb] : -1;
		}
	}
	__syncthreads();

	/* 4. features */
	__nv_bfloat16 *F = reinterpret_cast<__nv_bfloat16 *>(A.feats) + q * F_DIM;
	const float sp = 256.0f / (float)max(1, S.tot_p), sw = 256.0f / (float)max(1, S.tot_w);
	for (int i = tid; i < 512; i += THREADS) F[i] = __float2bfloat16_rn((float)S.bins[i] * (i < 256 ? sp : sw));
	for (int i = 532 + tid; i < F_DIM; i += THREADS) F[i] = __float2bfloat16_rn(0.0f);
	if (tid == 0) {
		const int32_t len = S.chain[0], fc = S.chain[1], cov = S.chain[2];
		const int32_t fp = S.chain[3], lp = S.chain[4], fr = S.chain[5], lr = S.chain[6];
		const float fnl = (float)max(nl, 1), fal = (float)max(al, 1);
		float v[20];
		v[0] = log2f(1.0f + al) / 12.0f;
		v[1] = log2f(1.0f + nl) / 16.0f;
		v[2] = log2f(1.0f + na_all) / 10.0f;
		v[3] = (float)len / (float)max(1, al - 4);
		v[4] = log2f(1.0f + len) / 10.0f;
		v[5] = (float)cov / fal;
		v[6] = len > 0 ? (float)(lp - fp) / fnl : 0.0f;
		v[7] = len > 0 ? (float)fp / fnl : 0.0f;
		v[8] = len > 0 ? (float)lp / fnl : 0.0f;
		v[9] = len > 0 ? (float)fr / fal : 0.0f;
		v[10] = len > 0 ? (float)lr / fal : 0.0f;
		v[11] = (float)fc / 8.0f;
		v[12] = len > 0 ? log2f(1.0f + (lp - fp)) / 16.0f : 0.0f;
		v[13] = len > 0 ? fminf(fmaxf((float)(fp - 3 * fr - 2) / fnl, -1.0f), 2.0f) : 0.0f;
		v[14] = len > 0 ? fminf(fmaxf((float)(lp + 3 * (al - 1 - lr)) / fnl, -1.0f), 2.0f) : 0.0f;
		v[15] = (float)min(na_all, 65535) * 1000.0f / fnl / 8.0f;
		v[16] = (float)len / (float)max(1, na);
		v[17] = 1.0f;
		v[18] = len >= 2 ? 1.0f : 0.0f;
		v[19] = na_all > MAXA ? 1.0f : 0.0f;
#pragma unroll
		for (int i = 0; i < 20; ++i) F[512 + i] = __float2bfloat16_rn(v[i]);
		int32_t *ci = A.chain + 4 * q;
		ci[0] = len > 0 ? fp : -1, ci[1] = len > 0 ? lp : -1, ci[2] = len > 0 ? fr : -1, ci[3] = len > 0 ? lr : -1;
	}
}

}  // namespace

extern "C" int plk_pf_features(const plk_pf_feat_args_t *a, void *stream)
{
	if (a->n <= 0) return 0;
	const int smem = (int)sizeof(FeatSmem);
	cudaError_t e = cudaFuncSetAttribute(k_pf_features, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
	if (e != cudaSuccess) return (int)e;
	k_pf_features<<<(unsigned)a->n, THREADS, smem, (cudaStream_t)stream>>>(*a);
	plk_add_launches(1);
	return (int)cudaGetLastError();
}
