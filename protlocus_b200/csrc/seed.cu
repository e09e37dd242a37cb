/*
 * seed.cu -- the coarse mapper's seeding on the device (mp_map_coarse's sketch and
 * anchor stages, map.c:565-572, default mode): per protein the k-mer sketch
 * (mp_sketch_prot, sketch.c:18-37), the occurrence cap (mp_cal_max_occ,
 * map.c:304-320, and map.c:566-569), the anchors of every seed whose bucket holds at
 * most the cap (mp_collect_anchors without the rescue, map.c:346-397) and their sort
 * (map.c:571).  The index is the reference's own (index.c:74-98), on the device:
 * ki[b] the first entry of bucket b in kb, the bucket's end ki[b+1] (n_kb for the last).
 *
 *   k_seed_sketch  one warp per protein: the 4-bit k-mers over the 13-letter alphabet of
 *                  32 positions at a time, the masked integer hash, the seeds compacted
 *                  in position order, their bucket sizes (32 lookups in flight), the cap
 *                  (the 25 % and 75 % order statistics of the sizes by a warp radix
 *                  select) and the anchor count.
 *   k_seed_anchors one CTA per protein of at most 16,384 anchors: the blocks of its kept
 *                  buckets as block << 32 | position into shared memory (32 seeds at a time
 *                  per warp, laid out by a warp scan), sorted there, written once.
 *   k_seed_emit    the larger proteins' anchors to memory, for the segmented sort.
 * HMM-profile queries (the query the profile's consensus, mp_sketch_query with a profile,
 * map.c:332-343) add the profile-derived seeds of mp_sketch_hmm (sketch.c:40-118) before
 * the cap: k_seed_hmm_alts (a thread per match state: its offered groups), k_seed_hmm_enum
 * (a warp per protein, a lane per window: the seeds appended after the protein's own), a
 * segmented sort and k_seed_unique (duplicates removed, then the cap as in the sketch).
 * The anchors of each protein are sorted ascending as 64-bit keys (equal keys are equal
 * values, so any sort leaves the reference's array).
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include <cub/cub.cuh>
#include "plk.h"
#include "seed_hmm.cuh"

extern "C" void plk_add_launches(uint64_t n);

namespace {

/* nasw-tab.c:9-12: residue letters, codes 0-21 and their 13-letter groups; other bytes 15 */
__constant__ uint8_t c_a2r[22] = { 0, 2, 4, 4, 6, 5, 5, 8, 3, 10, 11, 2, 11, 12, 7, 1, 1, 13, 12, 10, 14, 15 };
__constant__ char c_aa[23] = "ARNDCQEGHILKMFPSTWYV*X";

__device__ __forceinline__ uint32_t sd_hash(uint32_t key, const uint32_t mask)
{ /* sketch.c:7-16 */
	key = (key + ~(key << 15)) & mask;
	key ^= key >> 10;
	key = (key + (key << 3)) & mask;
	key ^= key >> 6;
	key = (key + ~(key << 11)) & mask;
	key ^= key >> 16;
	return key;
}

__device__ __forceinline__ int64_t sd_bucket_size(const int64_t *ki, const int64_t n_bucket, const int64_t n_kb, const int64_t b)
{
	return (b + 1 < n_bucket ? ki[b + 1] : n_kb) - ki[b];
}

__device__ __forceinline__ int64_t sd_warp_sum(int64_t v)
{
#pragma unroll
	for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
	return v;
}

/* the k-th smallest (0-based) of v[0..n), the whole warp: bit by bit from the top, the
 * values that share the bits chosen so far and have a 0 next are counted */
__device__ uint32_t sd_select(const uint32_t *v, const int32_t n, int64_t k, const int lane)
{
	uint32_t prefix = 0, top = 0;
	for (int32_t j = lane; j < n; j += 32) top |= v[j];
#pragma unroll
	for (int o = 16; o >= 1; o >>= 1) top |= __shfl_xor_sync(0xffffffffu, top, o);
	const int bits = 32 - __clz(top);  /* no value has a bit above these */
	uint32_t mask = bits < 32 ? ~0u << bits : 0;
	for (int bit = bits - 1; bit >= 0; --bit) {
		const uint32_t m = mask | 1u << bit;
		int64_t c = 0;
		for (int32_t j = lane; j < n; j += 32) c += (v[j] & m) == prefix;
		c = sd_warp_sum(c);
		if (k >= c) k -= c, prefix |= 1u << bit;
		mask = m;
	}
	return prefix;
}

/* the end of a protein's sketch, the whole warp: its n seeds' bucket sizes cnt (written
 * by the warp's lanes) give the occurrence cap, from 8 seeds on the box-plot bound over
 * the sizes' order statistics at these indices (map.c:310-319) limited by the option
 * (map.c:566-569); lane 0 records the count, the cap and the seeds' segment end */
__device__ __forceinline__ void sd_finish(const plk_seed_args_t &A, const int64_t q, const uint32_t *cnt, const int32_t n,
		const int lane)
{
	__syncwarp();
	int32_t max_occ = A.max_occ;
	if (n >= 8) {
		const int64_t k25 = (int64_t)(n * .25 + .499), k75 = (int64_t)(n * .75 + .499);
		const uint64_t q75 = sd_select(cnt, n, k75, lane), q25 = sd_select(cnt, n, k25, lane);
		max_occ = (int32_t)__dadd_rn(__dadd_rn((double)q75, __dmul_rn((double)(q75 - q25), 1.5)), 10.);
		if (max_occ > A.max_occ) max_occ = A.max_occ;
	}
	if (lane == 0) A.n_seed[q] = n, A.cap[q] = max_occ, A.seed_end[q] = A.soff[q] + n;
}

/* one warp per protein: the seeds in position order (a position's k-mer is its last kmer
 * residues when none of them restarts the k-mer, which is what the reference's rolling
 * k-mer holds), their bucket sizes, the cap and the anchor count */
__global__ void __launch_bounds__(256) k_seed_sketch(plk_seed_args_t A)
{
	__shared__ uint8_t tab[256];
	for (int x = threadIdx.x; x < 256; x += blockDim.x) tab[x] = 15;
	__syncthreads();
	if (threadIdx.x < 22) {
		const uint8_t c = (uint8_t)c_aa[threadIdx.x], g = c_a2r[threadIdx.x];
		tab[threadIdx.x] = g, tab[c] = g;
		if (c >= 'A' && c <= 'Z') tab[c + 32] = g;
	}
	__syncthreads();
	const int lane = threadIdx.x & 31;
	const int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	if (q >= A.n) return;  /* whole warps */
	const uint8_t *seq = A.seq + A.off[q];
	const int32_t len = A.len[q], kmer = A.kmer;
	uint64_t *sd = A.seeds + A.soff[q];
	uint32_t *cnt = A.cnt + A.soff[q];
	const uint32_t mask_k = (1U << kmer * 4) - 1, mask_mod = (1U << A.mod_bit) - 1;
	int32_t n = 0;
	for (int32_t i0 = 0; i0 < len; i0 += 32) {
		const int32_t i = i0 + lane;
		bool is_seed = false;
		uint64_t key = 0;
		if (i < len && i >= kmer - 1) {
			uint32_t x = 0;
			bool ok = true;
			for (int32_t t = i - kmer + 1; t <= i; ++t) {
				const uint32_t c = tab[seq[t]];
				ok = ok && c < 14;
				x = (x << 4 | c) & mask_k;
			}
			if (ok) {
				const uint32_t y = sd_hash(x, mask_k);
				if ((y & mask_mod) == 0) is_seed = true, key = (uint64_t)(y >> A.mod_bit) << 32 | (uint32_t)i;
			}
		}
		const unsigned bal = __ballot_sync(0xffffffffu, is_seed);
		if (is_seed) {
			const int32_t j = n + __popc(bal & ((1u << lane) - 1));
			sd[j] = key;
			cnt[j] = (uint32_t)sd_bucket_size(A.ki, A.n_bucket, A.n_kb, (int64_t)(key >> 32));
		}
		n += __popc(bal);
	}
	sd_finish(A, q, cnt, n, lane);
}

/* one warp per protein: the anchors each seed gives (mp_collect_anchors, map.c:352-384):
 * a bucket within the cap whole; with the repeat rescue, up to repeat_cap blocks of a
 * bucket over it, and when those exceed the budget, every share scaled down, then the rest
 * of the budget handed out one block at a time over the seeds in their sorted order from
 * the query name's hash onwards (lane 0, as the reference's loop) */
__global__ void __launch_bounds__(256) k_seed_take(plk_seed_args_t A)
{
	const int lane = threadIdx.x & 31;
	const int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	if (q >= A.n) return;  /* whole warps */
	const uint64_t *sd = A.seeds + A.soff[q];
	int32_t *take = A.take + A.soff[q];
	const int32_t n = A.n_seed[q], max_occ = A.cap[q], rcap = A.repeat_cap;
	int64_t n_base = 0, n_res = 0;
	for (int32_t j = lane; j < n; j += 32) {
		const int64_t sz = sd_bucket_size(A.ki, A.n_bucket, A.n_kb, (int64_t)(sd[j] >> 32));
		int32_t t = 0;
		if (sz <= max_occ) t = (int32_t)sz, n_base += sz;
		else if (rcap > 0) t = (int32_t)(sz < rcap ? sz : rcap), n_res += t;
		take[j] = t;
	}
	n_base = sd_warp_sum(n_base), n_res = sd_warp_sum(n_res);
	if (n_res > A.budget) {
		int64_t used = 0;
		for (int32_t j = lane; j < n; j += 32) {
			const int64_t sz = sd_bucket_size(A.ki, A.n_bucket, A.n_kb, (int64_t)(sd[j] >> 32));
			if (sz > max_occ && take[j] > 0) take[j] = (int32_t)((int64_t)take[j] * A.budget / n_res), used += take[j];
		}
		used = sd_warp_sum(used);
		__syncwarp();
		if (lane == 0) {
			const uint32_t start = n > 0 ? A.qhash[q] % (uint32_t)n : 0;
			for (int32_t i = 0; i < n && used < A.budget; ++i) {
				const int32_t j = (int32_t)((start + (uint32_t)i) % (uint32_t)n);
				const int64_t sz = sd_bucket_size(A.ki, A.n_bucket, A.n_kb, (int64_t)(sd[j] >> 32));
				const int64_t cap = sz < rcap ? sz : rcap;
				if (sz > max_occ && take[j] < cap) ++take[j], ++used;
			}
		}
		n_res = __shfl_sync(0xffffffffu, used, 0);
		__syncwarp();
	}
	if (lane == 0) A.n_anchor[q] = n_base + n_res;
}

/* what a warp holds of 32 seeds: exclusive scan of their takes, their buckets */
struct SdGroup {
	int64_t st[32], sz[32];
	int32_t pre[33];
	uint32_t pos[32];
};

/* seeds j0 .. j0+31 of a protein into G; returns their anchors */
__device__ __forceinline__ int32_t sd_group(const plk_seed_args_t &A, SdGroup &G, const uint64_t *sd, const int32_t *take,
		const int32_t n, const int32_t j0, const int lane)
{
	const int32_t j = j0 + lane;
	int64_t st = 0, sz = 0;
	int32_t tk = 0;
	uint32_t pos = 0;
	if (j < n) {
		const int64_t b = (int64_t)(sd[j] >> 32);
		st = A.ki[b];
		sz = (b + 1 < A.n_bucket ? A.ki[b + 1] : A.n_kb) - st;
		tk = take[j];
		pos = (uint32_t)sd[j];
	}
	int32_t inc = tk;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const int32_t t = __shfl_up_sync(0xffffffffu, inc, o);
		if (lane >= o) inc += t;
	}
	__syncwarp();
	G.pre[lane] = inc - tk, G.st[lane] = st, G.pos[lane] = pos, G.sz[lane] = sz;
	if (lane == 31) G.pre[32] = inc;
	__syncwarp();
	return __shfl_sync(0xffffffffu, inc, 31);
}

/* anchor t of the group: the seed is the last one whose offset is at most t; a whole bucket,
 * or take of its blocks evenly spaced (map.c:390-393) */
__device__ __forceinline__ uint64_t sd_anchor(const plk_seed_args_t &A, const SdGroup &G, const int32_t t)
{
	int lo = 0;
#pragma unroll
	for (int h = 16; h >= 1; h >>= 1) if (G.pre[lo + h] <= t) lo += h;
	const int64_t u = t - G.pre[lo], bsz = G.sz[lo], btk = G.pre[lo + 1] - G.pre[lo];
	const int64_t o = btk == bsz ? u : u * bsz / btk + bsz / (2 * btk);
	return (uint64_t)__ldg(A.kb + G.st[lo] + o) << 32 | G.pos[lo];
}

/* one warp per protein of the list: its anchors to memory, unsorted */
#define SD_EMIT_WARPS 8
__global__ void __launch_bounds__(32 * SD_EMIT_WARPS) k_seed_emit(plk_seed_args_t A, const int32_t *list, int32_t n_list)
{
	__shared__ SdGroup s_g[SD_EMIT_WARPS];
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	if (i >= n_list) return;  /* whole warps */
	const int32_t q = list[i];
	const uint64_t *sd = A.seeds + A.soff[q];
	const int32_t n = A.n_seed[q];
	const int32_t *take = A.take + A.soff[q];
	uint64_t *a = A.anchors + A.a_off[q];
	int64_t k = 0;
	for (int32_t j0 = 0; j0 < n; j0 += 32) {
		const int32_t total = sd_group(A, s_g[w], sd, take, n, j0, lane);
		for (int32_t t = lane; t < total; t += 32) a[k + t] = sd_anchor(A, s_g[w], t);
		k += total;
	}
}

/* One CTA of T threads per protein of the list, each with at most T * PER anchors: emitted into
 * shared memory and sorted there, so that they cross HBM once (emission, the segmented sort's
 * read and write were 3.5 times the traffic and a radix sort's passes).  A genome's blocks
 * spread a protein's anchors thinly, so one distribution over B buckets of equal width between
 * the smallest and the largest block leaves one or two keys a bucket, which a thread sorts by
 * insertion; a gene's cluster of up to 128 keys is ranked by a warp, and where a bucket holds
 * more (or more than SD_BIG of them are large) the CTA sorts all keys by a bitonic network.
 * Any order the seeds and the buckets come in is taken.  10,000 proteins, 26.5 M anchors:
 * emission and sort 2.16 -> 0.58 ms. */
#define SD_BIG 256
template <int T, int PER>
__global__ void __launch_bounds__(T) k_seed_anchors(plk_seed_args_t A, const int32_t *list, uint64_t *__restrict__ out)
{
	constexpr int NMAX = T * PER, B = NMAX / 2;
	extern __shared__ __align__(16) uint64_t s_key[];  /* [NMAX], then uint32 [B + 1] */
	uint32_t *s_cnt = (uint32_t*)(s_key + NMAX);
	__shared__ SdGroup s_g[T / 32];
	__shared__ uint32_t s_mn, s_mx, s_part[T / 32], s_big[SD_BIG];
	__shared__ int32_t s_n, s_nbig;
	const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
	const int32_t q = list[blockIdx.x];
	const int32_t n = (int32_t)(A.a_off[q + 1] - A.a_off[q]);
	if (n <= 0) return;
	if (tid == 0) s_n = 0, s_nbig = 0, s_mn = 0xffffffffu, s_mx = 0;
	for (int x = tid; x <= B; x += T) s_cnt[x] = 0;
	__syncthreads();
	{ /* emission: the groups of 32 seeds in any order */
		const uint64_t *sd = A.seeds + A.soff[q];
		const int32_t *take = A.take + A.soff[q], ns = A.n_seed[q];
		for (int32_t j0 = 32 * w; j0 < ns; j0 += T) {
			const int32_t total = sd_group(A, s_g[w], sd, take, ns, j0, lane);
			int32_t k = 0;
			if (lane == 0) k = atomicAdd(&s_n, total);
			k = __shfl_sync(0xffffffffu, k, 0);
			for (int32_t t = lane; t < total; t += 32)
				if (k + t < NMAX) s_key[k + t] = sd_anchor(A, s_g[w], t);
		}
	}
	__syncthreads();
	uint64_t key[PER];
	uint32_t mn = 0xffffffffu, mx = 0;
#pragma unroll
	for (int i = 0; i < PER; ++i) {
		key[i] = tid + i * T < n ? s_key[tid + i * T] : 0;
		if (tid + i * T < n) mn = min(mn, (uint32_t)(key[i] >> 32)), mx = max(mx, (uint32_t)(key[i] >> 32));
	}
#pragma unroll
	for (int o = 16; o >= 1; o >>= 1) {
		mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
		mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
	}
	if (lane == 0) atomicMin(&s_mn, mn), atomicMax(&s_mx, mx);
	__syncthreads();
	mn = s_mn, mx = s_mx;
	/* bucket of a block: d * B / range rounded down, the block itself where B covers the range */
	const uint64_t range = (uint64_t)mx - mn + 1;
	const uint32_t scale = range > B ? (uint32_t)(((uint64_t)B << 32) / range) : 0;
	uint32_t at[PER];
#pragma unroll
	for (int i = 0; i < PER; ++i)
		if (tid + i * T < n) {
			const uint32_t d = (uint32_t)(key[i] >> 32) - mn, b = scale ? __umulhi(d, scale) : d;
			at[i] = atomicAdd(&s_cnt[b], 1) << 16 | b;  /* its place in bucket b: n <= 16384, B <= 8192 */
		}
	__syncthreads();
	{ /* exclusive scan of the counts, B / T of them a thread */
		constexpr int C = B / T;
		uint32_t c[C], sum = 0;
#pragma unroll
		for (int x = 0; x < C; ++x) c[x] = s_cnt[tid * C + x], sum += c[x];
		uint32_t inc = sum;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
			if (lane >= o) inc += t;
		}
		if (lane == 31) s_part[w] = inc;
		__syncthreads();
		uint32_t base = 0;
		for (int x = 0; x < w; ++x) base += s_part[x];
		base += inc - sum;
#pragma unroll
		for (int x = 0; x < C; ++x) s_cnt[tid * C + x] = base, base += c[x];
		if (tid == T - 1) s_cnt[B] = base;
	}
	__syncthreads();
#pragma unroll
	for (int i = 0; i < PER; ++i)
		if (tid + i * T < n) s_key[s_cnt[at[i] & 0xffffu] + (at[i] >> 16)] = key[i];
	__syncthreads();
	for (int b = tid; b < B; b += T) {
		const int s0 = (int)s_cnt[b], m = (int)s_cnt[b + 1] - s0;
		if (m <= 1) continue;
		if (m > 12) {
			const int x = atomicAdd(&s_nbig, 1);
			if (x < SD_BIG) s_big[x] = (uint32_t)b;
			continue;
		}
		for (int i = 1; i < m; ++i) {
			const uint64_t v = s_key[s0 + i];
			int j = i;
			for (; j > 0 && s_key[s0 + j - 1] > v; --j) s_key[s0 + j] = s_key[s0 + j - 1];
			s_key[s0 + j] = v;
		}
	}
	__syncthreads();
	bool bad = s_nbig > SD_BIG;
	if (!bad)
		for (int x = w; x < s_nbig; x += T / 32) { /* ranks by counting, four keys a lane; equal keys by place */
			const int s0 = (int)s_cnt[s_big[x]], m = (int)s_cnt[s_big[x] + 1] - s0;
			if (m > 128) { bad = true; continue; }
			uint64_t v[4];
			int r[4];
#pragma unroll
			for (int i = 0; i < 4; ++i) v[i] = lane + 32 * i < m ? s_key[s0 + lane + 32 * i] : 0, r[i] = 0;
			for (int j = 0; j < m; ++j) {
				const uint64_t u = s_key[s0 + j];
#pragma unroll
				for (int i = 0; i < 4; ++i) r[i] += u < v[i] || (u == v[i] && j < lane + 32 * i);
			}
			__syncwarp();
#pragma unroll
			for (int i = 0; i < 4; ++i) if (lane + 32 * i < m) s_key[s0 + r[i]] = v[i];
			__syncwarp();
		}
	if (__syncthreads_or(bad)) {
		int np2 = 1;
		while (np2 < n) np2 <<= 1;  /* at most NMAX, a power of two */
		for (int i = n + tid; i < np2; i += T) s_key[i] = ~0ull;
		__syncthreads();
		for (int k = 2; k <= np2; k <<= 1)
			for (int j = k >> 1; j > 0; j >>= 1) {
				for (int i = tid; i < np2; i += T) {
					const int l = i ^ j;
					if (l > i) {
						const uint64_t a = s_key[i], c = s_key[l];
						if ((a > c) == ((i & k) == 0)) s_key[i] = c, s_key[l] = a;
					}
				}
				__syncthreads();
			}
	}
	uint64_t *o = out + A.a_off[q];
	for (int i = tid; i < n; i += T) o[i] = s_key[i];
}

/* HMM-profile queries: one thread per match state, its offered groups (seed_hmm.cuh) */
__global__ void __launch_bounds__(256) k_seed_hmm_alts(plk_seed_args_t A)
{
	const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (s >= A.n_state) return;
	((sh_alts_t*)A.alts)[s] = sh_state_alts(A.emit + s * 20, A.pos_loss);
}

/* one warp per protein, 32 windows of its profile at a time: each lane counts its window's
 * seeds, a warp scan places them after the protein's own seeds (the sketch's), and the lane
 * walks its window again to write them.  The protein's slots hold its own seeds (at most
 * len) and at most min(seed_max, 4^kmer) per window */
__global__ void __launch_bounds__(256) k_seed_hmm_enum(plk_seed_args_t A)
{
	const int lane = threadIdx.x & 31;
	const int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	if (q >= A.n) return;  /* whole warps */
	const int32_t kmer = A.kmer, el = A.e_len[q], mx = A.seed_max;
	const int32_t n_win = mx > 0 && el >= kmer ? el - kmer + 1 : 0;
	const sh_alts_t *al = (const sh_alts_t*)A.alts + A.e_off[q];
	const int32_t n0 = A.n_seed[q];
	uint64_t *out = A.seeds + A.soff[q] + n0;
	int64_t k = 0;
	for (int32_t w0 = 0; w0 < n_win; w0 += 32) {
		const int32_t w = w0 + lane;
		int64_t c = 0;
		if (w < n_win) c = sh_window_seeds(al + w, kmer, A.mod_bit, A.win_loss, mx, w + kmer - 1, 0);
		int64_t inc = c;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const int64_t t = __shfl_up_sync(0xffffffffu, inc, o);
			if (lane >= o) inc += t;
		}
		if (c > 0) sh_window_seeds(al + w, kmer, A.mod_bit, A.win_loss, mx, w + kmer - 1, out + k + inc - c);
		k += __shfl_sync(0xffffffffu, inc, 31);
	}
	__syncwarp();
	if (lane == 0) A.n_seed[q] = n0 + (int32_t)k, A.seed_end[q] = A.soff[q] + n0 + k;
}

/* one warp per protein: its seeds, sorted (sorted + soff, n_seed of them), without
 * duplicates into its slots (mp_sketch_query with a profile, map.c:338-342), their bucket
 * sizes, and the cap over them (sd_finish) */
__global__ void __launch_bounds__(256) k_seed_unique(plk_seed_args_t A, const uint64_t *sorted)
{
	const int lane = threadIdx.x & 31;
	const int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	if (q >= A.n) return;  /* whole warps */
	const int64_t base = A.soff[q];
	const int32_t n_in = A.n_seed[q];
	const uint64_t *in = sorted + base;
	uint64_t *sd = A.seeds + base;
	uint32_t *cnt = A.cnt + base;
	int32_t n = 0;
	uint64_t last = 0;
	for (int32_t j0 = 0; j0 < n_in; j0 += 32) {
		const int32_t j = j0 + lane;
		const uint64_t v = j < n_in ? in[j] : 0;
		uint64_t prev = __shfl_up_sync(0xffffffffu, v, 1);
		if (lane == 0) prev = last;
		const bool keep = j < n_in && (j == 0 || v != prev);
		const unsigned bal = __ballot_sync(0xffffffffu, keep);
		if (keep) {
			const int32_t t = n + __popc(bal & ((1u << lane) - 1));
			sd[t] = v;
			cnt[t] = (uint32_t)sd_bucket_size(A.ki, A.n_bucket, A.n_kb, (int64_t)(v >> 32));
		}
		n += __popc(bal);
		last = __shfl_sync(0xffffffffu, v, 31);
	}
	sd_finish(A, q, cnt, n, lane);
}

}  // namespace

extern "C" int plk_seed_hmm_alts(const plk_seed_args_t *a, void *stream)
{
	if (a->n_state <= 0) return 0;
	k_seed_hmm_alts<<<(unsigned)((a->n_state + 255) / 256), 256, 0, (cudaStream_t)stream>>>(*a);
	plk_add_launches(1);
	return (int)cudaGetLastError();
}

extern "C" int plk_seed_hmm_enum(const plk_seed_args_t *a, void *stream)
{
	if (a->n <= 0) return 0;
	k_seed_hmm_enum<<<(unsigned)(((int64_t)a->n * 32 + 255) / 256), 256, 0, (cudaStream_t)stream>>>(*a);
	plk_add_launches(1);
	return (int)cudaGetLastError();
}

extern "C" int plk_seed_unique(const plk_seed_args_t *a, const uint64_t *sorted, void *stream)
{
	if (a->n <= 0) return 0;
	k_seed_unique<<<(unsigned)(((int64_t)a->n * 32 + 255) / 256), 256, 0, (cudaStream_t)stream>>>(*a, sorted);
	plk_add_launches(1);
	return (int)cudaGetLastError();
}

extern "C" int plk_seed_sketch(const plk_seed_args_t *a, void *stream)
{
	if (a->n <= 0) return 0;
	k_seed_sketch<<<(unsigned)(((int64_t)a->n * 32 + 255) / 256), 256, 0, (cudaStream_t)stream>>>(*a);
	plk_add_launches(1);
	return (int)cudaGetLastError();
}

extern "C" int plk_seed_take(const plk_seed_args_t *a, void *stream)
{
	if (a->n <= 0) return 0;
	k_seed_take<<<(unsigned)(((int64_t)a->n * 32 + 255) / 256), 256, 0, (cudaStream_t)stream>>>(*a);
	plk_add_launches(1);
	return (int)cudaGetLastError();
}

extern "C" int plk_seed_emit(const plk_seed_args_t *a, const int32_t *list, int32_t n_list, void *stream)
{
	if (n_list <= 0) return 0;
	k_seed_emit<<<(unsigned)(((int64_t)n_list * 32 + 32 * SD_EMIT_WARPS - 1) / (32 * SD_EMIT_WARPS)), 32 * SD_EMIT_WARPS, 0,
			(cudaStream_t)stream>>>(*a, list, n_list);
	plk_add_launches(1);
	return (int)cudaGetLastError();
}

template <int T, int PER>
static int seed_anchors(const plk_seed_args_t *a, const int32_t *list, int32_t n_list, uint64_t *out, cudaStream_t st)
{
	const int smem = 8 * T * PER + 4 * (T * PER / 2 + 4);
	cudaError_t e = cudaFuncSetAttribute(k_seed_anchors<T, PER>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
	if (e != cudaSuccess) return (int)e;
	k_seed_anchors<T, PER><<<(unsigned)n_list, T, smem, st>>>(*a, list, out);
	plk_add_launches(1);
	return (int)cudaGetLastError();
}

/* the sorted anchors of the list's proteins, each at most PLK_SEED_CLASS(cls) of them, into out */
extern "C" int plk_seed_anchors(const plk_seed_args_t *a, const int32_t *list, int32_t n_list, int32_t cls, uint64_t *out,
		void *stream)
{
	cudaStream_t st = (cudaStream_t)stream;
	if (n_list <= 0) return 0;
	/* the least shared memory that holds a class: 23 to 187 KB a CTA */
	switch (cls) {
	case 0: return seed_anchors<256, 8>(a, list, n_list, out, st);
	case 1: return seed_anchors<256, 16>(a, list, n_list, out, st);
	case 2: return seed_anchors<512, 16>(a, list, n_list, out, st);
	case 3: return seed_anchors<1024, 16>(a, list, n_list, out, st);
	default: return (int)cudaErrorInvalidValue;
	}
}

/* per-segment ascending sort of keys_in into keys_out, segment i at [seg_off[i],
 * seg_end[i]) (seg_end 0: up to seg_off[i + 1]); tmp == 0 asks for the scratch size */
extern "C" int plk_seed_sort(const uint64_t *keys_in, uint64_t *keys_out, int64_t n_items, int32_t n_seg,
		const int64_t *seg_off, const int64_t *seg_end, void *tmp, size_t *tmp_bytes, void *stream)
{
	cudaError_t e = cub::DeviceSegmentedSort::SortKeys(tmp, *tmp_bytes, keys_in, keys_out, n_items, n_seg, seg_off,
			seg_end ? seg_end : seg_off + 1, (cudaStream_t)stream);
	if (tmp) plk_add_launches(1);
	return (int)e;
}
