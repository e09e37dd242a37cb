/*
 * plhmm.c -- host layer of the integer profile DP (the device replacement of
 * hmm-gpu.c; semantics of mp_hmm_dp_score, hmm.c:252-291).
 *
 * Bulk entry points take the profile as plain tables (pl_hmm_profile_create);
 * the reference's entry points (mppriv.h:128-134) take its opaque mp_hmm_t and
 * read the tables through hmm.c's accessors, caching the device copy in the
 * profile's GPU slot (mp_hmm_gpu_slot) until mp_hmm_gpu_release().  Those
 * accessors and the codon tables live in the host program (hmm.c, nasw-tab.c);
 * they are weak references here, so a caller without them (Python, tests) uses
 * the bulk entry points and the reference entry points report "not taken".
 * No CPU fallback: a failed batch returns 0 with the reason in pl_last_error().
 */
#define _POSIX_C_SOURCE 200809L
#include <limits.h>
#include <pthread.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "plhost.h"

struct pl_hmm_profile_s {
	int device;
	plk_hmm_prof_t k;      /* the profile for the paired kernel where it fits that, else for the 32-bit one */
	plk_hmm_prof_t k32;    /* a paired profile for the 32-bit kernel, where that can be the faster one */
	void *dev;             /* their tables, one block */
	uint8_t *codon_dev;    /* codon index -> HMMER column, 20 = no emission (in dev) */
	uint8_t codon[64];     /* the same, on the host */
};

/* Columns a lane (2-8) when the paired 16-bit kernel can take the profile, else 0.  With no
 * transition above 0 a state is at most bound = m * (largest emission); a transition below
 * -(bound + emax + 1) or an emission below -(bound + 1) then sends every state to the DP's
 * clamp at 0 as that floor does, and with 2 * bound + emax + 2 <= 32767 no sum of a state and
 * the two wraps. */
static int pl_hmm_cols(int32_t m, const int16_t *emit, const int16_t *trans, int32_t *t_floor, int32_t *e_floor)
{
	int64_t bound;
	int32_t emax = 0, cols, tiles = (m + PLK_HMM_TILE - 1) / PLK_HMM_TILE;
	size_t x;
	for (x = 0; x < (size_t)m * 20; ++x) if (emit[x] > emax) emax = emit[x];
	for (x = 0; x < (size_t)m * 7; ++x) if (trans[x] > 0) return 0;
	bound = (int64_t)m * emax;
	if (2 * bound + emax + 2 > 32767) return 0;
	*t_floor = -(int32_t)(bound + emax + 1), *e_floor = -(int32_t)(bound + 1);
	cols = plk_hmm_smem_bytes(tiles * PLK_HMM_TILE, 8) > 0 ? (m + 32 * tiles - 1) / (32 * tiles) : 8;
	return cols < 2 ? 2 : cols;
}

/* the 32-bit kernel's tables: column j holds profile position j (the DP's column j+1) */
static void pl_hmm_tables32(int32_t m, int32_t mpad, const int16_t *emit, const int16_t *trans, int16_t *e, int32_t *t)
{
	int32_t j, k;
	for (j = 0; j < m; ++j)
		for (k = 0; k < 20; ++k) e[(size_t)k * mpad + j] = emit[(size_t)j * 20 + k];
	for (k = 0; k < 7; ++k)
		for (j = 0; j < mpad; ++j) t[(size_t)k * mpad + j] = j < m ? trans[(size_t)j * 7 + k] : -(1 << 28);
}

/* With one region a warp on a scheduler of its own, the 32-bit kernel takes 0.11 us a row and tile and
 * the paired one 0.08 to 0.16, by its columns a lane: 2,000 rows of 250 columns 0.23 and 0.32 ms, of
 * 400 0.46 and 0.53, of 300 (five columns a lane) 0.46 and 0.44.  So profiles of more than five columns
 * a lane have both kernels' tables, and scans of at most a region a scheduler take the 32-bit one. */
#define PL_HMM_BOTH 6

PL_EXPORT pl_hmm_profile_t *pl_hmm_profile_create(int32_t device, int32_t m, const int16_t *emit,
		const int16_t *trans, const uint8_t *codon_alpha)
{
	pl_hmm_profile_t *p;
	char *host = 0;
	int32_t mpad, j, k, cols, t_floor = 0, e_floor = 0;
	size_t row, o_t, o_codon, o_e32, o_t32, size;
	if (m <= 0 || !emit || !trans || !codon_alpha) { pl_set_error("pl_hmm_profile_create: empty profile"); return 0; }
	for (k = 0; k < 64; ++k)
		if (codon_alpha[k] > 20) { pl_set_error("codon_alpha[%d] = %d (HMMER columns 0-19, 20 = none)", k, codon_alpha[k]); return 0; }
	mpad = (m + PLK_HMM_TILE - 1) / PLK_HMM_TILE * PLK_HMM_TILE;
	cols = pl_hmm_cols(m, emit, trans, &t_floor, &e_floor);
	/* emissions | transitions | codons, then the 32-bit kernel's of a paired profile */
	row = (size_t)mpad;
	o_t = (cols ? sizeof(uint32_t) : sizeof(int16_t)) * 21 * row, o_codon = o_t + sizeof(int32_t) * 7 * row;
	o_e32 = o_codon + 64, o_t32 = o_e32 + sizeof(int16_t) * 21 * row;
	size = cols >= PL_HMM_BOTH ? o_t32 + sizeof(int32_t) * 7 * row : o_e32;
	p = (pl_hmm_profile_t*)calloc(1, sizeof(*p));
	host = (char*)calloc(size, 1);
	if (!p || !host) { pl_set_error("out of host memory"); goto fail; }
	if (cols == 0) pl_hmm_tables32(m, mpad, emit, trans, (int16_t*)host, (int32_t*)(host + o_t));
	else {
		uint32_t *e = (uint32_t*)host;
		int32_t *t = (int32_t*)(host + o_t);
		const uint32_t none = ((uint32_t)t_floor & 0xffffu) * 0x10001u;
		for (j = 0; j < 7 * mpad; ++j) t[j] = (int32_t)none;
		for (j = 0; j < m; ++j) { /* the slot of column j in the paired kernel's tables */
			const size_t x = (size_t)(j / (32 * cols)) * PLK_HMM_TILE + (size_t)(j % (32 * cols) / cols) * 8 + j % cols;
			for (k = 0; k < 20; ++k) {
				const int32_t v = emit[(size_t)j * 20 + k];
				e[(size_t)k * mpad + x] = (uint32_t)(v < e_floor ? e_floor : v) & 0xffffu;
			}
			for (k = 0; k < 7; ++k) {
				const int32_t v = trans[(size_t)j * 7 + k];
				t[(size_t)k * mpad + x] = (int32_t)(((uint32_t)(v < t_floor ? t_floor : v) & 0xffffu) * 0x10001u);
			}
		}
		if (cols >= PL_HMM_BOTH)
			pl_hmm_tables32(m, mpad, emit, trans, (int16_t*)(host + o_e32), (int32_t*)(host + o_t32));
	}
	memcpy(host + o_codon, codon_alpha, 64);
	memcpy(p->codon, codon_alpha, 64);
	p->device = device, p->k.m = p->k32.m = m, p->k.mpad = p->k32.mpad = mpad, p->k.cols = cols;
	p->k.hi = p->k32.hi = 65536;
	CK(cudaSetDevice(device));
	CK(cudaMalloc(&p->dev, size));
	CK(cudaMemcpy(p->dev, host, size, cudaMemcpyHostToDevice));
	p->k.emit_t = p->dev, p->k.trans_t = (const int32_t*)((char*)p->dev + o_t), p->codon_dev = (uint8_t*)p->dev + o_codon;
	if (cols >= PL_HMM_BOTH)
		p->k32.emit_t = (char*)p->dev + o_e32, p->k32.trans_t = (const int32_t*)((char*)p->dev + o_t32);
	free(host);
	return p;
fail:
	free(host);
	if (p) {
		if (p->dev) cudaFree(p->dev);
		free(p);
	}
	return 0;
}

PL_EXPORT void pl_hmm_profile_destroy(pl_hmm_profile_t *p)
{
	if (!p) return;
	cudaSetDevice(p->device);
	cudaFree(p->dev);
	free(p);
}

void pl_hmm_engine_free(pl_engine_t *e)
{
	dbuf_free(&e->h_off), dbuf_free(&e->h_len), dbuf_free(&e->h_rowoff), dbuf_free(&e->h_rows);
	dbuf_free(&e->h_order), dbuf_free(&e->h_counter), dbuf_free(&e->h_edge), dbuf_free(&e->h_nt);
	dbuf_free(&e->h_score);
	{
		int s;
		for (s = 0; s < PL_HMM_STREAMS; ++s) {
			if (e->h_st[s]) cudaStreamDestroy(e->h_st[s]), e->h_st[s] = 0;
		}
		for (s = 0; s <= PL_HMM_STREAMS; ++s)
			if (e->h_ev[s]) cudaEventDestroy(e->h_ev[s]), e->h_ev[s] = 0;
	}
	free(e->h_hbuf);
	e->h_hbuf = 0, e->h_hcap = 0;
}

/* longest region first; one counting pass over the length (bounded buckets) */
static int pl_hmm_plan(pl_engine_t *e, int32_t n, const int32_t *len, int64_t **row_off, int32_t **order,
		int64_t *rows_total, int32_t *max_rows)
{
	const size_t need = sizeof(int64_t) * (size_t)n + sizeof(int32_t) * (size_t)n + sizeof(int32_t) * 4097;
	int32_t q, *cnt;
	int64_t acc = 0;
	if (need > e->h_hcap) {
		free(e->h_hbuf);
		e->h_hbuf = malloc(need);
		e->h_hcap = e->h_hbuf ? need : 0;
		if (!e->h_hbuf) { pl_set_error("out of host memory"); return 0; }
	}
	*row_off = (int64_t*)e->h_hbuf;
	*order = (int32_t*)(*row_off + n);
	cnt = *order + n;
	memset(cnt, 0, sizeof(int32_t) * 4097);
	*max_rows = 0;
	for (q = 0; q < n; ++q) {
		const int32_t r = len[q] >= 3 ? len[q] / 3 : 0;
		int b;
		if (len[q] < 0) { pl_set_error("region %d: negative length", q); return 0; }
		(*row_off)[q] = acc, acc += (r + 15) / 16 * 16;
		if (r > *max_rows) *max_rows = r;
		b = 4095 - (r >> 4 > 4095 ? 4095 : r >> 4);
		++cnt[b + 1];
	}
	for (q = 0; q < 4096; ++q) cnt[q + 1] += cnt[q];
	for (q = 0; q < n; ++q) {
		const int32_t r = len[q] >= 3 ? len[q] / 3 : 0;
		(*order)[cnt[4095 - (r >> 4 > 4095 ? 4095 : r >> 4)]++] = q;
	}
	*rows_total = acc;
	return 1;
}

/* A profile's launch over n regions, one of n_st side by side: its kernel, and as few warps a CTA as
 * leave one CTA to an SM of its part of the GPU, so that the regions of a small scan spread over the
 * SMs and their schedulers (with eight warps to a CTA whatever their number, 186 regions of 12 kb
 * against 4 profiles of up to 800 columns took 2.1 ms, on 48 SMs; a second CTA on an SM puts two
 * warps on a scheduler where others have none). */
typedef struct { const plk_hmm_prof_t *k; int32_t ctas, warps; } pl_hmm_grid_t;
static int pl_hmm_grid(const pl_engine_t *e, const pl_hmm_profile_t *p, int32_t n, int32_t n_st, pl_hmm_grid_t *g)
{
	const int32_t most = plk_hmm_warps_per_cta(), part = e->n_sm > n_st ? e->n_sm / n_st : 1;
	int32_t units, all;
	g->k = p->k.cols >= PL_HMM_BOTH && n <= 4 * part ? &p->k32 : &p->k;
	units = g->k->cols ? (n + 1) / 2 : n;  /* the paired kernel: two regions a warp */
	all = plk_hmm_ctas_per_sm(g->k);
	if (all < 1) { pl_set_error("HMM DP kernel does not fit on an SM"); return 0; }
	all *= e->n_sm;
	g->warps = units > part * most ? most : (units + part - 1) / part;
	g->ctas = units > (int64_t)all * g->warps ? all : (units + g->warps - 1) / g->warps;
	return 1;
}
/* its edge buffer (columns handed from tile to tile, two rows of 16 bytes a warp, the rows in fours as
 * the paired kernel walks them): none for one tile */
static int64_t pl_hmm_edge_rows(int32_t max_rows) { return ((int64_t)max_rows + 3) / 4 * 4 + 4; }
static size_t pl_hmm_edge_bytes(int32_t max_rows, const pl_hmm_grid_t *g)
{
	if (g->k->mpad <= PLK_HMM_TILE) return 0;
	return (size_t)16 * 2 * (size_t)pl_hmm_edge_rows(max_rows) * (size_t)g->ctas * g->warps;
}

static int pl_hmm_run(pl_engine_t *e, const pl_hmm_profile_t *p, int32_t n, const uint8_t *nt_dev,
		const int32_t *off, const int32_t *len, int32_t *score_dev, cudaStream_t st)
{
	int64_t *row_off, rows_total, cells = 0;
	int32_t *order, max_rows, q;
	pl_hmm_grid_t g;
	if (n <= 0) return 1;
	if (!p) { pl_set_error("no profile"); return 0; }
	if (p->device != e->device) { pl_set_error("profile on device %d, engine on device %d", p->device, e->device); return 0; }
	if (!pl_hmm_plan(e, n, len, &row_off, &order, &rows_total, &max_rows)) return 0;
	for (q = 0; q < n; ++q) cells += (int64_t)(len[q] >= 3 ? len[q] / 3 : 0) * p->k.m;
	if (!pl_hmm_grid(e, p, n, 1, &g)) return 0;
	if (!dbuf_ensure(&e->h_off, sizeof(int32_t) * (size_t)n) || !dbuf_ensure(&e->h_len, sizeof(int32_t) * (size_t)n) ||
			!dbuf_ensure(&e->h_rowoff, sizeof(int64_t) * (size_t)n) || !dbuf_ensure(&e->h_order, sizeof(int32_t) * (size_t)n) ||
			!dbuf_ensure(&e->h_rows, (size_t)(rows_total > 0 ? rows_total : 16)) || !dbuf_ensure(&e->h_counter, 64) ||
			!dbuf_ensure(&e->h_edge, pl_hmm_edge_bytes(max_rows, &g)))
		return 0;
	CK(cudaMemcpyAsync(e->h_off.p, off, sizeof(int32_t) * (size_t)n, cudaMemcpyHostToDevice, st));
	CK(cudaMemcpyAsync(e->h_len.p, len, sizeof(int32_t) * (size_t)n, cudaMemcpyHostToDevice, st));
	CK(cudaMemcpyAsync(e->h_rowoff.p, row_off, sizeof(int64_t) * (size_t)n, cudaMemcpyHostToDevice, st));
	CK(cudaMemcpyAsync(e->h_order.p, order, sizeof(int32_t) * (size_t)n, cudaMemcpyHostToDevice, st));
	e->n_ev = 0;
	PL_TIME(e, st, 0);
	CKK(plk_hmm_codons(nt_dev, (const int32_t*)e->h_off.p, (const int32_t*)e->h_len.p, (const int64_t*)e->h_rowoff.p, n,
			p->codon_dev, (uint8_t*)e->h_rows.p, st));
	PL_TIME(e, st, 0);
	PL_TIME(e, st, 1);
	CKK(plk_hmm_dp(g.k, (const uint8_t*)e->h_rows.p, (const int64_t*)e->h_rowoff.p, (const int32_t*)e->h_len.p,
			(const int32_t*)e->h_order.p, n, (int32_t*)e->h_counter.p, e->h_edge.p, pl_hmm_edge_rows(max_rows), g.ctas, g.warps,
			score_dev, st));
	PL_TIME(e, st, 1);
	CK(cudaStreamSynchronize(st));
	if (e->timing) {
		int k;
		float ms;
		for (k = 0; k + 1 < e->n_ev; k += 2) {
			cudaEventElapsedTime(&ms, e->ev[k], e->ev[k + 1]);
			e->acc_ms[e->ev_kind[k]] += ms;
		}
		e->acc_dp_launches += 1, e->acc_cells += cells;
	}
	e->h_last_cells = cells;
	return 1;
fail:
	return 0;
}

PL_EXPORT int pl_hmm_score_device(pl_engine_t *e, const pl_hmm_profile_t *p, int32_t n, const uint8_t *nt,
		const int32_t *off, const int32_t *len, int32_t *score_dev, void *stream)
{
	if (!e) { pl_set_error("no engine"); return 0; }
	if (cudaSetDevice(e->device) != cudaSuccess) { pl_set_error("cudaSetDevice failed"); return 0; }
	return pl_hmm_run(e, p, n, nt, off, len, score_dev, stream ? (cudaStream_t)stream : e->stream);
}

/* Many profiles against one region set: the planning, the upload of the region tables and
 * the codon translation once (again only when a profile's codon table differs from the
 * previous one's), then one DP launch per profile, round-robin on up to PL_HMM_STREAMS streams
 * with their own queue counters and parts of the edge buffer, so that the launches of a region set
 * too small to fill the GPU run side by side.  All memory is there before the first launch (growing
 * a buffer waits for the launches under way), streams and events as many as there are profiles for. */
PL_EXPORT int pl_hmm_score_many_device(pl_engine_t *e, const pl_hmm_profile_t *const *ps, int32_t n_prof, int32_t n,
		const uint8_t *nt, const int32_t *off, const int32_t *len, int32_t *score_dev, void *stream)
{
	int64_t *row_off, rows_total, cells = 0, rows_sum = 0;
	size_t edge[PL_HMM_STREAMS + 1] = {0};  /* bytes of each stream's part, then where it starts */
	int32_t *order, max_rows, q, k, s;
	pl_hmm_grid_t *g = 0;
	const int32_t n_st = n_prof < PL_HMM_STREAMS ? n_prof : PL_HMM_STREAMS;
	int ok = 0;
	const uint8_t *codon = 0;
	cudaStream_t st;
	if (!e) { pl_set_error("no engine"); return 0; }
	if (n <= 0 || n_prof <= 0) return 1;
	if (!ps || !off || !len || !nt || !score_dev) { pl_set_error("pl_hmm_score_many_device: missing argument"); return 0; }
	for (k = 0; k < n_prof; ++k)
		if (!ps[k] || ps[k]->device != e->device) { pl_set_error("profile %d missing or on another device", k); return 0; }
	CK(cudaSetDevice(e->device));
	st = stream ? (cudaStream_t)stream : e->stream;
	if (!pl_hmm_plan(e, n, len, &row_off, &order, &rows_total, &max_rows)) return 0;
	for (q = 0; q < n; ++q) rows_sum += len[q] >= 3 ? len[q] / 3 : 0;
	g = (pl_hmm_grid_t*)malloc(sizeof(*g) * (size_t)n_prof);
	if (!g) { pl_set_error("out of host memory"); goto fail; }
	for (k = 0; k < n_prof; ++k) {
		size_t b;
		if (!pl_hmm_grid(e, ps[k], n, n_st, &g[k])) goto fail;
		b = pl_hmm_edge_bytes(max_rows, &g[k]);
		if (b > edge[k % PL_HMM_STREAMS + 1]) edge[k % PL_HMM_STREAMS + 1] = b;
	}
	for (s = 0; s < n_st; ++s) edge[s + 1] += edge[s];
	for (s = 0; s < n_st; ++s)
		if (!e->h_st[s]) CK(cudaStreamCreateWithFlags(&e->h_st[s], cudaStreamNonBlocking));
	for (s = 0; s <= PL_HMM_STREAMS; ++s)
		if ((s < n_st || s == PL_HMM_STREAMS) && !e->h_ev[s]) CK(cudaEventCreateWithFlags(&e->h_ev[s], cudaEventDisableTiming));
	if (!dbuf_ensure(&e->h_off, sizeof(int32_t) * (size_t)n) || !dbuf_ensure(&e->h_len, sizeof(int32_t) * (size_t)n) ||
			!dbuf_ensure(&e->h_rowoff, sizeof(int64_t) * (size_t)n) || !dbuf_ensure(&e->h_order, sizeof(int32_t) * (size_t)n) ||
			!dbuf_ensure(&e->h_rows, (size_t)(rows_total > 0 ? rows_total : 16)) ||
			!dbuf_ensure(&e->h_counter, 64 * PL_HMM_STREAMS) || !dbuf_ensure(&e->h_edge, edge[n_st]))
		goto fail;
	CK(cudaMemcpyAsync(e->h_off.p, off, sizeof(int32_t) * (size_t)n, cudaMemcpyHostToDevice, st));
	CK(cudaMemcpyAsync(e->h_len.p, len, sizeof(int32_t) * (size_t)n, cudaMemcpyHostToDevice, st));
	CK(cudaMemcpyAsync(e->h_rowoff.p, row_off, sizeof(int64_t) * (size_t)n, cudaMemcpyHostToDevice, st));
	CK(cudaMemcpyAsync(e->h_order.p, order, sizeof(int32_t) * (size_t)n, cudaMemcpyHostToDevice, st));
	e->n_ev = 0;
	PL_TIME(e, st, 1);
	for (k = 0; k < n_prof; ++k) {
		const pl_hmm_profile_t *p = ps[k];
		cudaStream_t sk;
		if (!codon || memcmp(codon, p->codon, 64) != 0) {  /* the rows of this codon table, then fork again */
			if (codon) {  /* every launch reading the previous rows has finished */
				for (s = 0; s < n_st; ++s) {
					CK(cudaEventRecord(e->h_ev[s], e->h_st[s]));
					CK(cudaStreamWaitEvent(st, e->h_ev[s], 0));
				}
			}
			CKK(plk_hmm_codons(nt, (const int32_t*)e->h_off.p, (const int32_t*)e->h_len.p, (const int64_t*)e->h_rowoff.p,
					n, p->codon_dev, (uint8_t*)e->h_rows.p, st));
			CK(cudaEventRecord(e->h_ev[PL_HMM_STREAMS], st));
			for (s = 0; s < n_st; ++s) CK(cudaStreamWaitEvent(e->h_st[s], e->h_ev[PL_HMM_STREAMS], 0));
			codon = p->codon;
		}
		s = k % PL_HMM_STREAMS, sk = e->h_st[s];
		CKK(plk_hmm_dp(g[k].k, (const uint8_t*)e->h_rows.p, (const int64_t*)e->h_rowoff.p, (const int32_t*)e->h_len.p,
				(const int32_t*)e->h_order.p, n, (int32_t*)e->h_counter.p + 16 * s,
				(char*)e->h_edge.p + edge[s], pl_hmm_edge_rows(max_rows), g[k].ctas, g[k].warps,
				score_dev + (int64_t)k * n, sk));
		cells += rows_sum * p->k.m;
	}
	for (s = 0; s < n_st; ++s) {  /* join */
		CK(cudaEventRecord(e->h_ev[s], e->h_st[s]));
		CK(cudaStreamWaitEvent(st, e->h_ev[s], 0));
	}
	PL_TIME(e, st, 1);
	CK(cudaStreamSynchronize(st));
	if (e->timing) {
		float ms;
		if (e->n_ev >= 2 && cudaEventElapsedTime(&ms, e->ev[0], e->ev[1]) == cudaSuccess) e->acc_ms[1] += ms;
		e->acc_dp_launches += n_prof, e->acc_cells += cells;
	}
	e->h_last_cells = cells;
	ok = 1;
fail:
	free(g);
	return ok;
}

/* pl_hmm_score_many_device from host buffers: the region set uploaded once, the
 * n_prof x n scores copied back. */
PL_EXPORT int pl_hmm_score_many_host(pl_engine_t *e, const pl_hmm_profile_t *const *ps, int32_t n_prof, int32_t n,
		const uint8_t *nt, int64_t l_nt, const int32_t *off, const int32_t *len, int32_t *score)
{
	cudaStream_t st;
	int32_t q;
	if (!e) { pl_set_error("no engine"); return 0; }
	if (n <= 0 || n_prof <= 0) return 1;
	for (q = 0; q < n; ++q)
		if (off[q] < 0 || len[q] < 0 || (int64_t)off[q] + len[q] > l_nt) {
			pl_set_error("region %d [%d, +%d) outside the %lld-byte buffer", q, off[q], len[q], (long long)l_nt);
			return 0;
		}
	st = e->stream;
	CK(cudaSetDevice(e->device));
	if (!dbuf_ensure(&e->h_nt, (size_t)(l_nt > 0 ? l_nt : 1)) ||
			!dbuf_ensure(&e->h_score, sizeof(int32_t) * (size_t)n * (size_t)n_prof))
		return 0;
	if (l_nt > 0) CK(cudaMemcpyAsync(e->h_nt.p, nt, (size_t)l_nt, cudaMemcpyHostToDevice, st));
	if (!pl_hmm_score_many_device(e, ps, n_prof, n, (const uint8_t*)e->h_nt.p, off, len, (int32_t*)e->h_score.p, st))
		return 0;
	CK(cudaMemcpyAsync(score, e->h_score.p, sizeof(int32_t) * (size_t)n * (size_t)n_prof, cudaMemcpyDeviceToHost, st));
	CK(cudaStreamSynchronize(st));
	return 1;
fail:
	return 0;
}

PL_EXPORT int pl_hmm_score_host(pl_engine_t *e, const pl_hmm_profile_t *p, int32_t n, const uint8_t *nt,
		int64_t l_nt, const int32_t *off, const int32_t *len, int32_t *score)
{
	cudaStream_t st;
	int32_t q;
	if (!e) { pl_set_error("no engine"); return 0; }
	if (n <= 0) return 1;
	for (q = 0; q < n; ++q)
		if (off[q] < 0 || len[q] < 0 || (int64_t)off[q] + len[q] > l_nt) {
			pl_set_error("region %d [%d, +%d) outside the %lld-byte buffer", q, off[q], len[q], (long long)l_nt);
			return 0;
		}
	st = e->stream;
	CK(cudaSetDevice(e->device));
	if (!dbuf_ensure(&e->h_nt, (size_t)(l_nt > 0 ? l_nt : 1)) || !dbuf_ensure(&e->h_score, sizeof(int32_t) * (size_t)n)) return 0;
	if (l_nt > 0) CK(cudaMemcpyAsync(e->h_nt.p, nt, (size_t)l_nt, cudaMemcpyHostToDevice, st));
	if (!pl_hmm_run(e, p, n, (const uint8_t*)e->h_nt.p, off, len, (int32_t*)e->h_score.p, st)) return 0;
	CK(cudaMemcpyAsync(score, e->h_score.p, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToHost, st));
	CK(cudaStreamSynchronize(st));
	return 1;
fail:
	return 0;
}

PL_EXPORT int64_t pl_hmm_last_cells(const pl_engine_t *e) { return e ? e->h_last_cells : 0; }

/* ------------------------------------------------------------------ reference entry points (mppriv.h:128-134) */

typedef struct mp_hmm_s mp_hmm_t;
/* provided by the host program's hmm.c and nasw-tab.c */
extern int32_t mp_hmm_length(const mp_hmm_t *h) __attribute__((weak));
extern const int16_t *mp_hmm_emissions(const mp_hmm_t *h) __attribute__((weak));
extern const int16_t *mp_hmm_transitions(const mp_hmm_t *h) __attribute__((weak));
extern void **mp_hmm_gpu_slot(const mp_hmm_t *h, int which) __attribute__((weak));
extern const int8_t *mp_hmm_aa20_to_alpha_table(void) __attribute__((weak));
extern uint8_t ns_tab_codon[64] __attribute__((weak));

static pthread_mutex_t hm_mu = PTHREAD_MUTEX_INITIALIZER;
static pl_engine_t *hm_engine;
static int hm_ready = -1;

static int hm_init(void)
{ /* called with hm_mu held */
	const char *env = getenv("PLGPU_DEVICE");
	int count = 0, dev = env ? atoi(env) : 0;
	if (hm_ready >= 0) return hm_ready;
	hm_ready = 0;
	if (!mp_hmm_length || !mp_hmm_emissions || !mp_hmm_transitions || !mp_hmm_gpu_slot ||
			!mp_hmm_aa20_to_alpha_table || !ns_tab_codon) {
		pl_set_error("the host program provides no hmm.c accessors: use pl_hmm_profile_create");
		return 0;
	}
	if (cudaGetDeviceCount(&count) != cudaSuccess || dev < 0 || dev >= count) { cudaGetLastError(); return 0; }
	hm_engine = pl_engine_create(dev, 0);
	hm_ready = hm_engine != 0;
	return hm_ready;
}

/* the device copy of h's tables, built once and kept in h's GPU slot 0 (called with hm_mu held) */
static pl_hmm_profile_t *hm_profile(const mp_hmm_t *h)
{
	void **slot = mp_hmm_gpu_slot(h, 0);
	uint8_t codon[64];
	const int8_t *alpha;
	int k;
	if (!slot) return 0;
	if (*slot) return (pl_hmm_profile_t*)*slot;
	alpha = mp_hmm_aa20_to_alpha_table();
	for (k = 0; k < 64; ++k) { /* hmm.c:269-270 */
		const int a = ns_tab_codon[k];
		codon[k] = a < 20 && alpha[a] >= 0 ? (uint8_t)alpha[a] : 20;
	}
	*slot = pl_hmm_profile_create(hm_engine->device, mp_hmm_length(h), mp_hmm_emissions(h), mp_hmm_transitions(h), codon);
	return (pl_hmm_profile_t*)*slot;
}

/* mppriv.h:132 -- 1 = every score filled, exactly mp_hmm_dp_score() of each region. */
PL_EXPORT int mp_hmm_dp_score_gpu_batch(const mp_hmm_t *h, int32_t n, const uint8_t *nt, int64_t l_nt,
		const int32_t *off, const int32_t *len, int32_t *score)
{
	pl_hmm_profile_t *p;
	int ok = 0;
	if (!h || n <= 0 || !nt || !off || !len || !score) return 0;
	pthread_mutex_lock(&hm_mu);
	if (hm_init() && mp_hmm_length(h) > 0 && (p = hm_profile(h)) != 0)
		ok = pl_hmm_score_host(hm_engine, p, n, nt, l_nt, off, len, score);
	pthread_mutex_unlock(&hm_mu);
	return ok;
}

/* mppriv.h:129 -- INT32_MIN when not taken (the caller then runs the CPU). */
PL_EXPORT int32_t mp_hmm_dp_score_gpu(const mp_hmm_t *h, const uint8_t *nt, int32_t nlen)
{
	int32_t off = 0, score = INT32_MIN;
	if (nlen < 3) return INT32_MIN;
	return mp_hmm_dp_score_gpu_batch(h, 1, nt, nlen, &off, &nlen, &score) ? score : INT32_MIN;
}

/* mppriv.h:134 -- drop the cached device tables (called from mp_hmm_destroy, hmm.c:207-212). */
PL_EXPORT void mp_hmm_gpu_release(mp_hmm_t *h)
{
	void **slot;
	if (!h || !mp_hmm_gpu_slot) return;
	slot = mp_hmm_gpu_slot(h, 0);
	if (!slot || !*slot) return;
	pthread_mutex_lock(&hm_mu);
	pl_hmm_profile_destroy((pl_hmm_profile_t*)*slot);
	*slot = 0;
	pthread_mutex_unlock(&hm_mu);
}
