/*
 * kma_serve.cu -- the served form (include/kma_serve.h): a host request
 * loop over one device-resident heap.  Each slot owns a CUDA stream and a
 * per-vertex list table; a request runs as a build kernel and a kernel that
 * checks and frees on its slot's stream, so requests admitted at different
 * times overlap on the device.  Admission is FIFO and waits for a free slot and for the
 * heap room its estimate needs (reserved bytes <= limit * heap bytes);
 * completion times come from CUDA events on the device timeline.
 */
#include <string.h>
#include <stdlib.h>
#include <math.h>
#include <chrono>
#include <deque>
#include <thread>
#include <vector>

#include "kma_internal.h"
#include "kma_scratch.h"
#include "kma_serve.h"
#include "kma_structs.cuh"
#include "kma_wl_common.cuh"

#define SV_MAX_SLOTS 64
#define SV_MAX_CHUNKS 16
#define SV_FROM_BITS 12u
#define SV_FROM_COUNT ((1u << SV_FROM_BITS) + 1u)

namespace {

using namespace kma_wl;

struct sv_params {
	uint32_t n;
	uint32_t deg_max;
	uint64_t seed;
	const uint32_t *deg_cdf;  /* [deg_max] cumulative thresholds of 2^32 */
	const uint16_t *deg_from; /* [2^SV_FROM_BITS + 1] see sv_degree */
	const uint32_t *chunks;   /* [nchunks] objects of the k-th page of a list */
	uint32_t nchunks;
	kma_heap *heap;
	kma_clarraylist *lists;   /* [n] */
	unsigned long long *acc;  /* [SV_WORDS], zero before the request */
	unsigned long long *host; /* [SV_WORDS] pinned: where they go at its end */
};

/* a request's counters */
enum { SV_CHECKSUM, SV_EDGES, SV_MALLOCS, SV_FREES, SV_NULLS, SV_BAD, SV_FREE_SB, SV_BLOCKS, SV_WORDS };

/* The first degree whose threshold is not below the draw.  deg_from holds it
 * for the draws 0, 2^20, 2 * 2^20 ... (and deg_max's at the end), so that all
 * but the highest degrees, thousands of which share the last few of these
 * steps, are found in two or three dependent loads; bisection of the whole
 * law takes log2(deg_max), in both kernels (64 requests of 1000 to 1000000
 * vertices, 16 at a time, degrees to 4096: 3450 -> 3383 us). */
__device__ __forceinline__ uint32_t sv_degree(const sv_params &p, uint64_t d)
{
	uint32_t u = (uint32_t)(d >> 32);
	const uint16_t *from = p.deg_from + (u >> (32 - SV_FROM_BITS));
	uint32_t lo = __ldg(&from[0]), hi = __ldg(&from[1]);
	while (lo < hi) {
		uint32_t mid = (lo + hi) >> 1;
		if (u <= __ldg(&p.deg_cdf[mid]))
			hi = mid;
		else
			lo = mid + 1;
	}
	return lo + 1;
}
/* uniform in [0, n) by multiply-shift of the draw's high half */
__device__ __forceinline__ uint32_t sv_neighbour(uint64_t d, uint32_t n)
{
	return (uint32_t)(((d >> 32) * (uint64_t)n) >> 32);
}
__device__ __forceinline__ uint64_t sv_rng0(uint64_t seed, uint32_t v)
{
	return seed ^ ((uint64_t)(v + 1) * 0x9E3779B97F4A7C15ull);
}
__device__ __forceinline__ uint64_t sv_hash_init(uint32_t v, uint32_t d)
{
	return ((uint64_t)(v + 1) * 0xD6E8FEB86659FD93ull) ^ d;
}
__device__ __forceinline__ uint64_t sv_hash_step(uint64_t h, uint32_t nb)
{
	h = (h ^ nb) * 0x9E3779B97F4A7C15ull;
	return h ^ (h >> 29);
}
__device__ __forceinline__ void sv_flush(unsigned long long *acc, int k, unsigned long long v)
{
	for (int d = 16; d > 0; d >>= 1)
		v += __shfl_down_sync(0xffffffffu, v, d);
	if ((threadIdx.x & 31) == 0 && v)
		atomicAdd(&acc[k], v);
}

/* The k-th draw (k >= 0) behind rng state s: what splitmix gives on its
 * k + 1-st call, without the calls before it. */
__device__ __forceinline__ uint64_t sv_draw(uint64_t s, uint32_t k)
{
	s += (uint64_t)k * SPLITMIX_STEP;
	return splitmix(s);
}

/*
 * What bounds a request is its few vertices of high degree (up to deg_max;
 * the others have 3 or 4 neighbours): one thread that draws, stores, loads
 * or hashes 4096 ids one after the other is busy for 0.3 ms while its warp
 * waits.  So
 *   - a page of SV_WARP_IDS ids and more is written by its whole warp (each
 *     id is its own draw, and the stores of a warp are consecutive);
 *   - a vertex of SV_WARP_DEGREE ids and more is checked by its whole warp,
 *     32 ids to a load, the next 32 loaded before this 32 go through the
 *     hash, whose chain of dependent multiplies is then all that is left;
 *   - other vertices are checked by their threads, eight ids to a batch;
 *   - a list is its vertex's thread's alone until the request is done, so it
 *     is linked and walked with plain stores and loads, not with the queue's
 *     atomics.
 * Measured on 64 requests of 1000 to 1000000 vertices (sums over the
 * requests, 16 at a time): build 4.4 ms (10.8 before), check and free 8.5
 * (23.5).
 */
#define SV_WARP_IDS 32u
#define SV_WARP_DEGREE 128u
#define SV_BATCH 8u

/* Neighbours first .. first+n-1 of each calling lane's vertex (rng state
 * behind its degree draw) into o; every lane of the warp calls, n 0: nothing. */
__device__ __forceinline__ void sv_fill(uint32_t *o, uint32_t n, uint32_t first, uint64_t rng, uint32_t verts)
{
	const uint32_t lane = threadIdx.x & 31, full = 0xffffffffu;
	const bool big = n >= SV_WARP_IDS;
	if (!big)
		for (uint32_t j = 0; j < n; j++)
			o[j] = sv_neighbour(sv_draw(rng, first + j), verts);
	for (uint32_t mb = __ballot_sync(full, big); mb; mb &= mb - 1) {
		const uint32_t l = __ffs(mb) - 1;
		uint32_t *ol = (uint32_t *)__shfl_sync(full, (unsigned long long)o, l);
		const uint32_t nl = __shfl_sync(full, n, l), fl = __shfl_sync(full, first, l);
		const uint64_t rl = __shfl_sync(full, rng, l);
		for (uint32_t j = lane; j < nl; j += 32)
			ol[j] = sv_neighbour(sv_draw(rl, fl + j), verts);
	}
}

/* the link of a page (kma_clarraylist's: see clq_link_aligned) */
__device__ __forceinline__ unsigned long long *sv_link(unsigned long long page)
{
	return kma_detail::clq_link_aligned::at(page);
}

/* WARP: the pages of a warp's vertices come from one warp-collaborative
 * heap call per step (kma_malloc_warp); otherwise every vertex's thread
 * calls kma_malloc itself (the reference's per-work-item calls, the
 * denominator the served form is measured against). */
template <bool WARP>
__global__ void __launch_bounds__(1024) k_sv_build(sv_params p)
{
	uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
	bool act = v < p.n;
	uint64_t rng = sv_rng0(p.seed, v);
	const uint64_t dd = splitmix(rng);
	uint32_t deg = act ? sv_degree(p, dd) : 0;
	uint32_t written = 0, page = 0;
	unsigned long long mallocs = 0, nulls = 0, head = 0, tail = 0;
	while (__any_sync(0xffffffffu, written < deg)) {
		uint32_t chunk = 0;
		if (written < deg) {
			chunk = __ldg(&p.chunks[page < p.nchunks ? page : p.nchunks - 1]);
			chunk = chunk < deg - written ? chunk : deg - written;
		}
		/* one warp-collaborative heap call for every lane's page, without the
		 * sweep for scattered slots: most of a request's pages come from
		 * superblocks that nobody has freed into yet, and the registers it
		 * takes cost more than it finds (3383 -> 3270 us) */
		const size_t req = (size_t)chunk * 4 + KMA_AL_PAGE_HDR;
		void *blk = WARP ? kma_malloc_warp_t<false>(p.heap, chunk ? req : ~(size_t)0, nullptr, nullptr)
				 : (chunk ? kma_malloc(p.heap, req) : nullptr);
		if (chunk) {
			mallocs++;
			if (!blk) {
				nulls++;
				chunk = 0;
				deg = written; /* give up on this vertex; verify reports it */
			} else {
				const unsigned long long pg = (unsigned long long)blk;
				*kma_detail::al_page_count(pg) = chunk;
				*sv_link(pg) = 0;
				if (tail)
					*sv_link(tail) = pg;
				else
					head = pg;
				tail = pg;
				page++;
			}
		}
		__syncwarp();
		sv_fill((uint32_t *)((unsigned char *)blk + KMA_AL_PAGE_HDR), chunk, written, rng, p.n);
		written += chunk;
	}
	if (act) {
		kma_clarraylist *l = &p.lists[v];
		kma_clarraylist_init(l, 4, p.heap, KMA_AL_HEAP_KMA);
		l->queue.head = head;
		l->queue.tail = tail;
	}
	sv_flush(p.acc, SV_MALLOCS, mallocs);
	sv_flush(p.acc, SV_NULLS, nulls);
}

/* Check one vertex's list by the whole warp: all lanes call with the same
 * arguments.  Returns its hash; *seen: ids found, *bad: of this lane, those
 * that are not the draws. */
__device__ __forceinline__ uint64_t sv_check_warp(unsigned long long pg, uint32_t deg, uint64_t rng, uint64_t h,
		uint32_t verts, uint32_t *seen, unsigned long long *bad)
{
	const uint32_t lane = threadIdx.x & 31, full = 0xffffffffu;
	uint32_t k = 0;
	while (pg && k < deg) {
		const unsigned long long next = kma_detail::clq_next<kma_detail::clq_link_aligned>(pg);
		const uint32_t c = *kma_detail::al_page_count(pg), m = c < deg - k ? c : deg - k;
		const uint32_t *o = (const uint32_t *)(pg + KMA_AL_PAGE_HDR);
		uint32_t nb = lane < m ? o[lane] : 0u;
		for (uint32_t j = 0; j < m; j += 32) {
			const uint32_t ahead = j + 32 + lane < m ? o[j + 32 + lane] : 0u;
			if (j + lane < m && nb != sv_neighbour(sv_draw(rng, k + j + lane), verts))
				(*bad)++;
			if (j + 32 <= m) {
#pragma unroll
				for (uint32_t i = 0; i < 32; i++)
					h = sv_hash_step(h, __shfl_sync(full, nb, i));
			} else {
				for (uint32_t i = 0; i < m - j; i++)
					h = sv_hash_step(h, __shfl_sync(full, nb, i));
			}
			nb = ahead;
		}
		k += m;
		pg = next;
	}
	*seen = k;
	return h;
}

/* Check every vertex's list and give it back: the request's last kernel.  Its
 * last block hands the request's counters to the host and clears them for
 * the slot's next request, so that neither takes a copy of its own.
 * PER_SM 2: 32 registers a thread, 64 warps an SM, some values spilled.  For
 * requests that fill the GPU at 32 warps an SM by themselves: the more of
 * their pages' round trips are on their way at a time, the better, while
 * smaller ones only pay for the spills (64 requests of 1000 to 1000000
 * vertices, 16 at a time: 3297 us without, 3180 for those above, 3040 for
 * all; 30 requests of at most 400000, 4 at a time: 1785, 1722 and 1847). */
template <bool WARP, int PER_SM>
__global__ void __launch_bounds__(1024, PER_SM) k_sv_finish(sv_params p)
{
	const uint32_t full = 0xffffffffu, lane = threadIdx.x & 31;
	uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
	unsigned long long sum = 0, edges = 0, bad = 0, frees = 0;
	uint64_t rng = 0, h = 0;
	uint32_t deg = 0, seen = 0;
	unsigned long long pg = 0;
	/* the superblocks still free when the request's whole graph is there */
	if (v == 0 && (p.heap->flags & KMA_HEAP_RING))
		p.acc[SV_FREE_SB] = kma_detail::ld_relaxed(&p.heap->ring_avail.v);
	if (v < p.n) {
		rng = sv_rng0(p.seed, v);
		deg = sv_degree(p, splitmix(rng));
		h = sv_hash_init(v, deg);
		pg = kma_detail::qp_ptr(p.lists[v].queue.head);
	}
	for (uint32_t mb = __ballot_sync(full, deg >= SV_WARP_DEGREE); mb; mb &= mb - 1) {
		const uint32_t l = __ffs(mb) - 1;
		uint32_t s;
		const uint64_t x = sv_check_warp(__shfl_sync(full, pg, l), __shfl_sync(full, deg, l),
						 __shfl_sync(full, rng, l), __shfl_sync(full, h, l), p.n, &s, &bad);
		if (lane == l) {
			h = x;
			seen = s;
		}
	}
	const bool check = deg < SV_WARP_DEGREE;
	while (__any_sync(full, pg != 0)) {
		unsigned long long next = 0;
		if (pg) {
			/* the link before the block is given back */
			next = kma_detail::clq_next<kma_detail::clq_link_aligned>(pg);
			const uint32_t c = *kma_detail::al_page_count(pg), left = check ? deg - seen : 0u;
			const uint32_t m = c < left ? c : left;
			const uint32_t *o = (const uint32_t *)(pg + KMA_AL_PAGE_HDR);
			for (uint32_t j = 0; j < m; j += SV_BATCH) {
				uint32_t nb[SV_BATCH];
#pragma unroll
				for (uint32_t i = 0; i < SV_BATCH; i++)
					nb[i] = j + i < m ? o[j + i] : 0u;
#pragma unroll
				for (uint32_t i = 0; i < SV_BATCH; i++)
					if (j + i < m) {
						if (nb[i] != sv_neighbour(sv_draw(rng, seen + j + i), p.n))
							bad++;
						h = sv_hash_step(h, nb[i]);
					}
			}
			seen += m;
			frees++;
		}
		__syncwarp();
		if (WARP)
			kma_free_warp(p.heap, reinterpret_cast<void *>(pg));
		else if (pg)
			kma_free(p.heap, reinterpret_cast<void *>(pg));
		pg = next;
	}
	if (v < p.n) {
		kma_clqueue_init(&p.lists[v].queue);
		if (seen != deg)
			bad++;
		sum = h;
		edges = seen;
	}
	sv_flush(p.acc, SV_CHECKSUM, sum);
	sv_flush(p.acc, SV_EDGES, edges);
	sv_flush(p.acc, SV_BAD, bad);
	sv_flush(p.acc, SV_FREES, frees);
	__shared__ bool last;
	__syncthreads();
	if (threadIdx.x == 0) {
		__threadfence();
		last = atomicAdd(&p.acc[SV_BLOCKS], 1ull) == gridDim.x - 1;
		__threadfence();
	}
	__syncthreads();
	if (last && threadIdx.x < SV_WORDS) {
		const unsigned long long x = atomicExch(&p.acc[threadIdx.x], 0ull);
		if (threadIdx.x != SV_BLOCKS)
			p.host[threadIdx.x] = x;
	}
}

struct sv_slot {
	cudaStream_t st;
	cudaEvent_t end;
	kma_clarraylist *lists;
	unsigned long long *acc;   /* device [SV_WORDS] */
	unsigned long long *host;  /* pinned [SV_WORDS] */
	int req;
	uint64_t reserved;
};

} /* namespace */

struct kma_serve_s {
	kma_heap_s *heap;
	kma_serve_cfg cfg;
	int mode; /* KMA_MODE_WARP (default) or KMA_MODE_PLAIN */
	uint32_t *deg_cdf;
	uint16_t *deg_from;
	uint32_t dense; /* requests of more vertices: k_sv_finish at 64 warps an SM */
	uint32_t *chunks;
	uint32_t nchunks;
	double bytes_per_vertex;
	sv_slot slot[SV_MAX_SLOTS];
	unsigned long long *host_all; /* pinned, SV_WORDS per slot */
};

static void sv_teardown(kma_serve_s *s)
{
	for (uint32_t i = 0; i < s->cfg.slots; i++) {
		sv_slot &sl = s->slot[i];
		if (sl.end)
			cudaEventDestroy(sl.end);
		if (sl.st)
			cudaStreamDestroy(sl.st);
		if (sl.lists)
			cudaFree(sl.lists);
		if (sl.acc)
			cudaFree(sl.acc);
	}
	if (s->host_all)
		cudaFreeHost(s->host_all);
	if (s->deg_cdf)
		cudaFree(s->deg_cdf);
	if (s->deg_from)
		cudaFree(s->deg_from);
	if (s->chunks)
		cudaFree(s->chunks);
	free(s);
}

extern "C" int kma_serve_create(kma_heap_t h, const kma_serve_cfg *cfg, kma_serve_t *out)
{
	if (!out)
		return KMA_EINVAL;
	*out = NULL;
	if (!h || !cfg || cfg->slots == 0 || cfg->slots > SV_MAX_SLOTS || cfg->max_vertices == 0 ||
	    cfg->max_vertices > (1u << 28) || cfg->deg_max == 0 || cfg->deg_max > 65535 || !(cfg->gamma > 1.0f) ||
	    !(cfg->occupancy_limit > 0.0f) || cfg->occupancy_limit > 1.0f)
		return KMA_EINVAL;
	uint32_t bd = cfg->block_dim ? cfg->block_dim : 256;
	if (bd % 32 || bd > 1024)
		return KMA_EINVAL;
	kma_device_guard g(h->device);
	kma_serve_s *s = (kma_serve_s *)calloc(1, sizeof(*s));
	if (!s)
		return KMA_ENOMEM;
	s->heap = h;
	s->mode = KMA_MODE_WARP;
	s->cfg = *cfg;
	s->cfg.block_dim = bd;
	/* pages fill their size class: objects = (class bytes - header) / 4 */
	std::vector<uint32_t> chunks, chunk_bytes;
	for (uint32_t c = 0; c < h->hh.nclasses; c++) {
		uint32_t sz = h->hh.cls_size[c];
		if (sz < KMA_AL_PAGE_HDR + 8 * 4)
			continue;
		chunks.push_back((sz - KMA_AL_PAGE_HDR) / 4);
		chunk_bytes.push_back(sz);
		if (chunks.size() == SV_MAX_CHUNKS)
			break;
	}
	if (chunks.empty()) {
		free(s);
		return KMA_EINVAL;
	}
	s->nchunks = (uint32_t)chunks.size();
	/* degree law and the expected heap bytes of one vertex */
	std::vector<double> pd(cfg->deg_max);
	double tot = 0;
	for (uint32_t d = 1; d <= cfg->deg_max; d++)
		tot += (pd[d - 1] = pow((double)d, -(double)cfg->gamma));
	std::vector<uint32_t> cdf(cfg->deg_max);
	double run = 0, bpv = 0;
	for (uint32_t d = 1; d <= cfg->deg_max; d++) {
		double p = pd[d - 1] / tot;
		run += p;
		double t = run * 4294967296.0;
		cdf[d - 1] = d == cfg->deg_max ? 0xffffffffu : (uint32_t)(t >= 4294967295.0 ? 4294967295.0 : t);
		uint64_t left = d, bytes = 0;
		for (uint32_t k = 0; left; k++) {
			uint32_t i = k < s->nchunks ? k : s->nchunks - 1;
			left -= left < chunks[i] ? left : chunks[i];
			bytes += chunk_bytes[i];
		}
		bpv += p * (double)bytes;
	}
	s->bytes_per_vertex = bpv;
	int sms = 0;
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device);
	s->dense = (uint32_t)sms * 1024u;
	std::vector<uint16_t> from(SV_FROM_COUNT);
	for (uint32_t i = 0, d = 0; i < SV_FROM_COUNT; i++) {
		while (d + 1 < cfg->deg_max && cdf[d] < (uint64_t)i << (32 - SV_FROM_BITS))
			d++;
		from[i] = (uint16_t)d;
	}
	int rc = KMA_OK;
	if (kma_device_malloc((void **)&s->deg_cdf, cfg->deg_max * 4) != cudaSuccess ||
	    kma_device_malloc((void **)&s->deg_from, SV_FROM_COUNT * 2) != cudaSuccess ||
	    kma_device_malloc((void **)&s->chunks, s->nchunks * 4) != cudaSuccess ||
	    cudaMallocHost(&s->host_all, (size_t)cfg->slots * SV_WORDS * 8) != cudaSuccess)
		rc = KMA_ENOMEM;
	if (rc == KMA_OK && (cudaMemcpy(s->deg_cdf, cdf.data(), cfg->deg_max * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
			     cudaMemcpy(s->deg_from, from.data(), SV_FROM_COUNT * 2, cudaMemcpyHostToDevice) != cudaSuccess ||
			     cudaMemcpy(s->chunks, chunks.data(), s->nchunks * 4, cudaMemcpyHostToDevice) != cudaSuccess))
		rc = KMA_ECUDA;
	for (uint32_t i = 0; i < cfg->slots && rc == KMA_OK; i++) {
		sv_slot &sl = s->slot[i];
		sl.req = -1;
		sl.host = s->host_all + SV_WORDS * i;
		if (cudaStreamCreateWithFlags(&sl.st, cudaStreamNonBlocking) != cudaSuccess ||
		    cudaEventCreateWithFlags(&sl.end, cudaEventDefault) != cudaSuccess)
			rc = KMA_ECUDA;
		else if (kma_device_malloc((void **)&sl.lists, (size_t)cfg->max_vertices * sizeof(kma_clarraylist)) != cudaSuccess ||
			 kma_device_malloc((void **)&sl.acc, SV_WORDS * 8) != cudaSuccess)
			rc = KMA_ENOMEM;
		else if (cudaMemset(sl.acc, 0, SV_WORDS * 8) != cudaSuccess)
			rc = KMA_ECUDA;
	}
	if (rc != KMA_OK) {
		cudaGetLastError();
		sv_teardown(s);
		return rc;
	}
	*out = s;
	return KMA_OK;
}

extern "C" int kma_serve_destroy(kma_serve_t s)
{
	if (!s)
		return KMA_EINVAL;
	kma_device_guard g(s->heap->device);
	for (uint32_t i = 0; i < s->cfg.slots; i++)
		cudaStreamSynchronize(s->slot[i].st);
	sv_teardown(s);
	return KMA_OK;
}

extern "C" int kma_serve_set_mode(kma_serve_t s, int mode)
{
	if (!s || (mode != KMA_MODE_WARP && mode != KMA_MODE_PLAIN))
		return KMA_EINVAL;
	s->mode = mode;
	return KMA_OK;
}

extern "C" uint64_t kma_serve_estimate(kma_serve_t s, uint32_t n)
{
	if (!s)
		return 0;
	/* expected bytes plus 10% for the spread of a request's degree draws */
	return (uint64_t)(s->bytes_per_vertex * (double)n * 1.10) + (64u << 10);
}

extern "C" int kma_serve_run(kma_serve_t s, const kma_serve_req *reqs, uint32_t n, int realtime,
		kma_serve_result *res, kma_serve_summary *sum)
{
	if (!s || (n && (!reqs || !res)) || !sum)
		return KMA_EINVAL;
	for (uint32_t i = 1; i < n; i++)
		if (reqs[i].arrival_s < reqs[i - 1].arrival_s)
			return KMA_EINVAL;
	kma_device_guard g(s->heap->device);
	memset(sum, 0, sizeof(*sum));
	memset(res, 0, sizeof(*res) * n);
	uint32_t pages = s->heap->hh.pages;
	uint64_t heap_bytes = s->heap->hh.region_bytes;
	const uint64_t limit = (uint64_t)((double)s->cfg.occupancy_limit * (double)heap_bytes);
	const bool ring = (s->heap->hh.flags & KMA_HEAP_RING) != 0;
	const uint32_t bd = s->cfg.block_dim;
	cudaEvent_t t0ev;
	KMA_CUDA(cudaEventCreate(&t0ev));
	KMA_CUDA(cudaEventRecord(t0ev, s->slot[0].st));
	KMA_CUDA(cudaEventSynchronize(t0ev));
	auto t0 = std::chrono::steady_clock::now();
	auto now_s = [&]() {
		return std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
	};
	std::deque<uint32_t> waiting;
	uint32_t next = 0, done = 0, running = 0;
	uint64_t reserved = 0, max_reserved = 0;
	bool room_wait = false;
	int rc = KMA_OK;
	double last_done = 0;
	while (done < n && rc == KMA_OK) {
		bool progress = false;
		double t = now_s();
		while (next < n && (!realtime || reqs[next].arrival_s <= t))
			waiting.push_back(next++);
		/* completions */
		for (uint32_t i = 0; i < s->cfg.slots; i++) {
			sv_slot &sl = s->slot[i];
			if (sl.req < 0)
				continue;
			cudaError_t q = cudaEventQuery(sl.end);
			if (q == cudaErrorNotReady)
				continue;
			if (q != cudaSuccess) {
				rc = KMA_ECUDA;
				break;
			}
			kma_serve_result &r = res[sl.req];
			float ms = 0;
			cudaEventElapsedTime(&ms, t0ev, sl.end);
			r.done_s = ms / 1e3;
			r.checksum = sl.host[SV_CHECKSUM];
			r.edges = sl.host[SV_EDGES];
			r.mallocs = sl.host[SV_MALLOCS];
			r.frees = sl.host[SV_FREES];
			r.nulls = sl.host[SV_NULLS];
			r.status = r.nulls ? KMA_SERVE_NOMEM : (sl.host[SV_BAD] ? KMA_SERVE_MISMATCH : KMA_SERVE_OK);
			if (ring) {
				const uint32_t free_sb = (uint32_t)sl.host[SV_FREE_SB], in_use = pages - free_sb;
				if (in_use > sum->max_sb_in_use && free_sb <= pages)
					sum->max_sb_in_use = in_use;
			}
			sum->ops += r.mallocs + r.frees;
			last_done = r.done_s > last_done ? r.done_s : last_done;
			reserved -= sl.reserved;
			sl.req = -1;
			running--;
			done++;
			progress = true;
		}
		/* admissions, FIFO */
		while (rc == KMA_OK && !waiting.empty()) {
			uint32_t ri = waiting.front();
			const kma_serve_req &q = reqs[ri];
			uint64_t est = kma_serve_estimate(s, q.n_vertices);
			if (q.n_vertices == 0 || q.n_vertices > s->cfg.max_vertices || est > limit) {
				res[ri].status = KMA_SERVE_TOO_BIG;
				res[ri].admit_s = res[ri].done_s = now_s();
				waiting.pop_front();
				done++;
				progress = true;
				continue;
			}
			int free_slot = -1;
			for (uint32_t i = 0; i < s->cfg.slots; i++)
				if (s->slot[i].req < 0) {
					free_slot = (int)i;
					break;
				}
			if (reserved + est > limit) {
				/* counted once per wait: a slot was free, the room was not */
				if (free_slot >= 0 && !room_wait) {
					sum->admit_waits++;
					room_wait = true;
				}
				break;
			}
			room_wait = false;
			if (free_slot < 0)
				break;
			sv_slot &sl = s->slot[free_slot];
			sv_params p;
			p.n = q.n_vertices;
			p.deg_max = s->cfg.deg_max;
			p.seed = q.seed;
			p.deg_cdf = s->deg_cdf;
			p.deg_from = s->deg_from;
			p.chunks = s->chunks;
			p.nchunks = s->nchunks;
			p.heap = s->heap->dh;
			p.lists = sl.lists;
			p.acc = sl.acc;
			uint32_t blocks = (q.n_vertices + bd - 1) / bd;
			p.host = sl.host;
			if (s->mode == KMA_MODE_WARP) {
				k_sv_build<true><<<blocks, bd, 0, sl.st>>>(p);
				if (q.n_vertices > s->dense)
					k_sv_finish<true, 2><<<blocks, bd, 0, sl.st>>>(p);
				else
					k_sv_finish<true, 1><<<blocks, bd, 0, sl.st>>>(p);
			} else {
				k_sv_build<false><<<blocks, bd, 0, sl.st>>>(p);
				k_sv_finish<false, 1><<<blocks, bd, 0, sl.st>>>(p);
			}
			if (cudaGetLastError() != cudaSuccess || cudaEventRecord(sl.end, sl.st) != cudaSuccess) {
				rc = KMA_ECUDA;
				break;
			}
			sl.req = (int)ri;
			sl.reserved = est;
			reserved += est;
			if (reserved > max_reserved)
				max_reserved = reserved;
			res[ri].admit_s = now_s();
			res[ri].slot = (uint32_t)free_slot;
			res[ri].reserved_bytes = est;
			waiting.pop_front();
			running++;
			if (running > sum->max_running)
				sum->max_running = running;
			progress = true;
		}
		if (!progress) {
			if (running == 0 && waiting.empty() && next < n && realtime) {
				double wait = reqs[next].arrival_s - now_s();
				if (wait > 0)
					std::this_thread::sleep_for(std::chrono::duration<double>(wait < 0.001 ? wait : 0.001));
			} else {
				std::this_thread::sleep_for(std::chrono::microseconds(20));
			}
		}
	}
	for (uint32_t i = 0; i < s->cfg.slots; i++) {
		cudaStreamSynchronize(s->slot[i].st);
		if (rc != KMA_OK) /* a request cut short leaves its counters behind */
			cudaMemset(s->slot[i].acc, 0, SV_WORDS * 8);
	}
	cudaEventDestroy(t0ev);
	double first = n ? (realtime ? reqs[0].arrival_s : 0.0) : 0.0;
	sum->wall_s = last_done > first ? last_done - first : 0.0;
	sum->max_occupancy = pages ? (double)sum->max_sb_in_use / (double)pages : 0.0;
	sum->max_reserved = heap_bytes ? (double)max_reserved / (double)heap_bytes : 0.0;
	return rc;
}
