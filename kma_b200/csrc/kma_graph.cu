/*
 * kma_graph.cu -- the graph-build workload (include/kma_graph.h), after the
 * reference's tree driver (test/tb_clTree.cl:12-85).
 *
 * Build: threads stride over the edges; for each, clGraph_node_ensure both
 * endpoints (tree get; else malloc a node, init its links queue, tree add;
 * free the node again when another thread added the key first) and
 * enqueue a freshly malloc'd link on the source's queue.  Every inserted
 * node and every link is also recorded in a registry array: the teardown
 * frees them from there, and the walk starts in the middle of long queues.
 *
 * Every kernel is a template on the heap backend (kma_backend.cuh), as the
 * reference's driver builds the same tb_clTree.cl over kma.cl or pma.cl
 * (test/tb_clTree.c:441-446, 478-480).
 */
#include <string.h>
#include <stdlib.h>
#include <algorithm>
#include <numeric>
#include <vector>

#include "kma_internal.h"
#include "kma_scratch.h"
#include "kma_graph.h"
#include "kma_structs.h"
#include "kma_structs.cuh"
#include "kma_backend.cuh"
#include "kma_tree_check.cuh"

#define GR_LINK_REQ 16u /* the reference's clGraph_link size */

namespace {

/* 40 bytes, the reference's clGraph_node size (tb_clTree.h) */
struct gr_node {
	kma_clqueue links;
	kma_cltree_node tree;  /* key, state, left, right */
};

/* Where a node sits in its block.  KMA blocks are only 4-byte aligned, so
 * the node goes to align16(block) inside a 52-byte request, the same size
 * class as the reference's 40-byte request; PMA blocks of this build are
 * 8-byte aligned (40- and 16-byte requests from an aligned base), so the
 * node is the block and the request is the reference's own 40 bytes:
 * either way serial builds use the reference's blocks. */
template <class B> struct gr_layout;
template <> struct gr_layout<kma_backend_kma> {
	static constexpr uint32_t node_req = 52, node_align = 16;
};
template <> struct gr_layout<kma_backend_pma> {
	static constexpr uint32_t node_req = 40, node_align = 8;
};

__host__ __device__ __forceinline__ uint64_t gr_mix(uint32_t a, uint32_t b)
{
	uint64_t z = ((uint64_t)a << 32 | b) + 0x9E3779B97F4A7C15ull;
	z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
	z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
	return z ^ (z >> 31);
}

__device__ __forceinline__ gr_node *gr_of_tree(kma_cltree_node *t)
{
	return reinterpret_cast<gr_node *>(reinterpret_cast<unsigned char *>(t) - offsetof(gr_node, tree));
}

template <class B>
struct gr_dev {
	typename B::heap *h;
	kma_cltree *tree;
	gr_node **reg;               /* [cap] inserted nodes */
	unsigned long long *link;    /* [n] edge i's link item, 0 when it has none */
	unsigned long long *nreg;
	unsigned long long *acc;     /* lost_adds, nulls */
	uint32_t *qerr;
};

/* The rest of clGraph_node_ensure (tb_clTree.cl:12-38) for a key that was not
 * in the tree when looked up; NULL when the heap is out of blocks (the
 * reference retries forever there) */
template <class B>
__device__ gr_node *gr_insert(const gr_dev<B> &g, uint32_t key, unsigned long long &lost, unsigned long long &nulls)
{
	for (int tries = 0; tries < 1 << 20; tries++) {
		void *b = B::alloc(g.h, gr_layout<B>::node_req);
		if (!b) {
			nulls++;
			return nullptr;
		}
		const uintptr_t al = gr_layout<B>::node_align - 1;
		gr_node *n = reinterpret_cast<gr_node *>(((uintptr_t)b + al) & ~al);
		n->tree.key = key;
		kma_clqueue_init(&n->links);
		if (kma_cltree_add(g.tree, &n->tree) == KMA_TREE_INSERTED) {
			unsigned long long i = atomicAdd(g.nreg, 1ull);
			g.reg[i] = n;
			return n;
		}
		B::release(g.h, b);
		lost++;
		kma_cltree_node *t = kma_cltree_get(g.tree, key);
		if (t)
			return gr_of_tree(t);
	}
	atomicOr(g.qerr, KMA_ERR_TIMEOUT);
	return nullptr;
}

/* An edge's two ends, looked up side by side: a search is one round trip a
 * level and nothing else, so two cost what the deeper one does. */
__device__ __forceinline__ void gr_find_both(kma_cltree *tree, uint32_t a, uint32_t b, gr_node **na, gr_node **nb)
{
	using namespace kma_detail;
	const unsigned long long root = ld_relaxed64(&tree->root);
	unsigned long long *la = &tree->root, *lb = &tree->root;
	unsigned long long ca = root, cb = root;
	bool fa = false, fb = false;
	while ((ca && !fa) || (cb && !fb)) {
		kma_cltree_node *xa = reinterpret_cast<kma_cltree_node *>(ca), *xb = reinterpret_cast<kma_cltree_node *>(cb);
		const bool ga = ca && !fa, gb = cb && !fb;
		/* a search that has ended reads the other's node again */
		const tree_step sa(ga ? xa : xb), sb(gb ? xb : xa);
		if (ga) {
			if (sa.key == a) {
				fa = true;
			} else {
				la = a < sa.key ? &xa->left : &xa->right;
				ca = a < sa.key ? sa.left : sa.right;
			}
		}
		if (gb) {
			if (sb.key == b) {
				fb = true;
			} else {
				lb = b < sb.key ? &xb->left : &xb->right;
				cb = b < sb.key ? sb.left : sb.right;
			}
		}
	}
	/* as kma_cltree_get: the links again, by acquire loads */
	if (fa)
		ld_acquire64(la);
	if (fb)
		ld_acquire64(lb);
	*na = fa ? gr_of_tree(reinterpret_cast<kma_cltree_node *>(ca)) : nullptr;
	*nb = fb ? gr_of_tree(reinterpret_cast<kma_cltree_node *>(cb)) : nullptr;
}

/* clTree_test (tb_clTree.cl:40-85).  At most 64 registers a thread: a search
 * is bound by its round trips, so the more warps an SM holds the better (2^22
 * uniform edges by 1024 threads an SM: 7.2 ms, 8.9 at 72 registers, where a
 * quarter of them waits for the others to end). */
template <class B>
__global__ void __launch_bounds__(256, 4) k_gr_build(gr_dev<B> g, const uint32_t *edges, uint64_t n)
{
	uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
	unsigned long long lost = 0, nulls = 0;
	for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
		const uint32_t from = edges[2 * i], to = edges[2 * i + 1];
		gr_node *src, *snk;
		gr_find_both(g.tree, from, to, &src, &snk);
		if (!src) {
			src = gr_insert(g, from, lost, nulls);
			if (from == to)
				snk = src;
		}
		if (!snk && (src || from != to))
			snk = gr_insert(g, to, lost, nulls);
		void *b = src && snk ? B::alloc(g.h, GR_LINK_REQ) : nullptr;
		if (!b) {
			nulls += src && snk;
			g.link[i] = 0;
			continue;
		}
		unsigned char *item = reinterpret_cast<unsigned char *>(((uintptr_t)b + 7) & ~(uintptr_t)7);
		g.link[i] = (unsigned long long)item;
		*reinterpret_cast<uint32_t *>(item + 8) = (uint32_t)(((unsigned char *)snk - B::base(g.h)) >> 3);
		/* (the append's exchange publishes the sink too) */
		kma_clqueue_enqueue(&src->links, reinterpret_cast<kma_clqueue_item *>(item), g.qerr);
	}
	if (lost)
		atomicAdd(&g.acc[0], lost);
	if (nulls)
		atomicAdd(&g.acc[1], nulls);
}

/*
 * The walk of every node's queue.  A queue is a linked list, one dependent
 * load per link, and with skewed edges one queue holds a large share of all
 * links: one thread per node took 30 ms for 2^20 Zipf(1.1) edges, all but a
 * little of it on the hottest node.  So the lists are cut (Helman and JaJa's
 * list ranking): every link whose address hashes to 0 mod GR_SPACING starts a
 * segment, and its thread walks to the next such link or the queue's end,
 * some GR_SPACING * ln(segments) links at most.  Pointer jumping then gives
 * every segment the totals from itself to the end of its queue (a chain of
 * the segments, 600 for the hottest node at a spacing of 128, was 1 of the
 * walk's 1.6 ms; now 0.4 in all), and a node's thread walks to its first
 * segment and adds those.
 *
 * While the walk runs, a segment's first link holds the segment's number in
 * place of its sink, which the segment keeps.
 */
struct gr_seg {
	unsigned long long item; /* its first link */
	uint32_t sink8;          /* that link's sink, as a link holds it */
	uint32_t key;            /* the source of that link's edge */
	unsigned long long end;  /* last segment of a queue: where the queue's
				    sinks end, ~0 when no node leads to it */
};
/* From a segment on: over the segments up to `next` (not included), `last`
 * being the one before; next GR_NO_SEG: to the end of the queue. */
struct gr_jump {
	uint32_t next, last, len, pad;
	unsigned long long x, s; /* edge hashes */
};
#define GR_NO_SEG 0xffffffffu
#define GR_SPACING 32u

struct gr_cut {
	gr_seg *seg;
	gr_jump *jump[2];   /* [cap] each; k_gr_jump leaves its result in jump[0] */
	unsigned int *nseg; /* may count past cap: the links past it stay ordinary */
	uint32_t cap;
	uint32_t n;         /* no queue is longer */
};

__device__ __forceinline__ uint32_t *gr_sink_word(unsigned long long item)
{
	return reinterpret_cast<uint32_t *>(item + 8);
}

__device__ __forceinline__ bool gr_hits(unsigned long long item)
{
	return (uint32_t)((item >> 3) * 0x9E3779B97F4A7C15ull >> 32) % GR_SPACING == 0;
}

/* The segment that starts at `item` (whose sink word is w), or GR_NO_SEG.
 * Only the segment's own record decides: w is a sink, and may be any number,
 * in a link that hits but found the records full. */
__device__ __forceinline__ uint32_t gr_seg_at(const gr_cut &c, uint32_t nseg, unsigned long long item, uint32_t w)
{
	return gr_hits(item) && w < nseg && c.seg[w].item == item ? w : GR_NO_SEG;
}
__device__ __forceinline__ uint32_t gr_nseg(const gr_cut &c)
{
	const uint32_t m = *c.nseg;
	return m < c.cap ? m : c.cap;
}

template <class B>
__global__ void k_gr_cut(gr_dev<B> g, const uint32_t *edges, uint64_t n, gr_cut c)
{
	const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
	for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
		const unsigned long long item = g.link[i];
		if (!item || !gr_hits(item))
			continue;
		const uint32_t s = atomicAdd(c.nseg, 1u);
		if (s >= c.cap)
			continue;
		gr_seg &r = c.seg[s];
		r.item = item;
		r.sink8 = *gr_sink_word(item);
		r.key = edges[2 * i];
		r.end = ~0ull;
		*gr_sink_word(item) = s;
	}
}

/* Put the sinks back into the segments' first links. */
__global__ void k_gr_uncut(gr_cut c)
{
	const uint32_t nseg = gr_nseg(c), stride = gridDim.x * blockDim.x;
	for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < nseg; s += stride)
		*gr_sink_word(c.seg[s].item) = c.seg[s].sink8;
}

template <class B>
__device__ __forceinline__ uint32_t gr_key_at(const gr_dev<B> &g, uint32_t off8)
{
	return reinterpret_cast<const gr_node *>(B::base(g.h) + ((size_t)off8 << 3))->tree.key;
}

/* Walk from `item` (0: nothing) to the next segment or the end of the queue;
 * first: item's own sink, when item starts a segment.  Visits the sink keys
 * in order; returns how many, *next: the segment it ended at.  A sink's key
 * is handed on one step late, so that its load runs beside the next link's. */
template <class B, class F>
__device__ __forceinline__ uint32_t gr_run(const gr_dev<B> &g, const gr_cut &c, uint32_t nseg, unsigned long long item,
		bool starts, uint32_t first, uint32_t *next, F visit)
{
	uint32_t len = 0, key = 0;
	*next = GR_NO_SEG;
	while (item && len < c.n) {
		uint32_t w = *gr_sink_word(item);
		const unsigned long long after = kma_detail::clq_next<kma_detail::clq_link_head>(item);
		if (starts && len == 0) {
			w = first;
		} else {
			const uint32_t s = gr_seg_at(c, nseg, item, w);
			if (s != GR_NO_SEG) {
				*next = s;
				break;
			}
		}
		const uint32_t k = gr_key_at(g, w);
		if (len)
			visit(len - 1, key);
		key = k;
		len++;
		item = after;
	}
	if (len)
		visit(len - 1, key);
	return len;
}

/* every segment's length and edge hashes */
template <class B>
__global__ void k_gr_walk_segs(gr_dev<B> g, gr_cut c)
{
	const uint32_t nseg = gr_nseg(c), stride = gridDim.x * blockDim.x;
	for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nseg; i += stride) {
		const gr_seg &r = c.seg[i];
		gr_jump j;
		j.x = j.s = 0;
		const uint32_t key = r.key;
		j.len = gr_run(g, c, nseg, r.item, true, r.sink8, &j.next, [&](uint32_t, uint32_t sk) {
			const uint64_t m = gr_mix(key, sk);
			j.x ^= m;
			j.s += m;
		});
		/* a segment of another source's edges is a link on the wrong queue:
		 * it is not counted, nor is anything behind it */
		if (j.next != GR_NO_SEG && c.seg[j.next].key != key)
			j.next = GR_NO_SEG;
		j.last = i;
		j.pad = 0;
		c.jump[0][i] = j;
	}
}

/* one round of pointer jumping */
__global__ void k_gr_jump(const gr_jump *in, gr_jump *out, gr_cut c)
{
	const uint32_t nseg = gr_nseg(c), stride = gridDim.x * blockDim.x;
	for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nseg; i += stride) {
		gr_jump a = in[i];
		if (a.next != GR_NO_SEG) {
			const gr_jump b = in[a.next];
			a.next = b.next;
			a.last = b.last;
			a.len += b.len;
			a.x ^= b.x;
			a.s += b.s;
		}
		out[i] = a;
	}
}

/* per node: its links in queue order -> count and edge hashes.  start (second
 * pass of an export): the node's place among the sinks, whose end goes to
 * its queue's last segment. */
template <class B>
__global__ void k_gr_walk(gr_dev<B> g, uint64_t nodes, gr_cut c, unsigned long long *counts, const uint64_t *start,
		unsigned long long *sums /* links, xor, sum */)
{
	const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	unsigned long long n = 0, x = 0, s = 0;
	if (i < nodes) {
		const gr_node *nd = g.reg[i];
		const uint32_t key = nd->tree.key, nseg = gr_nseg(c);
		uint32_t next;
		n = gr_run(g, c, nseg, (unsigned long long)kma_clqueue_first(&nd->links), false, 0, &next,
			   [&](uint32_t, uint32_t sk) {
				   const uint64_t m = gr_mix(key, sk);
				   x ^= m;
				   s += m;
			   });
		if (next != GR_NO_SEG && c.seg[next].key == key) {
			const gr_jump j = c.jump[0][next];
			n += j.len;
			x ^= j.x;
			s += j.s;
			if (start)
				c.seg[j.last].end = start[i] + n;
		}
		if (counts)
			counts[i] = n;
	}
	if (start)
		return;
	/* a warp's in one: every node's own, on three words, took 0.4 ms */
	for (int d = 16; d > 0; d >>= 1) {
		n += __shfl_down_sync(0xffffffffu, n, d);
		x ^= __shfl_down_sync(0xffffffffu, x, d);
		s += __shfl_down_sync(0xffffffffu, s, d);
	}
	if ((threadIdx.x & 31) == 0 && n) {
		atomicAdd(&sums[0], n);
		atomicXor(&sums[1], x);
		atomicAdd(&sums[2], s);
	}
}

/* every node's sinks, in queue order: from its head to its first segment,
 * and every segment at its place */
template <class B>
__global__ void k_gr_sinks(gr_dev<B> g, uint64_t nodes, gr_cut c, const uint64_t *start, uint32_t *sinks)
{
	const uint32_t nseg = gr_nseg(c);
	const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
	for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nodes + nseg; i += stride) {
		const bool seg = i >= nodes;
		const gr_seg *r = &c.seg[seg ? i - nodes : 0];
		unsigned long long pos;
		if (seg) {
			const gr_jump &j = c.jump[0][i - nodes];
			pos = c.seg[j.last].end;
			if (pos == ~0ull)
				continue;
			pos -= j.len;
		} else {
			pos = start[i];
		}
		uint32_t next;
		gr_run(g, c, nseg, seg ? r->item : (unsigned long long)kma_clqueue_first(&g.reg[i]->links), seg,
		       seg ? r->sink8 : 0u, &next, [&](uint32_t k, uint32_t sk) { sinks[pos + k] = sk; });
	}
}

/* offset of the block that holds node nd (PMA: of the node itself, its
 * blocks have no recorded start) */
__device__ __forceinline__ long long gr_block_off(kma_heap *h, const gr_node *nd)
{
	return (long long)((const unsigned char *)kma_block_of(h, nd) - h->sb_base);
}
__device__ __forceinline__ long long gr_block_off(kma_pma *p, const gr_node *nd)
{
	return (long long)((const unsigned char *)nd - p->base);
}

template <class B>
__global__ void k_gr_export(gr_dev<B> g, uint64_t nodes, uint32_t *keys, long long *offs)
{
	uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= nodes)
		return;
	const gr_node *nd = g.reg[i];
	keys[i] = nd->tree.key;
	offs[i] = gr_block_off(g.h, nd);
}

/* teardown: every link and every node is freed, from the registries: the
 * hottest queue emptied by its node's thread, one dequeue after the other,
 * took 480 ms of a 2^20-edge Zipf(1.1) graph.  Neighbouring edges' links come
 * from the same superblocks, so the warp form frees a warp's with a few
 * atomics: 0.05 ms. */
template <class B>
__global__ void k_gr_free(gr_dev<B> g, uint64_t nodes, uint64_t n)
{
	if constexpr (B::id == KMA_BACKEND_ID_KMA) {
		const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
		/* all lanes of a warp call every time, together */
		for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < n + nodes; base += stride) {
			const uint64_t i = base + threadIdx.x;
			void *b = B::block(g.h, i < n ? reinterpret_cast<void *>(g.link[i])
						      : i < n + nodes ? g.reg[i - n] : nullptr);
			__syncwarp();
			B::free_block_warp(g.h, b);
		}
	}
}

} /* namespace */

extern "C" uint64_t kma_graph_edge_mix(uint32_t source, uint32_t sink) { return gr_mix(source, sink); }

namespace {
/* The build on heap dh (device header) of either backend; region_bytes:
 * the heap's data bytes (sink offsets are 32-bit multiples of 8 bytes). */
template <class B>
int graph_build(typename B::heap *dh, int device, uint64_t region_bytes, const uint32_t *edges, uint64_t n,
		uint32_t threads, int free_after, kma_graph_stats *st, uint32_t *keys_out, int64_t *node_off,
		uint32_t *link_sinks, uint64_t *link_start)
{
	if (!dh || !edges || !st || n == 0 || n > (1ull << 30) || threads == 0)
		return KMA_EINVAL;
	if (region_bytes > (1ull << 35))
		return KMA_EINVAL;
	if (keys_out && (!node_off || !link_sinks || !link_start))
		return KMA_EINVAL;
	kma_device_guard gd(device);
	memset(st, 0, sizeof(*st));
	uint64_t cap = 2 * n;
	/* segments of the walk: records for twice as many as the hash should give */
	const uint32_t segs = (uint32_t)(2 * n / GR_SPACING) + 1024;
	size_t o_tree = 0, o_reg = 256, o_nreg = o_reg + cap * 8, o_acc = o_nreg + 8, o_err = o_acc + 16,
	       o_sums = (o_err + 8 + 255) & ~(size_t)255, o_nseg = o_sums + 24, o_tc = o_sums + 64, o_cnt = o_tc + 128, o_start = o_cnt + cap * 8,
	       o_sinks = o_start + (cap + 1) * 8, o_keys = o_sinks + n * 4, o_offs = (o_keys + cap * 4 + 7) & ~(size_t)7,
	       o_edges = o_offs + cap * 8, o_link = o_edges + n * 8, o_seg = o_link + n * 8,
	       o_jump = o_seg + (size_t)segs * sizeof(gr_seg), total = o_jump + 2 * (size_t)segs * sizeof(gr_jump);
	/* the tree check's work list (16 bytes a node, at most cap nodes) lies over
	 * the export arrays, which are written after it (44 n + 8 bytes, of which
	 * it needs 16 cap = 32 n behind a 16-byte boundary) */
	const size_t o_list = (o_start + 15) & ~(size_t)15;
	kma_dev_bufs bufs;
	unsigned char *m = bufs.alloc<unsigned char>(total);
	if (!m)
		return KMA_ENOMEM;
	int rc = KMA_OK;
	gr_dev<B> g;
	g.h = dh;
	g.tree = (kma_cltree *)(m + o_tree);
	g.reg = (gr_node **)(m + o_reg);
	g.link = (unsigned long long *)(m + o_link);
	g.nreg = (unsigned long long *)(m + o_nreg);
	g.acc = (unsigned long long *)(m + o_acc);
	g.qerr = (uint32_t *)(m + o_err);
	unsigned long long *sums = (unsigned long long *)(m + o_sums);
	gr_jump *jump = (gr_jump *)(m + o_jump);
	const gr_cut cut = {(gr_seg *)(m + o_seg), {jump, jump + segs}, (unsigned int *)(m + o_nseg), segs, (uint32_t)n};
	if (cudaMemset(m, 0, o_reg) != cudaSuccess || cudaMemset(m + o_nreg, 0, o_cnt - o_nreg) != cudaSuccess ||
	    cudaMemcpy(m + o_edges, edges, n * 8, cudaMemcpyHostToDevice) != cudaSuccess)
		rc = KMA_ECUDA;
	cudaEvent_t e0, e1;
	cudaEventCreate(&e0);
	cudaEventCreate(&e1);
	if (rc == KMA_OK) {
		uint32_t bd = threads < 256 ? threads : 256;
		uint32_t nb = (threads + bd - 1) / bd;
		cudaEventRecord(e0);
		k_gr_build<B><<<nb, bd>>>(g, (const uint32_t *)(m + o_edges), n);
		cudaEventRecord(e1);
		if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess)
			rc = KMA_ECUDA;
		cudaEventElapsedTime(&st->build_ms, e0, e1);
	}
	unsigned long long nodes = 0, acc[2] = {0, 0};
	uint32_t qerr = 0;
	if (rc == KMA_OK && (cudaMemcpy(&nodes, g.nreg, 8, cudaMemcpyDeviceToHost) != cudaSuccess ||
			     cudaMemcpy(acc, g.acc, 16, cudaMemcpyDeviceToHost) != cudaSuccess))
		rc = KMA_ECUDA;
	uint32_t gb = (uint32_t)((nodes + 255) / 256);
	/* grids of the kernels that stride over the edges, or over the segments */
	const uint64_t most = 148 * 8;
	const uint32_t eb = (uint32_t)std::min<uint64_t>((n + nodes + 255) / 256, most);
	const uint32_t sb = (uint32_t)std::min<uint64_t>((segs + 255) / 256, most);
	if (rc == KMA_OK && nodes) {
		unsigned long long *cnt = (unsigned long long *)(m + o_cnt);
		k_gr_cut<B><<<eb, 256>>>(g, (const uint32_t *)(m + o_edges), n, cut);
		k_gr_walk_segs<B><<<sb, 256>>>(g, cut);
		/* an even number of rounds, 2^rounds segments at least */
		for (uint32_t r = 0; r == 0 || (1ull << r) < segs; r += 2) {
			k_gr_jump<<<sb, 256>>>(cut.jump[0], cut.jump[1], cut);
			k_gr_jump<<<sb, 256>>>(cut.jump[1], cut.jump[0], cut);
		}
		k_gr_walk<B><<<gb, 256>>>(g, nodes, cut, keys_out ? cnt : NULL, NULL, sums);
		if (cudaGetLastError() != cudaSuccess)
			rc = KMA_ECUDA;
		unsigned long long *tc = (unsigned long long *)(m + o_tc);
		if (rc == KMA_OK)
			rc = tree_check(g.tree, m + o_list, nodes, tc, device, NULL);
		if (rc == KMA_OK && cudaDeviceSynchronize() != cudaSuccess)
			rc = KMA_ECUDA;
		unsigned long long sm[3], tcw[KMA_TC_WORDS];
		if (rc == KMA_OK && (cudaMemcpy(sm, sums, sizeof(sm), cudaMemcpyDeviceToHost) != cudaSuccess ||
				     cudaMemcpy(tcw, tc, sizeof(tcw), cudaMemcpyDeviceToHost) != cudaSuccess))
			rc = KMA_ECUDA;
		if (rc == KMA_OK) {
			st->links = sm[0];
			st->edge_xor = sm[1];
			st->edge_sum = sm[2];
			st->sorted = tcw[KMA_TC_UNSORTED] == 0 && tcw[KMA_TC_OVERFLOW] == 0;
		}
		if (rc == KMA_OK && keys_out) {
			/* export: nodes in key order, links in queue order */
			std::vector<unsigned long long> c(nodes);
			std::vector<uint32_t> k(nodes);
			std::vector<long long> o(nodes);
			k_gr_export<B><<<gb, 256>>>(g, nodes, (uint32_t *)(m + o_keys), (long long *)(m + o_offs));
			if (cudaDeviceSynchronize() != cudaSuccess ||
			    cudaMemcpy(c.data(), cnt, nodes * 8, cudaMemcpyDeviceToHost) != cudaSuccess ||
			    cudaMemcpy(k.data(), m + o_keys, nodes * 4, cudaMemcpyDeviceToHost) != cudaSuccess ||
			    cudaMemcpy(o.data(), m + o_offs, nodes * 8, cudaMemcpyDeviceToHost) != cudaSuccess)
				rc = KMA_ECUDA;
			std::vector<uint64_t> start(nodes + 1, 0);
			for (uint64_t i = 0; i < nodes; i++)
				start[i + 1] = start[i] + c[i];
			if (rc == KMA_OK && start[nodes] <= n) {
				if (cudaMemcpy(m + o_start, start.data(), (nodes + 1) * 8, cudaMemcpyHostToDevice) != cudaSuccess)
					rc = KMA_ECUDA;
				const uint64_t *dstart = (const uint64_t *)(m + o_start);
				k_gr_walk<B><<<gb, 256>>>(g, nodes, cut, NULL, dstart, sums);
				k_gr_sinks<B><<<eb, 256>>>(g, nodes, cut, dstart, (uint32_t *)(m + o_sinks));
				std::vector<uint32_t> sk(start[nodes] ? start[nodes] : 1);
				if (rc == KMA_OK && (cudaDeviceSynchronize() != cudaSuccess ||
						     cudaMemcpy(sk.data(), m + o_sinks, start[nodes] * 4,
								cudaMemcpyDeviceToHost) != cudaSuccess))
					rc = KMA_ECUDA;
				if (rc == KMA_OK) {
					std::vector<uint64_t> ord(nodes);
					std::iota(ord.begin(), ord.end(), 0);
					std::sort(ord.begin(), ord.end(), [&](uint64_t a, uint64_t b) { return k[a] < k[b]; });
					uint64_t pos = 0;
					for (uint64_t j = 0; j < nodes; j++) {
						uint64_t i = ord[j];
						keys_out[j] = k[i];
						node_off[j] = o[i];
						link_start[j] = pos;
						for (uint64_t q = start[i]; q < start[i + 1]; q++)
							link_sinks[pos++] = sk[q];
					}
					link_start[nodes] = pos;
				}
			} else if (rc == KMA_OK) {
				rc = KMA_EFAULT;
			}
		}
	}
	if (rc == KMA_OK && !free_after && nodes) {
		/* the graph stays in the heap as it was built */
		k_gr_uncut<<<sb, 256>>>(cut);
		if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess)
			rc = KMA_ECUDA;
	}
	if (rc == KMA_OK && free_after && nodes) {
		k_gr_free<B><<<eb, 256>>>(g, nodes, n);
		if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess)
			rc = KMA_ECUDA;
	}
	if (rc == KMA_OK)
		cudaMemcpy(&qerr, g.qerr, 4, cudaMemcpyDeviceToHost);
	st->nodes = nodes;
	st->lost_adds = acc[0];
	st->nulls = acc[1];
	st->err = qerr;
	cudaEventDestroy(e0);
	cudaEventDestroy(e1);
	return rc;
}
} /* namespace */

extern "C" int kma_graph_build(kma_heap_t h, const uint32_t *edges, uint64_t n, uint32_t threads, int free_after,
		kma_graph_stats *st, uint32_t *keys_out, int64_t *node_off, uint32_t *link_sinks,
		uint64_t *link_start)
{
	if (!h)
		return KMA_EINVAL;
	return graph_build<kma_backend_kma>(h->dh, h->device, h->hh.region_bytes, edges, n, threads, free_after, st,
					    keys_out, node_off, link_sinks, link_start);
}

extern "C" int kma_graph_build_pma(kma_pma_t p, const uint32_t *edges, uint64_t n, uint32_t threads,
		kma_graph_stats *st, uint32_t *keys_out, int64_t *node_off, uint32_t *link_sinks,
		uint64_t *link_start)
{
	if (!p)
		return KMA_EINVAL;
	return graph_build<kma_backend_pma>(p->dp, p->device, p->bytes, edges, n, threads, 0, st, keys_out, node_off,
					    link_sinks, link_start);
}
