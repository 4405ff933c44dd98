/*
 * kma_device.cuh -- device-side API of the B200 KMA heap (sm_100a).
 *
 * Drop-in for the reference's device API (clheap.h:37-39, kma.cl:279-373):
 *   void *kma_malloc(kma_heap *heap, size_t size);   NULL on failure
 *   void  kma_free(kma_heap *heap, void *p);         kma_free(h, NULL) is a no-op
 * plus warp-collaborative forms (any subset of a warp may call them, with
 * different sizes per lane):
 *   void *kma_malloc_warp(kma_heap *heap, size_t size);
 *   void  kma_free_warp(kma_heap *heap, void *p);
 * The lock-free structures (clqueue, clindexedqueue, cltree, clarraylist)
 * and the PMA bump heap are in kma_structs.cuh.
 *
 * Heap layout in HBM (one cudaMalloc per heap, owned by kma_create):
 *   [kma_heap header | sb_state[nsb] u32 | sb_home[nsb] u16 |
 *    free-list words | superblocks]
 *   Superblock s lives at sb_base + s*SB: bytes [0,12) are reserved so that
 *   every block offset equals the reference's (its in-band 12-byte header,
 *   kma.h:71-78); blocks start at +12; the allocation bitmap sits at the
 *   tail and grows downward (bitmap word k = slots 32k..32k+31 at u32 index
 *   SB/4-1-k, kma.cl:183-188).  The header fields live in coalesced side
 *   arrays: sb_state[s] = class<<28 | slots<<14 | free (the reference packs
 *   slots<<16 | free, kma.cl:180; the class field makes a stale reservation
 *   detectable) and sb_home[s] = the shard whose class table holds s.
 *
 * Class table (kma.h:84): each class c has cls_nsh[c] words ("shards"),
 * each 0 (empty), 1 (POISON, refill in progress) or s+2 (superblock s is
 * that shard's current superblock for class c), every one on its own
 * 128-byte line.  A warp uses shard (global warp id) % cls_nsh[c] (its
 * per-thread calls: thread_shard), so one thread of warp 0, lane 0 -- a
 * serial replay -- always uses shard 0; a heap with
 * one shard per class is the reference's single table.  Only a shard's
 * current superblock is contended, so kma_create gives every class
 * pages/32 shards (at most 2048): enough to spread a full GPU's warps,
 * few enough that the superblocks pinned as shards' current ones leave
 * the heap room.
 *
 * Superblock free list, FIFO with the reference's order and its rule that
 * one superblock always stays behind as the queue's dummy
 * (clIndexedQueue.cl:254-290 returns the old dummy; the first superblock
 * handed out is superblock 0):
 *   KMA_HEAP_RING (default): a ticket ring -- fetch-and-add on the head and
 *     tail tickets, one {seq:32 | sb:32} word per slot, an availability
 *     count -- so concurrent refills do not retry CAS loops on one word;
 *   otherwise: the Michael-Scott queue with a dummy node over superblock
 *     indices, links in sb_next[] as 64-bit {tag:32 | idx+1:32} words
 *     (ABA-safe), as the reference builds it (clIndexedQueue.cl:194-290).
 *
 * One-thread-at-a-time execution never observes POISON, a lost CAS or a
 * second shard, so every configuration returns the reference's offsets
 * under serial replay.
 *
 * Every spin (POISON wait, CAS retry, queue helpers) is bounded by
 * heap->spin_limit iterations; on expiry the call fails (NULL / 0), sets
 * KMA_ERR_TIMEOUT in heap->err and never traps.
 */
#ifndef KMA_DEVICE_CUH
#define KMA_DEVICE_CUH

#include <stdint.h>
#include <stddef.h>

#define KMA_MAX_CLASSES 16
#define KMA_MAX_SHARDS 2048    /* per class */
#define KMA_MAX_CLS_LINES 32768 /* sum over classes */
#define KMA_SB_HDR 12u
#define KMA_POISON 1u
#define KMA_CLS_BASE 2u
/* classes with at most this many slots per superblock refill privately
 * instead of queueing behind another warp's refill (kma_malloc_warp) */
#define KMA_PRIVATE_REFILL_SLOTS 8u

#define KMA_ST_FREE_MASK 0x3fffu
#define KMA_ST_SLOTS_SHIFT 14
#define KMA_ST_CLASS_SHIFT 28

/* heap->flags */
#define KMA_HEAP_RING 1u

/* heap->err bits */
#define KMA_ERR_TIMEOUT 1u
#define KMA_ERR_BADFREE 2u
/* with KMA_ERR_TIMEOUT: which bounded wait expired */
#define KMA_ERR_AT_MSQ (1u << 8)        /* MS-queue free list */
#define KMA_ERR_AT_RING_ENQ (1u << 9)   /* ring: slot not yet released */
#define KMA_ERR_AT_RING_AVAIL (1u << 10)/* ring: availability count */
#define KMA_ERR_AT_RING_DEQ (1u << 11)  /* ring: slot not yet filled */
#define KMA_ERR_AT_CLAIM (1u << 12)     /* plain malloc: bitmap claim */
#define KMA_ERR_AT_MALLOC (1u << 13)    /* plain malloc: reservation */
#define KMA_ERR_AT_FREE (1u << 14)      /* plain free: no wait of its own any more, never set */
#define KMA_ERR_AT_RESERVE (1u << 15)   /* warp malloc: reservation (POISON / stale waits) */
#define KMA_ERR_AT_WARP (1u << 16)      /* warp malloc: leader turns */

struct __align__(128) kma_line32 {
	uint32_t v;
	uint32_t pad_[31];
};
struct __align__(128) kma_line64 {
	unsigned long long v;
	unsigned long long pad_[15];
};

struct __align__(128) kma_heap {
	/* geometry: written by kma_create, read-only afterwards */
	unsigned char *sb_base;
	uint32_t *sb_state;
	uint16_t *sb_home;
	unsigned long long *sb_next; /* MS-queue links [nsb] (no KMA_HEAP_RING) */
	unsigned long long *ring;    /* ring slots [ring_cap] (KMA_HEAP_RING) */
	unsigned long long region_bytes; /* nsb << sb_log2 */
	uint32_t sb_log2;
	uint32_t sb_size;
	uint32_t nsb;        /* superblocks allocated (the reference's sblocks) */
	uint32_t pages;      /* superblocks on the free list: sblocks-1 (kma.cl:42) */
	uint32_t nclasses;   /* KMA_SB_SIZE_BUCKETS = log2 - 1 (kma.h:29) */
	uint32_t max_request;/* SB - 16 (kma.cl:126) */
	uint32_t spin_limit;
	uint32_t flags;
	uint32_t cls_lines;  /* sum of cls_nsh[] */
	uint32_t ring_cap;
	uint32_t cls_nsh[KMA_MAX_CLASSES];   /* shards per class */
	uint32_t cls_base[KMA_MAX_CLASSES];  /* first line of the class in cls[] */
	uint32_t cls_size[KMA_MAX_CLASSES];  /* kma.cl:55-90 */
	uint32_t cls_slots[KMA_MAX_CLASSES]; /* kma.cl:95-113 */
	uint32_t cls_magic[KMA_MAX_CLASSES]; /* floor(2^32/size)+1: exact x/size for x < 2^16 */
	uint32_t cls_words[KMA_MAX_CLASSES]; /* bitmap words = ceil(slots/32) */
	/* hot words, one line each */
	kma_line64 free_head; /* MS-queue head, or ring head ticket */
	kma_line64 free_tail; /* MS-queue tail, or ring tail ticket */
	kma_line32 ring_avail;
	kma_line32 err;
	kma_line32 cls[KMA_MAX_CLS_LINES];
};

/* ------------------------------------------------------------------ */
/* memory-model helpers (gpu scope)                                    */
/* ------------------------------------------------------------------ */
namespace kma_detail {

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t *p)
{
	uint32_t v;
	asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
	return v;
}
__device__ __forceinline__ uint32_t ld_relaxed16(const uint16_t *p)
{
	uint16_t v;
	asm volatile("ld.relaxed.gpu.global.u16 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
	return v;
}
__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p)
{
	uint32_t v;
	asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
	return v;
}
__device__ __forceinline__ unsigned long long ld_acquire64(const unsigned long long *p)
{
	unsigned long long v;
	asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
	return v;
}
__device__ __forceinline__ void st_release(uint32_t *p, uint32_t v)
{
	asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_release64(unsigned long long *p, unsigned long long v)
{
	asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint32_t cas_acqrel(uint32_t *p, uint32_t cmp, uint32_t val)
{
	uint32_t old;
	asm volatile("atom.acq_rel.gpu.global.cas.b32 %0, [%1], %2, %3;"
		     : "=r"(old) : "l"(p), "r"(cmp), "r"(val) : "memory");
	return old;
}
__device__ __forceinline__ unsigned long long cas64_acqrel(unsigned long long *p,
		unsigned long long cmp, unsigned long long val)
{
	unsigned long long old;
	asm volatile("atom.acq_rel.gpu.global.cas.b64 %0, [%1], %2, %3;"
		     : "=l"(old) : "l"(p), "l"(cmp), "l"(val) : "memory");
	return old;
}
__device__ __forceinline__ uint32_t add_acqrel(uint32_t *p, uint32_t v)
{
	uint32_t old;
	asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;"
		     : "=r"(old) : "l"(p), "r"(v) : "memory");
	return old;
}
__device__ __forceinline__ unsigned long long add64_acqrel(unsigned long long *p, unsigned long long v)
{
	unsigned long long old;
	asm volatile("atom.acq_rel.gpu.global.add.u64 %0, [%1], %2;"
		     : "=l"(old) : "l"(p), "l"(v) : "memory");
	return old;
}
__device__ __forceinline__ uint32_t or_acqrel(uint32_t *p, uint32_t v)
{
	uint32_t old;
	asm volatile("atom.acq_rel.gpu.global.or.b32 %0, [%1], %2;"
		     : "=r"(old) : "l"(p), "r"(v) : "memory");
	return old;
}
__device__ __forceinline__ uint32_t and_acqrel(uint32_t *p, uint32_t v)
{
	uint32_t old;
	asm volatile("atom.acq_rel.gpu.global.and.b32 %0, [%1], %2;"
		     : "=r"(old) : "l"(p), "r"(v) : "memory");
	return old;
}
__device__ __forceinline__ void fence_acqrel()
{
	asm volatile("fence.acq_rel.gpu;" ::: "memory");
}
/* Relaxed forms for the hot path.  Slot claims and releases are decided by
 * these atomics at L2, the coherence point; a claim is issued only after
 * the reservation it depends on has returned (the GPU does not speculate),
 * and the only plain stores another thread must see first -- a refill's
 * bitmap zeroing and a free's word-0 residue -- are released with their
 * publication (sb_format's state store, bm_and_release). */
__device__ __forceinline__ uint32_t cas_relaxed(uint32_t *p, uint32_t cmp, uint32_t val)
{
	uint32_t old;
	asm volatile("atom.relaxed.gpu.global.cas.b32 %0, [%1], %2, %3;"
		     : "=r"(old) : "l"(p), "r"(cmp), "r"(val) : "memory");
	return old;
}
/* Allocation-bitmap words sit at the superblock tails, in lines they
 * share with payload that the workloads write and read as evict-first
 * (streaming); their atomics ask L2 to keep the line (evict_last): the
 * claims and frees then find it in L2 (config 2's rounds launch measured
 * 7.58 vs 7.66 ms).  A cache hint only: ordering and results unchanged. */
__device__ __forceinline__ unsigned long long keep_policy()
{
	unsigned long long pol;
	asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
	return pol;
}
__device__ __forceinline__ uint32_t bm_or(uint32_t *p, uint32_t v)
{
	uint32_t old;
	asm volatile("atom.relaxed.gpu.global.or.L2::cache_hint.b32 %0, [%1], %2, %3;"
		     : "=r"(old) : "l"(p), "r"(v), "l"(keep_policy()) : "memory");
	return old;
}
__device__ __forceinline__ uint32_t bm_and(uint32_t *p, uint32_t v)
{
	uint32_t old;
	asm volatile("atom.relaxed.gpu.global.and.L2::cache_hint.b32 %0, [%1], %2, %3;"
		     : "=r"(old) : "l"(p), "r"(v), "l"(keep_policy()) : "memory");
	return old;
}
__device__ __forceinline__ uint32_t bm_and_release(uint32_t *p, uint32_t v)
{
	uint32_t old;
	asm volatile("atom.release.gpu.global.and.L2::cache_hint.b32 %0, [%1], %2, %3;"
		     : "=r"(old) : "l"(p), "r"(v), "l"(keep_policy()) : "memory");
	return old;
}
__device__ __forceinline__ uint32_t cas_release(uint32_t *p, uint32_t cmp, uint32_t val)
{
	uint32_t old;
	asm volatile("atom.release.gpu.global.cas.b32 %0, [%1], %2, %3;"
		     : "=r"(old) : "l"(p), "r"(cmp), "r"(val) : "memory");
	return old;
}
__device__ __forceinline__ unsigned long long add64_relaxed(unsigned long long *p, unsigned long long v)
{
	unsigned long long old;
	asm volatile("atom.relaxed.gpu.global.add.u64 %0, [%1], %2;"
		     : "=l"(old) : "l"(p), "l"(v) : "memory");
	return old;
}
__device__ __forceinline__ unsigned long long ld_relaxed64(const unsigned long long *p)
{
	unsigned long long v;
	asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
	return v;
}
__device__ __forceinline__ void st_relaxed64(unsigned long long *p, unsigned long long v)
{
	asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint32_t lane_id()
{
	uint32_t l;
	asm volatile("mov.u32 %0, %%laneid;" : "=r"(l));
	return l;
}
__device__ __forceinline__ uint32_t sm_id()
{
	uint32_t s;
	asm volatile("mov.u32 %0, %%smid;" : "=r"(s));
	return s;
}
__device__ __forceinline__ uint32_t lanemask_lt()
{
	uint32_t m;
	asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
	return m;
}
/* position of the n-th (0-based) set bit of m, counting from bit 0;
 * requires n < popc(m) */
__device__ __forceinline__ uint32_t nth_set_bit(uint32_t m, uint32_t n)
{
	uint32_t pos = 0;
#pragma unroll
	for (uint32_t w = 16; w > 0; w >>= 1) {
		uint32_t c = __popc((m >> pos) & ((1u << w) - 1u));
		if (n >= c) {
			n -= c;
			pos += w;
		}
	}
	return pos;
}
__device__ __forceinline__ void backoff(uint32_t it)
{
	if (it > 4)
		__nanosleep(it < 64 ? 32u : 256u);
}
__device__ __forceinline__ void set_err(kma_heap *h, uint32_t e)
{
	atomicOr(&h->err.v, e);
}

/* state word */
__device__ __forceinline__ uint32_t st_free(uint32_t s) { return s & KMA_ST_FREE_MASK; }
__device__ __forceinline__ uint32_t st_slots(uint32_t s) { return (s >> KMA_ST_SLOTS_SHIFT) & KMA_ST_FREE_MASK; }
__device__ __forceinline__ uint32_t st_class(uint32_t s) { return s >> KMA_ST_CLASS_SHIFT; }
__device__ __forceinline__ uint32_t st_make(uint32_t c, uint32_t slots, uint32_t fr)
{
	return (c << KMA_ST_CLASS_SHIFT) | (slots << KMA_ST_SLOTS_SHIFT) | fr;
}

/* tagged index words {tag:32 | idx:32}, idx 0 = null, idx = item + 1 */
__device__ __forceinline__ uint32_t tw_idx(unsigned long long w) { return (uint32_t)w; }
__device__ __forceinline__ uint32_t tw_tag(unsigned long long w) { return (uint32_t)(w >> 32); }
__device__ __forceinline__ unsigned long long tw_make(uint32_t tag, uint32_t idx)
{
	return ((unsigned long long)tag << 32) | idx;
}

/* (Plain loads of the geometry: through the read-only path the compiler
 * keeps more of it in registers across a call, and the batched form measured
 * 39.1 ms instead of 37.7 for 64 jobs, spills and all.) */
__device__ __forceinline__ unsigned char *sb_addr(const kma_heap *h, uint32_t s)
{
	return h->sb_base + ((size_t)s << h->sb_log2);
}
/* bitmap word k of superblock sb (u32 index SB/4-1-k from the SB start) */
__device__ __forceinline__ uint32_t *bitmap_word(const kma_heap *h, unsigned char *sb, uint32_t k)
{
	return reinterpret_cast<uint32_t *>(sb + h->sb_size) - 1 - k;
}
/* linear id of the calling warp in the grid (stable for its lifetime) */
__device__ __forceinline__ unsigned long long global_warp()
{
	unsigned long long blk = ((unsigned long long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
	uint32_t tpb = blockDim.x * blockDim.y * blockDim.z;
	uint32_t t = (threadIdx.z * blockDim.y + threadIdx.y) * blockDim.x + threadIdx.x;
	return blk * ((tpb + 31) / 32) + t / 32;
}
__device__ __forceinline__ uint32_t my_shard(const kma_heap *h, uint32_t c)
{
	const uint32_t n = h->cls_nsh[c];
	const unsigned long long w = global_warp();
	/* a 64-bit remainder is some hundred instructions: only for grids of
	 * 2^32 warps and more */
	return (w >> 32) ? (uint32_t)(w % n) : (uint32_t)w % n;
}
/* The shard of a per-thread call.  Lanes that reserve each for itself collide
 * on one superblock's count, so a warp spreads over eight shards, lane % 8:
 * config 2's program per thread (24 rounds, 300 / 50021 / 250000 items) took
 * 0.80 / 1.13 / 3.06 ms, with one shard a warp 1.24 / 1.23 / 3.12, with one a
 * lane 0.67 / 1.10 / 3.67 (a full GPU's lanes then touch as many lines). */
__device__ __forceinline__ uint32_t thread_shard(const kma_heap *h, uint32_t c)
{
	const uint32_t n = h->cls_nsh[c];
	const unsigned long long t = global_warp() * 8 + lane_id() % 8;
	return (t >> 32) ? (uint32_t)(t % n) : (uint32_t)t % n;
}
__device__ __forceinline__ uint32_t *cls_word(kma_heap *h, uint32_t c, uint32_t shard)
{
	return &h->cls[h->cls_base[c] + shard].v;
}

} /* namespace kma_detail */

/* ------------------------------------------------------------------ */
/* size classes (kma.cl:55-148)                                        */
/* ------------------------------------------------------------------ */

/* The reference's _kma_sbid_by_size (kma.cl:119-148) returns the smallest
 * class whose block size is >= size (its MSB approximation never starts
 * above that class, and it only ever walks up); sizes above SB-16 give -1.
 * Sizes 0..3 read an uninitialised variable there; here they map to
 * class 0, which is what a zero-initialised reference build returns. */
__device__ __forceinline__ int kma_class_of(const kma_heap *h, size_t size)
{
	if (size > h->max_request)
		return -1;
	uint32_t s = (uint32_t)size;
	int c = s < 4 ? 0 : (int)(29 - __clz(s)); /* floor(log2 s) - 2 */
	while (h->cls_size[c] < s)
		c++;
	return c;
}

/* ------------------------------------------------------------------ */
/* superblock free list                                                */
/* ------------------------------------------------------------------ */
namespace kma_detail {

/* MS queue (clIndexedQueue.cl:194-247 idxd_enqueue).  Returns 1, or 0 on
 * spin-limit expiry. */
__device__ __forceinline__ int msq_enqueue(kma_heap *h, uint32_t s)
{
	unsigned long long *link = &h->sb_next[s];
	uint32_t idx = s + 1;
	unsigned long long old = *((volatile unsigned long long *)link);
	st_release64(link, tw_make(tw_tag(old) + 1, 0));
	uint32_t lim = h->spin_limit;
	for (uint32_t it = 0; it < lim; it++) {
		unsigned long long t = ld_acquire64(&h->free_tail.v);
		unsigned long long *tl = &h->sb_next[tw_idx(t) - 1];
		unsigned long long n = ld_acquire64(tl);
		if (t != ld_acquire64(&h->free_tail.v))
			continue;
		if (tw_idx(n) == 0) {
			if (cas64_acqrel(tl, n, tw_make(tw_tag(n) + 1, idx)) == n) {
				cas64_acqrel(&h->free_tail.v, t, tw_make(tw_tag(t) + 1, idx));
				return 1;
			}
		} else {
			cas64_acqrel(&h->free_tail.v, t, tw_make(tw_tag(t) + 1, tw_idx(n)));
		}
		backoff(it);
	}
	set_err(h, KMA_ERR_TIMEOUT | KMA_ERR_AT_MSQ);
	return 0;
}

/* MS queue dequeue (clIndexedQueue.cl:249-290): the superblock index, -1
 * when only the dummy is left, -2 on spin-limit expiry. */
__device__ __forceinline__ int64_t msq_dequeue(kma_heap *h)
{
	uint32_t lim = h->spin_limit;
	for (uint32_t it = 0; it < lim; it++) {
		unsigned long long hd = ld_acquire64(&h->free_head.v);
		unsigned long long t = ld_acquire64(&h->free_tail.v);
		unsigned long long n = ld_acquire64(&h->sb_next[tw_idx(hd) - 1]);
		if (hd != ld_acquire64(&h->free_head.v))
			continue;
		if (tw_idx(hd) == tw_idx(t)) {
			if (tw_idx(n) == 0)
				return -1;
			cas64_acqrel(&h->free_tail.v, t, tw_make(tw_tag(t) + 1, tw_idx(n)));
		} else if (cas64_acqrel(&h->free_head.v, hd, tw_make(tw_tag(hd) + 1, tw_idx(n))) == hd) {
			return (int64_t)tw_idx(hd) - 1;
		}
		backoff(it);
	}
	set_err(h, KMA_ERR_TIMEOUT | KMA_ERR_AT_MSQ);
	return -2;
}

/* Ticket ring.  Slot p % cap holds {seq:32 | sb:32}; seq == p+1 means
 * "filled by the enqueue with ticket p", seq == p means "free for the
 * enqueue with ticket p".  ring_avail counts completed enqueues not yet
 * claimed by a dequeue; a dequeue needs two (one stays behind, as the
 * reference's dummy does).  The ring carries only superblock numbers: the
 * enqueuer stores one after its detach of the superblock has returned
 * (ring_put), and everything a dequeuer then writes is addressed
 * through the number it read, so tickets, counts and slots are relaxed; a
 * count seen before its slot store only makes a dequeuer wait
 * on the slot's sequence number. */
/* ticket -> slot: as the 64-bit remainder, which only tickets past 2^32 take */
__device__ __forceinline__ uint32_t ring_slot(unsigned long long pos, uint32_t cap)
{
	return (pos >> 32) ? (uint32_t)(pos % cap) : (uint32_t)pos % cap;
}
/* Put superblock s into the slot of tail ticket `pos`.  detached: the value
 * an atomic that detached s returned.  It must have returned before s can be
 * handed out again (a late clearing of s's old class slot would hit its next
 * incarnation); the store waits for it by using it -- no class slot holds
 * 0xffffffff -- where a release store would wait out a fence. */
__device__ __forceinline__ int ring_put(kma_heap *h, unsigned long long pos, uint32_t s, uint32_t detached)
{
	unsigned long long *slot = h->ring + ring_slot(pos, h->ring_cap);
	uint32_t lim = h->spin_limit;
	for (uint32_t it = 0; it < lim; it++) {
		unsigned long long w = ld_relaxed64(slot);
		if ((uint32_t)(w >> 32) == (uint32_t)pos && detached != 0xffffffffu) {
			st_relaxed64(slot, ((unsigned long long)(uint32_t)(pos + 1) << 32) | s);
			return 1;
		}
		backoff(it);
	}
	set_err(h, KMA_ERR_TIMEOUT | KMA_ERR_AT_RING_ENQ);
	return 0;
}
__device__ __forceinline__ void ring_enqueue(kma_heap *h, uint32_t s, uint32_t detached)
{
	if (ring_put(h, add64_relaxed(&h->free_tail.v, 1ull), s, detached))
		atomicAdd(&h->ring_avail.v, 1u);
}
/* The calling lanes (`active`) that `want` to put theirs take tickets
 * together.  Every lane of `active` calls. */
__device__ __forceinline__ void ring_enqueue_lanes(kma_heap *h, uint32_t active, bool want, uint32_t s,
		uint32_t detached)
{
	const uint32_t m = __ballot_sync(active, want);
	const uint32_t first = __ffs(m) - 1;
	unsigned long long pos = 0;
	if (lane_id() == first)
		pos = add64_relaxed(&h->free_tail.v, (unsigned long long)__popc(m));
	pos = __shfl_sync(active, pos, first) + __popc(m & lanemask_lt());
	if (want && ring_put(h, pos, s, detached))
		atomicAdd(&h->ring_avail.v, 1u);
}

/* the superblock of head ticket `pos` (claimed against ring_avail) */
__device__ __forceinline__ int64_t ring_take(kma_heap *h, unsigned long long pos)
{
	const uint32_t cap = h->ring_cap;
	unsigned long long *slot = h->ring + ring_slot(pos, cap);
	uint32_t lim = h->spin_limit;
	for (uint32_t it = 0; it < lim; it++) {
		unsigned long long w = ld_relaxed64(slot);
		if ((uint32_t)(w >> 32) == (uint32_t)(pos + 1)) {
			st_relaxed64(slot, (unsigned long long)(uint32_t)(pos + cap) << 32);
			return (int64_t)(uint32_t)w;
		}
		backoff(it);
	}
	set_err(h, KMA_ERR_TIMEOUT | KMA_ERR_AT_RING_DEQ);
	return -2;
}

__device__ __forceinline__ int64_t ring_dequeue(kma_heap *h)
{
	int32_t *avail = reinterpret_cast<int32_t *>(&h->ring_avail.v);
	int32_t old = atomicSub(avail, 1);
	if (old < 2) {
		/* near empty: undo, then claim only a count that is really there */
		atomicAdd(avail, 1);
		int32_t a = (int32_t)ld_relaxed(&h->ring_avail.v);
		uint32_t lim = h->spin_limit, it = 0;
		for (;;) {
			if (a < 2)
				return -1;
			int32_t seen = (int32_t)atomicCAS((unsigned *)&h->ring_avail.v, (uint32_t)a, (uint32_t)(a - 1));
			if (seen == a)
				break;
			a = seen;
			if (++it >= lim) {
				set_err(h, KMA_ERR_TIMEOUT | KMA_ERR_AT_RING_AVAIL);
				return -2;
			}
		}
	}
	return ring_take(h, add64_relaxed(&h->free_head.v, 1ull));
}

/* The calling lanes (`active`) that `want` one each take superblocks
 * together: one claim of the availability count and one ticket add for all
 * of them.  Each gets what a ring_dequeue in lane order would: lanes beyond
 * the count go through ring_dequeue's own near-empty path. */
__device__ __forceinline__ int64_t ring_dequeue_lanes(kma_heap *h, uint32_t active, bool want)
{
	const uint32_t m = __ballot_sync(active, want);
	if (!m)
		return -1;
	const uint32_t first = __ffs(m) - 1, rank = __popc(m & lanemask_lt());
	int32_t granted = 0;
	unsigned long long pos = 0;
	if (lane_id() == first) {
		int32_t *avail = reinterpret_cast<int32_t *>(&h->ring_avail.v);
		const int32_t n = __popc(m);
		const int32_t old = atomicSub(avail, n);
		/* of n single claims the ones that find at least two succeed */
		granted = old - 1 < 0 ? 0 : old - 1 < n ? old - 1 : n;
		if (granted < n)
			atomicAdd(avail, n - granted);
		if (granted)
			pos = add64_relaxed(&h->free_head.v, (unsigned long long)granted);
	}
	granted = __shfl_sync(active, granted, first);
	pos = __shfl_sync(active, pos, first);
	if (!want)
		return -1;
	if ((int32_t)rank >= granted)
		return ring_dequeue(h);
	return ring_take(h, pos + rank);
}

__device__ __forceinline__ int64_t sb_dequeue(kma_heap *h)
{
	return (h->flags & KMA_HEAP_RING) ? ring_dequeue(h) : msq_dequeue(h);
}
/* for the calling lanes that want one; every lane of `active` calls */
__device__ __forceinline__ int64_t sb_dequeue_lanes(kma_heap *h, uint32_t active, bool want)
{
	if (h->flags & KMA_HEAP_RING)
		return ring_dequeue_lanes(h, active, want);
	return want ? msq_dequeue(h) : -1;
}

/* Prepare superblock s for class c: zero its bitmap except the bits in
 * [pre_lo, slots), which are pre-set (claimed by the refiller), record its
 * home shard, then publish state = (c, slots, free).  kma.cl:177-189, with
 * the bitmap written before the state becomes visible: the state alone lets
 * others in, before any class slot names s.  A warp whose hint names s, or a
 * thread that read a class slot before s was recycled, reserves as soon as it
 * sees a free count of its class, and a bitmap store that came after its
 * claim would give the claimed slots to somebody else too.  So the store is a
 * release: whoever reserves finds the bitmap and the home at L2, where its
 * claims and its recycle read them.  (The reserving CAS stays relaxed, as the
 * claims behind it are atomics issued after it has returned; as an acquire,
 * which drops the SM's L1 each time, it cost config 2 2.7% in its warp form
 * and 7% per thread, and 64 jobs 0.9%.  The release costs nothing that could
 * be measured: 6.42 ms for config 2.) */
__device__ __forceinline__ void sb_format(kma_heap *h, uint32_t s, uint32_t c, uint32_t pre_lo,
		uint32_t fr, uint32_t shard)
{
	unsigned char *sb = sb_addr(h, s);
	uint32_t slots = h->cls_slots[c];
	uint32_t words = h->cls_words[c];
	for (uint32_t k = 0; k < words; k++) {
		uint32_t lo = k * 32, hi = lo + 32;
		uint32_t v = 0;
		if (pre_lo < hi && slots > lo) {
			uint32_t a = pre_lo > lo ? pre_lo : lo;
			uint32_t b = slots < hi ? slots : hi;
			if (b > a) {
				uint32_t n = b - a;
				v = (n == 32 ? 0xffffffffu : ((1u << n) - 1u)) << (a - lo);
			}
		}
		*bitmap_word(h, sb, k) = v;
	}
	h->sb_home[s] = (uint16_t)shard;
	st_release(&h->sb_state[s], st_make(c, slots, fr));
}

} /* namespace kma_detail */

/* ------------------------------------------------------------------ */
/* plain per-thread malloc/free: the reference algorithm                */
/* (kma.cl:150-373) with its atomics, made safe against recycling:      */
/*  - a reservation CAS only succeeds on a state word whose class field */
/*    is the requested class (a stale cursor whose superblock was       */
/*    recycled for another class fails and retries);                   */
/*  - taking the last free slot detaches with CAS(cls, cursor, 0), not  */
/*    an unconditional exchange (kma.cl:217).                           */
/* In one-thread-at-a-time execution both are identical to the         */
/* reference, so serial replay returns the reference's offsets.         */
/* ------------------------------------------------------------------ */
namespace kma_detail {

/* A class slot that names a superblock which cannot serve its class (no
 * free count left, or recycled for another class) is cleared by the
 * thread that finds it, not waited on.  The thread that takes a
 * superblock's last slots clears the slot it read the superblock from;
 * if the superblock was recycled meanwhile and republished in another
 * shard's slot of the same class, that slot keeps naming it, full, until
 * all its blocks are freed -- and the threads waiting on that slot may be
 * the ones holding them.  Clearing at worst hides a superblock whose
 * slots were freed again since the read; it returns to the free list
 * when all its blocks are freed, as any detached one.  One-thread
 * execution never finds such a slot (a taker always clears the slot it
 * read), so serial replay is unchanged. */
__device__ __forceinline__ void clear_stale(uint32_t *clsw, uint32_t cur)
{
	cas_relaxed(clsw, cur, 0);
}

/* kma.cl:232-273: claim a bitmap bit at or above `hint` (wrapping),
 * write the hint into word 0 of the block.  v: the hint's bitmap word as the
 * caller has seen it, perhaps before its reservation: bits that look free
 * are tried first, and the atomicOr decides. */
__device__ __forceinline__ void *sb_get_block(kma_heap *h, uint32_t s, uint32_t c, uint32_t hint, uint32_t v)
{
	unsigned char *sb = sb_addr(h, s);
	uint32_t slots = h->cls_slots[c];
	uint32_t size = h->cls_size[c];
	uint32_t words = h->cls_words[c];
	uint32_t k = hint >> 5, lo = hint & 31;
	uint32_t lim = h->spin_limit;
	for (uint32_t it = 0; it < lim; it++) {
		uint32_t *wp = bitmap_word(h, sb, k);
		uint32_t valid = (k == words - 1 && (slots & 31)) ? ((1u << (slots & 31)) - 1u) : 0xffffffffu;
		uint32_t cand = ~v & valid & (0xffffffffu << lo);
		while (cand) {
			uint32_t b = __ffs(cand) - 1;
			uint32_t bit = 1u << b;
			uint32_t old = bm_or(wp, bit);
			if (!(old & bit)) {
				unsigned char *p = sb + KMA_SB_HDR + (size_t)(k * 32 + b) * size;
				*reinterpret_cast<uint32_t *>(p) = hint;
				return p;
			}
			cand &= ~old;
			cand &= ~bit;
		}
		/* the first of the next four words that looks as if it had a free
		 * bit: the used slots of a class with many stand together, and a word
		 * to a round trip was most of a malloc's time there */
		uint32_t x[4];
#pragma unroll
		for (uint32_t i = 0; i < 4; i++)
			x[i] = ld_relaxed(bitmap_word(h, sb, (k + 1 + i) % words));
		uint32_t i = x[0] != 0xffffffffu ? 0u : x[1] != 0xffffffffu ? 1u : x[2] != 0xffffffffu ? 2u : 3u;
		v = i == 0 ? x[0] : i == 1 ? x[1] : i == 2 ? x[2] : x[3];
		k = (k + 1 + i) % words;
		lo = 0;
	}
	set_err(h, KMA_ERR_TIMEOUT | KMA_ERR_AT_CLAIM);
	return NULL;
}

/* The free list is empty: one slot of class c from the current superblock of
 * one of the next shards, or NULL.  A warp's per-thread calls spread over
 * eight shards, so the slots that are left are spread too: without a look at
 * the neighbours a heap of 224 MiB that just held 60 k items' blocks refused
 * 100 of 600 k requests.  A thread alone fills no other shard than its own,
 * so serial replay is unchanged.
 *
 * A refusal pays for the look, so KMA_STEAL_ROW class words are read at a time:
 * a refused call by one thread takes 6.7 us (18 a word at a time, 1.0 without
 * the look), by 148 x 256 threads on 16 MiB / 224 MiB of heap 713 / 109 us
 * (943 / 141; 454 / 155), by 592 x 512 7.7 / 1.3 ms (7.9 / 1.4; 47 / 1.3).
 * Longer rows are no faster, and their registers are the caller's: with the
 * words of 8 at hand until they are tried, the graph build had 72 instead of
 * 64, and 22% more time. */
#define KMA_STEAL_SHARDS 64u
#define KMA_STEAL_ROW 4u
/* (below 2 n) */
__device__ __forceinline__ uint32_t *steal_word(kma_heap *h, uint32_t c, uint32_t shard, uint32_t n)
{
	return cls_word(h, c, shard < n ? shard : shard - n);
}
static __device__ __noinline__ void *steal_block(kma_heap *h, uint32_t c, uint32_t shard)
{
	const uint32_t n = h->cls_nsh[c], most = n - 1 < KMA_STEAL_SHARDS ? n - 1 : KMA_STEAL_SHARDS;
	for (uint32_t base = 1; base <= most; base += KMA_STEAL_ROW) {
		uint32_t named = 0; /* those that name a superblock */
#pragma unroll
		for (uint32_t i = 0; i < KMA_STEAL_ROW; i++)
			if (base + i <= most)
				named |= (uint32_t)(ld_relaxed(steal_word(h, c, shard + base + i, n)) >= KMA_CLS_BASE) << i;
		for (; named; named &= named - 1) {
			uint32_t *clsw = steal_word(h, c, shard + base + (__ffs(named) - 1), n);
			const uint32_t cur = ld_relaxed(clsw);
			if (cur < KMA_CLS_BASE)
				continue;
			const uint32_t s = cur - KMA_CLS_BASE;
			for (uint32_t tries = 0; tries < 4; tries++) {
				const uint32_t st = ld_relaxed(&h->sb_state[s]);
				if (st_class(st) != c || st_free(st) == 0)
					break;
				const uint32_t fr = st_free(st) - 1;
				const uint32_t v = ld_relaxed(bitmap_word(h, sb_addr(h, s), fr >> 5));
				if (cas_relaxed(&h->sb_state[s], st, st - 1) != st)
					continue;
				if (fr == 0)
					cas_relaxed(clsw, cur, 0);
				return sb_get_block(h, s, c, fr, v);
			}
		}
	}
	return NULL;
}

} /* namespace kma_detail */

/* kma.cl:279-303 (with _kma_reserve_block, kma.cl:150-225) */
__device__ inline void *kma_malloc(kma_heap *h, size_t size)
{
	using namespace kma_detail;
	int c = kma_class_of(h, size);
	if (c < 0)
		return NULL;
	uint32_t shard = thread_shard(h, (uint32_t)c);
	uint32_t *clsw = cls_word(h, (uint32_t)c, shard);
	uint32_t lim = h->spin_limit;
	for (uint32_t it = 0; it < lim; it++) {
		/* kma.cl:163 reads the slot with its CAS 0 -> POISON; here only an
		 * empty one is CASed, so that threads on one slot do not queue */
		uint32_t cur = ld_relaxed(clsw);
		if (cur == 0) {
			if (cas_relaxed(clsw, 0, KMA_POISON) != 0)
				continue;
			/* refill, kma.cl:166-195 */
			int64_t s = sb_dequeue(h);
			if (s < 0) {
				atomicExch(clsw, 0);
				return s == -1 ? steal_block(h, (uint32_t)c, shard) : NULL;
			}
			uint32_t slots = h->cls_slots[c];
			sb_format(h, (uint32_t)s, c, slots, slots - 1, shard);
			/* kma.cl:191 publishes the superblock even when the refill
			 * took its only slot (1-slot classes); every later request
			 * of that class then spins on a full superblock until the
			 * block is freed (kma.cl:203-204).  Leave the class empty
			 * instead, which is what taking the last slot does. */
			cas_release(clsw, KMA_POISON, slots == 1 ? 0u : (uint32_t)s + KMA_CLS_BASE);
			return sb_get_block(h, (uint32_t)s, c, slots - 1, 0u);
		}
		if (cur == KMA_POISON) {
			backoff(it);
			continue;
		}
		uint32_t s = cur - KMA_CLS_BASE;
		uint32_t *stp = &h->sb_state[s];
		uint32_t st = ld_relaxed(stp); /* kma.cl:198: atom_add(.., 0) */
		if (st_class(st) != (uint32_t)c || st_free(st) == 0) {
			clear_stale(clsw, cur);
			continue;
		}
		uint32_t fr = st_free(st) - 1;
		/* the hint's bitmap word beside the reservation, not after it */
		const uint32_t v = ld_relaxed(bitmap_word(h, sb_addr(h, s), fr >> 5));
		if (cas_relaxed(stp, st, st - 1) != st)
			continue;
		if (fr == 0)
			cas_relaxed(clsw, cur, 0); /* kma.cl:216-218 */
		return sb_get_block(h, s, c, fr, v);
	}
	set_err(h, KMA_ERR_TIMEOUT | KMA_ERR_AT_MALLOC);
	return NULL;
}

namespace kma_detail {
/* Locate the superblock / class / slot of a live block. */
__device__ __forceinline__ bool block_locate(const kma_heap *h, const void *p, uint32_t &s,
		uint32_t &c, uint32_t &slot)
{
	size_t off = (const unsigned char *)p - h->sb_base;
	if (off >= h->region_bytes)
		return false;
	s = (uint32_t)(off >> h->sb_log2);
	uint32_t in = (uint32_t)(off & (h->sb_size - 1));
	uint32_t st = ld_relaxed(&h->sb_state[s]);
	c = st_class(st);
	if (st == 0 || in < KMA_SB_HDR || c >= h->nclasses)
		return false;
	slot = (uint32_t)(((unsigned long long)(in - KMA_SB_HDR) * h->cls_magic[c]) >> 32);
	return slot < h->cls_slots[c];
}

/* Detach superblock s (class c, state word `full`: every slot free) from its
 * class, unless a reservation gets in first: kma.cl:350-367.  True: it is the
 * caller's to put on the free list; *seen: what its class slot held.
 *
 * The CAS that takes the count away detaches s: from then on, until it is on
 * the free list, nobody else can reserve from it, recycle it or give it another
 * home.  So the home is read after that CAS has returned.  Before it, s may be
 * recycled, formatted for the same class under another shard and freed again,
 * which the CAS cannot tell from nothing having happened: the old home's slot
 * would be cleared and the current one left naming a superblock on the free
 * list.  The home was stored before the state (sb_format), and a gpu-scope
 * relaxed load is served at L2, where that store already was; a plain one may
 * be served from this SM's L1, where a line of sb_home read during an earlier
 * incarnation can still sit. */
__device__ __forceinline__ bool sb_detach(kma_heap *h, uint32_t s, uint32_t c, uint32_t full, uint32_t *seen)
{
	if (cas_relaxed(&h->sb_state[s], full, st_make(c, st_slots(full), 0)) != full)
		return false;
	*seen = cas_relaxed(cls_word(h, c, ld_relaxed16(&h->sb_home[s])), s + KMA_CLS_BASE, 0);
	return true;
}
/* Recycle it, by one thread. */
__device__ __forceinline__ void sb_recycle(kma_heap *h, uint32_t s, uint32_t c, uint32_t full)
{
	uint32_t seen = 0;
	if (!sb_detach(h, s, c, full, &seen))
		return;
	if (h->flags & KMA_HEAP_RING)
		ring_enqueue(h, s, seen);
	else
		msq_enqueue(h, s);
}
/* The lanes of `active` that have one (all_free) recycle theirs together;
 * every lane of it calls. */
__device__ __forceinline__ void sb_recycle_lanes(kma_heap *h, uint32_t active, bool all_free, uint32_t s, uint32_t c,
		uint32_t full)
{
	uint32_t seen = 0;
	const bool mine = all_free && sb_detach(h, s, c, full, &seen);
	if (!__any_sync(active, mine))
		return;
	if (h->flags & KMA_HEAP_RING)
		ring_enqueue_lanes(h, active, mine, s, seen);
	else if (mine)
		msq_enqueue(h, s);
}
} /* namespace kma_detail */

/* The start of the heap block that contains p (p may point inside it), or
 * NULL when p is not inside a superblock in use.  For structures that
 * place an aligned object inside a 4-byte aligned block and must free the
 * block itself.  No counterpart in the reference. */
__device__ __forceinline__ void *kma_block_of(kma_heap *h, const void *p)
{
	using namespace kma_detail;
	uint32_t s, c, slot;
	if (!p || !block_locate(h, p, s, c, slot))
		return NULL;
	return sb_addr(h, s) + KMA_SB_HDR + (size_t)slot * h->cls_size[c];
}

/* kma.cl:305-373 */
__device__ inline void kma_free(kma_heap *h, void *p)
{
	using namespace kma_detail;
	if (p == NULL)
		return;
	uint32_t s, c, slot;
	if (!block_locate(h, p, s, c, slot)) {
		set_err(h, KMA_ERR_BADFREE);
		return;
	}
	unsigned char *sb = sb_addr(h, s);
	uint32_t bit = 1u << (slot & 31);
	uint32_t *wp = bitmap_word(h, sb, slot >> 5);
	/* kma.cl:336-338 leaves the bitmap word as it was before the clear in
	 * word 0 of the block, but stores it after the clear: by then another
	 * thread may already own the slot and have written that word.  Store
	 * the same value first, then clear the bit with release semantics. */
	uint32_t cur = ld_relaxed(wp);
	if (!(cur & bit)) {
		/* double free: the reference increments the free count anyway
		 * and corrupts the superblock (kma.cl:333-335); refuse it */
		set_err(h, KMA_ERR_BADFREE);
		return;
	}
	*reinterpret_cast<volatile uint32_t *>(p) = cur;
	uint32_t old = bm_and_release(wp, ~bit);
	if (!(old & bit)) {
		set_err(h, KMA_ERR_BADFREE); /* a concurrent double free */
		return;
	}
	/* kma.cl:343-367 re-reads and CASes the count until it fits; an add
	 * cannot miss, and lanes that free into one superblock need not queue */
	const uint32_t full = atomicAdd(&h->sb_state[s], 1u) + 1u;
	/* by itself: a per-thread call stands in whatever divergent code its caller
	 * has, where the lanes that seem to run with it need not take part in a
	 * vote or a shuffle with it (recycling together, threads of the graph build
	 * got tickets that nobody had drawn) */
	if (st_free(full) == st_slots(full))
		sb_recycle(h, s, c, full);
}

/* ------------------------------------------------------------------ */
/* warp-collaborative malloc/free                                      */
/* ------------------------------------------------------------------ */
/* Lanes are grouped by size class with __match_any_sync.  The group   */
/* leader reserves k slots with one CAS on the current superblock's     */
/* state word (refilling from the free list when needed; a group that   */
/* needs a whole superblock takes a fresh one without touching the      */
/* class table), then claims the bitmap bits one word at a time with    */
/* one atomicOr per word; the claimed (superblock, word, mask) is       */
/* broadcast with __shfl_sync and each lane picks its bit by rank.  All  */
/* leaders take these steps side by side, one of each per iteration.  One */
/* atomic per warp per superblock (and per bitmap word) reaches L2      */
/* instead of two or three per lane.  A single calling lane follows     */
/* exactly the plain path's choices.                                    */
/* ------------------------------------------------------------------ */
/* Optional event counts of the warp-collaborative calls (diagnostics):
 * pass a pointer to a per-thread tally to kma_malloc_warp/kma_free_warp;
 * with the default null pointer the counting compiles away. */
struct kma_tally {
	uint32_t n[8];
};
#define KMA_T_ITER 0      /* leader turns in kma_malloc_warp */
#define KMA_T_TRY 1       /* reservation attempts */
#define KMA_T_POISON 2    /* waits on a refill in progress */
#define KMA_T_STALE 3     /* class slot pointing at a full or stale superblock */
#define KMA_T_CASFAIL 4   /* lost reservation CASes */
#define KMA_T_REFILL 5    /* superblocks taken from the free list */
#define KMA_T_CLAIM 6     /* bitmap claim steps */
#define KMA_T_EMPTY 7     /* claim steps that got no bit */

namespace kma_detail {

__device__ __forceinline__ void tally(kma_tally *t, int k)
{
	if (t)
		t->n[k]++;
}

/* Leader-side state of one group's reservation.  known: the bitmap word at
 * the cursor as it was last seen, if knows (claims go blind on a word not
 * seen: setting a bit that is already set changes nothing, and the returned
 * word says what is free); pre: the slots from the cursor up are set already,
 * by the refill. */
struct warp_resv {
	uint32_t sb, left, cursor, hint, known;
	bool pre, knows;
};

/* A superblock that is no class slot's current one is reserved from, when a
 * hint names it, if it serves the whole request and its free bits are quick
 * to find: in at most two bitmap words, or a quarter of its slots. */
__device__ __forceinline__ bool hint_serves(const kma_heap *h, uint32_t c, uint32_t slots, uint32_t want, uint32_t st)
{
	const uint32_t fr = st_free(st);
	return st_class(st) == c && fr >= want && (h->cls_words[c] <= 2 || fr * 4 >= slots);
}

/* The bits of bitmap word `word` that reservation r takes next, given what
 * is known of it: the lowest `left` candidates at or above the cursor. */
__device__ __forceinline__ uint32_t claim_pick(const kma_heap *h, const warp_resv &r, uint32_t c, uint32_t slots,
		uint32_t &cand)
{
	const uint32_t k = r.cursor >> 5, lo = r.cursor & 31;
	const uint32_t valid = ((k + 1) * 32 > slots) ? ((1u << (slots & 31)) - 1u) : 0xffffffffu;
	/* first visit of a word: assume its bits are clear; the atomicOr's
	 * result then says which ones really were */
	const uint32_t v = r.knows ? r.known : 0u;
	cand = ~v & valid & (0xffffffffu << lo);
	if (__popc(cand) <= (int)r.left)
		return cand;
	const uint32_t top = nth_set_bit(cand, r.left - 1);
	return cand & (top == 31 ? 0xffffffffu : ((2u << top) - 1u));
}

/* Exclusive prefix sum over the 32 lanes of a full warp; *total: the sum. */
__device__ __forceinline__ uint32_t warp_excl_sum(uint32_t x, uint32_t *total)
{
	uint32_t incl = x;
#pragma unroll
	for (uint32_t d = 1; d < 32; d <<= 1) {
		const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
		if (lane_id() >= d)
			incl += v;
	}
	*total = __shfl_sync(0xffffffffu, incl, 31);
	return incl - x;
}
/* Of the 32 lanes with `n` items each, excl those before: the lane that has
 * item j (which one of them does). */
__device__ __forceinline__ uint32_t warp_owner_of(uint32_t excl, uint32_t j)
{
	uint32_t l = 0;
#pragma unroll
	for (uint32_t d = 16; d > 0; d >>= 1)
		if (__shfl_sync(0xffffffffu, excl, l + d) <= j)
			l += d;
	return l;
}

/* Claim up to `left` slots of superblock s (class c) by a whole warp, all
 * lanes with the same arguments but j: 32 bitmap words at a time, one a lane,
 * are loaded, the free bits numbered over the lanes, and the first `left` of
 * them claimed with one atomicOr a word.  A lane with j < the number claimed
 * gets the j-th as its block (word 0: hint - j).
 *
 * A superblock serves its class until its last slot is taken, so its last
 * slots are single bits all over its words; one leader that tried a word per
 * round trip made 44 claims a warp and round for 64 jobs (Zipf sizes, mostly
 * 8 to 32 bytes: 64 to 8 words), 37 of them for nothing, and the run took
 * 35.2 ms instead of 24.9. */
struct sweep_got {
	void *p;
	uint32_t n;
};
__device__ __forceinline__ sweep_got warp_sweep(kma_heap *h, uint32_t s, uint32_t c, uint32_t first, uint32_t left, uint32_t j,
		uint32_t hint)
{
	const uint32_t words = h->cls_words[c], slots = h->cls_slots[c], lane = lane_id(), full = 0xffffffffu;
	unsigned char *sb = sb_addr(h, s);
	sweep_got g = {NULL, 0};
	for (uint32_t base = 0; base < words && !g.n; base += 32) {
		const uint32_t o = base + lane;
		uint32_t w = first + o, cand = 0, total, old = 0;
		w = w >= words ? w - words : w;
		if (o < words) {
			const uint32_t valid = (w + 1) * 32 > slots ? (1u << (slots & 31)) - 1u : 0xffffffffu;
			cand = ~ld_relaxed(bitmap_word(h, sb, w)) & valid;
		}
		const uint32_t before = warp_excl_sum(__popc(cand), &total);
		if (total == 0)
			continue;
		const uint32_t room = before < left ? left - before : 0u;
		if (__popc(cand) > room)
			cand = room ? cand & (0xffffffffu >> (31u - nth_set_bit(cand, room - 1))) : 0u;
		if (cand)
			old = bm_or(bitmap_word(h, sb, w), cand);
		cand &= ~old;
		const uint32_t excl = warp_excl_sum(__popc(cand), &g.n);
		if (!g.n)
			continue;
		const uint32_t from = warp_owner_of(excl, j < g.n ? j : 0u);
		const uint32_t bits = __shfl_sync(full, cand, from), wo = __shfl_sync(full, w, from);
		const uint32_t i = j - __shfl_sync(full, excl, from);
		if (j < g.n) {
			const uint32_t slot = wo * 32 + nth_set_bit(bits, i);
			g.p = sb + KMA_SB_HDR + (size_t)slot * h->cls_size[c];
			*reinterpret_cast<uint32_t *>(g.p) = hint - j;
		}
	}
	return g;
}

/* One lane's part in a step of kma_malloc_warp: */
#define KMA_R_NONE 0u   /* nothing to reserve, or nothing got */
#define KMA_R_TAKE 1u   /* reserve from superblock s */
#define KMA_R_LOCK 2u   /* refill an empty class slot (POISON) */
#define KMA_R_OWN 3u    /* take a superblock without the class slot */
#define KMA_R_WAIT 4u   /* another refill is in progress */

} /* namespace kma_detail */

/* hint (optional): this warp's KMA_MAX_CLASSES words, zeroed once, best
 * in shared memory; the warp's leaders remember there, per class, the
 * superblock they last reserved from.  Its state is loaded together with the
 * class word on the next call, and if it still serves the request it is
 * reserved from, current or not (hint_serves): the class slot does not get
 * back a detached superblock whose blocks are freed one by one.  (Not for a
 * single calling lane, which follows the reference's choices.)  Words an
 * earlier call left are safe whatever has become of their superblocks, as a
 * reservation's CAS checks class and count. */
template <bool SWEEP>
__device__ __forceinline__ void *kma_malloc_warp_t(kma_heap *h, size_t size, kma_tally *tl, uint32_t *hint)
{
	using namespace kma_detail;
	const uint32_t active = __activemask();
	const uint32_t lane = lane_id();
	const bool sweep = SWEEP && active == 0xffffffffu;
	const int cls = kma_class_of(h, size);
	const uint32_t peers = __match_any_sync(active, cls);
	const uint32_t leader = __ffs(peers) - 1;
	const uint32_t rank = __popc(peers & lanemask_lt());
	const uint32_t gsize = __popc(peers);
	bool need = cls >= 0;
	void *res = NULL;

	/* leader-only state: the leader serves its whole group, not only itself */
	const bool leads = lane == leader && need;
	const uint32_t c = need ? (uint32_t)cls : 0u;
	const uint32_t slots = h->cls_slots[c];
	const uint32_t shard = my_shard(h, c);
	warp_resv r;
	r.left = 0;
	uint32_t served = 0, idle = 0;
	bool failed = false;

	/* Every lane runs every iteration, and each group's leader takes one step
	 * of its own reservation in it.  The steps of different leaders are the
	 * same instructions, or are issued before any of their results is used,
	 * so that an iteration costs the round trips of its longest step (a
	 * refill), not the sum over the groups.  A leader gives up, for its whole
	 * group, after spin_limit steps in a row that got nothing, which ends the
	 * loop. */
	while (__any_sync(active, need)) {
		const bool open = leads && served < gsize && !failed;
		const uint32_t want = gsize - served;
		uint32_t kind = KMA_R_NONE, cur = 0, s = 0, st = 0;
		bool known = false;
		/* 1. the class slot, and beside it the state of the superblock this
		 * warp last reserved from in the class */
		if (open && r.left == 0) {
			tally(tl, KMA_T_ITER);
			tally(tl, KMA_T_TRY);
			if (++idle > h->spin_limit) {
				failed = true;
				set_err(h, KMA_ERR_TIMEOUT | KMA_ERR_AT_RESERVE);
			} else if (want >= slots && slots > 1) {
				/* the group fills a whole superblock: take a fresh one
				 * privately (it would be detached at once anyway) */
				kind = KMA_R_OWN;
			} else {
				const uint32_t guess = hint ? hint[c] : 0u;
				cur = ld_relaxed(cls_word(h, c, shard));
				if (guess)
					st = ld_relaxed(&h->sb_state[guess - KMA_CLS_BASE]);
				if (guess && hint_serves(h, c, slots, want, st) && (active & (active - 1u))) {
					kind = KMA_R_TAKE;
					known = true;
					cur = guess;
				} else if (cur == 0) {
					/* the reference's refill under POISON (kma.cl:166-195) */
					kind = KMA_R_LOCK;
				} else if (cur != KMA_POISON) {
					kind = KMA_R_TAKE;
					known = cur == guess && st_class(st) == c && st_free(st) != 0;
				} else if (slots <= KMA_PRIVATE_REFILL_SLOTS) {
					/* a class with few slots per superblock: the refill in
					 * flight yields about one group's worth, so rather than
					 * queue behind it take a fresh superblock without the
					 * class slot, and publish the leftover slots only if the
					 * slot is empty by then.  Serial execution never
					 * observes POISON. */
					kind = KMA_R_OWN;
				} else {
					tally(tl, KMA_T_POISON);
					kind = KMA_R_WAIT;
				}
				s = cur - KMA_CLS_BASE;
			}
		}
		/* 2. its state, where step 1 did not have it */
		if (kind == KMA_R_TAKE && !known) {
			st = ld_relaxed(&h->sb_state[s]);
			if (st_class(st) != c || st_free(st) == 0) {
				tally(tl, KMA_T_STALE);
				clear_stale(cls_word(h, c, shard), cur);
				kind = KMA_R_NONE;
			}
		}
		/* 3. the reservation, with the first bitmap word the claim will visit
		 * loaded beside it; and the locks of empty class slots */
		uint32_t got = 0, spec = 0, t = 0;
		if (kind == KMA_R_TAKE) {
			t = want < st_free(st) ? want : st_free(st);
			spec = ld_relaxed(bitmap_word(h, sb_addr(h, s), (st_free(st) - t) >> 5));
			got = cas_relaxed(&h->sb_state[s], st, st - t);
		}
		if (kind == KMA_R_LOCK)
			got = cas_relaxed(cls_word(h, c, shard), 0, KMA_POISON);
		if (kind == KMA_R_TAKE) {
			if (got == st) {
				const uint32_t fr = st_free(st);
				if (fr == t)
					cas_relaxed(cls_word(h, c, shard), cur, 0);
				if (hint)
					hint[c] = cur;
				idle = 0;
				r.sb = s;
				r.left = t;
				r.cursor = fr - t; /* lowest of the t serial hints fr-1 .. fr-t */
				r.pre = false;
				r.knows = true;
				r.known = spec;
				r.hint = fr - 1;
			} else {
				tally(tl, KMA_T_CASFAIL);
			}
		}
		if (kind == KMA_R_LOCK && got != 0)
			kind = KMA_R_NONE;
		/* 4. claim bits of the word at the cursor; the result is used after
		 * the refills */
		uint32_t pick = 0, cand = 0, old = 0, word = 0;
		bool claims = open && r.left && !r.pre, sweeps = false;
		if (claims) {
			word = r.cursor >> 5;
			pick = claim_pick(h, r, c, slots, cand);
			/* a full warp looks over the other words at once */
			sweeps = sweep && (!r.knows || __popc(cand) < (int)r.left);
			claims = !sweeps;
			if (pick && claims)
				old = bm_or(bitmap_word(h, sb_addr(h, r.sb), word), pick);
		}
		/* 5. refills: superblocks for all leaders that need one */
		const bool refill = kind == KMA_R_LOCK || kind == KMA_R_OWN;
		if (__any_sync(active, refill)) {
			const int64_t f = sb_dequeue_lanes(h, active, refill);
			if (refill) {
				tally(tl, KMA_T_REFILL);
				if (f < 0) {
					if (kind == KMA_R_LOCK)
						atomicExch(cls_word(h, c, shard), 0);
					failed = true;
				} else {
					/* the refiller takes the top t slots, which are exactly
					 * the hints slots-1 .. slots-t of t serial reservations */
					t = want < slots ? want : slots;
					sb_format(h, (uint32_t)f, c, slots - t, slots - t, shard);
					const uint32_t pub = t == slots ? 0u : (uint32_t)f + KMA_CLS_BASE;
					/* release: a thread that finds f in the slot must find
					 * its bitmap and its state (a stale one would read as
					 * full and get f detached with free slots nobody can
					 * reach) */
					if (kind == KMA_R_LOCK)
						cas_release(cls_word(h, c, shard), KMA_POISON, pub);
					else if (pub)
						cas_release(cls_word(h, c, shard), 0, pub);
					if (hint && pub)
						hint[c] = pub;
					idle = 0;
					r.sb = (uint32_t)f;
					r.left = t;
					r.cursor = slots - t;
					r.hint = slots - 1;
					r.pre = true;
					r.knows = false;
				}
			}
		}
		/* 6. what was claimed: from the atomicOr of step 4, or the bits that
		 * a refill has set already */
		uint32_t bgot = 0;
		const uint32_t bbase = served, bhint = r.hint;
		if (claims) {
			tally(tl, KMA_T_CLAIM);
			bgot = pick & ~old;
			if (!bgot) {
				tally(tl, KMA_T_EMPTY);
				if (++idle > h->spin_limit) {
					failed = true;
					set_err(h, KMA_ERR_TIMEOUT | KMA_ERR_AT_WARP);
				}
			} else {
				idle = 0;
			}
			r.left -= __popc(bgot);
			if (pick) {
				r.knows = true;
				r.known = old | pick;
			}
			if (bgot == pick && r.left && pick == cand) {
				/* every candidate is ours and more are needed: move on.  What
				 * is known of this word may predate the reservation (the
				 * load beside it): the next visit, possibly of this same
				 * word after a wrap, claims afresh.  An atomicOr's result
				 * always shows at least `left` clear bits, which is what
				 * guarantees progress. */
				r.cursor = (word + 1) * 32;
				if (r.cursor >= slots)
					r.cursor = 0;
				r.knows = false;
			}
		} else if (leads && r.left && r.pre) {
			/* bits from the cursor up were set by sb_format */
			word = r.cursor >> 5;
			const uint32_t hi = slots < (word + 1) * 32 ? slots - word * 32 : 32u, lo = r.cursor & 31;
			const uint32_t n = hi - lo;
			bgot = (n == 32 ? 0xffffffffu : ((1u << n) - 1u)) << lo;
			r.cursor = word * 32 + hi;
			r.left -= n;
			tally(tl, KMA_T_CLAIM);
		}
		served += __popc(bgot);
		r.hint -= __popc(bgot);
		/* 7. hand them out: rank j of the claim takes the j-th highest bit,
		 * matching the serial hint order fr-1, fr-2, ... */
		const uint32_t gsb = __shfl_sync(active, r.sb, leader);
		const uint32_t gword = __shfl_sync(active, word, leader);
		const uint32_t ggot = __shfl_sync(active, bgot, leader);
		const uint32_t gbase = __shfl_sync(active, bbase, leader);
		const uint32_t ghint = __shfl_sync(active, bhint, leader);
		const bool gfail = __shfl_sync(active, (int)failed, leader);
		if (need) {
			const uint32_t n = __popc(ggot), j = rank - gbase;
			if (j < n) {
				const uint32_t slot = gword * 32 + nth_set_bit(ggot, n - 1 - j);
				unsigned char *p = sb_addr(h, gsb) + KMA_SB_HDR + (size_t)slot * h->cls_size[c];
				*reinterpret_cast<uint32_t *>(p) = ghint - j;
				res = p;
				need = false;
			} else if (gfail) {
				need = false;
			}
		}
		/* 8. reservations whose slots are not in one word: by the whole warp,
		 * one group after the other */
		bool swept = false;
		for (uint32_t m = sweep ? __ballot_sync(active, sweeps) : 0u; m; m &= m - 1) {
			const uint32_t l = __ffs(m) - 1;
			const uint32_t base = __shfl_sync(active, served, l);
			const uint32_t j = need && leader == l ? rank - base : 0xffffffffu;
			const sweep_got g = warp_sweep(h, __shfl_sync(active, r.sb, l), __shfl_sync(active, c, l),
						       __shfl_sync(active, r.cursor, l) >> 5, __shfl_sync(active, r.left, l),
						       j, __shfl_sync(active, r.hint, l));
			if (g.p) {
				res = g.p;
				need = false;
			}
			swept |= g.n != 0;
			if (lane == l) {
				tally(tl, KMA_T_CLAIM);
				if (!g.n) {
					tally(tl, KMA_T_EMPTY);
					if (++idle > h->spin_limit) {
						failed = true;
						set_err(h, KMA_ERR_TIMEOUT | KMA_ERR_AT_WARP);
					}
				} else {
					idle = 0;
				}
				r.left -= g.n;
				r.hint -= g.n;
				served += g.n;
				r.knows = false;
			}
		}
		/* nobody got anything and somebody waits */
		if (__any_sync(active, kind == KMA_R_WAIT) && !__any_sync(active, ggot != 0) && !swept)
			backoff(idle);
	}
	/* a leader's plain stores (a refill's bitmap and state) before its peers'
	 * use of the blocks */
	__syncwarp(active);
	return res;
}

/* The call: with the sweep, which any mix of sizes may need. */
__device__ inline void *kma_malloc_warp(kma_heap *h, size_t size, kma_tally *tl = nullptr, uint32_t *hint = nullptr)
{
	return kma_malloc_warp_t<true>(h, size, tl, hint);
}

__device__ inline void kma_free_warp(kma_heap *h, void *p)
{
	using namespace kma_detail;
	const uint32_t active = __activemask();
	const uint32_t lane = lane_id();
	uint32_t s = 0xffffffffu, c = 0, slot = 0;
	bool valid = false;
	if (p != NULL) {
		valid = block_locate(h, p, s, c, slot);
		if (!valid)
			set_err(h, KMA_ERR_BADFREE);
	}
	/* 1) clear bitmap bits: one atomicAnd per (superblock, word) */
	uint32_t word = slot >> 5;
	/* (a superblock of SB bytes has at most SB / 128 bitmap words, and a
	 * heap 2^31 of them: 256 GiB) */
	const uint32_t key = valid ? (s << (h->sb_log2 - 7)) | word : 0xffffffffu;
	uint32_t wpeers = __match_any_sync(active, key);
	uint32_t bit = valid ? (1u << (slot & 31)) : 0u;
	uint32_t mask = __reduce_or_sync(wpeers, bit);
	uint32_t wleader = __ffs(wpeers) - 1;
	uint32_t *wp = valid ? bitmap_word(h, sb_addr(h, s), word) : NULL;
	uint32_t old = 0;
	if (__popc(__ballot_sync(active, valid)) == 1) {
		/* one block: the reference's side effect, the bitmap word as it
		 * was before the clear, in word 0 of the block (kma.cl:338) --
		 * stored before the release, as in kma_free.  Every call of a
		 * one-thread-at-a-time execution takes this path. */
		if (valid) {
			uint32_t cur = ld_relaxed(wp);
			if (cur & bit) {
				*reinterpret_cast<volatile uint32_t *>(p) = cur;
				old = bm_and_release(wp, ~mask);
			} else {
				old = cur;
			}
		}
	} else if (valid && lane == wleader) {
		/* several blocks at once: freed memory has no defined contents,
		 * so the residue (a load, a store and a fence) is skipped */
		old = bm_and(wp, ~mask);
	}
	old = __shfl_sync(active, old, wleader);
	bool good = valid && (old & bit);
	if (valid && !good)
		set_err(h, KMA_ERR_BADFREE); /* double free, see kma_free */
	/* 2) return k slots to the superblock: one fetch-and-add per
	 * superblock, after the bits are clear (a count that reaches `slots`
	 * lets the superblock be recycled and reformatted) */
	uint32_t speers = __match_any_sync(active, good ? s : 0xffffffffu);
	uint32_t k = __popc(speers);
	uint32_t sleader = __ffs(speers) - 1;
	uint32_t full = 0;
	bool all_free = false;
	if (good && lane == sleader) {
		full = atomicAdd(&h->sb_state[s], k) + k;
		all_free = st_free(full) == st_slots(full);
	}
	/* 3) kma.cl:350-367: all free -- recycle */
	if (__any_sync(active, all_free))
		sb_recycle_lanes(h, active, all_free, s, c, full);
}

#endif /* KMA_DEVICE_CUH */
