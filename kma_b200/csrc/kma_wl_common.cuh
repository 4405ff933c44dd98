/*
 * kma_wl_common.cuh -- device helpers shared by the workload kernels
 * (kma_workload.cu, kma_batch.cu, kma_serve.cu): the SplitMix64 PRNG, the
 * ordered offset hash, and the warp-cooperative tag fill / verify of
 * payload blocks.
 */
#ifndef KMA_WL_COMMON_CUH
#define KMA_WL_COMMON_CUH

#include <stdint.h>

namespace kma_wl {

const uint64_t SPLITMIX_STEP = 0x9E3779B97F4A7C15ull;
__device__ __forceinline__ uint64_t splitmix(uint64_t &s)
{
	uint64_t z = (s += SPLITMIX_STEP);
	z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
	z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
	return z ^ (z >> 31);
}

__device__ __forceinline__ uint64_t hash_step(uint64_t h, int64_t off)
{
	return h ^ ((uint64_t)off + 0x9E3779B97F4A7C15ull + (h << 6) + (h >> 2));
}

/* Cache policy of the payload words (tag fill and verify): 0 default,
 * 1 at L2 only (.cg), 2 streaming (.cs: evict first).  Streaming both
 * measured 1-2% faster on config 2's rounds kernel than the default;
 * .cg loads alone 1.4% slower. */
#ifndef WL_PAYLOAD_LD
#define WL_PAYLOAD_LD 2
#endif
#ifndef WL_PAYLOAD_ST
#define WL_PAYLOAD_ST 2
#endif
template <class T>
__device__ __forceinline__ T pl_ld(const T *p)
{
#if WL_PAYLOAD_LD == 1
	return __ldcg(p);
#elif WL_PAYLOAD_LD == 2
	return __ldcs(p);
#else
	return *p;
#endif
}
template <class T>
__device__ __forceinline__ void pl_st(T *p, T v)
{
#if WL_PAYLOAD_ST == 1
	__stcg(p, v);
#elif WL_PAYLOAD_ST == 2
	__stcs(p, v);
#else
	*p = v;
#endif
}
/* Blocks of at least this many bytes are filled by the whole warp, one row of
 * consecutive 16-byte stores after the other; below, a lane's own loop is
 * shorter than the shuffles.  A loop of its own for every block (a warp's
 * largest decides how long) took 3.16 instead of 2.81 ms for 24 jobs on the
 * bump heap and 7.77 instead of 7.49 for config 2; from 128 / 256 / 1024 bytes
 * up config 2 took 7.52 / 7.47 / 7.48 ms, the per-thread program of 50021
 * items 1.80 / 1.74 / 1.67 (1.70 at 512). */
#ifndef WL_FILL_BYTES
#define WL_FILL_BYTES 512u
#endif
/* Tag fill of every calling lane's block (p may be NULL). */
__device__ __forceinline__ void coop_fill(uint32_t mask, uint32_t lane, void *p, uint32_t n, uint32_t tag)
{
	uint32_t *w = (uint32_t *)p;
	const bool big = p && n >= WL_FILL_BYTES;
	const uint32_t nw = p ? n >> 2 : 0u;
	uint32_t head = (uint32_t)((16u - ((uintptr_t)p & 15u)) & 15u) >> 2;
	head = head < nw ? head : nw;
	const uint32_t nv = (nw - head) >> 2, t0 = head + 4 * nv;
	uint4 *v = reinterpret_cast<uint4 *>(w + head);
	const uint4 t4 = make_uint4(tag, tag, tag, tag);
#pragma unroll
	for (uint32_t i = 0; i < 3; i++) {
		if (i < head)
			pl_st(&w[i], tag);
		if (t0 + i < nw)
			pl_st(&w[t0 + i], tag);
	}
	const uint32_t own = big ? 0u : nv;
#pragma unroll 4
	for (uint32_t k = 0; k < own; k++)
		pl_st(&v[k], t4);
	const uint32_t width = __popc(mask), rank = __popc(mask & ((1u << lane) - 1u));
	for (uint32_t mb = __ballot_sync(mask, big); mb; mb &= mb - 1) {
		const uint32_t j = __ffs(mb) - 1;
		uint4 *vj = (uint4 *)__shfl_sync(mask, (unsigned long long)v, j) + rank;
		const uint32_t nj = __shfl_sync(mask, nv, j), t = __shfl_sync(mask, tag, j);
		const uint4 tj = make_uint4(t, t, t, t);
#pragma unroll 4
		for (uint32_t k = rank; k < nj; k += width, vj += width)
			pl_st(vj, tj);
	}
}

/* Blocks of at least this many bytes are verified by the whole warp (64 jobs:
 * 35.1 ms at 128, 35.6 at 256, 36.9 at 512; config 2 within 1%). */
#ifndef WL_COOP_BYTES
#define WL_COOP_BYTES 128u
#endif

/* Vectors each lane has in flight per batch of coop_verify: config 2
 * (64 registers) took 6.58 / 6.53 / 6.83 / 6.96 ms at 2 / 3 / 4 / 5; deeper
 * batches cost more spills than they hide latency. */
#ifndef WL_VERIFY_SLOTS
#define WL_VERIFY_SLOTS 3
#endif
/* Vectors of its own small block that a lane has in flight, beside the words
 * before and after them: 6.86 / 6.53 / 6.74 ms at 2 / 4 / 5. */
#ifndef WL_SMALL_SLOTS
#define WL_SMALL_SLOTS 4
#endif

/* Verify every lane's block (p may be NULL) against its tag; true in the
 * owner lane of a block with a word that differs.  Every lane of `mask`
 * calls it.
 *
 * Small blocks, and the few words of any block before and after its 16-byte
 * aligned body: the owner reads its own, every load issued before the first
 * is compared (word by word and vector by vector, a lane with 64 bytes had up
 * to nine round trips in a row; config 2 took 7.54 ms, with this and the fill
 * above 6.59).
 * Blocks of WL_COOP_BYTES or more: their 16-byte aligned bodies are cut
 * into rows of one vector per calling lane, rows of all big blocks laid
 * end to end in lane order; the r-th calling lane reads vector r of each
 * row.  A batch is the next
 * SLOTS rows, whichever blocks they belong to: every lane issues
 * all the batch's loads before it compares any, so a pass over the warp's
 * blocks costs one memory round trip per batch rather than one per block
 * (a loop over blocks consumes each block's loads before it can issue the
 * next block's).  The row schedule is the same in every lane, so which
 * block a row belongs to, its base and its tag are broadcast by shuffles. */
template <int SLOTS = WL_VERIFY_SLOTS>
__device__ __forceinline__ bool coop_verify(uint32_t mask, uint32_t lane, const void *p, uint32_t n,
		uint32_t tag)
{
	const uint32_t *w = (const uint32_t *)p;
	const bool big = p && n >= WL_COOP_BYTES;
	const uint32_t nw = p ? n >> 2 : 0u;
	uint32_t head = (uint32_t)((16u - ((uintptr_t)p & 15u)) & 15u) >> 2;
	head = head < nw ? head : nw;
	const uint32_t nv = (nw - head) >> 2;
	uint32_t bad = 0;
	if (p) {
		/* head and tail words and (small blocks) the body, four vectors at a
		 * time: every load is issued before the first is compared */
		const uint4 *v = reinterpret_cast<const uint4 *>(w + head);
		const uint32_t t0 = head + 4 * nv, own = big ? 0u : nv;
		uint32_t e[6];
		uint4 x[WL_SMALL_SLOTS];
#pragma unroll
		for (uint32_t i = 0; i < 3; i++) {
			e[i] = i < head ? pl_ld(&w[i]) : tag;
			e[3 + i] = t0 + i < nw ? pl_ld(&w[t0 + i]) : tag;
		}
		uint32_t k = 0;
		do {
#pragma unroll
			for (uint32_t i = 0; i < WL_SMALL_SLOTS; i++) {
				x[i] = make_uint4(tag, tag, tag, tag);
				if (k + i < own)
					x[i] = pl_ld(&v[k + i]);
			}
#pragma unroll
			for (uint32_t i = 0; i < WL_SMALL_SLOTS; i++)
				bad |= (x[i].x ^ tag) | (x[i].y ^ tag) | (x[i].z ^ tag) | (x[i].w ^ tag);
			k += WL_SMALL_SLOTS;
		} while (k < own);
#pragma unroll
		for (uint32_t i = 0; i < 6; i++)
			bad |= e[i] ^ tag;
	}
	uint32_t mb = __ballot_sync(mask, big);
	uint32_t badbits = 0;
	const uint32_t width = __popc(mask), rank = __popc(mask & ((1u << lane) - 1u));
	/* the block whose rows are being scheduled (warp-uniform) */
	const uint4 *cb = nullptr;
	uint32_t cj = 0, cnv = 0, crow = 0, crows = 0;
	while (mb || crow < crows) {
		uint4 x[SLOTS];
		uint32_t sj[SLOTS];
		uint32_t valid = 0;
#pragma unroll
		for (int s = 0; s < SLOTS; s++) {
			if (crow >= crows && mb) {
				cj = __ffs(mb) - 1;
				mb &= mb - 1;
				const uint32_t *pj = (const uint32_t *)__shfl_sync(mask, (unsigned long long)w, cj);
				cnv = __shfl_sync(mask, nv, cj);
				const uint32_t hj = __shfl_sync(mask, head, cj);
				cb = reinterpret_cast<const uint4 *>(pj + hj);
				crow = 0;
				crows = (cnv + width - 1) / width;
			}
			sj[s] = cj;
			x[s] = make_uint4(0, 0, 0, 0);
			if (crow < crows) {
				const uint32_t k = crow * width + rank;
				if (k < cnv) {
					x[s] = pl_ld(&cb[k]);
					valid |= 1u << s;
				}
				crow++;
			}
		}
#pragma unroll
		for (int s = 0; s < SLOTS; s++) {
			const uint32_t tj = __shfl_sync(mask, tag, sj[s]);
			const uint32_t d = (x[s].x ^ tj) | (x[s].y ^ tj) | (x[s].z ^ tj) | (x[s].w ^ tj);
			if (((valid >> s) & 1u) && d)
				badbits |= 1u << sj[s];
		}
	}
	badbits = __reduce_or_sync(mask, badbits);
	return bad != 0 || ((badbits >> lane) & 1u);
}

/* Position of the (k+1)-th set bit of m; requires k < popc(m). */
__device__ __forceinline__ uint32_t nth_bit(uint32_t m, uint32_t k)
{
	uint32_t pos = 0;
#pragma unroll
	for (uint32_t s = 16; s; s >>= 1) {
		uint32_t lo = __popc(m & ((1u << s) - 1u));
		if (k >= lo) {
			k -= lo;
			m >>= s;
			pos += s;
		}
	}
	return pos;
}

/* Packed numbering of a full warp's work bits: the set bits of every
 * lane's `bits`, in lane order and within a lane in increasing bit index,
 * are numbered 0..total-1 by a warp prefix sum, so that pass k serves
 * numbers 32k..32k+31 with lane l taking number 32k+l.  Used for the
 * frees of a round: one pass per set bit of the busiest lane would leave
 * most lanes idle through about twice as many passes, each a chain of
 * dependent round trips (table load, payload loads, free atomics). */
struct warp_pack {
	uint32_t bits, excl, incl, total;
};

/* Every lane of the warp calls it. */
__device__ __forceinline__ warp_pack warp_pack_init(uint32_t lane, uint32_t bits)
{
	warp_pack wp;
	wp.bits = bits;
	const uint32_t c = __popc(bits);
	uint32_t incl = c;
#pragma unroll
	for (uint32_t o = 1; o < 32; o <<= 1) {
		uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
		if (lane >= o)
			incl += v;
	}
	wp.incl = incl;
	wp.excl = incl - c;
	wp.total = __shfl_sync(0xffffffffu, incl, 31);
	return wp;
}

/* Lane `lane`'s number in the pass starting at `base` (a multiple of 32
 * below total): true with the lane that owns it and its bit index, or
 * false (owner = lane) when the pass has no number for this lane.  Every
 * lane of the warp calls it. */
__device__ __forceinline__ bool warp_pack_slot(const warp_pack &wp, uint32_t lane, uint32_t base, uint32_t &owner,
		uint32_t &bit)
{
	const uint32_t full = 0xffffffffu;
	/* lanes owning numbers in this pass, and the pass slot of each one's
	 * first number (distinct slots, increasing with the lane) */
	const bool in = wp.incl > wp.excl && wp.excl < base + 32 && wp.incl > base;
	const uint32_t lanes = __ballot_sync(full, in);
	const uint32_t starts = __reduce_or_sync(full, in ? 1u << (wp.excl > base ? wp.excl - base : 0u) : 0u);
	const uint32_t s = base + lane;
	const bool mine = s < wp.total;
	owner = mine ? nth_bit(lanes, __popc(starts & (full >> (31 - lane))) - 1) : lane;
	const uint32_t o_excl = __shfl_sync(full, wp.excl, owner);
	const uint32_t o_bits = __shfl_sync(full, wp.bits, owner);
	bit = mine ? nth_bit(o_bits, s - o_excl) : 0u;
	return mine;
}

} /* namespace kma_wl */

#endif /* KMA_WL_COMMON_CUH */
