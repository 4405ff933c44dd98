/*
 * kma_tree_check.cuh -- in-order check of a whole kma_cltree by all SMs
 * (kma_structs.cu, kma_graph.cu).
 *
 * The keys of an in-order walk increase strictly exactly when every node's
 * key lies in the open interval its ancestors leave it, so the walk need not
 * be one thread's: the tree is visited level by level, each entry of the
 * work list carrying its node's interval, and the list holds every reachable
 * node once.
 *
 * Bound: one dependent node load per level (a random tree of n keys has
 * about 4.3 ln n levels at most, 60 at a million) plus a grid barrier; the
 * node bytes themselves are a few percent of HBM time.  Levels narrower
 * than one block (the top ones, and every level of a degenerate tree) are
 * walked by block 0 alone, with block barriers only, so that a chain of n
 * nodes costs n loads as a serial walk does.  Measured on the tree of 2^21
 * mixed ops (0.6 M nodes): 0.16 ms, 254 ms by one thread with a stack; on a
 * graph of 20000 nodes 0.08 against 4.7 ms.
 */
#ifndef KMA_TREE_CHECK_CUH
#define KMA_TREE_CHECK_CUH

#include <cooperative_groups.h>

#include "kma_internal.h"
#include "kma_structs.cuh"

/* words of the result */
#define KMA_TC_LIVE 0     /* nodes not removed: their number, */
#define KMA_TC_XOR 1      /* the xor */
#define KMA_TC_SUM 2      /* and the sum of their keys */
#define KMA_TC_UNSORTED 3 /* nodes outside their interval */
#define KMA_TC_OVERFLOW 4 /* more nodes reachable than the list holds */
#define KMA_TC_COUNT 5    /* [3] entries pushed by a level, by level number mod 3 */
#define KMA_TC_BEGIN 8    /* the level block 0 stopped at: first entry */
#define KMA_TC_END 9      /* and end */
#define KMA_TC_WORDS 10

namespace {

const uint32_t TC_THREADS = 512;

/* One work-list entry: {node, lo | hi << 32}, lo <= key <= hi. */
__device__ __forceinline__ void tc_visit(ulonglong2 e, unsigned long long &live, unsigned long long &x,
		unsigned long long &sum, unsigned long long &unsorted, ulonglong2 &l, ulonglong2 &r)
{
	/* the three words by independent loads: one round trip per level */
	const unsigned long long *w = reinterpret_cast<const unsigned long long *>(e.x);
	const unsigned long long ks = __ldg(&w[0]);
	const unsigned long long left = __ldg(&w[1]), right = __ldg(&w[2]);
	const uint32_t key = (uint32_t)ks, lo = (uint32_t)e.y, hi = (uint32_t)(e.y >> 32);
	l.x = r.x = 0;
	if ((uint32_t)(ks >> 32) == 0) {
		live++;
		x ^= key;
		sum += key;
	}
	/* an empty interval, or a key outside it: nothing below is followed, so
	 * that a damaged tree ends too */
	if (key < lo || key > hi || (left && key == lo) || (right && key == hi)) {
		unsorted++;
		return;
	}
	l.x = left;
	l.y = (unsigned long long)lo | ((unsigned long long)(key - 1u) << 32);
	r.x = right;
	r.y = (unsigned long long)(key + 1u) | ((unsigned long long)hi << 32);
}

/* Append a warp's children behind `base`; every lane of the warp calls. */
__device__ __forceinline__ void tc_push(ulonglong2 *list, uint64_t cap, uint64_t base, unsigned long long *count,
		unsigned long long *overflow, ulonglong2 l, ulonglong2 r)
{
	const uint32_t full = 0xffffffffu, lt = kma_detail::lanemask_lt();
	const uint32_t ml = __ballot_sync(full, l.x != 0), mr = __ballot_sync(full, r.x != 0);
	if (!(ml | mr))
		return;
	unsigned long long at = 0;
	if (kma_detail::lane_id() == 0)
		at = atomicAdd(count, (unsigned long long)(__popc(ml) + __popc(mr)));
	at = base + __shfl_sync(full, at, 0);
	const uint64_t il = at + __popc(ml & lt), ir = at + __popc(ml) + __popc(mr & lt);
	if (l.x && il < cap)
		__stcg(&list[il], l);
	if (r.x && ir < cap)
		__stcg(&list[ir], r);
	if ((l.x && il >= cap) || (r.x && ir >= cap))
		atomicOr(overflow, 1ull);
}

__global__ void __launch_bounds__(TC_THREADS, 2) k_tree_check(const kma_cltree *t, ulonglong2 *list, uint64_t cap,
		unsigned long long *out)
{
	cooperative_groups::grid_group grid = cooperative_groups::this_grid();
	unsigned long long live = 0, x = 0, sum = 0, unsorted = 0;
	const uint64_t stride = (uint64_t)gridDim.x * TC_THREADS;
	uint64_t begin = 0, end = 1, level = 0;
	const unsigned long long root = t->root;
	if (!root || cap == 0)
		end = 0;
	else if (blockIdx.x == 0 && threadIdx.x == 0)
		__stcg(&list[0], make_ulonglong2(root, 0xffffffff00000000ull));
	grid.sync();
	/* begin, end and level are the same in every thread of the grid */
	while (begin < end) {
		if (end - begin <= TC_THREADS) {
			if (blockIdx.x == 0) {
				__shared__ unsigned long long s_count[3];
				if (threadIdx.x < 3)
					s_count[threadIdx.x] = 0;
				__syncthreads();
				for (uint32_t k = 0; begin < end && end - begin <= TC_THREADS; k++) {
					ulonglong2 l = make_ulonglong2(0, 0), r = l;
					if (begin + threadIdx.x < end)
						tc_visit(__ldcg(&list[begin + threadIdx.x]), live, x, sum, unsorted, l, r);
					/* cleared here, counted in the next level but one */
					if (threadIdx.x == 0)
						s_count[(k + 1) % 3] = 0;
					tc_push(list, cap, end, &s_count[k % 3], &out[KMA_TC_OVERFLOW], l, r);
					__syncthreads();
					begin = end;
					end += s_count[k % 3];
					end = end < cap ? end : cap;
				}
				if (threadIdx.x == 0) {
					__stcg(&out[KMA_TC_BEGIN], (unsigned long long)begin);
					__stcg(&out[KMA_TC_END], (unsigned long long)end);
				}
			}
			grid.sync();
			begin = __ldcg(&out[KMA_TC_BEGIN]);
			end = __ldcg(&out[KMA_TC_END]);
			/* nobody may rewrite the two words before all have read them */
			grid.sync();
		} else {
			unsigned long long *count = &out[KMA_TC_COUNT + level % 3];
			if (blockIdx.x == 0 && threadIdx.x == 0)
				__stcg(&out[KMA_TC_COUNT + (level + 1) % 3], 0ull);
			for (uint64_t i = begin + (uint64_t)blockIdx.x * TC_THREADS; i < end; i += stride) {
				ulonglong2 l = make_ulonglong2(0, 0), r = l;
				if (i + threadIdx.x < end)
					tc_visit(__ldcg(&list[i + threadIdx.x]), live, x, sum, unsorted, l, r);
				tc_push(list, cap, end, count, &out[KMA_TC_OVERFLOW], l, r);
			}
			grid.sync();
			begin = end;
			end += __ldcg(count);
			end = end < cap ? end : cap;
			level++;
		}
	}
	for (int d = 16; d > 0; d >>= 1) {
		live += __shfl_down_sync(0xffffffffu, live, d);
		x ^= __shfl_down_sync(0xffffffffu, x, d);
		sum += __shfl_down_sync(0xffffffffu, sum, d);
		unsorted += __shfl_down_sync(0xffffffffu, unsorted, d);
	}
	if ((threadIdx.x & 31) == 0) {
		if (live) {
			atomicAdd(&out[KMA_TC_LIVE], live);
			atomicXor(&out[KMA_TC_XOR], x);
			atomicAdd(&out[KMA_TC_SUM], sum);
		}
		if (unsorted)
			atomicAdd(&out[KMA_TC_UNSORTED], unsorted);
	}
}

/* Check tree t (quiescent) on stream st: list holds cap entries (16 bytes
 * each, 16-byte aligned; cap >= the nodes a sound tree can have), out
 * KMA_TC_WORDS words. */
inline int tree_check(const kma_cltree *t, void *list, uint64_t cap, unsigned long long *out, int device,
		cudaStream_t st)
{
	int per_sm = 0, sms = 0;
	KMA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tree_check, (int)TC_THREADS, 0));
	KMA_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
	if (per_sm < 1 || sms < 1)
		return KMA_ECUDA;
	/* no more blocks than there are nodes for: each takes part in every barrier */
	uint64_t nb = (cap + TC_THREADS - 1) / TC_THREADS;
	const uint64_t most = (uint64_t)per_sm * sms;
	nb = nb < 1 ? 1 : nb > most ? most : nb;
	KMA_CUDA(cudaMemsetAsync(out, 0, KMA_TC_WORDS * 8, st));
	ulonglong2 *l = (ulonglong2 *)list;
	void *args[] = {(void *)&t, (void *)&l, (void *)&cap, (void *)&out};
	KMA_CUDA(cudaLaunchCooperativeKernel((const void *)k_tree_check, dim3((unsigned)nb), dim3(TC_THREADS), args, 0,
					     st));
	return KMA_OK;
}

} /* namespace */

#endif /* KMA_TREE_CHECK_CUH */
