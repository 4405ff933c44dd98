/*
 * device_calls.cu -- kernels that call the device headers as a user's do, for
 * tests/test_device_calls.py.  Every entry returns a cudaError_t.
 */
#include <stdint.h>
#include "kma_device.cuh"
#include "kma_structs.cuh"

namespace {
__global__ void k_replay_hint(kma_heap *h, const long long *ops, long long n, long long *out)
{
	__shared__ uint32_t hint[KMA_MAX_CLASSES];
	for (int c = 0; c < KMA_MAX_CLASSES; c++)
		hint[c] = 0;
	for (long long i = 0; i < n; i++) {
		const long long kind = ops[2 * i], arg = ops[2 * i + 1];
		if (kind == 0) {
			const size_t sz = arg < 0 ? ~(size_t)0 : (size_t)arg;
			unsigned char *p = (unsigned char *)kma_malloc_warp(h, sz, nullptr, hint);
			out[i] = p ? (long long)(p - h->sb_base) : -1;
		} else {
			kma_free_warp(h, arg >= 0 && arg < i && out[arg] >= 0 ? h->sb_base + out[arg] : nullptr);
			out[i] = 0;
		}
	}
}

/* One thread, lane `lane` of warp `warp` of the grid, mallocs up to `count`
 * blocks of n bytes, until it is refused one. */
__global__ void k_malloc_at(kma_heap *h, unsigned warp, unsigned lane, unsigned n, unsigned count, unsigned *got)
{
	if (blockIdx.x != warp || threadIdx.x != lane)
		return;
	unsigned k = 0;
	while (k < count && kma_malloc(h, n))
		k++;
	*got = k;
}

/* One warp: lane 0 puts n items on each of nq queues, the head of each then
 * held for good if `stuck`; every lane takes one from queue lane % nq, with an
 * error word of its own and a limit that `step` makes differ.  out: the item's
 * number in its queue, -1 for none. */
__global__ void k_lanes_dequeue(kma_clqueue *q, unsigned long long *items, int nq, int n, int stuck, uint32_t step,
		int *out, uint32_t *err)
{
	const int lane = threadIdx.x;
	if (lane == 0)
		for (int k = 0; k < nq; k++) {
			kma_clqueue_init(&q[k]);
			for (int i = 0; i < n; i++)
				kma_clqueue_enqueue(&q[k], reinterpret_cast<kma_clqueue_item *>(&items[2 * (k * n + i)]));
			if (stuck)
				items[2 * k * n] = kma_q::POISON;
		}
	__syncwarp();
	unsigned long long *it = reinterpret_cast<unsigned long long *>(
		kma_clqueue_dequeue(&q[lane % nq], &err[lane], 1024u + step * (lane % 3)));
	out[lane] = it ? (int)((it - items) / 2) - (lane % nq) * n : -1;
}

/* a user's kernels of one per-thread dequeue each, without launch bounds */
__global__ void k_user_clqueue(kma_clqueue *q, unsigned long long *sum)
{
	kma_clqueue_item *it = kma_clqueue_dequeue(q + threadIdx.x % 7);
	if (it)
		atomicAdd(sum, reinterpret_cast<unsigned long long *>(it)[1]);
}
__global__ void k_user_iqueue(kma_iqueue *q, unsigned long long *sum)
{
	void *it = kma_iqueue_dequeue(q);
	if (it)
		atomicAdd(sum, reinterpret_cast<unsigned long long *>(it)[1]);
}
} /* namespace */

extern "C" int t_malloc_at(kma_heap *h, unsigned warp, unsigned lane, unsigned n, unsigned count, unsigned *got)
{
	k_malloc_at<<<warp + 1, 32>>>(h, warp, lane, n, count, got);
	const cudaError_t e = cudaGetLastError();
	return e != cudaSuccess ? e : cudaDeviceSynchronize();
}

extern "C" int t_lanes_dequeue(void *q, unsigned long long *items, int nq, int n, int stuck, uint32_t step, int *out,
		uint32_t *err)
{
	k_lanes_dequeue<<<1, 32>>>((kma_clqueue *)q, items, nq, n, stuck, step, out, err);
	const cudaError_t e = cudaGetLastError();
	return e != cudaSuccess ? e : cudaDeviceSynchronize();
}

extern "C" void t_user_kernels(kma_clqueue *q, kma_iqueue *iq, unsigned long long *sum)
{
	k_user_clqueue<<<1, 1024>>>(q, sum);
	k_user_iqueue<<<1, 1024>>>(iq, sum);
}

/* one lane replays ops through the warp calls, with hints */
extern "C" int t_replay_hint(kma_heap *h, const long long *ops, long long n, long long *out)
{
	k_replay_hint<<<1, 1>>>(h, ops, n, out);
	const cudaError_t e = cudaGetLastError();
	return e != cudaSuccess ? e : cudaDeviceSynchronize();
}
