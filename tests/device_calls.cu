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
} /* namespace */

/* one lane replays ops through the warp calls, with hints */
extern "C" int t_replay_hint(kma_heap *h, const long long *ops, long long n, long long *out)
{
	k_replay_hint<<<1, 1>>>(h, ops, n, out);
	const cudaError_t e = cudaGetLastError();
	return e != cudaSuccess ? e : cudaDeviceSynchronize();
}
