/*
 * kma_scratch.cu -- see kma_scratch.h.
 */
#include <cuda.h>
#include <mutex>

#include "kma_scratch.h"

namespace {

struct kept {
	void *p;
	size_t bytes;
	int device;
	unsigned long long ctx;
};

std::mutex g_mu;
std::vector<kept> g_kept; /* oldest first */
size_t g_bytes = 0;

/* A number of the current context that no later one has (0: unknown, and
 * then nothing is kept). */
unsigned long long context_id()
{
	typedef CUresult (*get_id_t)(CUcontext, unsigned long long *);
	static get_id_t get_id = []() -> get_id_t {
		void *f = NULL;
		cudaDriverEntryPointQueryResult r;
		if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &r) != cudaSuccess) {
			cudaGetLastError();
			return NULL;
		}
		return r == cudaDriverEntryPointSuccess ? (get_id_t)f : NULL;
	}();
	unsigned long long id = 0;
	return get_id && get_id(NULL, &id) == CUDA_SUCCESS ? id : 0;
}

void drop(size_t i)
{
	g_bytes -= g_kept[i].bytes;
	g_kept.erase(g_kept.begin() + (ptrdiff_t)i);
}

} /* namespace */

void kma_scratch_trim(void)
{
	std::vector<kept> all;
	{
		std::lock_guard<std::mutex> lk(g_mu);
		all.swap(g_kept);
		g_bytes = 0;
	}
	if (all.empty())
		return;
	int prev = 0;
	if (cudaGetDevice(&prev) != cudaSuccess)
		return;
	for (const kept &k : all)
		if (cudaSetDevice(k.device) == cudaSuccess && context_id() == k.ctx)
			cudaFree(k.p);
	cudaSetDevice(prev);
	cudaGetLastError();
}

cudaError_t kma_device_malloc(void **p, size_t bytes)
{
	cudaError_t e = cudaMalloc(p, bytes);
	if (e == cudaErrorMemoryAllocation) {
		cudaGetLastError();
		kma_scratch_trim();
		e = cudaMalloc(p, bytes);
	}
	return e;
}

void *kma_dev_bufs::take(size_t bytes)
{
	int dev = 0;
	if (cudaGetDevice(&dev) != cudaSuccess)
		return NULL;
	/* also brings the device's context up, where it is not */
	void *p = NULL;
	if (cudaFree(NULL) != cudaSuccess) {
		cudaGetLastError();
		return NULL;
	}
	const unsigned long long ctx = context_id();
	{
		std::lock_guard<std::mutex> lk(g_mu);
		/* the smallest that fits */
		size_t best = g_kept.size();
		for (size_t i = 0; i < g_kept.size(); i++)
			if (ctx && g_kept[i].device == dev && g_kept[i].ctx == ctx && g_kept[i].bytes >= bytes &&
			    (best == g_kept.size() || g_kept[i].bytes < g_kept[best].bytes))
				best = i;
		if (best < g_kept.size()) {
			p = g_kept[best].p;
			bytes = g_kept[best].bytes;
			drop(best);
		}
	}
	if (!p && kma_device_malloc(&p, bytes) != cudaSuccess) {
		cudaGetLastError();
		return NULL;
	}
	v_.push_back({p, bytes});
	return p;
}

kma_dev_bufs::~kma_dev_bufs()
{
	if (v_.empty())
		return;
	int dev = 0;
	/* nothing may still use them; after an error they are not kept */
	const bool idle = cudaDeviceSynchronize() == cudaSuccess && cudaGetDevice(&dev) == cudaSuccess;
	const unsigned long long ctx = idle ? context_id() : 0;
	std::vector<void *> gone;
	{
		std::lock_guard<std::mutex> lk(g_mu);
		for (const buf &b : v_) {
			if (!ctx || b.bytes > KMA_SCRATCH_KEEP) {
				gone.push_back(b.p);
				continue;
			}
			/* make room: the oldest of this context leave, those of a
			 * context that is gone are forgotten with their memory */
			for (size_t i = 0; i < g_kept.size() && g_bytes + b.bytes > KMA_SCRATCH_KEEP;) {
				if (g_kept[i].device == dev && g_kept[i].ctx != ctx) {
					drop(i);
				} else if (g_kept[i].device == dev) {
					gone.push_back(g_kept[i].p);
					drop(i);
				} else {
					i++;
				}
			}
			if (g_bytes + b.bytes > KMA_SCRATCH_KEEP) {
				gone.push_back(b.p);
				continue;
			}
			g_kept.push_back({b.p, b.bytes, dev, ctx});
			g_bytes += b.bytes;
		}
	}
	for (void *p : gone)
		cudaFree(p);
}
