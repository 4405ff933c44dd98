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
/* oldest first.  (Arrays: these calls are made from C, which no exception of a
 * container may reach.) */
kept g_kept[KMA_SCRATCH_LIST];
size_t g_n = 0, g_bytes = 0;

/* The driver's context calls. */
struct driver {
	CUresult (*get_id)(CUcontext, unsigned long long *);
	CUresult (*get)(CUcontext *);
	CUresult (*set)(CUcontext);
	CUresult (*retain)(CUcontext *, CUdevice);
	CUresult (*release)(CUdevice);
	CUresult (*state)(CUdevice, unsigned int *, int *);
	bool ok;

	driver() : ok(true)
	{
		find("cuCtxGetId", (void **)&get_id);
		find("cuCtxGetCurrent", (void **)&get);
		find("cuCtxSetCurrent", (void **)&set);
		find("cuDevicePrimaryCtxRetain", (void **)&retain);
		find("cuDevicePrimaryCtxRelease", (void **)&release);
		find("cuDevicePrimaryCtxGetState", (void **)&state);
	}
	void find(const char *name, void **f)
	{
		cudaDriverEntryPointQueryResult r;
		*f = NULL;
		if (cudaGetDriverEntryPoint(name, f, cudaEnableDefault, &r) != cudaSuccess)
			cudaGetLastError();
		else if (r != cudaDriverEntryPointSuccess)
			*f = NULL;
		ok = ok && *f;
	}
};
const driver &drv()
{
	static const driver d;
	return d;
}

/* A number of device dev's primary context, which no later one has, if that
 * is the current context; else 0, and then nothing is kept: another context
 * may end at any time, and its memory with it, without a sign. */
unsigned long long context_id(int dev)
{
	const driver &d = drv();
	CUcontext now = NULL, primary = NULL;
	unsigned long long id = 0;
	unsigned int flags;
	int active = 0;
	if (!d.ok || d.get(&now) != CUDA_SUCCESS || d.state(dev, &flags, &active) != CUDA_SUCCESS || !active ||
	    d.retain(&primary, dev) != CUDA_SUCCESS)
		return 0;
	d.release(dev);
	return now == primary && d.get_id(now, &id) == CUDA_SUCCESS ? id : 0;
}

void drop(size_t i)
{
	g_bytes -= g_kept[i].bytes;
	for (g_n--; i < g_n; i++)
		g_kept[i] = g_kept[i + 1];
}
bool full(size_t bytes) { return g_n == KMA_SCRATCH_LIST || g_bytes + bytes > KMA_SCRATCH_KEEP; }

} /* namespace */

void kma_scratch_trim(void)
{
	kept all[KMA_SCRATCH_LIST];
	size_t n;
	{
		std::lock_guard<std::mutex> lk(g_mu);
		for (size_t i = 0; i < g_n; i++)
			all[i] = g_kept[i];
		n = g_n;
		g_n = g_bytes = 0;
	}
	if (!n)
		return;
	const driver &d = drv();
	CUcontext now = NULL;
	if (d.get(&now) != CUDA_SUCCESS)
		return;
	for (size_t i = 0; i < n; i++) {
		const kept &k = all[i];
		/* (the memory of a context that was reset went with it) */
		unsigned int flags;
		int active = 0;
		if (d.state(k.device, &flags, &active) == CUDA_SUCCESS && active && cudaSetDevice(k.device) == cudaSuccess &&
		    context_id(k.device) == k.ctx)
			cudaFree(k.p);
	}
	d.set(now);
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
	if (n_ == KMA_SCRATCH_PER_CALL || cudaGetDevice(&dev) != cudaSuccess)
		return NULL;
	/* also brings the device's context up, where it is not */
	void *p = NULL;
	if (cudaFree(NULL) != cudaSuccess) {
		cudaGetLastError();
		return NULL;
	}
	const unsigned long long ctx = context_id(dev);
	{
		std::lock_guard<std::mutex> lk(g_mu);
		/* the smallest that fits */
		size_t best = g_n;
		for (size_t i = 0; i < g_n; i++)
			if (ctx && g_kept[i].device == dev && g_kept[i].ctx == ctx && g_kept[i].bytes >= bytes &&
			    (best == g_n || g_kept[i].bytes < g_kept[best].bytes))
				best = i;
		if (best < g_n) {
			p = g_kept[best].p;
			bytes = g_kept[best].bytes;
			drop(best);
		}
	}
	if (!p && kma_device_malloc(&p, bytes) != cudaSuccess) {
		cudaGetLastError();
		return NULL;
	}
	v_[n_++] = {p, bytes};
	return p;
}

kma_dev_bufs::~kma_dev_bufs()
{
	if (!n_)
		return;
	int dev = 0;
	/* nothing may still use them; after an error they are not kept.  (The
	 * calls work on the default stream: a wait for the whole device would
	 * break any capture that another thread has under way on it.) */
	const bool idle = cudaStreamSynchronize(NULL) == cudaSuccess && cudaGetDevice(&dev) == cudaSuccess;
	const unsigned long long ctx = idle ? context_id(dev) : 0;
	for (unsigned j = 0; j < n_; j++) {
		const buf &b = v_[j];
		void *gone[KMA_SCRATCH_LIST + 1];
		size_t ngone = 0;
		if (!ctx || b.bytes > KMA_SCRATCH_KEEP) {
			gone[ngone++] = b.p;
		} else {
			std::lock_guard<std::mutex> lk(g_mu);
			/* make room: the oldest of this context leave; others of the
			 * device are of primary contexts that were reset, and are
			 * forgotten as their memory is gone */
			for (size_t i = 0; i < g_n && full(b.bytes);) {
				if (g_kept[i].device == dev && g_kept[i].ctx != ctx) {
					drop(i);
				} else if (g_kept[i].device == dev) {
					gone[ngone++] = g_kept[i].p;
					drop(i);
				} else {
					i++;
				}
			}
			if (full(b.bytes)) {
				gone[ngone++] = b.p;
			} else {
				g_kept[g_n++] = {b.p, b.bytes, dev, ctx};
				g_bytes += b.bytes;
			}
		}
		for (size_t i = 0; i < ngone; i++)
			cudaFree(gone[i]);
	}
}
