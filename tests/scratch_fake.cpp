/*
 * scratch_fake.cpp -- kma_b200/csrc/kma_scratch.cu over a CUDA runtime and
 * driver made up here, for tests/test_scratch_host.py: two devices, each with
 * a primary context that may be reset and any number of others, memory that
 * belongs to a context, and captures that a device-wide wait breaks.
 *
 *   scratch_fake SCENARIO     prints what went wrong; exits 0 when nothing did
 */
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <new>

#include "kma_scratch.h"

struct CUctx_st {
	unsigned long long id;
	int device;
	bool alive;
	std::map<void *, size_t> mem;
};

static int bad = 0;
#define CHECK(x) ((x) ? 0 : (printf("line %d: %s\n", __LINE__, #x), bad++))

static unsigned long long next_id = 1;
static CUctx_st *primary[2];
static CUctx_st *current;
static int device_now;
static bool capturing, capture_broken;
static int fail_new = -1; /* allocations of the host until one fails */
static size_t device_bytes = (size_t)8 << 30;

static CUctx_st *primary_of(int d)
{
	if (!primary[d])
		primary[d] = new CUctx_st{next_id++, d, true, {}};
	if (!primary[d]->alive) { /* reset: the same handle, another id */
		primary[d]->alive = true;
		primary[d]->id = next_id++;
	}
	return primary[d];
}
static void reset_primary(int d)
{
	primary[d]->mem.clear();
	primary[d]->alive = false;
}
static size_t live(CUctx_st *c) { return c ? c->mem.size() : 0; }

void *operator new(size_t n)
{
	if (fail_new >= 0 && fail_new-- == 0)
		throw std::bad_alloc();
	return malloc(n);
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

extern "C" {
static CUctx_st *working() { return current ? current : current = primary_of(device_now); }
cudaError_t cudaGetDevice(int *d)
{
	*d = current ? current->device : device_now;
	return cudaSuccess;
}
cudaError_t cudaSetDevice(int d)
{
	device_now = d;
	current = primary_of(d);
	return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n)
{
	const int armed = fail_new;
	fail_new = -1;
	CUctx_st *c = working();
	size_t used = 0;
	for (auto &m : c->mem)
		used += m.second;
	cudaError_t e = cudaErrorMemoryAllocation;
	if (used + n <= device_bytes) {
		static uintptr_t at = 4096;
		*p = (void *)at;
		at += (n + 4095) / 4096 * 4096;
		c->mem[*p] = n;
		e = cudaSuccess;
	}
	fail_new = armed;
	return e;
}
cudaError_t cudaFree(void *p)
{
	CUctx_st *c = working();
	if (!p)
		return cudaSuccess;
	return c->mem.erase(p) ? cudaSuccess : (CHECK(!"freed in a context that does not have it"), cudaErrorInvalidValue);
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize()
{
	if (capturing) {
		capture_broken = true;
		return cudaErrorStreamCaptureUnsupported;
	}
	return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }

static CUresult get_id(CUcontext c, unsigned long long *id)
{
	*id = (c ? c : current)->id;
	return CUDA_SUCCESS;
}
static CUresult get_current(CUcontext *c)
{
	*c = current;
	return CUDA_SUCCESS;
}
static CUresult set_current(CUcontext c)
{
	current = c;
	return CUDA_SUCCESS;
}
static CUresult retain(CUcontext *c, CUdevice d)
{
	*c = primary_of(d);
	return CUDA_SUCCESS;
}
static CUresult release(CUdevice) { return CUDA_SUCCESS; }
static CUresult state(CUdevice d, unsigned *flags, int *active)
{
	*flags = 0;
	*active = primary[d] && primary[d]->alive;
	return CUDA_SUCCESS;
}
cudaError_t cudaGetDriverEntryPoint(const char *name, void **f, unsigned long long, cudaDriverEntryPointQueryResult *r)
{
	static const struct {
		const char *name;
		void *f;
	} all[] = {{"cuCtxGetId", (void *)get_id},		 {"cuCtxGetCurrent", (void *)get_current},
		   {"cuCtxSetCurrent", (void *)set_current},	 {"cuDevicePrimaryCtxRetain", (void *)retain},
		   {"cuDevicePrimaryCtxRelease", (void *)release}, {"cuDevicePrimaryCtxGetState", (void *)state}};
	*f = nullptr;
	for (auto &a : all)
		if (!strcmp(a.name, name))
			*f = a.f;
	*r = *f ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
	return cudaSuccess;
}
}

/* one host call: two buffers */
static void *call(size_t a, size_t b)
{
	kma_dev_bufs bufs;
	char *p = bufs.alloc<char>(a), *q = bufs.alloc<char>(b);
	CHECK(p && q && p != q);
	CHECK(!p || working()->mem.count(p));
	return p;
}

/* a context of the program's own beside the primary one */
static void contexts()
{
	CUctx_st *mine = new CUctx_st{next_id++, 0, true, {}};
	for (int i = 0; i < 3; i++) {
		current = mine;
		call(1000, 3000);
		CHECK(current == mine);
		current = primary_of(0);
		call(1000, 3000);
		CHECK(current == primary[0]);
	}
	current = mine;
	kma_scratch_trim();
	CHECK(current == mine);
	CHECK(live(mine) == 0);
	CHECK(live(primary[0]) == 0);
}
/* a primary context that is reset between calls, and a device never used */
static void reset()
{
	cudaSetDevice(0);
	call(5000, 100);
	CHECK(live(primary[0]) == 2);
	reset_primary(0);
	current = nullptr;
	call(5000, 100);
	kma_scratch_trim();
	CHECK(live(primary[0]) == 0);
	call(5000, 100);
	reset_primary(0);
	current = nullptr;
	kma_scratch_trim();
	CHECK(!primary[0]->alive && !primary[1]);
}
static void two_devices()
{
	cudaSetDevice(0);
	void *p = call(7000, 100);
	cudaSetDevice(1);
	call(7000, 100);
	cudaSetDevice(0);
	CHECK(call(7000, 100) == p);
	kma_scratch_trim();
	CHECK(current == primary[0] && live(primary[0]) == 0 && live(primary[1]) == 0);
}
/* another thread captures a graph on the device meanwhile */
static void capture()
{
	cudaSetDevice(0);
	capturing = true;
	void *p = call(7000, 100);
	CHECK(call(7000, 100) == p);
	CHECK(!capture_broken);
}
/* the host is out of memory: no exception leaves a call, nothing is lost */
static void no_host_memory()
{
	cudaSetDevice(0);
	for (int n = 0; n < 12; n++)
		for (int before = 0; before < 2; before++) {
			if (before)
				call(1 << 20, 100);
			{
				kma_dev_bufs bufs;
				fail_new = n;
				char *p = bufs.alloc<char>(1 << 20);
				char *q = p ? bufs.alloc<char>((1 << 20) + n) : nullptr;
				CHECK(!p || live(primary[0]) >= 1);
				(void)q;
			}
			fail_new = -1;
			kma_scratch_trim();
			CHECK(live(primary[0]) == 0);
		}
}
static void bounded()
{
	cudaSetDevice(0);
	for (int i = 0; i < 10; i++)
		call((size_t)300 << 20, (size_t)200 << 20);
	call((size_t)2 << 30, 1);
	size_t kept = 0;
	for (auto &m : primary[0]->mem)
		kept += m.second;
	CHECK(kept <= KMA_SCRATCH_KEEP);
	/* an allocation of the library that needs what is kept */
	void *p = nullptr;
	CHECK(kma_device_malloc(&p, device_bytes) == cudaSuccess);
}

int main(int argc, char **argv)
{
	static const struct {
		const char *name;
		void (*run)();
	} all[] = {{"contexts", contexts}, {"reset", reset}, {"two_devices", two_devices}, {"capture", capture},
		 {"no_host_memory", no_host_memory}, {"bounded", bounded}};
	for (auto &s : all)
		if (argc == 2 && !strcmp(argv[1], s.name)) {
			s.run();
			return bad != 0;
		}
	return 2;
}
