/*
 * kma_scratch.h -- device scratch of the library's own host calls (replays,
 * the structure runs, the graph build).
 *
 * Those calls used to cudaMalloc their buffers and cudaFree them again.  Each
 * of the two maps or unmaps memory and waits for the device: 0.4 to 5 ms,
 * whatever the size, measured on a shared B200, so nine pairs were 20 of the
 * 28 ms of a 2^21-operation tree run.  dev_bufs takes its buffers from a list
 * of ones that earlier calls returned.
 *
 *   - bounded: at most KMA_SCRATCH_KEEP bytes per process, in at most
 *     KMA_SCRATCH_LIST buffers, stay on the list, the oldest leave first; a
 *     larger buffer is never kept;
 *   - given back: when a heap or a PMA heap is destroyed, when the program asks
 *     for it (kma_trim_scratch), and whenever an allocation of the library
 *     fails (kma_device_malloc empties the list and tries again);
 *   - a buffer belongs to one call at a time (the list is behind a mutex) and
 *     returns to the list only when the default stream, on which all of these
 *     calls work, is idle, so nothing can still use it;
 *   - only buffers of a device's primary context are kept, and used only in
 *     that one (it may be reset in between); calls that a program makes in a
 *     context of its own allocate and free.
 */
#ifndef KMA_SCRATCH_H
#define KMA_SCRATCH_H

#include <cuda_runtime.h>
#include <stddef.h>

#define KMA_SCRATCH_KEEP ((size_t)1 << 30)
#define KMA_SCRATCH_LIST 64     /* buffers on the list, at most */
#define KMA_SCRATCH_PER_CALL 8  /* buffers of one call, at most */

/* cudaMalloc on the current device; on failure once more with an empty list. */
cudaError_t kma_device_malloc(void **p, size_t bytes);
/* cudaFree every buffer on the list (of all devices). */
void kma_scratch_trim(void);

/* The buffers of one host call on the current device, all returned when it
 * goes out of scope.  For use on the default stream only. */
class kma_dev_bufs {
public:
	kma_dev_bufs() {}
	~kma_dev_bufs();
	kma_dev_bufs(const kma_dev_bufs &) = delete;
	kma_dev_bufs &operator=(const kma_dev_bufs &) = delete;
	/* NULL when out of memory, or past KMA_SCRATCH_PER_CALL; contents undefined */
	template <typename T>
	T *alloc(size_t bytes)
	{
		return (T *)take(bytes ? bytes : 1);
	}

private:
	struct buf {
		void *p;
		size_t bytes;
	};
	void *take(size_t bytes);
	buf v_[KMA_SCRATCH_PER_CALL];
	unsigned n_ = 0;
};

#endif
