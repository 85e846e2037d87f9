// Shared device/host helpers of libspmv_b200: error plumbing, PTX wrappers for the
// Blackwell bulk-copy engine (cp.async.bulk + mbarrier), small integer utilities.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "spmv_b200.h"

namespace spmv {

// ------------------------------------------------------------------ host error plumbing
void set_error(int code, const char * fmt, ...);
void clear_error();
int  last_status();

#define SPMV_CUDA_TRY(expr)                                                                      \
	do {                                                                                     \
		cudaError_t _e = (expr);                                                         \
		if (_e != cudaSuccess) {                                                         \
			cudaGetLastError();      /* reported here, not by the next launch's check */ \
			spmv::set_error(_e == cudaErrorMemoryAllocation ? SPMV_ERR_NOMEM : SPMV_ERR_CUDA, \
				"%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e), __FILE__, __LINE__); \
			return spmv::last_status();                                              \
		}                                                                                \
	} while (0)

#define SPMV_TRY(expr)                                                                           \
	do {                                                                                     \
		int _s = (expr);                                                                 \
		if (_s != SPMV_OK)                                                               \
			return _s;                                                               \
	} while (0)

// ------------------------------------------------------------------ device memory
// Stream-ordered allocations on the current device, from two pools per device of the library's
// own: one for scratch, one for the arrays of handles up to POOL_MOST_BYTES each (larger ones are
// plain allocations).  Mapping and unmapping memory cost a conversion more than its kernels, so
// each pool keeps up to POOL_KEEP_BYTES that nothing uses; the driver takes that back by itself
// when another allocation of the process, in a pool or a plain one, finds no memory.  (One pool for both, or larger arrays in it,
// put live arrays above the bound, and every synchronisation unmapped the scratch: 34 ms
// against 12 for a 2M-row SELL conversion.)  A SELL-C-sigma conversion of 8.5 M host entries with
// one SpMV: 12.8 ms with cudaMalloc and the default pool, 5.9 so.  The pools reuse what a stream
// has freed by waiting for that stream, without asking every live stream how far it is: a batch
// of 48 matrices (34 M entries) takes 46 ms to create with none or three others alive, 104 and
// 420 with the asking, 135 and 139 with cudaMalloc.
constexpr unsigned long long POOL_KEEP_BYTES = 512ULL << 20;
constexpr size_t POOL_MOST_BYTES = (size_t) 128 << 20;
enum class Pool { SCRATCH, HANDLE };
cudaError_t pool_alloc(void ** p, size_t bytes, Pool pool, cudaStream_t s);
// Bytes of the HANDLE pool that handles took (or gave back, < 0): its release threshold, which
// counts memory in use, is kept that far above.  With the bare bound, handles that held more had
// every synchronisation unmap what was free: 48 conversions beside 3.5 GB of other matrices spent
// 6.1 ms allocating and 8.0 freeing, 2.4 and 4.9 so.
void pool_live(int64_t bytes);
cudaError_t pools_trim();      // gives the unused memory of the current device's pools back

// While it lives, memory calls of this thread go through beside a stream capture, its own or
// another thread's, which they otherwise end.
struct BesideCapture {
	cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
	BesideCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
	~BesideCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// Device-side error word (one per handle): first error wins.
#define DEV_ERR_TIMEOUT 1
#define DEV_ERR_BOUNDS  2
#define DEV_ERR_FORMAT  3

__device__ __forceinline__ void dev_flag_error(int * err, int code)
{
	if (err)
		atomicCAS(err, 0, code);
}

// ------------------------------------------------------------------ bulk copy / mbarrier
__device__ __forceinline__ uint32_t smem_u32(const void * p)
{
	return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t * bar, uint32_t count)
{
	asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_fence_init()
{
	asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t * bar, uint32_t bytes)
{
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
	             : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t * bar)
{
	asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t * bar, uint32_t parity)
{
	uint32_t ok;
	asm volatile(
	    "{\n\t.reg .pred p;\n\t"
	    "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
	    "selp.u32 %0, 1, 0, p;\n\t}"
	    : "=r"(ok)
	    : "r"(smem_u32(bar)), "r"(parity)
	    : "memory");
	return ok != 0;
}

// try_wait that suspends the warp in hardware (up to `hint_ns` nanoseconds, or until the
// phase completes) instead of returning at once: a waiting warp takes no issue slots from
// the warps that work.
__device__ __forceinline__ bool mbar_try_wait_sleep(uint64_t * bar, uint32_t parity, uint32_t hint_ns)
{
	uint32_t ok;
	asm volatile(
	    "{\n\t.reg .pred p;\n\t"
	    "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
	    "selp.u32 %0, 1, 0, p;\n\t}"
	    : "=r"(ok)
	    : "r"(smem_u32(bar)), "r"(parity), "r"(hint_ns)
	    : "memory");
	return ok != 0;
}

// Bounded wait on an mbarrier phase: gives up after ~`budget` clock cycles and returns
// false (the caller records DEV_ERR_TIMEOUT and leaves), so no wait can spin forever.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t * bar, uint32_t parity, long long budget)
{
	if (mbar_try_wait(bar, parity))
		return true;
	long long t0 = clock64();
	while (!mbar_try_wait_sleep(bar, parity, 20000u)) {
		if (clock64() - t0 > budget)
			return false;
	}
	return true;
}

// Before a CTA (or warp) that gave up on a wait leaves: waits, bounded, for the `pending`
// bulk copies it issued that nobody has waited for, ring slots s, s+1, ... (mod S) from
// phase `parity` on, so that no copy is still writing into the shared memory of a CTA
// that has exited.  A slot whose copy already landed returns at once.
__device__ __forceinline__ void drain_ring(uint64_t * bars, int S, int s, uint32_t parity, int pending,
		long long budget)
{
	for (int q = 0; q < pending; q++) {
		(void) mbar_wait_bounded(&bars[s], parity, budget);
		if (++s == S) {
			s = 0;
			parity ^= 1u;
		}
	}
}

// Named barrier over n threads (a multiple of 32) of the CTA.
__device__ __forceinline__ void named_bar_sync(int id, int n)
{
	asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// Named barrier over n threads that also returns whether any of them passed `pred` true
// (so a decision to leave is taken by all of them together).
__device__ __forceinline__ bool named_bar_or(int id, int n, bool pred)
{
	uint32_t out;
	asm volatile(
	    "{\n\t.reg .pred p, q;\n\t"
	    "setp.ne.u32 p, %1, 0;\n\t"
	    "bar.red.or.pred q, %2, %3, p;\n\t"
	    "selp.u32 %0, 1, 0, q;\n\t}"
	    : "=r"(out)
	    : "r"((uint32_t) pred), "r"(id), "r"(n)
	    : "memory");
	return out != 0;
}

__device__ __forceinline__ void fence_proxy_async_smem()
{
	asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Global -> shared bulk copy (TMA, non-tensor form) completing on `bar`.
// Requirements: both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void * dst_smem, const void * src_gmem, uint32_t bytes, uint64_t * bar)
{
	asm volatile(
	    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
	        smem_u32(dst_smem)),
	    "l"(src_gmem), "r"(bytes), "r"(smem_u32(bar))
	    : "memory");
}

// Read-only path load of x (L1/texture path, stays in L2 across CTAs).
template <typename T>
__device__ __forceinline__ T ldg(const T * p)
{
	return __ldg(p);
}

// ------------------------------------------------------------------ overlapped launches
// A kernel launched with launch_overlapped() may start while the kernel before it in the stream
// still runs: from when all of that kernel's CTAs have begun and called release_next() (or have
// exited), or from its end.  Until wait_previous() returns, a thread may touch only what no
// earlier kernel of the stream writes (the matrix and its tables); x and y only after it, and x
// with load_x(), not through the read-only path, whose lines may date from before.
// Every CTA calls wait_previous(), so a kernel never ends before the one it overlapped.
// What it saves is the launch gap and the chain of table loads at a kernel's start: in a loop,
// csr_naive with 2,000 rows 8.2 -> 6.1 us a pass, with 100,000 8.2 -> 6.5, with 4M 200 -> 191,
// csr_vec 1M rows 95.3 -> 92.6, sell_sorted 700k rows 65.3 -> 61.4, FP32 4M rows 168 -> 161-165.
__device__ __forceinline__ void release_next()
{
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_previous()
{
	asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <typename T>
__device__ __forceinline__ T load_x(const T * p)
{
	return __ldca(p);
}
// An SM divides its memory between L1 and shared memory when it is idle.  Overlapped, the kernels that
// want much shared memory (the staged ones: their ring is dynamic) and those that want the L1 (row
// tiles, DIV-RF) would run on each other's division: SELL on 1 M rows and SELL-C-sigma on 40,000 in turn
// 82 us apart, 152 overlapped.  So a kernel overlaps one of its own kind, or where either has too few CTAs to
// matter: overlaps_last() notes the calling thread's last launch on a stream (a hint: what others launch there
// in between costs time, not results).
constexpr unsigned FEW_CTAS = 64;
bool overlaps_last(cudaStream_t s, bool staged, bool few);
template <typename A>
cudaError_t launch_overlapped(void (*kernel)(A), unsigned grid, unsigned threads, size_t smem, cudaStream_t s, const A & args)
{
	const bool overlap = overlaps_last(s, smem > 0, grid <= FEW_CTAS);
	cudaLaunchAttribute attr{};
	attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr.val.programmaticStreamSerializationAllowed = overlap;
	cudaLaunchConfig_t cfg{};
	cfg.gridDim = dim3(grid);
	cfg.blockDim = dim3(threads);
	cfg.dynamicSmemBytes = smem;
	cfg.stream = s;
	cfg.attrs = &attr;
	cfg.numAttrs = 1;
	return cudaLaunchKernelEx(&cfg, kernel, args);
}

// ------------------------------------------------------------------ misc
__host__ __device__ __forceinline__ int64_t ceil_div(int64_t a, int64_t b)
{
	return (a + b - 1) / b;
}

// x loads a gather thread of the warp-specialised kernels keeps in flight per round.
#ifndef SPMV_WS_GATHER_SLOTS
#define SPMV_WS_GATHER_SLOTS 4
#endif
static constexpr int WS_GATHER_SLOTS = SPMV_WS_GATHER_SLOTS;

static constexpr long long kWaitBudgetCycles = 4000000000LL;  // ~2 s at 1.9 GHz

// Bound of a device wait in clock cycles for a limit given in microseconds (0: the default
// ~2 s).  2,000 cycles a microsecond is at or above the B200's top SM clock (1,965 MHz), so
// a wait lasts at least the stated time.
__host__ __device__ __forceinline__ long long wait_budget_cycles(int limit_us)
{
	return limit_us > 0 ? (long long) limit_us * 2000LL : kWaitBudgetCycles;
}


}  // namespace spmv
