// Asynchronous staging primitives (sm_80+/sm_90+): mbarrier objects in shared memory and 16-byte asynchronous copies
// global -> this block's shared memory (cp.async) whose completion arrives on an mbarrier.  Every copy here reads the
// launching GPU's own global memory and lands in the issuing block's shared memory.
//
// Every wait is bounded: mbar_wait gives up after MBAR_WAIT_TRIES polls and returns false, and the
// kernels then leave their loops through a block-uniform flag and set g_async_error (s3d_async_error()).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace s3d {

constexpr int MBAR_WAIT_TRIES = 1 << 22;

// Set when a bounded wait of this file's kernels ran out (it never should); one word per including source file.
static __device__ int g_async_error;

// Whether it is set on the current device, and clears it.  Waits for the device.
static inline cudaError_t take_async_error(bool &set)
{
    int v = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_async_error, sizeof(v));
    set = e == cudaSuccess && v != 0;
    if (set) {
        v = 0;
        e = cudaMemcpyToSymbol(g_async_error, &v, sizeof(v));
    }
    return e;
}

__device__ __forceinline__ uint32_t smem_addr(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

// Makes the initialised barriers visible to the asynchronous proxy.
__device__ __forceinline__ void mbar_init_fence()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// true once the phase with the given parity has completed, false if it did not within the bound.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity)
{
    for (int i = 0; i < MBAR_WAIT_TRIES; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// 16 bytes global -> shared by the load/store unit, without a register in between; zeros where !valid (src is not read).
// A row piece of 32 or 64 bytes is too small for the bulk copy engine: one bulk copy per row and array, 64 to 128 of
// them per item, took the producer warp longer than the consumers' work on the smaller items.
__device__ __forceinline__ void cp_async16(void *dst_smem, const void *src_gmem, bool valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst_smem)), "l"(src_gmem), "r"(valid ? 16 : 0) : "memory");
}

// One arrival on the barrier (counted in its initial count) once this thread's earlier cp_async16 have landed.
__device__ __forceinline__ void mbar_arrive_cp_async(uint64_t *bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// A warp fetches 32 rows of PIECES 16-byte pieces: row r (lane r holds its row number) from src + row * row_elems, to
// dst + r * dst_elems; rows from n on become zeros.
template <int PIECES, typename T>
__device__ __forceinline__ void stage_rows(T *dst, int dst_elems, const T *src, int64_t row_elems, int row, int n, int lane)
{
    constexpr int PER = 16 / sizeof(T);
#pragma unroll
    for (int i = 0; i < PIECES; ++i) {
        const int c = lane + 32 * i, r = c / PIECES, e = c % PIECES * PER;
        const int64_t from = __shfl_sync(0xffffffffu, row, r);
        cp_async16(dst + r * dst_elems + e, src + from * row_elems + e, r < n);
    }
}

// Barrier among the first `count` threads of the block (a multiple of 32), id 1; the producer warp,
// which runs ahead, does not take part.
template <int COUNT>
__device__ __forceinline__ void consumer_sync()
{
    asm volatile("bar.sync 1, %0;" ::"n"(COUNT) : "memory");
}

}  // namespace s3d
