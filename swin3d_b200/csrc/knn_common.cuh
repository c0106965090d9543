// The pieces every KNN kernel shares: the reference's distance expression and its heap.
#pragma once
#include "common.cuh"

namespace s3d {

constexpr float KNN_FAR = 2147483648.0f;   // (float)0x7fffffff, the reference's initial heap entry

__device__ __forceinline__ void knn_sift_down(float *heap, int *idx, int start, int end)
{
    int curr = start;
    int child = curr * 2 + 1;
    while (child < end) {
        if (child + 1 < end && heap[child] < heap[child + 1]) child++;
        if (heap[curr] > heap[child]) return;
        const float tf = heap[curr]; heap[curr] = heap[child]; heap[child] = tf;
        const int ti = idx[curr]; idx[curr] = idx[child]; idx[child] = ti;
        curr = child;
        child = curr * 2 + 1;
    }
}

// fp32 squared distance.  The reference writes dx*dx + dy*dy + dz*dz and lets nvcc contract it;
// its compiled kernel (nvcc 12.9, default -fmad=true, sm_100) evaluates
// fma(dz,dz, fma(dx,dx, dy*dy)), established by comparing bit patterns of its output with the
// three possible contractions.  The expression is spelled with intrinsics so that it cannot
// drift with compiler versions; the GPU parity test re-checks it against the compiled reference.
__device__ __forceinline__ float knn_dist2(float dx, float dy, float dz)
{
    return __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
}

// The heap sort that ends the reference's scan: ascending distances.
__device__ __forceinline__ void knn_heap_sort(float *heap, int *idx, int K)
{
    for (int i = K - 1; i > 0; --i) {
        const float tf = heap[0]; heap[0] = heap[i]; heap[i] = tf;
        const int ti = idx[0]; idx[0] = idx[i]; idx[i] = ti;
        knn_sift_down(heap, idx, 0, i);
    }
}

// Scene of query g: the first whose end lies above g (the last one if there is none), and the sources
// [s0, s1) of that scene.
__device__ __forceinline__ int knn_scene(int64_t g, const int32_t *__restrict__ query_offset, int B)
{
    int b = 0;
    for (; b < B; ++b)
        if (g < __ldg(query_offset + b)) break;
    return b >= B ? B - 1 : b;
}

}  // namespace s3d
