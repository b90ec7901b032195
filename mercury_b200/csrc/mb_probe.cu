// Shared-memory read bandwidth of the device: the roofline denominator of
// the resident step kernel, whose binding resource is shared memory (it keeps
// every robot on chip for a whole launch, so HBM carries only the state and
// topology once per launch).
//
// One 1,024-thread CTA per SM (the step kernel's shape) streams 128-bit
// loads from a 32 KB shared buffer: consecutive lanes read consecutive
// 16-byte words, so each warp load is four conflict-free 128-byte
// wavefronts.  The loaded words are folded into an XOR that is written out,
// so no load can be dropped.  Bytes counted = 16 x loads; time from CUDA
// events on the launching stream, and the SM clock cycles of each CTA from
// clock64 (bytes per clock per SM).
#include <cstdint>

#include <cuda_runtime.h>

#include "../../include/mercury_b200.h"
#include "mb_step_math.cuh"

namespace {

constexpr int kThreads = 1024;
constexpr int kWords = 2048;  // 16-byte words: 32 KB
constexpr int kUnroll = 8;

__global__ void __launch_bounds__(kThreads, 1)
smem_read_kernel(uint32_t iters, uint32_t* sink, unsigned long long* cycles) {
    __shared__ uint4 buf[kWords];
    const uint32_t tid = threadIdx.x;
    for (uint32_t i = tid; i < kWords; i += kThreads) buf[i] = make_uint4(i, 3 * i + 1, 5 * i + 2, 7 * i + 3);
    __syncthreads();
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(buf);
    uint32_t acc = 0;
    const long long c0 = clock64();
    for (uint32_t it = 0; it < iters; ++it) {
#pragma unroll
        for (int k = 0; k < kUnroll; ++k) {
            // lanes of a warp: 32 consecutive words; the 8 loads of an
            // iteration read 8 distinct words of each thread and the offset
            // moves each iteration; volatile loads, so that none is merged
            // with another or hoisted
            const uint32_t idx = (tid + (uint32_t)k * 128u + it * 32u) & (kWords - 1);
            uint32_t a, b, c, d;
            asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(a), "=r"(b), "=r"(c), "=r"(d)
                         : "r"(base + idx * 16u));
            acc ^= a ^ b ^ c ^ d;
        }
    }
    const long long c1 = clock64();
    __syncthreads();
    if (tid == 0) cycles[blockIdx.x] = (unsigned long long)(c1 - c0);
    if (acc == 0x9e3779b9u) sink[blockIdx.x] = acc;  // keeps the loads live
}

// Every non-negative float (and positive NaN) as a squared length: where the fast path is taken, its length
// and reciprocal against the intrinsics'; the packed form against both.
__global__ void __launch_bounds__(256) spring_math_kernel(unsigned long long* bad) {
    unsigned long long n = 0;
    for (unsigned long long b = blockIdx.x * 256ull + threadIdx.x; b < 1ull << 31; b += gridDim.x * 256ull) {
        const float ns = -__uint_as_float((uint32_t)b);
        float nd, e, q, xd, xq;
        mb::length_and_reciprocal_fast(ns, nd, e, q);
        mb::length_and_reciprocal_exact(ns, xd, xq);
        mb::f32x2 pd, pe, pq;
        mb::lengths_and_reciprocals_fast(mb::pack2(ns, -1.0f), pd, pe, pq);
        float d0, d1, e0, e1, q0, q1;
        mb::unpack2(pd, d0, d1);
        mb::unpack2(pe, e0, e1);
        mb::unpack2(pq, q0, q1);
        auto same = [](float x, float y) { return __float_as_uint(x) == __float_as_uint(y); };
        const bool fast = mb::length_is_fast(nd, e);
        n += fast != mb::length_is_fast(d0, e0) || d1 != -1.0f || q1 != 1.0f;
        if (fast) n += !(same(nd, xd) && same(q, xq) && same(d0, xd) && same(q0, xq));
    }
    if (n) atomicAdd(bad, n);
}

}  // namespace

extern "C" {

mb_status mb_check_spring_math(int device, uint64_t* mismatches) {
    if (!mismatches) return MB_ERR_ARGUMENT;
    if (cudaSetDevice(device) != cudaSuccess) return MB_ERR_CUDA;
    unsigned long long* bad = nullptr;
    unsigned long long n = 0;
    if (cudaMalloc(&bad, sizeof(*bad)) != cudaSuccess) return MB_ERR_CUDA;
    cudaError_t e = cudaMemset(bad, 0, sizeof(*bad));
    if (e == cudaSuccess) {
        spring_math_kernel<<<148 * 8, 256>>>(bad);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(&n, bad, sizeof(n), cudaMemcpyDeviceToHost);
    cudaFree(bad);
    *mismatches = n;
    return e == cudaSuccess ? MB_OK : MB_ERR_CUDA;
}

mb_status mb_measure_smem_bandwidth(int device, double* bytes_per_s, double* bytes_per_clk_sm) {
    if (!bytes_per_s) return MB_ERR_ARGUMENT;
    if (cudaSetDevice(device) != cudaSuccess) return MB_ERR_CUDA;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0)
        return MB_ERR_CUDA;
    uint32_t* sink = nullptr;
    unsigned long long* cycles = nullptr;
    cudaStream_t st = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    mb_status rc = MB_ERR_CUDA;
    const uint32_t iters = 4096;
    const double bytes = 16.0 * kUnroll * (double)iters * kThreads * sms;
    float best_ms = 0.0f;
    double best_cycles = 0.0;
    unsigned long long* host_cycles = new unsigned long long[sms];
    if (cudaMalloc(&sink, sizeof(uint32_t) * sms) != cudaSuccess) goto done;
    if (cudaMalloc(&cycles, sizeof(unsigned long long) * sms) != cudaSuccess) goto done;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) goto done;
    if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) goto done;
    smem_read_kernel<<<sms, kThreads, 0, st>>>(iters / 8, sink, cycles);  // warm-up
    for (int rep = 0; rep < 5; ++rep) {
        cudaEventRecord(e0, st);
        smem_read_kernel<<<sms, kThreads, 0, st>>>(iters, sink, cycles);
        cudaEventRecord(e1, st);
        if (cudaEventSynchronize(e1) != cudaSuccess) goto done;
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (cudaMemcpy(host_cycles, cycles, sizeof(unsigned long long) * sms, cudaMemcpyDeviceToHost) !=
            cudaSuccess)
            goto done;
        double mean_cycles = 0.0;
        for (int i = 0; i < sms; ++i) mean_cycles += (double)host_cycles[i] / sms;
        if (best_ms == 0.0f || ms < best_ms) {
            best_ms = ms;
            best_cycles = mean_cycles;
        }
    }
    if (cudaGetLastError() != cudaSuccess || best_ms <= 0.0f) goto done;
    *bytes_per_s = bytes / (best_ms * 1e-3);
    if (bytes_per_clk_sm) *bytes_per_clk_sm = bytes / sms / best_cycles;
    rc = MB_OK;
done:
    delete[] host_cycles;
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (st) cudaStreamDestroy(st);
    if (sink) cudaFree(sink);
    if (cycles) cudaFree(cycles);
    return rc;
}

}  // extern "C"
