// k-nearest-neighbour springs of point-cloud robots, built on the device
// (the springs of the reference's NNRobot, common/evolvables/knn.cu:62-145
// with knn_kernel.cu:34-60, as the third benchmark configuration uses them:
// every mass joined to its k nearest masses, each unordered pair once).
//
// Per robot:
//   select_kernel  one warp per mass: the lanes compute 32 squared distances
//                  at a time (the float32 sum (dx*dx + dy*dy) + dz*dz, the
//                  robot's positions in shared memory), the warp holds the k
//                  nearest in order of (squared distance, index) -- the order
//                  of a stable sort of the distance row -- one per lane, and
//                  inserts what is nearer than the last; then sets bit (min,
//                  max) of an upper-triangular bitset for every neighbour;
//   count_kernel   popcounts each row and scans the robot's rows; the host
//                  adds up the robots;
//   emit_kernel    writes the pairs row by row, partners ascending (the
//                  lexicographic order of the unique pairs), with the float32
//                  distance as mean length and the composite material of the
//                  two masses.
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <algorithm>
#include <cstring>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "../../include/mercury_b200.h"
#include "mb_pack.h"

namespace mb {
namespace {

constexpr uint32_t kKnnMaxK = 32;
constexpr uint32_t kKnnMaxMasses = 4096;
constexpr uint32_t kKnnThreads = 256;
constexpr uint32_t kKnnMasses = 64;  // masses per CTA of the selection

__device__ __forceinline__ float sqdist(float3 a, float3 b) {
    const float dx = __fsub_rn(a.x, b.x), dy = __fsub_rn(a.y, b.y), dz = __fsub_rn(a.z, b.z);
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

__device__ __forceinline__ int composite_knn(int m1, int m2) {
    if (m1 == 0 || m2 == 0) return 0;
    const int i = min(m1, m2) - 1, j = max(m1, m2) - 1;
    if (i == j) return i + 1;
    return 23 + i * 21 - i * (i - 1) / 2 + (j - i - 1);
}

struct KnnArgs {
    const float* pos;         // 3 per mass
    const int64_t* mass_off;  // n_robots + 1
    uint32_t k;
    uint32_t* bits;           // per robot: rows of ceil(m / 32) words
    const uint64_t* bit_off;  // per robot: first word
    uint32_t* row_first;      // per mass: first spring of its row within the robot
    uint32_t* n_springs;      // per robot
};

__device__ __forceinline__ void mark(const KnnArgs& a, uint32_t* bits, uint32_t words, uint32_t i, uint32_t j) {
    const uint32_t lo = min(i, j), hi = max(i, j);
    atomicOr(&bits[(size_t)lo * words + hi / 32], 1u << (hi % 32));
}

// A mass with a NaN distance, one thread: neighbours are inserted in index
// order before the first of the list that is farther, and a NaN compares
// farther than none, so the list depends on where the NaNs come.
__device__ __noinline__ void select_nan(const KnnArgs& a, const float3* pts, uint32_t m, uint32_t i, uint32_t k,
                                        uint32_t* bits, uint32_t words) {
    float kd[kKnnMaxK];
    uint32_t kj[kKnnMaxK];
    uint32_t n = 0;
    for (uint32_t j = 0; j < m; ++j) {
        if (j == i) continue;
        const float d = sqdist(pts[i], pts[j]);
        if (n == k && !(d < kd[k - 1])) continue;
        uint32_t p = n < k ? n++ : k - 1;
        while (p > 0 && d < kd[p - 1]) {
            kd[p] = kd[p - 1];
            kj[p] = kj[p - 1];
            --p;
        }
        kd[p] = d;
        kj[p] = j;
    }
    for (uint32_t q = 0; q < n; ++q) mark(a, bits, words, i, kj[q]);
}

// A thread per mass with the list in local memory took 17.1 ms for 256 clouds
// of 500-2,000 points (k = 25); a warp per mass inserts each of the about
// k (1 + ln(m / k)) candidates that enter the list in a dozen instructions, and
// the same clouds take 2.06 ms.  Bound by the insertions, a serial chain per
// mass; 64 masses share one copy of the points, so that loading them is 1/64
// of the scan and a cloud of 500 still fills 8 CTAs.
__global__ void __launch_bounds__(kKnnThreads) select_kernel(const KnnArgs a) {
    extern __shared__ float3 pts[];
    const uint32_t r = blockIdx.y, lane = threadIdx.x & 31;
    const int64_t m0 = a.mass_off[r];
    const uint32_t m = (uint32_t)(a.mass_off[r + 1] - m0), words = (m + 31) / 32;
    if (blockIdx.x * kKnnMasses >= m) return;
    for (uint32_t j = threadIdx.x; j < m; j += blockDim.x)
        pts[j] = make_float3(a.pos[3 * (m0 + j)], a.pos[3 * (m0 + j) + 1], a.pos[3 * (m0 + j) + 2]);
    __syncthreads();
    uint32_t* bits = a.bits + a.bit_off[r];
    const uint32_t k = min(a.k, m - 1), last = min(m, (blockIdx.x + 1) * kKnnMasses);
    if (k == 0) return;
    for (uint32_t i = blockIdx.x * kKnnMasses + threadIdx.x / 32; i < last; i += kKnnThreads / 32) {
        const float3 pi = pts[i];
        // lane l < k: the l-th nearest so far, (distance bits << 32) | index;
        // `far`: the k-th
        unsigned long long mine = ~0ull, far = ~0ull;
        bool nan = false;
        for (uint32_t j0 = 0; j0 < m; j0 += 32) {
            const uint32_t j = j0 + lane;
            unsigned long long key = ~0ull;
            if (j < m && j != i) {
                const float d = sqdist(pi, pts[j]);
                nan |= d != d;
                key = (unsigned long long)__float_as_uint(d) << 32 | j;
            }
            uint32_t in = __ballot_sync(0xffffffffu, key < far);
            while (in) {
                const int src = __ffs(in) - 1;
                in &= in - 1;
                const unsigned long long c = __shfl_sync(0xffffffffu, key, src);
                if (!(c < far)) continue;  // the list moved on
                const uint32_t at = __popc(__ballot_sync(0xffffffffu, mine < c));
                const unsigned long long up = __shfl_up_sync(0xffffffffu, mine, 1);
                mine = lane < at ? mine : lane == at ? c : up;
                if (lane >= k) mine = ~0ull;
                far = __shfl_sync(0xffffffffu, mine, k - 1);
            }
        }
        if (__any_sync(0xffffffffu, nan)) {
            if (lane == 0) select_nan(a, pts, m, i, k, bits, words);
            __syncwarp();
        } else if (lane < k) {
            mark(a, bits, words, i, (uint32_t)mine);
        }
    }
}

// One CTA per robot: springs per row, scanned, so that the host reads and sums
// one number per robot (86 us; 29 us without the scan, then 1.4 MB of row
// counts to the host and 2.7 MB of offsets back).
__global__ void __launch_bounds__(1024) count_kernel(const KnnArgs a) {
    __shared__ uint32_t warp_sum[32];
    const uint32_t r = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x / 32;
    const int64_t m0 = a.mass_off[r];
    const uint32_t m = (uint32_t)(a.mass_off[r + 1] - m0), words = (m + 31) / 32;
    const uint32_t* bits = a.bits + a.bit_off[r];
    uint32_t base = 0;
    for (uint32_t row0 = 0; row0 < m; row0 += 1024) {
        // a warp's rows one after another, its lanes over the row's words
        uint32_t c = 0;
        for (uint32_t q = 0; q < 32; ++q) {
            const uint32_t row = row0 + 32 * warp + q;
            if (row >= m) break;
            uint32_t n = 0;
            for (uint32_t w = lane; w < words; w += 32) n += __popc(bits[(size_t)row * words + w]);
            n = __reduce_add_sync(0xffffffffu, n);
            if (lane == q) c = n;
        }
        uint32_t inc = c;  // inclusive scan over the 1,024 rows
        for (uint32_t o = 1; o < 32; o *= 2) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        if (lane == 31) warp_sum[warp] = inc;
        __syncthreads();
        uint32_t before = 0, total = 0;
        for (uint32_t w = 0; w < 32; ++w) {
            if (w < warp) before += warp_sum[w];
            total += warp_sum[w];
        }
        if (row0 + threadIdx.x < m) a.row_first[m0 + row0 + threadIdx.x] = base + before + inc - c;
        base += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) a.n_springs[r] = base;
}

struct EmitArgs {
    const float* pos;
    const uint8_t* mass_mat;
    const int64_t* mass_off;
    const uint32_t* bits;
    const uint64_t* bit_off;
    const uint32_t* row_first;     // per mass: first spring of its row within the robot
    const int64_t* spring_off;     // per robot: its first spring
    uint16_t* pairs;               // robot-local indices
    uint8_t* mat;
    float* lbar;
};

// A warp per row: lane w takes the row's words w, w + 32, ...  Bound by the
// scattered stores; 114 us for 4.6 million springs (256 clouds of 500-2,000
// points, k = 25), a thread per row 197 us.
__global__ void __launch_bounds__(kKnnThreads) emit_kernel(const EmitArgs a) {
    const uint32_t r = blockIdx.y, lane = threadIdx.x & 31;
    const int64_t m0 = a.mass_off[r];
    const uint32_t m = (uint32_t)(a.mass_off[r + 1] - m0), words = (m + 31) / 32;
    const uint32_t* bits = a.bits + a.bit_off[r];
    for (uint32_t row = (blockIdx.x * blockDim.x + threadIdx.x) / 32; row < m; row += gridDim.x * blockDim.x / 32) {
        uint64_t s0 = (uint64_t)a.spring_off[r] + a.row_first[m0 + row];
        const float3 p = make_float3(a.pos[3 * (m0 + row)], a.pos[3 * (m0 + row) + 1], a.pos[3 * (m0 + row) + 2]);
        const int mp = a.mass_mat[m0 + row];
        for (uint32_t w0 = row / 32; w0 < words; w0 += 32) {  // partners are higher
            const uint32_t w = w0 + lane;
            uint32_t v = w < words ? bits[(size_t)row * words + w] : 0u;
            uint32_t n = __popc(v), inc = n;
            for (uint32_t o = 1; o < 32; o *= 2) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += u;
            }
            uint64_t s = s0 + inc - n;
            s0 += __shfl_sync(0xffffffffu, inc, 31);
            while (v) {
                const uint32_t b = w * 32 + (uint32_t)(__ffs(v) - 1);
                v &= v - 1;
                const int64_t g = m0 + b;
                const float3 q = make_float3(a.pos[3 * g], a.pos[3 * g + 1], a.pos[3 * g + 2]);
                reinterpret_cast<uint32_t*>(a.pairs)[s] = row | b << 16;
                a.lbar[s] = __fsqrt_rn(sqdist(p, q));
                a.mat[s] = (uint8_t)composite_knn(mp, a.mass_mat[g]);
                ++s;
            }
        }
    }
}

// Grow-only device buffer, kept between calls.
template <typename T>
struct Dev {
    T* p = nullptr;
    size_t n = 0;
    cudaError_t alloc(size_t count) {
        if (count <= n && p) return cudaSuccess;
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
        const size_t c = std::max<size_t>(count, 1);
        const cudaError_t e = cudaMalloc(&p, c * sizeof(T));
        if (e == cudaSuccess) n = c;
        return e;
    }
};

// Maps the pages of arrays about to receive a device copy, on several threads.
// The copy's one thread otherwise faults fresh pages in one by one: 41 MB
// of springs into fresh arrays 13.0 ms for the whole call, 7.8 ms with the pages
// mapped first (4.6 ms into arrays that were written before, either way).  What
// the arrays hold stays as it is; where the system cannot do this the copy
// faults the pages in itself.
struct HostRange {
    void* p;
    size_t bytes;
};
void map_pages(std::initializer_list<HostRange> ranges) {
#ifdef MADV_POPULATE_WRITE
    constexpr uintptr_t kPage = 4096, kPiece = 2 << 20;
    std::vector<HostRange> pieces;
    for (const HostRange& r : ranges) {
        const uintptr_t a = (reinterpret_cast<uintptr_t>(r.p) + kPage - 1) & ~(kPage - 1);
        const uintptr_t z = (reinterpret_cast<uintptr_t>(r.p) + r.bytes) & ~(kPage - 1);
        for (uintptr_t o = a; o < z; o += kPiece) pieces.push_back({reinterpret_cast<void*>(o), std::min(kPiece, z - o)});
    }
    const unsigned threads = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
    if (pieces.size() > 1)
        parallel_for(static_cast<uint32_t>(pieces.size()), threads,
                     [&](uint32_t i) { (void)madvise(pieces[i].p, pieces[i].bytes, MADV_POPULATE_WRITE); });
#endif
}

// Scratch and stream of one device, kept for the process: calls reuse them
// (one call at a time per device, under the lock), so a call allocates only
// when it needs more than any earlier one.
struct KnnScratch {
    std::mutex lock;
    cudaStream_t stream = nullptr;
    Dev<float> pos, lbar;
    Dev<uint8_t> mm, mat;
    Dev<int64_t> off, soff;
    Dev<uint16_t> pairs;
    Dev<uint32_t> bits, first, count;
    Dev<uint64_t> boff;
};

KnnScratch& knn_scratch(int device) {
    static std::mutex registry_lock;
    static std::vector<std::unique_ptr<KnnScratch>> per_device;
    std::lock_guard<std::mutex> g(registry_lock);
    if ((size_t)device >= per_device.size()) per_device.resize(device + 1);
    if (!per_device[device]) per_device[device] = std::make_unique<KnnScratch>();
    return *per_device[device];
}

}  // namespace
}  // namespace mb

extern "C" mb_status mb_knn_springs(int device, uint32_t n_robots, const int64_t* mass_offsets, const float* pos,
                                    const uint8_t* mass_material, uint32_t k, int64_t* spring_offsets,
                                    uint16_t* pairs, uint8_t* spring_material, float* lbar, uint64_t capacity) {
    using namespace mb;
    if (!mass_offsets || !pos || !mass_material || !spring_offsets || n_robots == 0) return MB_ERR_ARGUMENT;
    if (k == 0 || k > kKnnMaxK || mass_offsets[0] != 0) return MB_ERR_ARGUMENT;
    uint32_t max_m = 0;
    std::vector<uint64_t> bit_off(n_robots + 1, 0);
    for (uint32_t r = 0; r < n_robots; ++r) {
        if (mass_offsets[r + 1] < mass_offsets[r]) return MB_ERR_ARGUMENT;
        const uint64_t m = (uint64_t)(mass_offsets[r + 1] - mass_offsets[r]);
        if (m > kKnnMaxMasses) return MB_ERR_CAPACITY;
        max_m = std::max<uint32_t>(max_m, (uint32_t)m);
        bit_off[r + 1] = bit_off[r] + m * ((m + 31) / 32);
    }
    const uint64_t M = (uint64_t)mass_offsets[n_robots];
    if (device < 0 || cudaSetDevice(device) != cudaSuccess) return MB_ERR_CUDA;
    KnnScratch& sc = knn_scratch(device);
    std::lock_guard<std::mutex> held(sc.lock);
    if (!sc.stream && cudaStreamCreateWithFlags(&sc.stream, cudaStreamNonBlocking) != cudaSuccess) {
        sc.stream = nullptr;
        return MB_ERR_CUDA;
    }
    cudaStream_t st = sc.stream;
    auto& d_pos = sc.pos;
    auto& d_lbar = sc.lbar;
    auto& d_mm = sc.mm;
    auto& d_mat = sc.mat;
    auto& d_off = sc.off;
    auto& d_pairs = sc.pairs;
    auto& d_bits = sc.bits;
    auto& d_count = sc.count;
    auto& d_soff = sc.soff;
    auto& d_boff = sc.boff;
    auto& d_first = sc.first;
#define KNN_CUDA(x)                               \
    do {                                          \
        if ((x) != cudaSuccess) return MB_ERR_CUDA; \
    } while (0)
    KNN_CUDA(d_pos.alloc(3 * M));
    KNN_CUDA(d_mm.alloc(M));
    KNN_CUDA(d_off.alloc(n_robots + 1));
    KNN_CUDA(d_bits.alloc(bit_off[n_robots]));
    KNN_CUDA(d_boff.alloc(n_robots + 1));
    KNN_CUDA(d_first.alloc(M));
    KNN_CUDA(d_count.alloc(n_robots));
    KNN_CUDA(d_soff.alloc(n_robots + 1));
    KNN_CUDA(cudaMemcpyAsync(d_pos.p, pos, 3 * M * sizeof(float), cudaMemcpyHostToDevice, st));
    KNN_CUDA(cudaMemcpyAsync(d_mm.p, mass_material, M, cudaMemcpyHostToDevice, st));
    KNN_CUDA(cudaMemcpyAsync(d_off.p, mass_offsets, (n_robots + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, st));
    KNN_CUDA(cudaMemcpyAsync(d_boff.p, bit_off.data(), (n_robots + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
    KNN_CUDA(cudaMemsetAsync(d_bits.p, 0, bit_off[n_robots] * sizeof(uint32_t), st));
    const KnnArgs ka{d_pos.p, d_off.p, k, d_bits.p, d_boff.p, d_first.p, d_count.p};
    select_kernel<<<dim3((max_m + kKnnMasses - 1) / kKnnMasses, n_robots), kKnnThreads, max_m * sizeof(float3), st>>>(ka);
    KNN_CUDA(cudaGetLastError());
    count_kernel<<<n_robots, 1024, 0, st>>>(ka);
    KNN_CUDA(cudaGetLastError());
    std::vector<uint32_t> count(n_robots);
    KNN_CUDA(cudaMemcpyAsync(count.data(), d_count.p, n_robots * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    KNN_CUDA(cudaStreamSynchronize(st));
    uint64_t total = 0;
    spring_offsets[0] = 0;
    for (uint32_t r = 0; r < n_robots; ++r) {
        total += count[r];
        spring_offsets[r + 1] = (int64_t)total;
    }
    if (!pairs) return MB_OK;  // counting call
    if (total > capacity || !spring_material || !lbar) return MB_ERR_CAPACITY;
    KNN_CUDA(d_pairs.alloc(2 * total));
    KNN_CUDA(d_mat.alloc(total));
    KNN_CUDA(d_lbar.alloc(total));
    KNN_CUDA(cudaMemcpyAsync(d_soff.p, spring_offsets, (n_robots + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, st));
    const EmitArgs ea{d_pos.p, d_mm.p, d_off.p, d_bits.p, d_boff.p, d_first.p, d_soff.p, d_pairs.p, d_mat.p, d_lbar.p};
    emit_kernel<<<dim3((max_m + 63) / 64, n_robots), kKnnThreads, 0, st>>>(ea);
    KNN_CUDA(cudaGetLastError());
    map_pages({{pairs, 2 * total * sizeof(uint16_t)}, {spring_material, total}, {lbar, total * sizeof(float)}});
    KNN_CUDA(cudaMemcpyAsync(pairs, d_pairs.p, 2 * total * sizeof(uint16_t), cudaMemcpyDeviceToHost, st));
    KNN_CUDA(cudaMemcpyAsync(spring_material, d_mat.p, total, cudaMemcpyDeviceToHost, st));
    KNN_CUDA(cudaMemcpyAsync(lbar, d_lbar.p, total * sizeof(float), cudaMemcpyDeviceToHost, st));
    KNN_CUDA(cudaStreamSynchronize(st));
#undef KNN_CUDA
    return MB_OK;
}
