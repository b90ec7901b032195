// Step kernels of the batched soft-body simulator (sm_100a).
//
// The reference step (common/simulator/sim_kernel.cu:141-269) launches four
// kernels per step and re-stages every robot through shared memory each
// time, accumulating the spring corrections with shared-memory float
// atomics.  Here one CTA simulates one "bin" (a group of whole robots) for a
// whole chunk of steps without leaving the SM:
//
//   registers : each thread's masses (x, v);
//   tensor    : each thread's springs (packed pair + material slot, mean
//   memory      length, optional stress), two at a time into registers;
//   shared    : predicted positions x~ (SoA), per-spring corrections dp
//               (SoA), the bin's incidence lists (SELL-32), and the per-step
//               actuation factors and 1/K of the bin's materials.
//
// Per step: (1) warp 0 evaluates the actuation factor dL0*sin(omega*t+phi)
// of each material of the bin; every thread predicts x~ = x + v*dt for its
// masses; barrier.  (2) every thread solves its springs (XPBD distance
// constraint, sim_kernel.cu:209-243) and stores dp per spring; barrier.
// (3) every thread gathers, for each of its masses, the corrections of the
// incident springs in a fixed order from its SELL row (no atomics), then
// integrates x and v (sim_kernel.cu:246-252, 261-268).
//
// This kernel steps what the tensor-memory kernel (mb_tm.cu) does not: parts
// of robots split over a cluster, masses of more springs than a lattice has
// (point clouds), small shapes.  With the springs in registers, 1,024 threads
// of 64 registers spilled 28-300 bytes inside the step and held one load in
// flight; in tensor memory nothing spills at the 1,024-thread shapes and two
// springs and four row entries are in flight.  64 split robots of 11x11x11
// masses: 6.24 -> 5.80 us a step, 256 point clouds of 500-2,000 masses: 48.0
// -> 42.7, 30 clouds of 60: 9.4 -> 3.0.  Five or eight row entries in flight
// measured 6.03 and 5.92 (clouds 43.4 and 44.2), one at a time 6.45 (46.5).
// Split robots are bound by issue (71 %), clouds by the shared-memory pipe
// while it is used (40 % conflict wavefronts of the random rows) and the
// barriers between the parts.
//
// All arithmetic uses explicit round-to-nearest intrinsics so that the
// result is bit-identical to the CPU restatement in the oracle.
#include <cooperative_groups.h>

#include "mb_internal.h"
#include "mb_sin.cuh"
#include "mb_step_math.cuh"
#include "mb_tmem.cuh"

namespace mb {

namespace cg = cooperative_groups;

namespace {

// Packed spring word: a (12 bits) | b << 12 (12 bits) | slot << 24 (8 bits).
__device__ __forceinline__ uint32_t pk_a(uint32_t w) { return w & 0xFFFu; }
__device__ __forceinline__ uint32_t pk_b(uint32_t w) { return (w >> 12) & 0xFFFu; }
__device__ __forceinline__ uint32_t pk_slot(uint32_t w) { return w >> 24; }

template <int T, int SPT, int MPT, int MODE, bool TRACK, bool SPLIT>
__global__ void __launch_bounds__(T, 1024 / T) step_kernel(const StepParams p) {
    constexpr bool XPBD = MODE == kModeXpbd;
    constexpr bool FACES = MODE == kModeForceWaterFaces;  // face drag compiled in
    extern __shared__ float4 smem4[];
    const int tid = threadIdx.x;
    // 64 columns a warp: words of the thread's springs 2 i, 2 i + 1 at
    // column 4 i {packed word, mean length} x 2, their stresses at kStress + 2 i
    constexpr uint32_t kCols = T / 2, kPairs = (SPT + 1) / 2, kStress = 4 * kPairs;
    static_assert(kStress + 2 * kPairs <= 64 && kStress + 4 <= 64, "");
    const uint32_t tmem0 = tm_alloc(reinterpret_cast<uint32_t*>(smem4), kCols);
    const uint32_t tm = tmem0 + ((tid / 32 & 3u) << 21) + (tid / 128) * 64u;
    const float dt = p.dt;
    const double ddt = (double)dt;
    const double inv_dt = __drcp_rn(ddt);
    const float inv_dt_f = __frcp_rn(dt);

    for (uint32_t b = blockIdx.x; b < p.n_bins; b += gridDim.x) {
        const BinDesc bd = p.bins[b];
        // predicted positions x~, one float4 per mass (split bins: two
        // buffers, own masses then halo, alternating by step; with faces,
        // two velocity buffers of the same shape follow)
        float4* sxt = smem4;
        float4* sdp = sxt + (SPLIT ? (FACES ? 4u : 2u) * bd.x_stride : bd.n_mass);  // corrections dp, one float4 per spring
        float2* smat = reinterpret_cast<float2*>(sdp + bd.n_spring);  // {dL0 sin(..), 1/K} per slot
        // split bins: the buffer stride of every part of the cluster, then
        // the export list
        uint32_t* sstride = reinterpret_cast<uint32_t*>(smat + kMaxMaterialSlots);
        uint32_t* sexp = sstride + (SPLIT ? kMaxClusterParts : 0u);
        uint16_t* sinc = reinterpret_cast<uint16_t*>(sexp + (SPLIT ? bd.n_export : 0u));
        // face drag (water, bins with faces), after the rows at a 16-byte
        // boundary: velocities (resident bins; split bins keep them after
        // the positions), face forces, corners, face rows (first entry |
        // count << 24), incidence
        const uint32_t n_face = FACES && p.face_on ? bd.n_face : 0u;
        float4* sv = reinterpret_cast<float4*>((reinterpret_cast<uintptr_t>(sinc + bd.n_inc) + 15u) & ~uintptr_t(15));
        float4* sfd = SPLIT ? sv : sv + bd.n_mass;
        if (SPLIT) sv = sxt + 2u * bd.x_stride;
        uint2* sface = reinterpret_cast<uint2*>(sfd + n_face);
        uint32_t* sfrow = reinterpret_cast<uint32_t*>(sface + n_face);
        uint16_t* sfinc = reinterpret_cast<uint16_t*>(sfrow + bd.n_mass);

        const uint32_t n_mat = *p.n_mat;
        for (uint32_t i = tid; i < bd.n_inc; i += T) sinc[i] = __ldg(&p.inc[bd.inc_begin + i]);
        if (n_face) {
            for (uint32_t i = tid; i < n_face; i += T) sface[i] = __ldg(&p.faces[bd.face_begin + i]);
            for (uint32_t i = tid; i < bd.n_mass; i += T) sfrow[i] = __ldg(&p.face_row[bd.mass_begin + i]);
            for (uint32_t i = tid; i < bd.n_face_inc; i += T) sfinc[i] = __ldg(&p.face_inc[bd.face_inc_begin + i]);
        }
        if (SPLIT) {
            for (uint32_t i = tid; i < bd.n_export; i += T) sexp[i] = __ldg(&p.exports[bd.export_begin + i]);
            const cg::cluster_group cl = cg::this_cluster();
            if (tid < cl.num_blocks()) sstride[tid] = p.bins[b - cl.block_rank() + tid].x_stride;
        }
        float next_rate = 0.0f;  // actuation factor of material tid for the coming step
        if (tid < n_mat) {
            smat[tid].y = __ldg(&p.invk[tid]);  // 1/K (reference step) or k (force modes)
            next_rate = __ldg(&p.rates[tid]);
        }

        // Springs of this thread, s = tid + j T: packed word and mean length
        // (+ stress) into tensor memory; a missing one gets word 0.
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 2 * (int)kPairs; j += 2) {
            uint32_t sw[2] = {0, 0}, lb[2] = {0, 0}, st[2] = {0, 0};
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t s = tid + (j + u) * T;
                if (s < bd.n_spring) {
                    const uint32_t g = bd.spring_begin + s;
                    sw[u] = __ldg(&p.spring_pair[g]);
                    lb[u] = __float_as_uint(__ldg(&p.spring_lbar[g]));
                    if (TRACK) st[u] = __float_as_uint(p.stress[__ldg(&p.spring_gidx[g]) & 0x7FFFFFFFu]);
                }
            }
            __syncwarp();
            tm_st2(tm + 2 * j, sw[0], lb[0]);
            tm_st2(tm + 2 * j + 2, sw[1], lb[1]);
            if (TRACK) tm_st2(tm + kStress + j, st[0], st[1]);
        }
        tm_wait_st();
        // columns of pairs this warp has springs in
        const uint32_t s_warp = tid & ~31u;
        const uint32_t tm_end = tm + (bd.n_spring > s_warp ? 4u * (((bd.n_spring - s_warp + T - 1) / T + 1) / 2) : 0u);
        // Masses of this thread: x, v, mass and the SELL row (offset | width << 20).
        float3 x[MPT], v[MPT];
        float mass[MPT];
        uint32_t row[MPT];
#pragma unroll
        for (int j = 0; j < MPT; ++j) {
            const uint32_t m = tid + j * T;
            x[j] = make_float3(0.f, 0.f, 0.f);
            v[j] = make_float3(0.f, 0.f, 0.f);
            row[j] = 0;
            mass[j] = 1.0f;
            if (m < bd.n_mass) {
                const uint32_t g = __ldg(&p.mass_gidx[bd.mass_begin + m]);
                const float4 P = p.pos[g], V = p.vel[g];
                x[j] = make_float3(P.x, P.y, P.z);
                mass[j] = P.w;
                v[j] = make_float3(V.x, V.y, V.z);
                const uint32_t sl = bd.slice_begin + m / kSliceWidth;
                row[j] = (__ldg(&p.slice_off[sl]) + (m % kSliceWidth)) | (__ldg(&p.slice_width[sl]) << 20);
            }
        }
        if (SPLIT)
            cg::this_cluster().sync();  // every part of the robot has started
        else
            __syncthreads();

        for (uint32_t step = 0; step < p.steps; ++step) {
            float4* X = SPLIT ? sxt + (step & 1u) * bd.x_stride : sxt;
            float4* V = SPLIT ? sv + (step & 1u) * bd.x_stride : sv;  // velocities (face drag)
            // (1) actuation factors of this step (sim_kernel.cu:222), loaded one
            // step ahead from the launch's table
            if (tid < n_mat) {
                smat[tid].x = next_rate;
                if (step + 1 < p.steps) next_rate = __ldg(&p.rates[(step + 1) * n_mat + tid]);
            }
            // (1) reference step: predict x~ = x + v*dt (sim_kernel.cu:147-152);
            //     force modes: publish the current positions
#pragma unroll
            for (int j = 0; j < MPT; ++j) {
                const uint32_t m = tid + j * T;
                if (m >= bd.n_mass) break;
                if (XPBD)
                    X[m] = make_float4(__fadd_rn(x[j].x, __fmul_rn(v[j].x, dt)),
                                       __fadd_rn(x[j].y, __fmul_rn(v[j].y, dt)),
                                       __fadd_rn(x[j].z, __fmul_rn(v[j].z, dt)), 0.0f);
                else
                    X[m] = make_float4(x[j].x, x[j].y, x[j].z, 0.0f);
                // split bins publish every velocity: other parts' faces may
                // have corners here
                if (FACES && (SPLIT || n_face)) V[m] = make_float4(v[j].x, v[j].y, v[j].z, 0.0f);
            }
            __syncthreads();
            if (SPLIT) {
                // masses the other parts hold as halo, into their buffer of
                // this step (at the part's own stride); the cluster barrier
                // makes them visible.  A part is at most one step ahead of
                // another, so the other buffer is never read meanwhile.
                cg::cluster_group cl = cg::this_cluster();
                for (uint32_t i = tid; i < bd.n_export; i += T) {
                    const uint32_t ex = sexp[i], q = (ex >> 12) & 7u;
                    float4* dst = cl.map_shared_rank(sxt, q) + (step & 1u) * sstride[q];
                    dst[ex >> 15] = X[ex & 0xFFFu];
                    if (FACES) dst[2u * sstride[q] + (ex >> 15)] = V[ex & 0xFFFu];  // the velocity buffer
                }
                cl.sync();
            }
            // (2) distance constraints (sim_kernel.cu:209-243), two springs at a
            // time; the next two's words arrive during the arithmetic
            if (tm != tm_end) {
                uint32_t c[4], st[2], s = tid;
                tm_ld(tm, c);
                if (TRACK) tm_ld(tm + kStress, st);
                for (uint32_t ta = tm; ta != tm_end; s += 2 * T) {
                    if (TRACK)
                        asm volatile("tcgen05.wait::ld.sync.aligned;"
                                     : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(st[0]), "+r"(st[1]));
                    else
                        asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]));
                    // (a missing spring computes from mass 0 twice, and is not stored)
                    const float4 a0 = X[pk_a(c[0])], b0 = X[pk_b(c[0])], a1 = X[pk_a(c[2])], b1 = X[pk_b(c[2])];
                    const float2 m0 = smat[pk_slot(c[0])], m1 = smat[pk_slot(c[2])];
                    const float lb0 = __uint_as_float(c[1]), lb1 = __uint_as_float(c[3]);
                    const float st0 = __uint_as_float(st[0]), st1 = __uint_as_float(st[1]);
                    const uint32_t ts = tm + kStress + (ta - tm) / 2;
                    ta += 4;
                    tm_ld(ta, c);  // (past the last pair: words of this warp, not used)
                    if (TRACK) tm_ld(ts + 2, st);
                    const f32x2 minus = pack2(-1.0f, -1.0f);
                    const f32x2 d0 = fma2(pack2(b0.x, b0.y), minus, pack2(a0.x, a0.y));
                    const f32x2 d1 = fma2(pack2(b1.x, b1.y), minus, pack2(a1.x, a1.y));
                    const float z0 = __fsub_rn(a0.z, b0.z), z1 = __fsub_rn(a1.z, b1.z);
                    float x0, y0, x1, y1;
                    unpack2(d0, x0, y0);
                    unpack2(d1, x1, y1);
                    const float n0 = __fmaf_rn(-x0, x0, __fmaf_rn(-y0, y0, __fmul_rn(-z0, z0)));
                    const float n1 = __fmaf_rn(-x1, x1, __fmaf_rn(-y1, y1, __fmul_rn(-z1, z1)));
                    f32x2 nd, e, r;  // -d and 1 / (d + eps)
                    lengths_and_reciprocals_fast(pack2(n0, n1), nd, e, r);
                    float nd0, nd1, e0, e1, r0, r1;
                    unpack2(nd, nd0, nd1);
                    unpack2(e, e0, e1);
                    unpack2(r, r0, r1);
                    const bool has0 = s < bd.n_spring, has1 = s + T < bd.n_spring;
                    const bool ok0 = length_is_fast(nd0, e0) || !has0, ok1 = length_is_fast(nd1, e1) || !has1;
                    if (__any_sync(0xffffffffu, !ok0 || !ok1)) {
                        length_and_reciprocal_exact(n0, nd0, r0);
                        length_and_reciprocal_exact(n1, nd1, r1);
                        __syncwarp();
                    }
                    const float L0 = __fmaf_rn(lb0, m0.x, lb0), L1 = __fmaf_rn(lb1, m1.x, lb1);
                    // reference step: lambda = -C/K, dp = lambda n (sim_kernel.cu:230-232);
                    // force modes: Hooke force on the a end, -k (d - L) n
                    const float lam0 = __fmul_rn(-__fsub_rn(-nd0, L0), m0.y), lam1 = __fmul_rn(-__fsub_rn(-nd1, L1), m1.y);
                    const float f0 = __fmul_rn(lam0, r0), f1 = __fmul_rn(lam1, r1);
                    float px, py;
                    unpack2(mul2(pack2(f0, f0), d0), px, py);
                    if (has0) sdp[s] = make_float4(px, py, __fmul_rn(f0, z0), 0.0f);
                    unpack2(mul2(pack2(f1, f1), d1), px, py);
                    if (has1) sdp[s + T] = make_float4(px, py, __fmul_rn(f1, z1), 0.0f);
                    // stress: lambda/Lbar (reference, sim_kernel.cu:234); k (d - L)/Lbar (force)
                    if (TRACK) {
                        const float t0 = __fadd_rn(st0, __fmul_rn(XPBD ? lam0 : -lam0, __frcp_rn(lb0)));
                        const float t1 = __fadd_rn(st1, __fmul_rn(XPBD ? lam1 : -lam1, __frcp_rn(lb1)));
                        __syncwarp();
                        tm_st2(ts, __float_as_uint(t0), __float_as_uint(t1));
                    } else {
                        __syncwarp();  // the next wait wants the warp together
                    }
                }
                asm volatile("tcgen05.wait::ld.sync.aligned;"
                             : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(st[0]), "+r"(st[1])::"memory");
                if (TRACK) tm_wait_st();
            }
            // face drag: the share of each corner, per face
            for (uint32_t f = tid; f < n_face; f += T) {
                const uint2 c = sface[f];
                const uint32_t i0 = c.x & 0xFFFFu, i1 = c.x >> 16, i2 = c.y;
                sfd[f] = face_force(X[i0], X[i1], X[i2], V[i0], V[i1], V[i2], p.face_coef);
            }
            __syncthreads();
            // (3) gather in summation order and integrate (sim_kernel.cu:246-268).
            // acc + (+-c) is computed as fma(c, +-1, acc): c*(+-1) is exact, so
            // the single rounding equals that of the addition.
#pragma unroll
            for (int j = 0; j < MPT; ++j) {
                const uint32_t m = tid + j * T;
                if (m >= bd.n_mass) break;
                float ax = 0.0f, ay = 0.0f, az = 0.0f;
                const uint16_t* rp = sinc + (row[j] & 0xFFFFFu);
                const uint32_t w = row[j] >> 20;  // the same for the warp (one slice)
                uint32_t k = 0;
                for (; k + 4 <= w; k += 4) {
                    uint32_t e[4];
                    float4 c[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) e[u] = rp[(k + u) * kSliceWidth];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        c[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (e[u] != kPadEntry) c[u] = sdp[e[u] >> 1];
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const float sg = __uint_as_float(0x3f800000u | ((e[u] & 1u) << 31));
                        ax = __fmaf_rn(c[u].x, sg, ax);
                        ay = __fmaf_rn(c[u].y, sg, ay);
                        az = __fmaf_rn(c[u].z, sg, az);
                    }
                }
                for (; k < w; ++k) {
                    const uint32_t e = rp[k * kSliceWidth];
                    if (e != kPadEntry) {
                        const float4 c = sdp[e >> 1];
                        const float sg = __uint_as_float(0x3f800000u | ((e & 1u) << 31));
                        ax = __fmaf_rn(c.x, sg, ax);
                        ay = __fmaf_rn(c.y, sg, ay);
                        az = __fmaf_rn(c.z, sg, az);
                    }
                }
                if (XPBD) {
                    const float4 xt = X[m];
                    const float nx = __fadd_rn(xt.x, ax);
                    const float ny = __fadd_rn(xt.y, ay);
                    const float nz = __fadd_rn(xt.z, az);
                    // v = 0.99*(x~ - x)/dt in double (sim_kernel.cu:265-267)
                    v[j].x = velocity_of(__fsub_rn(nx, x[j].x), ddt, inv_dt);
                    v[j].y = velocity_of(__fsub_rn(ny, x[j].y), ddt, inv_dt);
                    v[j].z = velocity_of(__fsub_rn(nz, x[j].z), ddt, inv_dt);
                    x[j] = make_float3(nx, ny, nz);
                } else {
                    // face drag after the springs, faces in ascending order
                    // (the face row: first entry | count << 24)
                    const uint32_t fr = n_face ? sfrow[m] : 0u;
                    const uint16_t* fp = sfinc + (fr & 0xFFFFFFu);
                    for (uint32_t k = 0; k < (fr >> 24); ++k) {
                        const float4 c = sfd[fp[k]];
                        ax = __fadd_rn(ax, c.x);
                        ay = __fadd_rn(ay, c.y);
                        az = __fadd_rn(az, c.z);
                    }
                    force_integrate<MODE>(p, x[j], v[j], mass[j], inv_dt_f, ax, ay, az);
                }
            }
        }

        // Write back in the upload layout (w components unchanged); flag
        // non-finite positions.
        bool bad = false;
#pragma unroll
        for (int j = 0; j < MPT; ++j) {
            const uint32_t m = tid + j * T;
            if (m < bd.n_mass) {
                const uint32_t g = __ldg(&p.mass_gidx[bd.mass_begin + m]);
                p.pos[g] = make_float4(x[j].x, x[j].y, x[j].z, p.pos[g].w);
                p.vel[g] = make_float4(v[j].x, v[j].y, v[j].z, p.vel[g].w);
                bad |= !(isfinite(x[j].x) && isfinite(x[j].y) && isfinite(x[j].z));
            }
        }
        if (TRACK) {
            __syncwarp();
            for (uint32_t j = 0; 2 * j < tm_end - tm; j += 2) {
                uint32_t st[2];
                tm_ld(tm + kStress + j, st);
                asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(st[0]), "+r"(st[1]));
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint32_t s = tid + (j + u) * T;
                    if (s < bd.n_spring) {
                        const uint32_t g = __ldg(&p.spring_gidx[bd.spring_begin + s]);
                        if (!(g >> 31)) p.stress[g] = __uint_as_float(st[u]);  // bit 31: a copy in a split part
                    }
                }
                __syncwarp();
            }
        }
        if (__syncthreads_or(bad) && tid == 0) atomicOr(&p.bin_flags[b], 1u);
        if (SPLIT) cg::this_cluster().sync();
    }
    tm_free(tmem0, kCols);
}


// Streamed step: one CTA per bin (typically one large robot).  Shared memory
// holds the predicted positions and the material factors; every step reads
// the bin's springs and rows from global memory and exchanges the per-spring
// corrections through a global scratch array (L2-resident), with the same
// arithmetic and summation order as step_kernel.
template <int T, int MPT, int MODE, bool TRACK>
__global__ void __launch_bounds__(T, 1024 / T) stream_kernel(const StepParams p) {
    constexpr bool XPBD = MODE == kModeXpbd;
    constexpr bool FACES = MODE == kModeForceWaterFaces;  // face drag compiled in
    extern __shared__ float4 smem4[];
    const int tid = threadIdx.x;
    const float dt = p.dt;
    const double ddt = (double)dt;
    const double inv_dt = __drcp_rn(ddt);
    const float inv_dt_f = __frcp_rn(dt);

    for (uint32_t b = blockIdx.x; b < p.n_bins; b += gridDim.x) {
        const BinDesc bd = p.bins[b];
        float4* sxt = smem4;
        float2* smat = reinterpret_cast<float2*>(sxt + bd.n_mass);
        float4* dp = p.dp + bd.spring_begin;
        float* stp = p.st + bd.spring_begin;
        const uint32_t* pair = p.spring_pair + bd.spring_begin;
        const float* lbar = p.spring_lbar + bd.spring_begin;
        const uint32_t* inc = p.inc32 + bd.inc_begin;
        // face drag: velocities in shared memory after the material factors,
        // face forces through the global scratch like the corrections
        const uint32_t n_face = FACES && p.face_on ? bd.n_face : 0u;
        float4* sv = reinterpret_cast<float4*>(smat + kMaxMaterialSlots);
        float4* fd = p.fd + bd.face_begin;
        const uint2* fcorner = p.faces + bd.face_begin;
        const uint16_t* finc = p.face_inc + bd.face_inc_begin;
        const uint32_t n_mat = *p.n_mat;
        float next_rate = 0.0f;
        if (tid < n_mat) {
            smat[tid].y = __ldg(&p.invk[tid]);
            next_rate = __ldg(&p.rates[tid]);
        }
        if (TRACK)
            for (uint32_t s = tid; s < bd.n_spring; s += T)
                stp[s] = p.stress[__ldg(&p.spring_gidx[bd.spring_begin + s])];

        float3 x[MPT], v[MPT];
        float mass[MPT];
        uint32_t roff[MPT], rwid[MPT], frow[MPT];
#pragma unroll
        for (int j = 0; j < MPT; ++j) {
            const uint32_t m = tid + j * T;
            x[j] = make_float3(0.f, 0.f, 0.f);
            v[j] = make_float3(0.f, 0.f, 0.f);
            mass[j] = 1.0f;
            roff[j] = 0;
            rwid[j] = 0;
            frow[j] = 0;
            if (n_face && m < bd.n_mass) frow[j] = __ldg(&p.face_row[bd.mass_begin + m]);
            if (m < bd.n_mass) {
                const uint32_t g = __ldg(&p.mass_gidx[bd.mass_begin + m]);
                const float4 P = p.pos[g], V = p.vel[g];
                x[j] = make_float3(P.x, P.y, P.z);
                v[j] = make_float3(V.x, V.y, V.z);
                mass[j] = P.w;
                const uint32_t sl = bd.slice_begin + m / kSliceWidth;
                roff[j] = __ldg(&p.slice_off[sl]) + (m % kSliceWidth);
                rwid[j] = __ldg(&p.slice_width[sl]);
            }
        }
        __syncthreads();

        for (uint32_t step = 0; step < p.steps; ++step) {
            if (tid < n_mat) {
                smat[tid].x = next_rate;
                if (step + 1 < p.steps) next_rate = __ldg(&p.rates[(step + 1) * n_mat + tid]);
            }
#pragma unroll
            for (int j = 0; j < MPT; ++j) {
                const uint32_t m = tid + j * T;
                if (m >= bd.n_mass) break;
                if (XPBD)
                    sxt[m] = make_float4(__fadd_rn(x[j].x, __fmul_rn(v[j].x, dt)),
                                         __fadd_rn(x[j].y, __fmul_rn(v[j].y, dt)),
                                         __fadd_rn(x[j].z, __fmul_rn(v[j].z, dt)), 0.0f);
                else
                    sxt[m] = make_float4(x[j].x, x[j].y, x[j].z, 0.0f);
                if (n_face) sv[m] = make_float4(v[j].x, v[j].y, v[j].z, 0.0f);
            }
            __syncthreads();
            for (uint32_t s = tid; s < bd.n_spring; s += T) {
                const uint32_t w = __ldg(&pair[s]);
                const float lb = __ldg(&lbar[s]);
                const float4 pa = sxt[pk_a(w)], pb = sxt[pk_b(w)];
                const float2 mt = smat[pk_slot(w)];
                const float L = __fmaf_rn(lb, mt.x, lb);
                const float dx = __fsub_rn(pa.x, pb.x);
                const float dy = __fsub_rn(pa.y, pb.y);
                const float dz = __fsub_rn(pa.z, pb.z);
                float nd, r;  // -d and 1 / (d + eps)
                length_and_reciprocal(__fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz))), nd, r);
                const float lam = __fmul_rn(-__fsub_rn(-nd, L), mt.y);
                const float coef = __fmul_rn(lam, r);
                __stcg(&dp[s], make_float4(__fmul_rn(coef, dx), __fmul_rn(coef, dy), __fmul_rn(coef, dz), 0.0f));
                if (TRACK) stp[s] = __fadd_rn(stp[s], __fmul_rn(XPBD ? lam : -lam, __frcp_rn(lb)));
            }
            for (uint32_t f = tid; f < n_face; f += T) {
                const uint2 c = __ldg(&fcorner[f]);
                const uint32_t i0 = c.x & 0xFFFFu, i1 = c.x >> 16, i2 = c.y;
                __stcg(&fd[f], face_force(sxt[i0], sxt[i1], sxt[i2], sv[i0], sv[i1], sv[i2], p.face_coef));
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < MPT; ++j) {
                const uint32_t m = tid + j * T;
                if (m >= bd.n_mass) break;
                float ax = 0.0f, ay = 0.0f, az = 0.0f;
                for (uint32_t k = 0; k < rwid[j]; ++k) {
                    const uint32_t e = __ldg(&inc[roff[j] + k * kSliceWidth]);
                    if (e != kPadEntry32) {
                        const float4 c = __ldcg(&dp[e >> 1]);
                        const float sg = __uint_as_float(0x3f800000u | ((e & 1u) << 31));
                        ax = __fmaf_rn(c.x, sg, ax);
                        ay = __fmaf_rn(c.y, sg, ay);
                        az = __fmaf_rn(c.z, sg, az);
                    }
                }
                // face drag after the springs, faces in ascending order
                for (uint32_t k = 0; k < (frow[j] >> 24); ++k) {
                    const float4 c = __ldcg(&fd[__ldg(&finc[(frow[j] & 0xFFFFFFu) + k])]);
                    ax = __fadd_rn(ax, c.x);
                    ay = __fadd_rn(ay, c.y);
                    az = __fadd_rn(az, c.z);
                }
                if (XPBD) {
                    const float4 xt = sxt[m];
                    const float nx = __fadd_rn(xt.x, ax);
                    const float ny = __fadd_rn(xt.y, ay);
                    const float nz = __fadd_rn(xt.z, az);
                    v[j].x = velocity_of(__fsub_rn(nx, x[j].x), ddt, inv_dt);
                    v[j].y = velocity_of(__fsub_rn(ny, x[j].y), ddt, inv_dt);
                    v[j].z = velocity_of(__fsub_rn(nz, x[j].z), ddt, inv_dt);
                    x[j] = make_float3(nx, ny, nz);
                } else {
                    force_integrate<MODE>(p, x[j], v[j], mass[j], inv_dt_f, ax, ay, az);
                }
            }
        }

        bool bad = false;
#pragma unroll
        for (int j = 0; j < MPT; ++j) {
            const uint32_t m = tid + j * T;
            if (m < bd.n_mass) {
                const uint32_t g = __ldg(&p.mass_gidx[bd.mass_begin + m]);
                p.pos[g] = make_float4(x[j].x, x[j].y, x[j].z, p.pos[g].w);
                p.vel[g] = make_float4(v[j].x, v[j].y, v[j].z, p.vel[g].w);
                bad |= !(isfinite(x[j].x) && isfinite(x[j].y) && isfinite(x[j].z));
            }
        }
        if (TRACK) {
            __syncthreads();
            for (uint32_t s = tid; s < bd.n_spring; s += T)
                p.stress[__ldg(&p.spring_gidx[bd.spring_begin + s])] = stp[s];
        }
        if (__syncthreads_or(bad) && tid == 0) atomicOr(&p.bin_flags[b], 1u);
    }
}

// Actuation factors of one launch.  Block b covers steps [256 b, 256 b + 256):
// thread 0 accumulates the float clock from t0 (the clock is a sequential
// float sum, Simulator.cu:447, so it is not reassociated), then the threads
// share the steps' materials (4 steps of 10 materials: 5.4 -> 3.9 us).
__global__ void __launch_bounds__(256) actuation_kernel(const float4* __restrict__ table,
                                                        const uint8_t* __restrict__ mat_ids,
                                                        const uint32_t* __restrict__ n_mat_ptr,
                                                        float t0, float dt, uint32_t steps,
                                                        uint32_t mode, float* __restrict__ rates,
                                                        float* __restrict__ invk) {
    __shared__ float s_t[256];
    const uint32_t n_mat = *n_mat_ptr;
    const uint32_t base = blockIdx.x * 256u;
    if (threadIdx.x == 0) {
        float t = t0;
        for (uint32_t i = 0; i < base; ++i) t = __fadd_rn(t, dt);
        const uint32_t n = min(256u, steps - base);
        for (uint32_t i = 0; i < n; ++i) {
            s_t[i] = t;
            t = __fadd_rn(t, dt);
        }
    }
    if (blockIdx.x == 0) {
        for (uint32_t i = threadIdx.x; i < n_mat; i += 256u) {
            const float4 mt = table[mat_ids[i]];
            if (mode == kModeXpbd) {
                // alpha = 1/k/dt/dt, K = 2 + alpha (sim_kernel.cu:220, 225)
                const float alpha = __fdiv_rn(__fdiv_rn(__fdiv_rn(1.0f, mt.x), dt), dt);
                invk[i] = __frcp_rn(__fadd_rn(2.0f, alpha));
            } else {
                invk[i] = mt.x;
            }
        }
    }
    __syncthreads();
    // the block's (step, material) pairs over its threads, materials first
    const uint32_t pairs = min(256u, steps - base) * n_mat;
    for (uint32_t k = threadIdx.x; k < pairs; k += 256u) {
        const uint32_t n = k / n_mat, i = k - n * n_mat;
        const float4 mt = table[mat_ids[i]];
        const float arg = __fmaf_rn(mt.z, s_t[n], mt.w);
        rates[(size_t)base * n_mat + k] = __fmul_rn(mt.y, __double2float_rn(sin_cw((double)arg)));
    }
}

// Centre of mass of non-air masses, one warp per robot: lane l sums masses
// l, l+32, ... in double, then an xor butterfly; mean rounded to float.
__global__ void com_kernel(const float4* __restrict__ pos, const uint8_t* __restrict__ mat,
                           const int64_t* __restrict__ off, uint32_t n_robots,
                           float* __restrict__ com) {
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const uint32_t lane = threadIdx.x % 32;
    if (warp >= n_robots) return;
    const int64_t b = off[warp], n = off[warp + 1] - b;
    double sx = 0.0, sy = 0.0, sz = 0.0;
    long long cnt = 0;
    for (int64_t i = lane; i < n; i += 32) {
        if (!mat[b + i]) continue;
        const float4 q = pos[b + i];
        sx = __dadd_rn(sx, (double)q.x);
        sy = __dadd_rn(sy, (double)q.y);
        sz = __dadd_rn(sz, (double)q.z);
        ++cnt;
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        sx = __dadd_rn(sx, __shfl_xor_sync(0xffffffffu, sx, o));
        sy = __dadd_rn(sy, __shfl_xor_sync(0xffffffffu, sy, o));
        sz = __dadd_rn(sz, __shfl_xor_sync(0xffffffffu, sz, o));
        cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    }
    if (lane == 0) {
        const double dc = (double)cnt;
        com[3 * warp + 0] = cnt ? __double2float_rn(__ddiv_rn(sx, dc)) : 0.0f;
        com[3 * warp + 1] = cnt ? __double2float_rn(__ddiv_rn(sy, dc)) : 0.0f;
        com[3 * warp + 2] = cnt ? __double2float_rn(__ddiv_rn(sz, dc)) : 0.0f;
    }
}

// Per-robot status: bit 0 set when any position of the robot is NaN/Inf.
// One warp per robot.
__global__ void flags_kernel(const float4* __restrict__ pos, const int64_t* __restrict__ off,
                             uint32_t n_robots, uint32_t* __restrict__ out) {
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const uint32_t lane = threadIdx.x % 32;
    if (warp >= n_robots) return;
    bool bad = false;
    for (int64_t i = off[warp] + lane; i < off[warp + 1]; i += 32) {
        const float4 q = pos[i];
        bad |= !(isfinite(q.x) && isfinite(q.y) && isfinite(q.z));
    }
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) out[warp] = bad ? 1u : 0u;
}

using StepFn = void (*)(const StepParams);

struct ShapeEntry {
    uint32_t threads, spt, mpt;
    StepFn fn[4][2];  // [mode][track]; mode 3: water with face drag
};

#define MB_SHAPE(T, S, M, SPLIT)                                                               \
    {                                                                                          \
        T, S, M, {                                                                             \
            {step_kernel<T, S, M, kModeXpbd, false, SPLIT>,                                    \
             step_kernel<T, S, M, kModeXpbd, true, SPLIT>},                                    \
                {step_kernel<T, S, M, kModeForceLand, false, SPLIT>,                           \
                 step_kernel<T, S, M, kModeForceLand, true, SPLIT>},                           \
                {step_kernel<T, S, M, kModeForceWater, false, SPLIT>,                          \
                 step_kernel<T, S, M, kModeForceWater, true, SPLIT>},                          \
                {step_kernel<T, S, M, kModeForceWaterFaces, false, SPLIT>,                     \
                 step_kernel<T, S, M, kModeForceWaterFaces, true, SPLIT>},                     \
        }                                                                                      \
    }
const ShapeEntry kShapes[] = {
    MB_SHAPE(256, 8, 2, false),   MB_SHAPE(512, 4, 1, false),   MB_SHAPE(512, 8, 2, false),
    MB_SHAPE(512, 16, 4, false),  MB_SHAPE(1024, 4, 1, false),  MB_SHAPE(1024, 6, 2, false),
    MB_SHAPE(1024, 8, 2, false),  MB_SHAPE(1024, 10, 2, false), MB_SHAPE(1024, 12, 2, false),
};
// the parts of split robots (thread-block clusters)
const ShapeEntry kSplitShapes[] = {
    MB_SHAPE(1024, 8, 1, true),
    MB_SHAPE(1024, 10, 1, true),
    MB_SHAPE(1024, 8, 2, true),
    MB_SHAPE(1024, 10, 2, true),
    MB_SHAPE(1024, 12, 2, true),
};
#undef MB_SHAPE


struct StreamEntry {
    uint32_t threads, mpt;
    StepFn fn[4][2];  // [mode][track]; mode 3: water with face drag
};
#define MB_STREAM(T, M)                                                                          \
    {                                                                                            \
        T, M, {                                                                                  \
            {stream_kernel<T, M, kModeXpbd, false>, stream_kernel<T, M, kModeXpbd, true>},       \
                {stream_kernel<T, M, kModeForceLand, false>,                                     \
                 stream_kernel<T, M, kModeForceLand, true>},                                     \
                {stream_kernel<T, M, kModeForceWater, false>,                                    \
                 stream_kernel<T, M, kModeForceWater, true>},                                    \
                {stream_kernel<T, M, kModeForceWaterFaces, false>,                               \
                 stream_kernel<T, M, kModeForceWaterFaces, true>},                               \
        }                                                                                        \
    }
// up to threads * MPT masses per bin (2,048 or 4,096 with 1,024 threads)
const StreamEntry kStream[] = {MB_STREAM(1024, 2), MB_STREAM(1024, 4)};
#undef MB_STREAM

const StreamEntry* find_stream(uint32_t threads, uint32_t mpt) {
    for (const auto& e : kStream)
        if (e.threads == threads && e.mpt == mpt) return &e;
    return nullptr;
}

const ShapeEntry* find_shape(const KernelShape& s) {
    for (const auto& e : kShapes)
        if (e.threads == s.threads && e.spt == s.spt && e.mpt == s.mpt) return &e;
    return nullptr;
}

const ShapeEntry* find_split(const KernelShape& s) {
    for (const auto& e : kSplitShapes)
        if (e.threads == s.threads && e.spt == s.spt && e.mpt == s.mpt) return &e;
    return nullptr;
}

}  // namespace

uint32_t bin_smem_bytes(uint32_t n_mass, uint32_t n_spring, uint32_t n_inc) {
    return bin_smem_bytes_dev(n_mass, n_spring, n_inc);
}

uint32_t max_step_smem(int device) {
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    return (uint32_t)v;
}

cudaError_t allow_smem(const void* kernel, uint32_t smem_bytes) {
    int device = 0;
    const cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    const uint32_t most = max_step_smem(device);
    if (smem_bytes > most) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}

bool shape_supported(const KernelShape& shape) { return find_shape(shape) != nullptr; }

bool split_supported(const KernelShape& shape) { return find_split(shape) != nullptr; }

cudaError_t prepare_split(const KernelShape& shape, uint32_t mode, bool track, uint32_t smem_bytes) {
    const ShapeEntry* e = find_split(shape);
    if (!e || mode > kModeForceWater) return cudaErrorInvalidValue;
    cudaError_t r = allow_smem(reinterpret_cast<const void*>(e->fn[mode][track ? 1 : 0]), smem_bytes);
    if (r == cudaSuccess && mode == kModeForceWater)  // and the face-drag variant
        r = allow_smem(reinterpret_cast<const void*>(e->fn[kModeForceWaterFaces][track ? 1 : 0]), smem_bytes);
    return r;
}

// One CTA per part, the parts of a robot (bins r*C .. r*C + C-1) forming a
// cluster of C CTAs.
cudaError_t launch_split(const StepParams& p, const KernelShape& shape, uint32_t cluster, cudaStream_t s) {
    const ShapeEntry* e = find_split(shape);
    if (!e || p.mode > kModeForceWater || cluster < 2 || cluster > 8 || p.n_bins % cluster)
        return cudaErrorInvalidValue;
    if (p.n_bins == 0) return cudaSuccess;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(p.n_bins, 1, 1);
    cfg.blockDim = dim3(shape.threads, 1, 1);
    cfg.dynamicSmemBytes = p.smem_bytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const uint32_t variant = p.mode == kModeForceWater && p.face_on ? kModeForceWaterFaces : p.mode;
    return cudaLaunchKernelEx(&cfg, e->fn[variant][p.track ? 1 : 0], p);
}

cudaError_t prepare_step(const KernelShape& shape, uint32_t mode, bool track, uint32_t smem_bytes) {
    const ShapeEntry* e = find_shape(shape);
    if (!e || mode > kModeForceWater) return cudaErrorInvalidValue;
    cudaError_t r = allow_smem(reinterpret_cast<const void*>(e->fn[mode][track ? 1 : 0]), smem_bytes);
    if (r == cudaSuccess && mode == kModeForceWater)  // and the face-drag variant
        r = allow_smem(reinterpret_cast<const void*>(e->fn[kModeForceWaterFaces][track ? 1 : 0]), smem_bytes);
    return r;
}

int ctas_per_sm(const KernelShape& shape, uint32_t mode, bool track, uint32_t smem_bytes) {
    const ShapeEntry* e = find_shape(shape);
    if (!e || mode > kModeForceWater) return 0;
    StepFn fn = e->fn[mode][track ? 1 : 0];
    if (allow_smem(reinterpret_cast<const void*>(fn), smem_bytes) != cudaSuccess) return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, (int)shape.threads, smem_bytes) != cudaSuccess)
        return 0;
    return n;
}

int max_active_clusters(const KernelShape& shape, uint32_t mode, uint32_t cluster, uint32_t smem_bytes) {
    const ShapeEntry* e = find_split(shape);
    if (!e || mode > kModeForceWater || cluster < 1 || cluster > kMaxClusterParts) return 0;
    StepFn fn = e->fn[mode][0];
    if (allow_smem(reinterpret_cast<const void*>(fn), smem_bytes) != cudaSuccess) return 0;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(cluster, 1, 1);
    cfg.blockDim = dim3(shape.threads, 1, 1);
    cfg.dynamicSmemBytes = smem_bytes;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return n;
}

uint32_t list_shapes(KernelShape* out, uint32_t cap, bool streamed) {
    uint32_t n = 0;
    if (streamed) {
        for (const auto& e : kStream) {
            if (n < cap) out[n] = KernelShape{e.threads, 0, e.mpt};
            ++n;
        }
    } else {
        for (const auto& e : kShapes) {
            if (n < cap) out[n] = KernelShape{e.threads, e.spt, e.mpt};
            ++n;
        }
    }
    return n;
}

uint32_t stream_smem_bytes(uint32_t n_mass) { return 16u * n_mass + 8u * kMaxMaterialSlots; }

bool stream_supported(uint32_t threads, uint32_t mpt) { return find_stream(threads, mpt) != nullptr; }

cudaError_t prepare_stream(uint32_t threads, uint32_t mpt, uint32_t mode, bool track,
                           uint32_t smem_bytes) {
    const StreamEntry* e = find_stream(threads, mpt);
    if (!e || mode > kModeForceWater) return cudaErrorInvalidValue;
    cudaError_t r = allow_smem(reinterpret_cast<const void*>(e->fn[mode][track ? 1 : 0]), smem_bytes);
    if (r == cudaSuccess && mode == kModeForceWater)  // and the face-drag variant
        r = allow_smem(reinterpret_cast<const void*>(e->fn[kModeForceWaterFaces][track ? 1 : 0]), smem_bytes);
    return r;
}

cudaError_t launch_stream(const StepParams& p, uint32_t threads, uint32_t mpt, cudaStream_t s) {
    const StreamEntry* e = find_stream(threads, mpt);
    if (!e || p.mode > kModeForceWater) return cudaErrorInvalidValue;
    if (p.n_bins == 0) return cudaSuccess;
    const uint32_t variant = p.mode == kModeForceWater && p.face_on ? kModeForceWaterFaces : p.mode;
    e->fn[variant][p.track ? 1 : 0]<<<p.n_bins, threads, p.smem_bytes, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_step(const StepParams& p, const KernelShape& shape, cudaStream_t s) {
    const ShapeEntry* e = find_shape(shape);
    if (!e) return cudaErrorInvalidValue;
    if (p.n_bins == 0) return cudaSuccess;
    if (p.mode > kModeForceWater) return cudaErrorInvalidValue;
    const uint32_t grid = p.grid ? std::min(p.grid, p.n_bins) : p.n_bins;
    const uint32_t variant = p.mode == kModeForceWater && p.face_on ? kModeForceWaterFaces : p.mode;
    e->fn[variant][p.track ? 1 : 0]<<<grid, shape.threads, p.smem_bytes, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_actuation(const float4* table, const uint8_t* mat_ids, const uint32_t* n_mat,
                             float t0, float dt, uint32_t steps, uint32_t mode, float* rates,
                             float* coef, cudaStream_t s) {
    if (steps == 0) return cudaSuccess;
    actuation_kernel<<<(steps + 255) / 256, 256, 0, s>>>(table, mat_ids, n_mat, t0, dt, steps, mode,
                                                         rates, coef);
    return cudaGetLastError();
}

cudaError_t launch_com(const float4* pos, const uint8_t* mass_mat, const int64_t* mass_off,
                       uint32_t n_robots, float* com, cudaStream_t s) {
    if (n_robots == 0) return cudaSuccess;
    const uint32_t threads = 256, warps = threads / 32;
    com_kernel<<<(n_robots + warps - 1) / warps, threads, 0, s>>>(pos, mass_mat, mass_off,
                                                                   n_robots, com);
    return cudaGetLastError();
}

cudaError_t launch_flags(const float4* pos, const int64_t* mass_off, uint32_t n_robots,
                         uint32_t* out, cudaStream_t s) {
    if (n_robots == 0) return cudaSuccess;
    const uint32_t threads = 256, warps = threads / 32;
    flags_kernel<<<(n_robots + warps - 1) / warps, threads, 0, s>>>(pos, mass_off, n_robots, out);
    return cudaGetLastError();
}

}  // namespace mb
