// Resident step kernel with per-thread operands in tensor memory (sm_100a).
//
// The step of mb_kernels.cu (reference sim_kernel.cu:141-269) for resident
// bins, laid out for what bounded it there: the shared-memory pipe (71 % busy,
// 33 wavefronts per 32 springs) and the issue slots (70 %, 130 instructions
// per spring; counters of 512 robots of 3-8 cells).
//   - A mass sums its springs in ascending order of the other end, so first
//     those to lower masses.  The thread of a mass computes exactly these
//     (its own position stays in registers, one position load a spring
//     instead of two), adds them up as they come, and stores each for the
//     lower end; after a barrier it adds the springs to higher masses, read
//     from their owners.  Each correction is stored once and loaded once.
//   - Corrections are kept as {x, y} and z (3 wavefronts a warp instead of 4)
//     at slot 32 k + lane of the owner's slice: consecutive masses read
//     consecutive slots, free of bank conflicts in every direction of a
//     lattice.
//   - Operands that belong to one thread for a whole launch (address of the
//     other end, material, mean length, stress, slots to gather) live in
//     tensor memory, which is read beside the shared-memory pipe: 32 warps x
//     8 words in 81 cycles, no slower next to LDS.128 at full rate.
//   - A CTA is split into warp groups with their own bins and barriers, so
//     that one bin's latencies run under another's work.
//   - Square root and reciprocal come from one approximation and are
//     correctly rounded without branches (mb_step_math.cuh).
// A step of those 512 robots then takes 21 wavefronts per 32 springs and 98
// instructions per spring, 5.3 us instead of 7.3.  What bounds it now is issue
// (69 %) and the warps waiting at barriers (a quarter of the stalls).  Two
// kernels: at most 24 warps of 80 registers (without tracking they spill 4-28
// bytes a thread and load 4-52; 28 warps of 72 registers and 32 of 64 measured
// 7.4 and 8.3 us there), and at
// most 16 of up to 128 (WIDE, below); the plan takes the one whose estimated
// step is shorter.
// With stress tracking the same 512 robots take 7.8 us (8.5 with the springs
// in registers and shared memory); bins of 769-1,024 masses, such as two robots
// of 5-8 cells, run two masses a thread on 16 warps: 260 such robots 5.2 us
// instead of 6.1.
// With the face drag, a face is one more correction slot: computed by any
// thread beside the springs (velocities ride in the positions' w and one more
// plane: 3 x 24 bytes of loads a face instead of 3 x 32), gathered after the
// springs' slots by words in the same columns.  The 512 robots with 215,000
// faces: 16.5 -> 10.0 us a step; bound by the shared-memory pipe (73 %, of it
// 29 % bank conflicts of the faces' corners and gathers).
// Same operations in the same order as the oracle: same bits.
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <type_traits>

#include "mb_step_math.cuh"
#include "mb_tm.h"
#include "mb_tmem.cuh"

namespace mb {

namespace {

template <bool WIDE>
__device__ __forceinline__ void group_sync(uint32_t id, uint32_t threads) {
    if (WIDE && threads == 32)
        __syncwarp();  // a group of one warp
    else
        asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Shared memory by 32-bit address: operands hold addresses, so that an
// access needs no address arithmetic.
__device__ __forceinline__ float2 lds2(uint32_t a) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ float lds1(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ float4 lds4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts4(uint32_t a, float x, float y, float z, float w) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}
__device__ __forceinline__ void sts2(uint32_t a, float x, float y) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ void lds_xyz(uint32_t a, f32x2& xy, float& z) {  // 16-byte position
    f32x2 zw;
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(xy), "=l"(zw) : "r"(a));
    float w;
    unpack2(zw, z, w);
}
__device__ __forceinline__ f32x2 lds_pair(uint32_t a) {
    f32x2 v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts_pair(uint32_t a, f32x2 v) {
    asm volatile("st.shared.b64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
__device__ __forceinline__ uint4 lds_info(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts_info(uint32_t a, uint4 v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void sts1(uint32_t a, float x) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(x) : "memory");
}

// What a group needs of its bin outside the hot path of a step, in shared
// memory so that the step loop holds no registers for it.
struct TmBin {
    uint32_t bin, mass_begin, n_mass, slice_begin;
    uint32_t n_mat;     // material factors of the bin; the next one is zero
    uint32_t x0, mat0;  // shared addresses of the positions and the factors
    uint32_t xy0, z0;   // of slot 0's correction
    uint32_t row;       // row length of the actuation table
    // face drag: faces of the bin, their corners, the velocities' address less
    // half that of the positions, slot 0's force
    uint32_t n_face, face0, v_base, face_xy, face_z;
};
static_assert(sizeof(TmBin) * kTmMaxGroups + sizeof(uint32_t) <= kTmHeadBytes, "");
template <int OFFSET>
__device__ __forceinline__ uint32_t bin_word(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(OFFSET));
    return v;
}
template <int OFFSET>
__device__ __forceinline__ void set_bin_word(uint32_t a, uint32_t v) {
    asm volatile("st.shared.b32 [%0+%1], %2;" ::"r"(a), "n"(OFFSET), "r"(v) : "memory");
}
// (through one 32-bit address: as a C++ object at the start of the dynamic
// shared memory it cost the 24-warp kernels registers, and 3 % of a step)
#define TM_BIN(field) bin_word<(int)offsetof(TmBin, field)>(bin_mine)
#define TM_BIN_SET(field, v) set_bin_word<(int)offsetof(TmBin, field)>(bin_mine, v)

// Operand of an own spring: address of the other end | of the material
// factors << 16.
__device__ __forceinline__ uint32_t spring_word(uint32_t entry, uint32_t x0, uint32_t mat0, uint32_t n_mat) {
    const bool pad = entry >> 31;
    return (x0 + 16u * (pad ? entry & 7u : kTmStandIns + (entry & 0xFFFFu))) | (mat0 + 8u * (pad ? n_mat : entry >> 16)) << 16;
}

// Gather word k of a mass's faces (`row`: first entry | count << 24): slots
// from `slot0` in face order, then zero slots.
__device__ __forceinline__ uint32_t face_word(const uint16_t* inc, uint32_t row, uint32_t k, uint32_t slot0, uint32_t lane) {
    const uint32_t n = row >> 24, at = (row & 0xFFFFFFu) + 2 * k;
    const uint32_t lo = 2 * k < n ? slot0 + __ldg(&inc[at]) : lane;
    return lo | (2 * k + 1 < n ? slot0 + __ldg(&inc[at + 1]) : lane) << 16;
}

// Columns of one mass: `own` springs in pairs {address of the other end |
// of the material factors << 16} x 2, {mean length} x 2, their stresses in
// pairs, the gather words.
struct TmColumns {
    uint32_t stress, gather, end;
    __host__ __device__ TmColumns(uint32_t own, uint32_t words, bool track) {
        stress = 4 * ((own + 1) / 2);
        gather = (stress + (track ? 2 * ((own + 1) / 2) : 0u) + 3u) & ~3u;
        end = (gather + words + 3u) & ~3u;
    }
};

// WIDE: at most kTmWideWarps warps, so registers for four springs at a time:
// with few warps an SM, latency has to be hidden within the warp (32 robots of
// 4x4x4 cells, one an SM: 1.84 -> 1.55 us a step; 282 robots of 5-8 cells, two
// masses a thread: 4.3 us, 5.0 on 24 warps).  The last three of a row go
// together too, and with one mass a thread the first words are read before the
// barriers: a robot of one cell, seven springs a row, 1.18 -> 1.08 us, with
// tracking 1.52 -> 1.16.
template <int MODE, bool TRACK, int MPT, bool WIDE>
__global__ void __launch_bounds__(32 * (WIDE ? kTmWideWarps : kTmMaxWarps), 1) tm_step_kernel(const __grid_constant__ TmParams q) {
    constexpr bool XPBD = MODE == kModeXpbd;
    constexpr bool FACES = MODE == kModeForceWaterFaces;  // face drag compiled in
    // one mass a thread and registers to spare: the slice's data stay in
    // registers, and the first words are read ahead of the barriers
    constexpr bool AHEAD = WIDE && MPT == 1;
    // (all shared memory is dynamic, so that the plan's sum is what a launch asks
    // for; its first kTmHeadBytes: every group's TmBin, the allocation's word)
    extern __shared__ __align__(128) uint8_t tm_smem[];
    const StepParams& p = q.p;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // the CTA's columns, a power of two, shared by its warps' four lane quarters
    const uint32_t per_quarter = (blockDim.x / 32 + 3) / 4;
    const uint32_t cols = per_quarter <= 2 ? 256u : 512u, my_cols = (cols / per_quarter) & ~3u;
    const uint32_t tmem0 = tm_alloc(reinterpret_cast<uint32_t*>(tm_smem + kTmMaxGroups * sizeof(TmBin)), cols);
    const uint32_t tm = tmem0 + ((warp & 3u) << 21) + (warp >> 2) * my_cols;  // this warp's words

    // this warp's group (lane g of 8 looks at group g); warps without one wait
    // for the others at the end
    uint32_t gi;
    TmGroup grp;
    {
        const TmGroup mine = q.groups[blockIdx.x * kTmMaxGroups + (lane & 7u)];
        const uint32_t in = __ballot_sync(0xffffffffu, warp >= mine.warp0 && warp < mine.warp0 + mine.warps) & 0xFFu;
        gi = in ? (uint32_t)__ffs(in) - 1u : 0u;
        auto of = [&](uint32_t v) { return __shfl_sync(0xffffffffu, v, gi); };
        grp.first = of(mine.first);
        grp.count = in ? of(mine.count) : 0u * of(mine.count);
        grp.warp0 = of(mine.warp0);
        grp.warps = of(mine.warps);
        grp.mat_off = of(mine.mat_off);
        grp.x_off = of(mine.x_off);
        grp.xy_off = of(mine.xy_off);
        grp.z_off = of(mine.z_off);
        grp.info_off = of(mine.info_off);
        grp.spare_off = of(mine.spare_off);
        if (FACES) {
            grp.v_off = of(mine.v_off);
            grp.face_off = of(mine.face_off);
        }
    }
    const uint32_t gw = warp - grp.warp0;  // warp of the group
    const uint32_t gt = gw * 32 + lane;    // thread of the group
    const uint32_t GT = 32u * grp.warps;   // the group's threads
    const uint32_t bar = 1 + gi;
    const uint32_t bin_mine = smem_addr(tm_smem) + gi * (uint32_t)sizeof(TmBin);
    const float dt = p.dt;
    // shared memory of the group: material factors {dL0 sin(..), 1/K}, the
    // positions, the corrections
    const uint32_t smem0 = smem_addr(tm_smem), mat_mine = smem0 + grp.mat_off + 8u * gt;
    const uint32_t x_mine = smem0 + grp.x_off + 16u * (kTmStandIns + gt);
    // What the warp's slices (sl = gw, gw + warps) need in a step is read from
    // shared memory, 32 bytes a slice, rather than held in registers:
    //   {first address of the own corrections {x, y}, of z, own springs kept
    //    in tensor memory | all << 16, their first column}
    //   {column of the gather words, words kept | all << 16, address of the
    //    words kept in shared memory, or 0}
    const uint32_t info_mine = smem0 + grp.info_off + 32u * gw;

    for (uint32_t bi = 0; bi < grp.count; ++bi) {
        // ---- the bin, its materials and one of stiffness 0, the zero slots
        // and the stand-in positions (far from any robot)
        const TmBinRef ref = q.bins[grp.first + bi];
        const uint32_t n_mat = __ldg(&q.r.n_mat[ref.bin]);
        const uint32_t x0 = smem0 + grp.x_off, mat0 = smem0 + grp.mat_off, xy0 = smem0 + grp.xy_off, z0 = smem0 + grp.z_off;
        // the actuation factor of material gt, loaded one step ahead; further
        // materials (more than threads): loaded when needed
        uint32_t rate_at = gt < 256u ? __ldg(&q.r.mat[256u * ref.bin + gt]) : 0u;
        const bool my_mat = gt < n_mat, more_mats = gt + GT < n_mat;
        float next_rate = my_mat ? __ldg(p.rates + rate_at) : 0.0f;
        if (my_mat) sts1(mat_mine + 4u, __ldg(&p.invk[rate_at]));  // 1/K (reference step) or k (force modes)
        for (uint32_t i = gt + GT; i < n_mat; i += GT)
            sts1(mat0 + 8u * i + 4u, __ldg(&p.invk[__ldg(&q.r.mat[256u * ref.bin + i])]));
        if (gt == 0) {
            TM_BIN_SET(bin, ref.bin);
            TM_BIN_SET(mass_begin, ref.mass_begin);
            TM_BIN_SET(n_mass, ref.n_mass);
            TM_BIN_SET(slice_begin, ref.slice_begin);
            TM_BIN_SET(n_mat, n_mat);
            TM_BIN_SET(x0, x0);
            TM_BIN_SET(mat0, mat0);
            TM_BIN_SET(xy0, xy0);
            TM_BIN_SET(z0, z0);
            TM_BIN_SET(row, *p.n_mat);
            if (FACES) {
                const uint32_t slots = __ldg(&q.r.n_slots[ref.bin]);
                TM_BIN_SET(n_face, ref.n_face);
                TM_BIN_SET(face0, smem0 + grp.face_off);
                TM_BIN_SET(v_base, smem0 + grp.v_off - x0 / 2);
                TM_BIN_SET(face_xy, xy0 + 8u * slots);
                TM_BIN_SET(face_z, z0 + 4u * slots);
            }
            sts2(mat0 + 8u * n_mat, 0.0f, 0.0f);
        }
        if (gt < kTmZeros) {
            sts2(xy0 + 8u * gt, 0.0f, 0.0f);
            sts1(z0 + 4u * gt, 0.0f);
        }
        if (gt < kTmStandIns) sts4(x0 + 16u * gt, 1.0e6f, 0.0f, 0.0f, 0.0f);
        if (FACES)  // addresses of the corners' positions, {first | second << 16, third}
            for (uint32_t f = gt; f < ref.n_face; f += GT) {
                const uint2 c = __ldg(&p.faces[ref.face_begin + f]);
                const uint32_t m0 = x0 + 16u * kTmStandIns, c0 = m0 + 16u * (c.x & 0xFFFFu), c1 = m0 + 16u * (c.x >> 16);
                sts2(smem0 + grp.face_off + 8u * f, __uint_as_float(c0 | c1 << 16), __uint_as_float(m0 + 16u * c.y));
            }
        // ---- masses m = gt + j GT, and their operands into tensor memory
        const uint32_t n_slices = (ref.n_mass + 31) / 32;
        // slices of this warp
        const uint32_t mine = gw >= n_slices ? 0u : 1u + (MPT > 1 && gw + grp.warps < n_slices);
        float3 x[MPT], v[MPT];
        float mass[MPT];
        uint32_t gidx = 0;  // WIDE: the mass's index and w components, for the write-back
        float vw = 0.0f;
        uint32_t free_col = 0;
        uint4 info_own = make_uint4(0, 0, 0, 0), info_gather = info_own;  // AHEAD
#pragma unroll
        for (int j = 0; j < MPT; ++j) {
            const uint32_t m = gt + j * GT, sl = gw + j * grp.warps;
            x[j] = make_float3(0.f, 0.f, 0.f);
            v[j] = make_float3(0.f, 0.f, 0.f);
            mass[j] = 1.0f;
            if (j >= mine) continue;
            const uint4 h = __ldg(&q.r.head[ref.slice_begin + sl]);
            uint32_t face_row = 0;
            if (FACES && ref.n_face && m < ref.n_mass) face_row = __ldg(&p.face_row[ref.mass_begin + m]);
            if (m < ref.n_mass) {
                const uint32_t g = __ldg(&p.mass_gidx[ref.mass_begin + m]);
                const float4 P = p.pos[g], V = p.vel[g];
                x[j] = make_float3(P.x, P.y, P.z);
                mass[j] = P.w;
                v[j] = make_float3(V.x, V.y, V.z);
                if (WIDE && MPT == 1) {
                    gidx = g;
                    vw = V.w;
                }
            }
            __syncwarp();
            const uint32_t own = h.x & 0xFFFFu, spring_words = h.x >> 16, rw = h.z + lane;
            // the faces' forces are gathered after the springs' (sim_kernel.cu:246-252)
            const uint32_t words = spring_words + (FACES ? (__reduce_max_sync(0xffffffffu, face_row >> 24) + 1) / 2 : 0u);
            // what fits the columns left: own springs first (in pairs), then
            // the gather words
            // (the step loop reads up to two pairs past the last one: room for them)
            constexpr uint32_t kPast = WIDE ? 8u : 4u;
            const uint32_t left = my_cols - free_col, room = left - kPast;
            const uint32_t own_kept = left < kPast ? 0u : min(own, TRACK ? 2 * (room / 6u) : 2 * (room / 4u) + (WIDE ? 0u : 1u));
            const TmColumns tc(own_kept, words, TRACK);
            const uint32_t words_kept = tc.gather <= left ? min(words, left - tc.gather) : 0u;
            // gather words that the columns do not hold: in the group's spare
            // shared memory, else in global memory
            const uint32_t spare = j && words > words_kept && words - words_kept <= kTmSpareWords
                                       ? smem0 + grp.spare_off + (128u * kTmSpareWords) * gw : 0u;
            const uint32_t c0 = tm + free_col;
            uint32_t odd = 0;  // tracking: some mean length's reciprocal needs the general one
            auto check_length = [&](uint32_t lb) {
                const float x = __uint_as_float(lb);
                if (TRACK) odd |= __float_as_uint(rcp_fast(x)) != __float_as_uint(__frcp_rn(x));
            };
            __syncwarp();
#pragma unroll 4
            for (uint32_t k = 0; k < own_kept; k += 2) {
                const uint2 e0 = __ldg(&q.r.own[rw + 32 * k]);
                const uint2 e1 = k + 1 < own_kept ? __ldg(&q.r.own[rw + 32 * (k + 1)]) : make_uint2(1u << 31, __float_as_uint(1.0f));
                tm_st2(c0 + 2 * k, spring_word(e0.x, x0, mat0, n_mat), spring_word(e1.x, x0, mat0, n_mat));
                tm_st2(c0 + 2 * k + 2, e0.y, e1.y);
                check_length(e0.y);
                check_length(e1.y);
                __syncwarp();
            }
            if (TRACK) {
                for (uint32_t k = own_kept; k < own; ++k) check_length(__ldg(&q.r.own[rw + 32 * k]).y);
                odd = __any_sync(0xffffffffu, odd);
                // stresses, eight at a time (loads of two latencies in a chain)
                for (uint32_t k = 0; k < own_kept; k += 8) {
                    uint32_t g[8], st[8];
#pragma unroll
                    for (uint32_t u = 0; u < 8; ++u) g[u] = k + u < own_kept ? __ldg(&q.r.gidx[rw + 32 * (k + u)]) : ~0u;
#pragma unroll
                    for (uint32_t u = 0; u < 8; ++u) st[u] = g[u] != ~0u ? __float_as_uint(p.stress[g[u] & 0x7FFFFFFFu]) : 0u;
                    __syncwarp();
#pragma unroll
                    for (uint32_t u = 0; u < 8; u += 2)
                        if (k + u < own_kept) tm_st2(c0 + tc.stress + k + u, st[u], st[u + 1]);
                }
            }
            info_own = make_uint4(xy0 + 8u * h.y, z0 + 4u * h.y, own_kept | own << 16 | odd << 31, c0);
            info_gather = make_uint4(c0 + tc.gather, words_kept | words << 16, spare, 0u);
            if (lane == 0) {
                sts_info(info_mine + j * GT, info_own);
                sts_info(info_mine + j * GT + 16u, info_gather);
            }
            __syncwarp();
#pragma unroll 4
            for (uint32_t k = 0; k < words; ++k) {
                const uint32_t w = !FACES || k < spring_words
                                       ? __ldg(&q.r.gather[rw + 32 * k])
                                       : face_word(p.face_inc + ref.face_inc_begin, face_row, k - spring_words,
                                                   __ldg(&q.r.n_slots[ref.bin]), lane);
                if (FACES) __syncwarp();
                if (k < words_kept)
                    tm_st(c0 + tc.gather + k, w);
                else if (spare)
                    sts1(spare + 128u * (k - words_kept) + 4u * lane, __uint_as_float(w));
            }
            free_col = min(my_cols, (tc.gather + words_kept + 3u + free_col) & ~3u);
        }
        tm_wait_st();
        __syncwarp();
        group_sync<WIDE>(bar, GT);

        for (uint32_t step = 0; step < p.steps; ++step) {
            // (1) actuation factors (sim_kernel.cu:222); predicted positions
            // x~ = x + v dt (sim_kernel.cu:147-152), or the current ones
            if (my_mat) {
                sts1(mat_mine, next_rate);
                rate_at += TM_BIN(row);
                if (step + 1 < p.steps) next_rate = __ldg(p.rates + rate_at);
            }
            if (more_mats)
                for (uint32_t i = gt + GT; i < TM_BIN(n_mat); i += GT)
                    sts1(TM_BIN(mat0) + 8u * i, __ldg(p.rates + (size_t)step * TM_BIN(row) + __ldg(&q.r.mat[256u * TM_BIN(bin) + i])));
            float ax[MPT], ay[MPT], az[MPT];
#pragma unroll
            for (int j = 0; j < MPT; ++j) {
                if (j >= mine) break;
                const float3 xt = XPBD ? make_float3(__fadd_rn(x[j].x, __fmul_rn(v[j].x, dt)), __fadd_rn(x[j].y, __fmul_rn(v[j].y, dt)),
                                                     __fadd_rn(x[j].z, __fmul_rn(v[j].z, dt)))
                                       : x[j];
                sts4(x_mine + 16u * j * GT, xt.x, xt.y, xt.z, FACES ? v[j].x : 0.0f);
                if (FACES) sts2(x_mine / 2 + 8u * j * GT + TM_BIN(v_base), v[j].y, v[j].z);
            }
            __syncwarp();
            // a slice's next own springs {words, lengths} x 2 (and stresses), the two
            // after them, and gather words: a block of four, then two and one
            struct Words {
                uint32_t c[4], st[2], c2[4], st2[2], g4[4], g2[2], g1[1];
            } ahead;
            auto first_springs = [&](const uint4& info, Words& w) {
                const uint32_t kept = info.z & 0xFFFFu, ta = info.w, ts = ta + 4 * ((kept + 1) / 2);
                if (!kept) return;
                tm_ld(ta, w.c);
                if (TRACK) tm_ld(ts, w.st);
                if (WIDE) {
                    tm_ld(ta + 4, w.c2);
                    if (TRACK) tm_ld(ts + 2, w.st2);
                }
            };
            if (TRACK) tm_wait_st();  // the last step's stresses
            if (AHEAD && mine) first_springs(info_own, ahead);
            group_sync<WIDE>(bar, GT);
            if (FACES) {  // the share of each corner, per face, stored like a correction
                const uint32_t n = TM_BIN(n_face), face0 = TM_BIN(face0), vb = TM_BIN(v_base), fxy = TM_BIN(face_xy), fz = TM_BIN(face_z);
                for (uint32_t f = gt; f < n; f += GT) {
                    const float2 c = lds2(face0 + 8u * f);
                    const uint32_t a0 = __float_as_uint(c.x) & 0xFFFFu, a1 = __float_as_uint(c.x) >> 16, a2 = __float_as_uint(c.y);
                    const float4 x0 = lds4(a0), x1 = lds4(a1), x2 = lds4(a2);  // (w: the velocity's x)
                    const float2 u0 = lds2(a0 / 2 + vb), u1 = lds2(a1 / 2 + vb), u2 = lds2(a2 / 2 + vb);
                    const float4 r = face_force(x0, x1, x2, make_float4(x0.w, u0.x, u0.y, 0.0f), make_float4(x1.w, u1.x, u1.y, 0.0f),
                                                make_float4(x2.w, u2.x, u2.y, 0.0f), p.face_coef);
                    sts2(fxy + 8u * f, r.x, r.y);
                    sts1(fz + 4u * f, r.z);
                }
                __syncwarp();
            }
            // (2) distance constraints to lower masses (sim_kernel.cu:209-243)
#pragma unroll
            for (int j = 0; j < MPT; ++j) {
                if (j >= mine) break;
                const uint4 info = AHEAD ? info_own : lds_info(info_mine + j * GT);
                const uint32_t kept = info.z & 0xFFFFu, own = TRACK ? (info.z >> 16) & 0x7FFFu : info.z >> 16, x_first = x_mine - 16u * gt;
                const bool plain_rcp = TRACK && info.z >> 31;
                // this mass's position, negated: differences are sums then
                f32x2 nxy;
                float nz;
                if (XPBD) {
                    nxy = pack2(__fsub_rn(-x[j].x, __fmul_rn(v[j].x, dt)), __fsub_rn(-x[j].y, __fmul_rn(v[j].y, dt)));
                    nz = __fsub_rn(-x[j].z, __fmul_rn(v[j].z, dt));
                } else {
                    nxy = pack2(-x[j].x, -x[j].y);
                    nz = -x[j].z;
                }
                // from the lower end's position to this mass: the operands'
                // order only negates the correction, exactly; sums of what
                // is subtracted here
                f32x2 sxy = 0;
                float sz = 0.0f;
                uint32_t a_xy = info.x + 8u * lane, a_z = info.y + 4u * lane;
                bool fast = true;
                {
                    auto delta = [&](uint32_t w, f32x2& dxy, float& dz) {
                        f32x2 oxy;
                        float oz;
                        lds_xyz(w & 0xFFFFu, oxy, oz);
                        dxy = add2(oxy, nxy);
                        dz = __fadd_rn(oz, nz);
                        float dx, dy;
                        unpack2(dxy, dx, dy);
                        return __fmaf_rn(-dx, dx, __fmaf_rn(-dy, dy, __fmul_rn(-dz, dz)));  // -|d|^2
                    };
                    // correction of the lower end, stored and summed
                    auto apply = [&](float f, f32x2 dxy, float dz, uint32_t off) {
                        float dx, dy;
                        unpack2(dxy, dx, dy);
                        const f32x2 pxy = pack2(__fmul_rn(f, dx), __fmul_rn(f, dy));
                        const float pz = __fmul_rn(f, dz);
                        sts_pair(a_xy + 256u * off, pxy);
                        sts1(a_z + 128u * off, pz);
                        sxy = add2(sxy, pxy);
                        sz = __fadd_rn(sz, pz);
                    };
                    // stress: lambda/Lbar (reference, sim_kernel.cu:234); k (d - L)/Lbar (force)
                    auto stressed = [&](uint32_t st, float lam, float inv) {
                        return __float_as_uint(__fadd_rn(__uint_as_float(st), __fmul_rn(XPBD ? lam : -lam, inv)));
                    };
                    // reference step: lambda = -C/K, dp = lambda n (sim_kernel.cu:230-232);
                    // force modes: Hooke force, -k (d - L) n
                    // A row's padding computes a correction of +-0 -- unless
                    // the mass is so far away or not finite that the length
                    // is not, when it takes the exact path and is cleared.
                    auto stand_in = [&](uint32_t w) { return (w & 0xFFFFu) < x_first; };
                    auto clear = [&](f32x2& d, float& dz, float& nd, float& r, float L) {
                        d = 0;
                        dz = 0.0f;
                        nd = -L;
                        r = 0.0f;
                    };
                    struct Pair {
                        f32x2 d0, d1, ns, L, nd, r;
                        float z0, z1, k0, k1, i0, i1;  // (i: 1 / mean length, for the stress)
                    };
                    auto load = [&](Pair& u, const uint32_t (&c)[4]) {
                        const float2 m0 = lds2(c[0] >> 16), m1 = lds2(c[1] >> 16);
                        const float n0 = delta(c[0], u.d0, u.z0), n1 = delta(c[1], u.d1, u.z1);
                        u.ns = pack2(n0, n1);
                        const float l0 = __uint_as_float(c[2]), l1 = __uint_as_float(c[3]);
                        u.L = pack2(__fmaf_rn(l0, m0.x, l0), __fmaf_rn(l1, m1.x, l1));
                        if (TRACK) {
                            u.i0 = rcp_fast(l0);
                            u.i1 = rcp_fast(l1);
                        }
                        u.k0 = m0.y;
                        u.k1 = m1.y;
                    };
                    auto lengths = [&](Pair& u) {
                        f32x2 e;
                        lengths_and_reciprocals_fast(u.ns, u.nd, e, u.r);
                        float nd0, nd1, e0, e1;
                        unpack2(u.nd, nd0, nd1);
                        unpack2(e, e0, e1);
                        return length_is_fast(nd0, e0) && length_is_fast(nd1, e1);
                    };
                    // (plain_rcp: kept out of the common path, where even a
                    // branch around the general reciprocal cost 0.3 us of a
                    // one-warp step)
                    auto exact = [&](Pair& u, uint32_t w0, uint32_t w1, float l0, float l1) {
                        float n0, n1, d0, d1, r0, r1, L0, L1;
                        unpack2(u.ns, n0, n1);
                        unpack2(u.L, L0, L1);
                        length_and_reciprocal_exact(n0, d0, r0);
                        length_and_reciprocal_exact(n1, d1, r1);
                        if (stand_in(w0)) clear(u.d0, u.z0, d0, r0, L0);
                        if (stand_in(w1)) clear(u.d1, u.z1, d1, r1, L1);
                        u.nd = pack2(d0, d1);
                        u.r = pack2(r0, r1);
                        u.i0 = __frcp_rn(l0);
                        u.i1 = __frcp_rn(l1);
                        __syncwarp();
                    };
                    auto finish = [&](const Pair& u, uint32_t off, const uint32_t (&st)[2], uint32_t ts, bool both = true) {
                        float t0, t1, f0, f1;
                        unpack2(add2(u.L, u.nd), t0, t1);  // -C
                        const float lam0 = __fmul_rn(t0, u.k0), lam1 = __fmul_rn(t1, u.k1);
                        unpack2(mul2(pack2(lam0, lam1), u.r), f0, f1);
                        apply(f0, u.d0, u.z0, off);
                        if (both) apply(f1, u.d1, u.z1, off + 1);
                        if (TRACK)
                            tm_st2(ts, stressed(st[0], lam0, u.i0), stressed(st[1], lam1, u.i1));
                    };
                    uint32_t ta = info.w, ts = ta + 4 * ((kept + 1) / 2);
                    const uint32_t end = ta + 2 * (kept & ~1u);
                    Words own_words, &w0 = AHEAD ? ahead : own_words;
                    uint32_t(&c)[4] = w0.c, (&c2)[4] = w0.c2, (&st)[2] = w0.st, (&st2)[2] = w0.st2;
                    if (!AHEAD) first_springs(info, w0);
                    if (WIDE) {  // four springs at a time, then the rest together
                        auto wait = [&] {
                            if (TRACK)
                                asm volatile("tcgen05.wait::ld.sync.aligned;"
                                             : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c2[0]), "+r"(c2[1]), "+r"(c2[2]), "+r"(c2[3]),
                                               "+r"(st[0]), "+r"(st[1]), "+r"(st2[0]), "+r"(st2[1]));
                            else
                                asm volatile("tcgen05.wait::ld.sync.aligned;"
                                             : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c2[0]), "+r"(c2[1]), "+r"(c2[2]), "+r"(c2[3]));
                        };
                        // springs ta .. (the last one of four missing unless `all`), the next four's words in flight
                        auto four = [&](bool all) {
                            Pair u, w;
                            wait();
                            load(u, c);
                            load(w, c2);
                            const uint4 k0 = make_uint4(c[0], c[1], c[2], c[3]), k1 = make_uint4(c2[0], c2[1], c2[2], c2[3]);
                            const uint32_t s0[2] = {st[0], st[1]}, s1[2] = {st2[0], st2[1]};
                            ta += 8;
                            tm_ld(ta, c);
                            tm_ld(ta + 4, c2);
                            if (TRACK) {
                                tm_ld(ts + 4, st);
                                tm_ld(ts + 6, st2);
                            }
                            const bool ok0 = lengths(u), ok1 = lengths(w);
                            fast = fast && ok0 && ok1;
                            // (the warp together: tensor-memory accesses want it converged)
                            if (TRACK && __any_sync(0xffffffffu, !ok0 || !ok1 || plain_rcp)) {
                                exact(u, k0.x, k0.y, __uint_as_float(k0.z), __uint_as_float(k0.w));
                                exact(w, k1.x, k1.y, __uint_as_float(k1.z), __uint_as_float(k1.w));
                            }
                            finish(u, 0, s0, ts);
                            finish(w, 2, s1, ts + 2, all);
                            a_xy += all ? 1024u : 768u;
                            a_z += all ? 512u : 384u;
                            ts += 4;
                        };
                        while (end - ta >= 8) four(true);
                        if ((kept & 3u) == 3u) four(false);
                        wait();
                    }
                    while (WIDE ? (int32_t)(end - ta) > 0 : ta != end) {
                        Pair u;
                        if (TRACK)
                            asm volatile("tcgen05.wait::ld.sync.aligned;"
                                         : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(st[0]), "+r"(st[1]));
                        else
                            asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]));
                        load(u, c);
                        const uint32_t st0[2] = {st[0], st[1]};
                        const uint4 k0 = make_uint4(c[0], c[1], c[2], c[3]);
                        ta += 4;
                        tm_ld(ta, c);  // the next pair (or words past the last one), in flight during this one's arithmetic
                        if (TRACK) tm_ld(ts + 2, st);
                        const bool ok = lengths(u);
                        fast = fast && ok;
                        // (the warp together: tensor-memory accesses want it converged)
                        if (TRACK && __any_sync(0xffffffffu, !ok || plain_rcp))
                            exact(u, k0.x, k0.y, __uint_as_float(k0.z), __uint_as_float(k0.w));
                        finish(u, 0, st0, ts);
                        a_xy += 512u;
                        a_z += 256u;
                        ts += 2;
                    }
                    // one spring from words {w, length}; returns the stress after it
                    auto single = [&](uint32_t w, float lb, uint32_t st) {
                        f32x2 d;
                        float dz, nd, e, r, inv = TRACK ? rcp_fast(lb) : 0.0f;
                        const float2 mt = lds2(w >> 16);
                        const float n = delta(w, d, dz), L = __fmaf_rn(lb, mt.x, lb);
                        length_and_reciprocal_fast(n, nd, e, r);
                        if (__any_sync(0xffffffffu, !length_is_fast(nd, e) || plain_rcp)) {
                            length_and_reciprocal_exact(n, nd, r);
                            if (stand_in(w)) clear(d, dz, nd, r, L);
                            if (TRACK) inv = __frcp_rn(lb);
                            __syncwarp();
                        }
                        const float lam = __fmul_rn(__fadd_rn(L, nd), mt.y);
                        apply(__fmul_rn(lam, r), d, dz, 0);
                        a_xy += 256u;
                        a_z += 128u;
                        return stressed(st, lam, inv);
                    };
                    if (kept)  // (loads past the last pair included)
                        asm volatile("tcgen05.wait::ld.sync.aligned;"
                                     : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(st[0]), "+r"(st[1])::"memory");
                    if (!TRACK && __any_sync(0xffffffffu, !fast)) {
                        // some length needs the general square root or
                        // reciprocal: the row again, one spring at a time
                        sxy = 0;
                        sz = 0.0f;
                        a_xy = info.x + 8u * lane;
                        a_z = info.y + 4u * lane;
                        for (uint32_t k = 0; k < kept; ++k) {
                            uint32_t w[1], lb[1];
                            tm_ld(info.w + 4 * (k / 2) + (k & 1u), w);
                            tm_ld(info.w + 4 * (k / 2) + (k & 1u) + 2, lb);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(w[0]), "+r"(lb[0]));
                            single(w[0], __uint_as_float(lb[0]), 0u);
                        }
                    } else if (WIDE ? (kept & 3u) == 1u : kept & 1u) {
                        const uint32_t s = single(c[0], __uint_as_float(c[2]), st[0]);
                        if (TRACK) tm_st(ts, s);
                    }
                    // springs beyond the columns (rows grown by development): from global memory
                    for (uint32_t k = kept; k < own; ++k) {
                        const uint32_t at = __ldg(&q.r.head[TM_BIN(slice_begin) + gw + j * grp.warps]).z + 32 * k + lane;
                        const uint2 e = __ldg(&q.r.own[at]);
                        const float lb = __uint_as_float(e.y);
                        float* sp = nullptr;
                        if (TRACK) {
                            const uint32_t g = __ldg(&q.r.gidx[at]);
                            if (g != ~0u) sp = &p.stress[g & 0x7FFFFFFFu];
                            __syncwarp();
                        }
                        const uint32_t s = single(spring_word(e.x, TM_BIN(x0), TM_BIN(mat0), TM_BIN(n_mat)), lb, sp ? __float_as_uint(*sp) : 0u);
                        if (sp) *sp = __uint_as_float(s);
                        __syncwarp();
                    }
                }
                float sx, sy;
                unpack2(sxy, sx, sy);
                ax[j] = __fsub_rn(0.0f, sx);
                ay[j] = __fsub_rn(0.0f, sy);
                az[j] = __fsub_rn(0.0f, sz);
            }
            if (AHEAD && mine && (info_gather.y & 0xFFFCu)) tm_ld(info_gather.x, ahead.g4);
            group_sync<WIDE>(bar, GT);
            // (3) add the corrections of the springs to higher masses, in
            // summation order, and integrate (sim_kernel.cu:246-268)
#pragma unroll
            for (int j = 0; j < MPT; ++j) {
                if (j >= mine) break;
                if (j) __syncwarp();  // (the integration before may diverge)
                const uint4 info = AHEAD ? info_gather : lds_info(info_mine + j * GT + 16u);
                f32x2 fxy = pack2(ax[j], ay[j]);
                float fz = az[j];
                const uint32_t sxy0 = AHEAD ? xy0 : TM_BIN(xy0), sz0 = AHEAD ? z0 : TM_BIN(z0);
                auto add = [&](uint32_t w) {
                    const uint32_t i0 = w & 0xFFFFu, i1 = w >> 16;
                    const f32x2 c0 = lds_pair(sxy0 + 8u * i0), c1 = lds_pair(sxy0 + 8u * i1);
                    const float e0 = lds1(sz0 + 4u * i0), e1 = lds1(sz0 + 4u * i1);
                    fxy = add2(add2(fxy, c0), c1);
                    fz = __fadd_rn(__fadd_rn(fz, e0), e1);
                };
                const uint32_t n = info.y & 0xFFFFu, words = info.y >> 16;
                uint32_t at = info.x;
                const uint32_t end = at + (n & ~3u);
                Words own_words, &w0 = AHEAD ? ahead : own_words;
                uint32_t(&g4)[4] = w0.g4, (&g2)[2] = w0.g2, (&g1)[1] = w0.g1;
                if (n & 2u) tm_ld(end, g2);
                if (n & 1u) tm_ld(end + (n & 2u), g1);
                while (at != end) {
                    if (!AHEAD || at != info.x) tm_ld(at, g4);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(g4[0]), "+r"(g4[1]), "+r"(g4[2]), "+r"(g4[3]));
                    at += 4;
#pragma unroll
                    for (int u = 0; u < 4; ++u) add(g4[u]);
                }
                asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(g2[0]), "+r"(g2[1]), "+r"(g1[0]));
                if (n & 2u) {
                    add(g2[0]);
                    add(g2[1]);
                }
                if (n & 1u) add(g1[0]);
                if (words > n) {  // beyond the columns
                    const uint4 h = __ldg(&q.r.head[TM_BIN(slice_begin) + gw + j * grp.warps]);
                    auto word = [&](uint32_t k) {
                        if (info.z) return __float_as_uint(lds1(info.z + 128u * (k - n) + 4u * lane));
                        if (!FACES || k < h.x >> 16) return __ldg(&q.r.gather[h.z + lane + 32 * k]);
                        const uint32_t m = gt + j * GT;
                        return face_word(p.face_inc + p.bins[TM_BIN(bin)].face_inc_begin,
                                         m < TM_BIN(n_mass) ? __ldg(&p.face_row[TM_BIN(mass_begin) + m]) : 0u, k - (h.x >> 16),
                                         __ldg(&q.r.n_slots[TM_BIN(bin)]), lane);
                    };
                    for (uint32_t k = n; k < words; ++k) add(word(k));
                    if (FACES) __syncwarp();
                }
                float fx, fy;
                unpack2(fxy, fx, fy);
                if (XPBD) {
                    const float nx = __fadd_rn(__fadd_rn(x[j].x, __fmul_rn(v[j].x, dt)), fx);
                    const float ny = __fadd_rn(__fadd_rn(x[j].y, __fmul_rn(v[j].y, dt)), fy);
                    const float nz = __fadd_rn(__fadd_rn(x[j].z, __fmul_rn(v[j].z, dt)), fz);
                    // v = 0.99*(x~ - x)/dt in double (sim_kernel.cu:265-267)
                    v[j].x = velocity_of(__fsub_rn(nx, x[j].x), (double)dt, p.inv_dt);
                    v[j].y = velocity_of(__fsub_rn(ny, x[j].y), (double)dt, p.inv_dt);
                    v[j].z = velocity_of(__fsub_rn(nz, x[j].z), (double)dt, p.inv_dt);
                    x[j] = make_float3(nx, ny, nz);
                } else {
                    force_integrate<MODE>(p, x[j], v[j], mass[j], p.inv_dt_f, fx, fy, fz);
                }
            }
        }

        // ---- write back in the upload layout; flag non-finite positions
        if (TRACK) tm_wait_st();
        bool bad = false;
#pragma unroll
        for (int j = 0; j < MPT; ++j) {
            const uint32_t m = gt + j * GT;
            if (m < TM_BIN(n_mass)) {
                const uint32_t g = WIDE && MPT == 1 ? gidx : __ldg(&p.mass_gidx[TM_BIN(mass_begin) + m]);
                p.pos[g] = make_float4(x[j].x, x[j].y, x[j].z, WIDE && MPT == 1 ? mass[j] : p.pos[g].w);
                p.vel[g] = make_float4(v[j].x, v[j].y, v[j].z, WIDE && MPT == 1 ? vw : p.vel[g].w);
                bad |= !(isfinite(x[j].x) && isfinite(x[j].y) && isfinite(x[j].z));
            }
            __syncwarp();
            if (TRACK && j < mine) {
                const uint32_t rw = __ldg(&q.r.head[TM_BIN(slice_begin) + gw + j * grp.warps]).z + lane;
                const uint4 info = lds_info(info_mine + j * GT);
                const uint32_t kept = info.z & 0xFFFFu, ts = info.w + 4 * ((kept + 1) / 2);
#pragma unroll 2
                for (uint32_t k = 0; k < kept; k += 4) {
                    uint32_t st[4], g[4];
                    __syncwarp();
                    tm_ld(ts + k, st);  // (past the last one: words of this warp, not used)
#pragma unroll
                    for (uint32_t u = 0; u < 4; ++u) g[u] = k + u < kept ? __ldg(&q.r.gidx[rw + 32 * (k + u)]) : ~0u;
                    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(st[0]), "+r"(st[1]), "+r"(st[2]), "+r"(st[3]));
#pragma unroll
                    for (uint32_t u = 0; u < 4; ++u)  // bit 31: a copy in a split part, or padding
                        if (!(g[u] >> 31)) p.stress[g[u]] = __uint_as_float(st[u]);
                }
            }
        }
        __syncwarp();
        if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&p.bin_flags[TM_BIN(bin)], 1u);
        __syncwarp();
        group_sync<WIDE>(bar, GT);  // the group's shared memory is free for its next bin
    }
    tm_free(tmem0, cols);
}

// One CTA per bin, a warp per slice of 32 masses.  Bound by latency: three passes
// over the rows that look every entry's spring up, so the springs' words and
// columns lie in shared memory and lengths are loaded four entries at a time.
// 444 bins of 512 robots of 3-8 cells: 102 us with 32 warps a CTA (most bins have
// 11 slices), 89 with 16, 87 with 12, 126 with 8.
constexpr uint32_t kRowBytes = sizeof(uint32_t) + sizeof(uint16_t);  // shared memory of a spring
constexpr uint32_t kRowThreads = 384;
__global__ void __launch_bounds__(kRowThreads) tm_rows_kernel(const TmSource in, const TmRows r) {
    extern __shared__ uint32_t tm_rows_smem[];
    __shared__ uint32_t n_own[kTmMaxSlices], first_slot[kTmMaxSlices];
    __shared__ uint32_t used[8];
    __shared__ uint8_t rank_of[256];
    const uint32_t b = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const BinDesc bd = in.bins[b];
    const uint32_t n_slices = (bd.n_mass + 31) / 32;
    uint32_t* pairs = tm_rows_smem;
    uint16_t* col = reinterpret_cast<uint16_t*>(pairs + bd.n_spring);
    uint32_t room;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(room));
    if (bd.n_spring > room / kRowBytes) {  // the launch was sized for fewer: no plan takes the bin
        if (tid == 0) r.n_slots[b] = ~0u;
        return;
    }
    // 1. the materials in use, numbered in slot order
    if (tid < 8) used[tid] = 0;
    __syncthreads();
    for (uint32_t s = tid; s < bd.n_spring; s += blockDim.x) {
        const uint32_t w = in.spring_pair[bd.spring_begin + s], slot = w >> 24;
        pairs[s] = w;
        if (!((((volatile uint32_t*)used)[slot >> 5] >> (slot & 31u)) & 1u)) atomicOr(&used[slot >> 5], 1u << (slot & 31u));
    }
    __syncthreads();
    auto rank = [&](uint32_t slot) {
        uint32_t i = __popc(used[slot >> 5] & ((1u << (slot & 31u)) - 1u));
        for (uint32_t k = 0; k < (slot >> 5); ++k) i += __popc(used[k]);
        return i;
    };
    if (tid < 256) {
        rank_of[tid] = (uint8_t)rank(tid);
        if ((used[tid >> 5] >> (tid & 31u)) & 1u) r.mat[256u * b + rank_of[tid]] = (uint8_t)tid;
    }
    if (tid == 0) {
        uint32_t n = 0;
        for (uint32_t k = 0; k < 8; ++k) n += __popc(used[k]);
        r.n_mat[b] = n;
    }
    __syncthreads();
    // an entry of mass m: 0 padding, 1 its own (other end lower), 2 to gather
    auto kind = [&](uint32_t e, uint32_t m, uint32_t& pw, uint32_t& other) {
        pw = other = 0;
        if (e == kPadEntry) return 0u;
        pw = pairs[e >> 1];
        other = (e & 1u) ? pw & 0xFFFu : (pw >> 12) & 0xFFFu;
        // a spring from a mass to itself (no force): owned once
        return other < m || (other == m && (e & 1u)) ? 1u : other == m ? 0u : 2u;
    };
    // 2. own springs: columns, and every spring's column for its lower end
    for (uint32_t sl = tid / 32; sl < n_slices; sl += blockDim.x / 32) {
        const uint32_t gs = bd.slice_begin + sl, w = in.slice_width[gs], m = sl * 32 + lane;
        const uint32_t off = bd.inc_begin + in.slice_off[gs], at0 = off + 32u * gs + lane;
        const uint16_t* inc = in.inc + off + lane;
        uint32_t nneg = 0, npos = 0, cneg = 0, cpos = 0, pw, o;
        bool pure = true;  // every column is all own or all to gather
#pragma unroll 8
        for (uint32_t k = 0; k < w; ++k) {
            const uint32_t t = kind(inc[32 * k], m, pw, o);
            const bool an = __any_sync(0xffffffffu, t == 1u), ap = __any_sync(0xffffffffu, t == 2u);
            nneg += t == 1u;
            npos += t == 2u;
            pure &= !(an && ap);
            cneg += an;
            cpos += ap;
        }
        const uint32_t own = pure ? cneg : __reduce_max_sync(0xffffffffu, nneg);
        const uint32_t gat = pure ? cpos : __reduce_max_sync(0xffffffffu, npos);
        if (lane == 0) n_own[sl] = own | (gat + 1) / 2 << 16 | (pure ? 1u << 31 : 0u);
        if (!pure)
            for (uint32_t k = nneg; k < own; ++k) {
                r.own[at0 + 32 * k] = make_uint2(1u << 31, __float_as_uint(1.0f));
                r.gidx[at0 + 32 * k] = ~0u;
            }
        uint32_t at = 0;  // next own column: of the slice when pure, else of the lane
        for (uint32_t k0 = 0; k0 < w; k0 += 4) {
            uint32_t es[4], ts[4], os[4], ms[4], gi[4];
            float lb[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) es[u] = k0 + u < w ? inc[32 * (k0 + u)] : kPadEntry;
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                ts[u] = kind(es[u], m, pw, os[u]);
                ms[u] = rank_of[pw >> 24];
                gi[u] = ts[u] == 1u ? in.spring_gidx[bd.spring_begin + (es[u] >> 1)] : ~0u;
                lb[u] = ts[u] == 1u ? in.spring_lbar[bd.spring_begin + (es[u] >> 1)] : 1.0f;
            }
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                if (k0 + u >= w) break;
                const uint32_t t = ts[u];
                o = os[u];
                const bool an = __any_sync(0xffffffffu, t == 1u);
                if (t == 1u) {
                    r.own[at0 + 32 * at] = make_uint2(o | ms[u] << 16, __float_as_uint(lb[u]));
                    r.gidx[at0 + 32 * at] = gi[u];
                    col[es[u] >> 1] = (uint16_t)at;
                }
                if (pure && an) {  // stand-ins of a bank group the quarter-warp's others leave free
                    uint32_t mask = t == 1u ? 1u << (o & 7u) : 0u;
                    for (uint32_t x = 1; x < 8; x *= 2) mask |= __shfl_xor_sync(0xffffffffu, mask, x);
                    if (t != 1u) {
                        r.own[at0 + 32 * at] = make_uint2(1u << 31 | (mask == 0xFFu ? 0u : (uint32_t)__ffs(~mask & 0xFFu) - 1u),
                                                          __float_as_uint(1.0f));
                        r.gidx[at0 + 32 * at] = ~0u;
                    }
                }
                at += pure ? an : t == 1u;
            }
        }
    }
    __syncthreads();
    if (tid == 0) {
        uint32_t s = kTmZeros;
        for (uint32_t sl = 0; sl < n_slices; ++sl) {
            first_slot[sl] = s;
            s += 32u * (n_own[sl] & 0xFFFFu);
        }
        r.n_slots[b] = s;
    }
    __syncthreads();
    // 3. gather words
    for (uint32_t sl = tid / 32; sl < n_slices; sl += blockDim.x / 32) {
        const uint32_t gs = bd.slice_begin + sl, w = in.slice_width[gs], m = sl * 32 + lane;
        const uint32_t off = bd.inc_begin + in.slice_off[gs];
        const uint16_t* inc = in.inc + off + lane;
        const bool pure = n_own[sl] >> 31;
        const uint32_t words = (n_own[sl] >> 16) & 0x7FFFu;
        if (lane == 0) r.head[gs] = make_uint4((n_own[sl] & 0xFFFFu) | words << 16, first_slot[sl], off + 32u * gs, 0u);
        uint32_t* out = r.gather + off + 32u * gs;
        uint16_t* half = reinterpret_cast<uint16_t*>(out);
        for (uint32_t k = 0; k < words; ++k) out[32 * k + lane] = 0xFFFFFFFFu;
        __syncwarp();
        uint32_t at = 0, pw, o;
#pragma unroll 4
        for (uint32_t k = 0; k < w; ++k) {
            const uint32_t e = inc[32 * k], t = kind(e, m, pw, o);
            const bool ap = __any_sync(0xffffffffu, t == 2u);
            if (t == 2u) {
                const uint32_t slot = first_slot[o / 32] + 32u * col[e >> 1] + (o & 31u);
                half[2 * (32 * (at / 2) + lane) + (at & 1u)] = (uint16_t)slot;
            }
            at += pure ? ap : t == 2u;
        }
        __syncwarp();
        // padding: a zero slot of a bank (of 16 for {x, y}) that no entry of the half-warp uses
        for (uint32_t k = 0; k < words; ++k) {
            uint32_t v = out[32 * k + lane];
#pragma unroll
            for (uint32_t u = 0; u < 2; ++u) {
                const uint32_t s = (v >> (16 * u)) & 0xFFFFu;
                uint32_t mask = s != 0xFFFFu ? 1u << (s & 15u) : 0u;
                for (uint32_t x = 1; x < 16; x *= 2) mask |= __shfl_xor_sync(0xffffffffu, mask, x);
                if (s == 0xFFFFu) {
                    const uint32_t z = (mask == 0xFFFFu ? 0u : (uint32_t)__ffs(~mask & 0xFFFFu) - 1u) + (lane & 16u);
                    v = (v & ~(0xFFFFu << (16 * u))) | z << (16 * u);
                }
            }
            out[32 * k + lane] = v;
        }
    }
}

using TmFn = void (*)(const TmParams);
#define MB_TM(M)                                                                                                   \
    {                                                                                                              \
        {{tm_step_kernel<M, false, 1, false>, tm_step_kernel<M, false, 2, false>},                                 \
         {tm_step_kernel<M, false, 1, true>, tm_step_kernel<M, false, 2, true>}},                                  \
            {{tm_step_kernel<M, true, 1, false>, nullptr},                                                         \
             {tm_step_kernel<M, true, 1, true>, tm_step_kernel<M, true, 2, true>}},                                \
    }
const TmFn kTm[4][2][2][2] = {MB_TM(kModeXpbd), MB_TM(kModeForceLand), MB_TM(kModeForceWater), MB_TM(kModeForceWaterFaces)};
#undef MB_TM

TmFn tm_kernel(uint32_t mode, bool track, const TmPlan& plan) {
    if (mode > kModeForceWater || !plan.ok || plan.mpt < 1 || plan.mpt > kTmMaxMpt) return nullptr;
    if (plan.faces) {
        if (mode != kModeForceWater) return nullptr;
        mode = kModeForceWaterFaces;
    }
    return kTm[mode][track ? 1 : 0][plan.threads <= 32 * kTmWideWarps ? 1 : 0][plan.mpt - 1];
}

}  // namespace

cudaError_t launch_tm_rows(const TmSource& in, const TmRows& r, cudaStream_t s) {
    if (in.n_bins == 0) return cudaSuccess;
    // (one value for every launch: the attribute is the process's)
    const cudaError_t e = cudaFuncSetAttribute(tm_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)(kMaxBinSprings * kRowBytes));
    if (e != cudaSuccess) return e;
    tm_rows_kernel<<<in.n_bins, kRowThreads, std::min(in.max_bin_springs, kMaxBinSprings) * kRowBytes, s>>>(in, r);
    return cudaGetLastError();
}

cudaError_t prepare_tm(uint32_t mode, bool track, const TmPlan& plan) {
    const TmFn f = tm_kernel(mode, track, plan);
    return f ? allow_smem(reinterpret_cast<const void*>(f), plan.smem) : cudaErrorInvalidValue;
}

cudaError_t launch_tm(const TmParams& q, const TmPlan& plan, cudaStream_t s) {
    const TmFn f = tm_kernel(q.p.mode, q.p.track != 0, plan);
    if (!f) return cudaErrorInvalidValue;
    f<<<plan.ctas, plan.threads, plan.smem, s>>>(q);
    return cudaGetLastError();
}

uint32_t tm_count_slots(const BinDesc& d, const uint32_t* pair, const uint16_t* inc, const uint32_t* slice_off,
                        const uint32_t* slice_width) {
    uint32_t slots = kTmZeros;
    for (uint32_t sl = 0; sl < (d.n_mass + 31) / 32; ++sl) {
        const uint32_t gs = d.slice_begin + sl;
        const uint16_t* row = inc + d.inc_begin + slice_off[gs];
        uint32_t n[32] = {}, own_columns = 0;
        bool pure = true;  // every column is all own or all to gather
        for (uint32_t k = 0; k < slice_width[gs]; ++k) {
            bool own = false, gather = false;
            for (uint32_t l = 0; l < 32; ++l) {
                const uint32_t e = row[32 * k + l], m = 32 * sl + l;
                if (e == kPadEntry) continue;
                const uint32_t w = pair[d.spring_begin + (e >> 1)], other = (e & 1u) ? w & 0xFFFu : (w >> 12) & 0xFFFu;
                const bool mine = other < m || (other == m && (e & 1u));
                own |= mine;
                gather |= other > m;
                n[l] += mine;
            }
            own_columns += own;
            pure &= !(own && gather);
        }
        slots += 32 * (pure ? own_columns : *std::max_element(n, n + 32));
    }
    return slots;
}

namespace {

// One CTA's arrangement: its warp groups.
struct TmCta {
    uint32_t n_groups = 0;
    uint32_t warps[kTmMaxGroups], most[kTmMaxGroups];   // warps; slices of the largest bin
    uint32_t slots[kTmMaxGroups], faces[kTmMaxGroups];  // most slots (faces' included) and faces of a bin
};

// Shared memory of a CTA; 0 when its addresses do not fit 16 bits.
uint32_t layout(const TmCta& a, uint32_t n_mat, bool faces, TmGroup* out) {
    uint32_t off = kTmHeadBytes, w0 = 0;
    auto take = [&](uint32_t bytes) {
        const uint32_t at = off;
        off += (bytes + 127u) & ~127u;
        return at;
    };
    for (uint32_t g = 0; g < a.n_groups; ++g) {
        out[g].mat_off = take(8u * (n_mat + 1));
        out[g].x_off = take(16u * (kTmStandIns + 32 * a.most[g]));
    }
    if (off + kTmSmemBase > 65536u) return 0;
    for (uint32_t g = 0; g < a.n_groups; ++g) {
        TmGroup& t = out[g];
        if (faces) {
            t.v_off = take(8u * (kTmStandIns + 32 * a.most[g]));
            t.face_off = take(8u * a.faces[g]);
        }
        if (a.slots[g] > 65535u) return 0;
        t.xy_off = take(8u * a.slots[g]);
        t.z_off = take(4u * a.slots[g]);
        t.info_off = take(32u * a.most[g]);
        t.spare_off = take(128u * kTmSpareWords * (a.most[g] - a.warps[g]));
        t.warp0 = w0;
        t.warps = a.warps[g];
        w0 += a.warps[g];
    }
    return off;
}

// The compiled kernels, and the time of a step of one CTA, us: the group that
// takes longest for its bins (per bin: a fixed part; each slice of a warp and
// each own column of it; each warp its barriers wait for) and the CTA's issue
// (per slice, per own column).  Fitted to 990 arrangements of 40 populations of
// 1-8 cells and of clouds, the reference step, within 5-7 % (one standard
// deviation); what it picks took 0.8 % longer than the best on average, 11 %
// at most.
struct TmKernel {
    uint32_t max_warps, max_mpt;
    struct Cost {
        double bin, slice, column, warp, cta_slice, cta_column;
    } cost[2];  // without and with stress tracking
};
constexpr TmKernel kTmKernels[] = {
    {kTmWideWarps, kTmMaxMpt, {{0.070, 0.540, 0.0539, 0.0168, 0.0265, 0.0021}, {0.088, 0.528, 0.0590, 0.0101, 0.0384, 0.0033}}},
    {kTmMaxWarps, 1, {{0.0, 0.0, 0.0975, 0.0191, 0.0682, 0.0}, {0.0, 0.0, 0.1128, 0.0187, 0.0669, 0.0009}}},
    // (not with tracking: stresses add to a thread's words, and two masses' do
    // not fit a column share of 24 warps)
    {kTmMaxWarps, kTmMaxMpt, {{0.372, 0.0, 0.0801, 0.0170, 0.0714, 0.0005}, {}}},
};

struct TmArrangement {
    bool ok = false;
    double us = 0.0;
    std::vector<TmCta> ctas;
    std::vector<uint8_t> group_of;  // per bin
};

// Arranges every CTA for one of the kernels; not ok when a CTA's bins do not fit
// or take `bound` us.
void arrange(const std::vector<TmBinSize>& bins, uint32_t ctas, uint32_t n_mat, uint32_t smem_cap, const TmKernel& kernel,
             bool faces, bool track, double bound, TmArrangement& out) {
    const uint32_t max_warps = kernel.max_warps, max_mpt = kernel.max_mpt;
    const TmKernel::Cost& k = kernel.cost[track];
    out = TmArrangement{};
    out.ctas.resize(ctas);
    out.group_of.assign(bins.size(), 0);
    auto slices = [&](uint32_t b) { return (bins[b].n_mass + 31) / 32; };
    // a face counts as two springs' instructions
    auto columns = [&](uint32_t b) { return (bins[b].slots - kTmZeros + (faces ? 2u * bins[b].n_face : 0u)) / 32.0; };
    auto cost = [&](uint32_t b) { return columns(b) + 2.0 * slices(b); };
    std::vector<uint32_t> mine;
    std::vector<uint8_t> group;
    std::vector<double> work;
    for (uint32_t c = 0; c < ctas; ++c) {
        mine.clear();
        double issue = 0.0;
        for (uint32_t b = c; b < bins.size(); b += ctas) {
            if (bins[b].n_mass == 0) continue;
            mine.push_back(b);
            issue += k.cta_slice * slices(b) + k.cta_column * columns(b);
        }
        std::stable_sort(mine.begin(), mine.end(), [&](uint32_t a, uint32_t b) { return cost(a) > cost(b); });
        const uint32_t n = (uint32_t)mine.size();
        group.resize(n);
        double best = -1.0;
        if (n == 0) best = 0.0;
        for (uint32_t G = std::min(n, kTmMaxGroups); G >= 1; --G) {
            TmCta a;
            a.n_groups = G;
            double load[kTmMaxGroups] = {};
            for (uint32_t g = 0; g < G; ++g) a.warps[g] = a.most[g] = 1, a.slots[g] = kTmZeros, a.faces[g] = 0;
            for (uint32_t i = 0; i < n; ++i) {
                const uint32_t b = mine[i], g = (uint32_t)(std::min_element(load, load + G) - load);
                group[i] = (uint8_t)g;
                load[g] += cost(b);
                a.most[g] = std::max(a.most[g], slices(b));
                a.slots[g] = std::max(a.slots[g], bins[b].slots + (faces ? bins[b].n_face : 0u));
                if (faces) a.faces[g] = std::max(a.faces[g], bins[b].n_face);
            }
            // warps: a slice each; where that is too many, one warp at a time
            // off the group with the most for its work
            uint32_t total = 0, least = 0;
            for (uint32_t g = 0; g < G; ++g) {
                total += a.warps[g] = a.most[g];
                least += (a.most[g] + max_mpt - 1) / max_mpt;
            }
            if (least > max_warps) continue;
            const bool all = total <= max_warps;
            while (total > max_warps) {
                int from = -1;
                for (uint32_t g = 0; g < G; ++g)
                    if (a.warps[g] > 1 && (a.warps[g] - 1) * max_mpt >= a.most[g] &&
                        (from < 0 || load[g] * a.warps[from] < load[from] * a.warps[g]))
                        from = (int)g;
                if (from < 0) break;
                --a.warps[from];
                --total;
            }
            TmGroup unused[kTmMaxGroups];
            const uint32_t bytes = total <= max_warps ? layout(a, n_mat, faces, unused) : 0;
            if (!bytes || bytes > smem_cap) continue;
            double busy[kTmMaxGroups] = {};
            for (uint32_t i = 0; i < n; ++i) {
                const uint32_t b = mine[i], sl = slices(b), m = (sl + a.warps[group[i]] - 1) / a.warps[group[i]];
                busy[group[i]] += k.bin + m * (k.slice + k.column * columns(b) / sl) + k.warp * sl;
            }
            const double us = issue + *std::max_element(busy, busy + G);
            if (best >= 0.0 && us >= best) continue;
            best = us;
            out.ctas[c] = a;
            for (uint32_t i = 0; i < n; ++i) out.group_of[mine[i]] = group[i];
            if (all && G == n) break;  // every bin at once, a warp a slice
        }
        if (best < 0.0 || best >= bound) return;
        out.us = std::max(out.us, best);
    }
    out.ok = true;
}

TmArrangement arrange_best(const std::vector<TmBinSize>& bins, uint32_t ctas, uint32_t n_mat, uint32_t smem_cap,
                           bool track, bool faces, double bound = 1e30) {
    TmArrangement best, a;
    for (const TmKernel& kernel : kTmKernels) {
        if (track && kernel.max_warps > kTmWideWarps && kernel.max_mpt > 1) continue;
        arrange(bins, ctas, n_mat, smem_cap, kernel, faces, track, best.ok ? best.us : bound, a);
        if (a.ok) best = std::move(a);
    }
    return best;
}

}  // namespace

double tm_estimate(const std::vector<TmBinSize>& bins, uint32_t ctas, uint32_t n_mat, uint32_t smem_cap, bool track,
                   bool faces, double bound) {
    const TmArrangement a = arrange_best(bins, ctas, n_mat, smem_cap, track, faces, bound);
    return a.ok ? a.us : 0.0;
}

void tm_plan(const std::vector<BinDesc>& bins, const std::vector<uint32_t>& slots, uint32_t ctas, uint32_t n_mat,
             uint32_t smem_cap, bool track, bool faces, TmPlan& out) {
    out = TmPlan{};
    out.faces = faces;
    if (bins.empty() || ctas == 0) return;
    ctas = std::min(ctas, (uint32_t)bins.size());
    std::vector<TmBinSize> sizes;
    for (size_t b = 0; b < bins.size(); ++b) sizes.push_back({bins[b].n_mass, slots[b], faces ? bins[b].n_face : 0u});
    const TmArrangement a = arrange_best(sizes, ctas, n_mat, smem_cap, track, faces);
    if (!a.ok) return;
    out.groups.assign((size_t)ctas * kTmMaxGroups, TmGroup{});
    for (uint32_t c = 0; c < ctas; ++c) {
        const TmCta& t = a.ctas[c];
        TmGroup* g = &out.groups[(size_t)c * kTmMaxGroups];
        out.smem = std::max(out.smem, layout(t, n_mat, faces, g));
        for (uint32_t i = 0; i < t.n_groups; ++i) {
            g[i].first = (uint32_t)out.bins.size();
            for (uint32_t b = c; b < bins.size(); b += ctas) {
                const BinDesc& d = bins[b];
                if (d.n_mass && a.group_of[b] == i)
                    out.bins.push_back({b, d.mass_begin, d.n_mass, d.slice_begin, d.face_begin, sizes[b].n_face, d.face_inc_begin});
            }
            g[i].count = (uint32_t)out.bins.size() - g[i].first;
            out.mpt = std::max(out.mpt, (t.most[i] + t.warps[i] - 1) / t.warps[i]);
            out.threads = std::max(out.threads, 32 * (g[i].warp0 + g[i].warps));
        }
    }
    out.threads = std::max(out.threads, 32u);
    out.ctas = ctas;
    out.ok = true;
}

}  // namespace mb
