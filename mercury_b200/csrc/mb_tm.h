// Resident step kernel with per-thread operands in tensor memory
// (mb_tm.cu); internal to the library.
#pragma once
#include <cstdint>
#include <vector>
#include <cuda_runtime.h>

#include "mb_internal.h"

namespace mb {

// Bins one warp group of a CTA steps, one after another, and its shared
// memory (byte offsets from the start of the dynamic shared memory).
struct alignas(16) TmGroup {
    uint32_t first, count;     // range of the bin list
    uint32_t warp0, warps;     // warps of the CTA (0: no such group)
    uint32_t mat_off;          // material factors
    uint32_t x_off;            // eight stand-in positions, then the masses'
    uint32_t xy_off, z_off;    // corrections of the bin's slots: {x, y} and z
    uint32_t info_off;         // 32 bytes per slice
    uint32_t spare_off;        // kTmSpareWords gather words per second slice of a warp
    uint32_t v_off, face_off;  // face drag: velocities {y, z} beside the positions, corners of the faces
};
// A bin of the list: what of its descriptor the kernel reads.
struct alignas(16) TmBinRef {
    uint32_t bin, mass_begin, n_mass, slice_begin;
    uint32_t face_begin, n_face, face_inc_begin;  // (n_face 0 without face drag)
};

constexpr uint32_t kTmMaxWarps = 24;      // warps per CTA: 80 registers a thread
constexpr uint32_t kTmWideWarps = 16;     // up to which the variant with more registers runs
constexpr uint32_t kTmMaxGroups = 8;      // groups (named barriers) per CTA
constexpr uint32_t kTmMaxMpt = 2;         // masses per thread
constexpr uint32_t kTmZeros = 32;         // zero slots before a bin's corrections, one per bank
constexpr uint32_t kTmStandIns = 8;       // stand-in positions before a bin's, one per bank group
constexpr uint32_t kTmSmemBase = 4096;    // bound on the address where dynamic shared memory starts
constexpr uint32_t kTmHeadBytes = 512;    // start of the dynamic shared memory: what the groups need of their bins
constexpr uint32_t kTmMaxSlices = 128;    // slices of 32 masses per bin
constexpr uint32_t kTmSpareWords = 8;     // gather words of a slice kept in shared memory when the columns are full

// Populations the kernel steps: resident bins of a 1,024-thread shape with at
// most one mass per thread, no mass with more springs than a lattice has.
constexpr uint32_t kTmMaxDegree = 26;
inline bool tm_shape(const KernelShape& s) { return s.threads == 1024 && (s.spt == 8 || s.spt == 10 || s.spt == 12); }
inline bool tm_holds(const KernelShape& s, bool streamed, uint32_t cluster, uint32_t max_bin_mass, uint32_t max_degree) {
    return !streamed && !cluster && tm_shape(s) && max_bin_mass <= s.threads && max_degree <= kTmMaxDegree;
}

// The launch of a population: which warps of which CTA step which bins.
struct TmPlan {
    bool ok = false;
    bool faces = false;  // with the face drag
    uint32_t ctas = 0, threads = 0, mpt = 1, smem = 0;
    std::vector<TmGroup> groups;  // kTmMaxGroups per CTA
    std::vector<TmBinRef> bins;   // the bin list
};

// Plans the launch over `bins` (slots[b]: correction slots of bin b, from
// launch_tm_rows): CTA c of `ctas` steps bins c, c + ctas, ...  Not ok when a
// CTA's bins fit no arrangement.
void tm_plan(const std::vector<BinDesc>& bins, const std::vector<uint32_t>& slots, uint32_t ctas, uint32_t n_mat,
             uint32_t smem_cap, bool track, bool faces, TmPlan& out);

// Estimated time of a step of such a launch, us (0: no arrangement, or none
// shorter than `bound`).
struct TmBinSize {
    uint32_t n_mass, slots, n_face;
};
double tm_estimate(const std::vector<TmBinSize>& bins, uint32_t ctas, uint32_t n_mat, uint32_t smem_cap, bool track,
                   bool faces, double bound);

// Correction slots of a bin from its SELL rows on the host, as the row kernel
// counts them (launch planning without a GPU).
uint32_t tm_count_slots(const BinDesc& bin, const uint32_t* pair, const uint16_t* inc, const uint32_t* slice_off,
                        const uint32_t* slice_width);

// Rows of the step kernel, from the SELL rows.  Every spring belongs to its
// end of higher index (the owner).  Per slice of 32 masses:
//   own springs   per mass its springs to lower masses, in summation order:
//                 {other end | material << 16, mean length}; the k-th of
//                 lane l has correction slot `slot` + 32 k + l.  Padding:
//                 1 << 31 | bank group of a stand-in position that the
//                 quarter-warp's others leave free;
//   gather words  per mass the slots of its springs to higher masses, in
//                 order, two 16-bit slots a word; padding names one of the
//                 zero slots 0..31.
// Columns of one neighbour offset stay columns (consecutive lanes then read
// consecutive slots).  Slice s of bin b starts at inc_begin + slice_off + 32 s
// in own, gidx and gather (one entry per SELL entry and 32 more a slice).
// Materials are numbered per bin.
struct TmRows {
    uint2* own;
    uint32_t* gidx;     // own springs: upload index (bit 31: a copy in a split part), or ~0
    uint32_t* gather;
    uint4* head;        // per slice: {own springs | gather words << 16, first correction slot, first entry}
    uint32_t* n_slots;  // per bin: correction slots
    uint32_t* n_mat;    // per bin: materials in use
    uint8_t* mat;       // per bin: 256 material slots, in order
};
struct TmSource {
    const BinDesc* bins;
    uint32_t n_bins;
    uint32_t max_bin_springs;  // packed springs of a bin, at most
    const uint32_t* spring_pair;
    const float* spring_lbar;
    const uint32_t* spring_gidx;
    const uint16_t* inc;
    const uint32_t* slice_off;
    const uint32_t* slice_width;
};

struct TmParams {
    StepParams p;
    const TmGroup* groups;
    const TmBinRef* bins;
    TmRows r;
};

cudaError_t launch_tm_rows(const TmSource& in, const TmRows& r, cudaStream_t s);
cudaError_t prepare_tm(uint32_t mode, bool track, const TmPlan& plan);
cudaError_t launch_tm(const TmParams& q, const TmPlan& plan, cudaStream_t s);

}  // namespace mb
