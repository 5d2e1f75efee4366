// Selection of the shape-specialised chunk kernels with fallback to the
// generic level-major kernel, and their launch variants (the autotuner in
// mgb_api.cu times the variants of a segment's kernel and keeps the fastest).
#pragma once

#include <vector>

#include "mgb_kernels.h"

namespace mgb {

struct TunedChoice {
    bool use = false;
    int family = 0;  // 1: registers, one to 32 lanes per chunk (d = 2, SpaceCurve); 2: group-tiled CTA kernel (mixed, d = 16 / 32); 3: tensor-core level-major (mixed, d = 64 / 128); 4 / 5: one thread per column (d = 3..8) / per 1 x 4 tile (d = 9..32), beside the generic kernel's variants
    int D = 0;
    int nmax = 0;
    int ctas_per_sm = 1;
    int variant = 0;    // launch variant of the family's kernel
    int nvariants = 1;  // variants the autotuner may choose from
};

// Scratch geometry of a segment: per-slot elements (compute type) and the
// number of slots (CTAs, or threads for the 4-element family).
struct SegSizing {
    int64_t slot_elems = 0;
    int64_t grid = 0;
    int lpc = 1;       // lanes or teams per chunk (d = 2..8, SpaceCurve)
    int64_t least = 1;  // slots a cut of the scratch must leave
    int64_t round = 1;  // grid is a multiple of this
};
SegSizing size_segment(bool plain, int kind, int rule, bool f64io, const std::vector<InstDev>& hi, int64_t nwork,
                       int sms, size_t budget_bytes);
cudaError_t launch_small_family(bool plain, int kind, int rule, int mode, const LaunchArgs& a);
int small_family_max_levels();
// Column kernel for d = 3..8 (mgb_col.cuh): whether an order fits, teams per
// chunk, VJP scratch (elements) wanted and needed.
bool col_ok(bool plain, int D, int nmax);
// Kernel for d = 9..32 outside the tensor-core kernels (mgb_dense.cuh; where it
// stands among the variants: dense_variant in mgb_tuned.cu); its VJP runs in the
// generic kernel's slots.
bool dense_ok(bool plain, int d, int nmax);
cudaError_t launch_dense(bool plain, int d, int rule, int mode, const LaunchArgs& a, int nmax, bool prepare_only);
int col_lanes(bool plain, int D, int nmax, int64_t nwork, int64_t kmax, int sms);
int64_t col_scratch(bool plain, int D, int nmax, int64_t nwork, int64_t kmax, int lpc, int sms);
int64_t col_scratch_min(bool plain, int D, int nmax, int64_t kmax, int lpc);
cudaError_t launch_col(bool plain, int D, int rule, int mode, const LaunchArgs& a, int nmax, bool prepare_only);
int small_family_lanes(int64_t nwork, int64_t kmax, int sms);
int64_t small_family_slot(int64_t kmax, int lpc);

TunedChoice choose_tuned(bool plain, int kind, int rule, int mode, bool f64io, const std::vector<InstDev>& hi,
                         int variant);
// Tensor-core chunk kernel (mgb_bigtc.cu) for the mixed form at d = 64 / 128.
// Variants: d = 64: 0 and 1 k-block 32 or 64 at 2 CTAs per SM, 2 the VJP of 1 (its
// forward pass is launch_cmma's), 3 k-block 64 at 1, 4 k-block 32 at 3; d = 128:
// k-block 32 or 64, or 32 with 2 CTAs per SM.  The grid is min(a.grid, sms x CTAs per SM).
cudaError_t launch_big(int D, int rule, int mode, const LaunchArgs& a, int sms, int variant, bool prepare_only);
int big_variants(int D);
int big_ctas_per_sm(int D, int variant);
// Group-tiled kernel (mgb_tuned.cu), variant 0: 2 CTAs per SM, 1: one;
// at d = 32 variant 2: the tcgen05 forward local pass (mgb_tiletc.cu) with
// the warp-MMA VJP (mgb_mma32.cu), variant 3: the warp-MMA forward pass
// (mgb_cmma.cu, launch_cmma) with it.
cudaError_t launch_tile(int D, int rule, int mode, const LaunchArgs& a, int grid, int variant, bool prepare_only);
cudaError_t launch_tiletc(int rule, const LaunchArgs& a, int grid, bool prepare_only);
// Warp-MMA VJP kernel at d = 32 (mgb_mma32.cu); two CTAs per SM.
cudaError_t launch_mma32(int rule, const LaunchArgs& a, int grid, bool prepare_only);
// Forward local pass at d = 32 / 64 with the prefix passes in the warp-MMA
// accumulators (mgb_cmma.cu); one slot (3 n d^2 elements) per CTA.
int cmma_ctas_per_sm(int D);
cudaError_t launch_cmma(int D, int rule, const LaunchArgs& a, int sms, bool prepare_only);
// Device address of the time-out flag the tensor-core kernels raise.
int* device_timeout_ptr();
// One CTA waits (limit_ns) on an mbarrier nothing arrives at and raises the
// time-out flag (mgb_selftest.cu).
cudaError_t launch_wait_selftest(uint64_t limit_ns, cudaStream_t st);
// Generic kernel variants: 8, 4 or 2 CTAs per SM (the column or tile kernel in
// place of the first, or, for the tile kernel in the mixed form at d = 9..12,
// after them).
constexpr int GENERIC_VARIANTS = 3;
int generic_ctas_per_sm(int variant);
// The variant a pass runs where nothing is timed (tc0: variant 0's choice).
int untimed_variant(const TunedChoice& tc0, bool plain, int mode, int nmax, int64_t nwork, int sms);
// The kernel a choice runs for a pass, and the CTAs per SM its grid is bounded
// to (0: as many as the chunks ask for).
const char* kernel_name(const TunedChoice& tc, int mode);
int kernel_ctas_per_sm(const TunedChoice& tc, int variant, int mode);
// 1 if a kernel gave up a bounded device-side wait since the last call.
int read_clear_device_timeout();
cudaError_t prepare_tuned(const TunedChoice& tc, int rule, int mode);
cudaError_t launch_tuned(const TunedChoice& tc, bool plain, int kind, int rule, int mode, const LaunchArgs& a, int sms);
cudaError_t launch_chunk_any(bool plain, int kind, int rule, int mode, const LaunchArgs& a,
                             const std::vector<InstDev>& hi, int sms, int variant);

}  // namespace mgb
