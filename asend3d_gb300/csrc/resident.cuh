// resident.cuh -- plan of the resident PCG (k_resident.cu) of one pattern.
#pragma once
#include "common.cuh"

namespace asend {

constexpr int kResLanes = 640;      // product lanes of a CTA at most
// threads of a CTA at most, by right-hand sides (their x and r are registers)
constexpr int res_threads(int nr) { return nr == 1 ? 1024 : 640; }
constexpr int kResMinThreads = 256; // warps for the sums and for fetching z beside them
constexpr int kResMaxLanes = 16;    // lanes of a row at most
constexpr int kResMinRows = 8;      // rows of a CTA at least

struct ResidentPlan {
    int64_t pattern = -1;           // pattern serial it was built for
    bool fits = false;              // the pattern can be spread over one CTA per SM
    int sms = 0, grid = 0;          // SMs; CTAs in use
    int rows = 0, T = 1, VT = 0;    // rows of a CTA, lanes of a row, rows x T
    int K = 0;                      // column steps: a row's blocks over its lanes
    int next = 0;                   // largest number of ext nodes of a CTA
    size_t smem = 0;                // shared memory a CTA may have
    unsigned long long epoch = 0;   // exchange numbers used so far
    DArr<int32_t> row0, ext_ptr, ext;
    DArr<uint16_t> lcol;
    DArr<ulonglong2> z, words;
    DArr<int> flags;                // [0]: a wait ran out
};

// A Newmark run's buffers (k_newmark.cu) and its outcome.
struct NewmarkState {
    int n_steps, probe, hist_fields;
    double c1, c2;
    const double *f0, *pen, *amp;  // amp: [n_steps] on the device
    double *u, *v, *a, *up, *vp, *ap, *du, *du_prev, *probe_hist, *hist;
};
struct ResidentRun {
    double rel_residual;
    int iterations, capped, nonfinite, next_step;
};
// The whole run in a few launches (after resident_usable and pcg_precondition).
ResidentRun resident_newmark(Ctx& c, const asend_solve_opts& o, const NewmarkState& N);

}  // namespace asend
