// box.cuh -- matrix-free products of the finest multigrid level on blocks of
// equal box elements (k_box.cu).
#pragma once
#include "pcg_common.cuh"

namespace asend {

struct BoxPlan;

// The plan of the assembled operator, built when needed; nullptr when some
// block is not made of equal box elements or the operator is more than
// sum E_e K^ + diagonal penalty.
BoxPlan* box_plan(Ctx& c, const std::vector<std::array<int, 5>>& blocks /* nx ny nz node0 el0 */);

// y = A p (FP32 pairs, natural layout) of the CG and the p.Ap reduction, as
// k_mg_spmv_dot_pair on the assembled values, for nr right-hand sides whose
// vectors follow each other.
void box_product(Ctx& c, const BoxPlan& P, pcg::PcgArgs a, int nr, int part_stride);
// r = b - A x; y4 = x + B^-1 (b - A x); and a power-iteration step y4 = D^-1 A x
// / nrm[k], nrm[k + 1] = |y4|, all FP32 on node-padded x.
void box_resid(Ctx& c, const BoxPlan& P, const float* b, const float4* x, float* r, const pcg::Control* ctl, int nr);
void box_post(Ctx& c, const BoxPlan& P, const float* binv, const float* b, const float4* x, float4* y4,
              const pcg::Control* ctl, int nr);
void box_power(Ctx& c, const BoxPlan& P, const float* dinv, const float4* x, float4* y4, float* nrm, int k,
               double* part, uint32_t* ticket);
const void* box_patterns(const BoxPlan& P);  // pattern blocks the launches read (a captured graph keeps them)
int box_ctas(const BoxPlan& P);  // CTAs of one launch (entries of a partials array)
double box_product_bytes(const Ctx& c);

}  // namespace asend
