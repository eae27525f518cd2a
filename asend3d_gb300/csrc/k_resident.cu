// k_resident.cu -- the point / block Jacobi PCG of k_pcg.cu as one cooperative
// kernel per solve (a few per Newmark run), its operator resident in shared memory.
//
// Reference: conj_grad_sparse, solverSrc/asend_run_job/src/matrix_functions.rs:285-362.
//
// What bounds the three-kernels-per-iteration PCG on models of up to some ten
// thousand nodes is neither bytes nor arithmetic but latency: a 525-node beam
// runs on 5 CTAs whose threads walk 27 block columns one dependent load after
// the other, between kernel boundaries and host looks at the scalars (38 us an
// iteration; 6.3 us here, two thirds of it the two exchanges below; 13.4 us on 9,744
// rows, FP64).  Here
//  * every SM gets one CTA and an equal run of rows; T lanes share a row;
//  * the CTA's operator values stay in shared memory for the whole solve (152
//    x 227 KB hold 34 MB); column steps that do not fit stream from L2;
//  * a CTA keeps the direction of its rows and of their neighbours ("ext"
//    nodes) in shared memory and updates all of them itself, p = z + beta p,
//    from the z = M r every owner publishes, so an iteration has two grid-wide
//    exchanges (p.Ap; r.z and r.r with the new z) instead of three launches;
//  * an exchange is one L2 round trip: CTA b stores (partial, epoch) as 16-byte
//    words, one for every CTA, and each CTA polls the words meant for it and
//    sums them in a fixed order, so every CTA holds bit-identical scalars and
//    takes the same branches.  Two sets of words alternate: set e is rewritten
//    two exchanges later, when every CTA has passed the one in between.  z
//    travels in such words too, so no fence stands on an iteration's path;
//  * x and r live in registers; convergence of the recurrence, the true
//    residual f - A64 x that has to confirm it, restarts and the iteration cap
//    are decided in the kernel, and the host reads the outcome once.
// Every wait is bounded: a CTA whose words do not arrive leaves with an error
// flag, and so do the others.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "pcg_common.cuh"
#include "resident.cuh"

namespace asend {
namespace {
using namespace pcg;

constexpr int kMaxCtas = 160;       // CTAs at most: five words a polling lane
constexpr int kPollLimit = 1 << 21; // polls (about 0.5 us each) before a wait gives up
// Exchanges (two an iteration, two a step) after which a Newmark run's launch ends.
// A launch takes every SM, so work of another context (another host thread's)
// waits for its end: a 9 ms solve beside a run of 21,948 steps waited for all of it
// (3.4 s) when the run was one launch, now 4 ms (the run on 525 rows) to 15 ms (on
// 9,744).  The launches' starts cost nothing to be seen (60 time steps of 10,201 shell
// rows, 40 of 1,225 hex8 rows: the times of one launch).
constexpr unsigned long long kLaunchExchanges = 2048;

struct ResArgs {
    int n_rows, n_dof, rows, T, K, KR, VT, next, cap, pc, zero_x, replace_every;
    int off_z, off_y, off_v, off_c, off_s;  // shared memory: fetched z, row products, values, column ids, scratch (p first)
    int n_words;                     // values an exchange may carry
    const int64_t* slice_off;
    const uint8_t* row_len;
    const int32_t* col;
    const double* v64;
    const float* v32;
    const int32_t* row0;     // [grid + 1] first row of each CTA
    const int32_t* ext_ptr;  // [grid + 1]
    const int32_t* ext;      // ext nodes of each CTA: its own rows, then their other neighbours
    const uint16_t* lcol;    // [grid][K][VT] place of a block's column among the ext nodes
    const double* f;
    double* x;
    double* r;
    ulonglong2* z;           // [NR][n_dof] published M r (value, epoch)
    const double* dinv;
    const float* binv;
    ulonglong2* words;       // [2][values][grid: from][grid: to] (partial, epoch)
    unsigned long long epoch0;
    double tol2;
    RhsScalars* sc;
    int* err;                // set when a wait ran out
};

// The Newmark loop of k_newmark.cu in the same kernel (DYN): its state vectors,
// mass and damping values, and its records.  A launch goes on from step0 until
// the last step or, after a whole step, kLaunchExchanges exchanges.
struct DynArgs {
    int n_steps, extrapolate, probe, hist_fields, step0;
    const double *m64, *d64, *f0, *pen, *amp;
    double cM, cD, dt, gamma, c1, c2;
    double *u, *v, *a, *up, *vp, *ap, *du_prev;
    double* probe_hist;  // [n_steps]
    double* hist;        // [n_steps][hist_fields][n_dof]
    ResidentRun* out;
};

__device__ __forceinline__ void st_word(ulonglong2* p, double v, unsigned long long e) {
    asm volatile(
        "{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(p),
        "l"((unsigned long long)__double_as_longlong(v)), "l"(e)
        : "memory");
}
__device__ __forceinline__ void ld_word(const ulonglong2* p, unsigned long long& v, unsigned long long& e) {
    asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
                 : "=l"(v), "=l"(e)
                 : "l"(p)
                 : "memory");
}

// Shared state of the solve, one set per right-hand side: kept by single
// lanes, since every FP64 instruction of every warp holds its quarter of the
// SM's FP64 pipe for 64 cycles.
struct ResShared {
    double red[32][kMaxRhs * 3];  // per-warp sums
    double tot[kMaxRhs * 3];                    // grid-wide sums of the last exchange
    double rz[kMaxRhs], rz_prev[kMaxRhs], rz_inv[kMaxRhs], alpha[kMaxRhs], beta[kMaxRhs];
    double rr[kMaxRhs], rr_true[kMaxRhs], target[kMaxRhs], bb[kMaxRhs];
    int flag_z[kMaxRhs], flag_r[kMaxRhs];       // kNonfinite | kConverged | kDropped
    int bad;
};
enum { kNonfinite = 1, kConverged = 2, kDropped = 4 };

// Sums of a over lanes 0-15's and b over lanes 16-31's side: lane 0 returns
// the warp's sum of a, lane 16 that of b, in 5 additions instead of 10 (an FP64
// instruction holds its quarter of the SM's FP64 pipe for 64 cycles).
__device__ __forceinline__ double warp_sum_pair(double a, double b, int lane) {
    const bool up = lane >= 16;
    double keep = up ? b : a;
    const double give = up ? a : b;
    keep += __shfl_xor_sync(0xffffffffu, give, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) keep += __shfl_xor_sync(0xffffffffu, keep, o);
    return keep;
}

enum { kSum = 0, kAlpha = 1, kBeta = 2 };

// Grid-wide sums of the NV per-thread values v of the first ndw warps into
// S.tot.  Warp q < NV carries value q: it stores a word with the CTA's partial
// for every CTA (next to each other: coalesced) and polls the ones meant for
// its own (on 152 CTAs an exchange took 10,900 cycles when all polled the same
// words, 3,900 with a word each).
// kAlpha: tot[k] is p.Ap, alpha[k] = rz[k] / tot[k] is formed on the way (and
// 1 / rz[k] while the words travel); kBeta: tot[k], k < NR, is the new r.z:
// beta[k] = tot[k] / rz[k], rz[k] = tot[k], and tot[NR + k] the new r.r with
// its flags (DROP: the mixed method's drop below the last true residual, too).  FENCE: what any thread stored
// before is visible to every CTA afterwards.  idle() is run by the other warps.
template <int NV, int NR, int WHAT, bool FENCE, bool DROP, typename Idle>
__device__ __forceinline__ bool exchange(const ResArgs& A, ResShared& S, int ndw, const double (&v)[NV],
                                         unsigned long long epoch, Idle&& idle) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int C = gridDim.x;
    if (warp < ndw) {
#pragma unroll
        for (int q = 0; q + 1 < NV; q += 2) {
            const double s = warp_sum_pair(v[q], v[q + 1], lane);
            if ((lane & 15) == 0) S.red[warp][q + (lane >> 4)] = s;
        }
        if constexpr (NV % 2 == 1) {
            const double s = warp_sum(v[NV - 1]);
            if (lane == 0) S.red[warp][NV - 1] = s;
        }
    }
    __syncthreads();
    if (warp >= NV) idle();
    ulonglong2* set = A.words + (size_t)(epoch & 1) * A.n_words * C * C;
    for (int q = warp; q < NV; q += nw) {
        double s = lane < ndw ? S.red[lane][q] : 0.0;
        int o = 1;
        while (o < ndw) o <<= 1;
        for (o >>= 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        s = __shfl_sync(0xffffffffu, s, 0);
        if (FENCE) __threadfence();
#pragma unroll
        for (int u = 0; u < 5; ++u)
            if (u * 32 + lane < C) st_word(set + ((size_t)q * C + blockIdx.x) * C + u * 32 + lane, s, epoch);
        if (WHAT == kAlpha && lane == 0) S.rz_inv[q] = 1.0 / S.rz[q];
    }
    for (int q = warp; q < NV; q += nw) {
        const ulonglong2* in = set + (size_t)q * C * C + blockIdx.x;
        unsigned long long val[5], ep[5];
        int spin = 0;
        bool all;
        do {
            all = true;
#pragma unroll
            for (int u = 0; u < 5; ++u) {
                val[u] = 0;
                ep[u] = epoch;
                if (u * 32 + lane < C) ld_word(in + (size_t)(u * 32 + lane) * C, val[u], ep[u]);
            }
#pragma unroll
            for (int u = 0; u < 5; ++u) all &= ep[u] == epoch;
        } while (!all && ++spin < kPollLimit);
        double s = __longlong_as_double((long long)val[0]);
        if (C > 32) {
            s += __longlong_as_double((long long)val[1]);
            if (C > 64)
                s += (__longlong_as_double((long long)val[2]) + __longlong_as_double((long long)val[3])) +
                     __longlong_as_double((long long)val[4]);
        }
        s = warp_sum(s);
        if (FENCE) __threadfence();
        if (!__all_sync(0xffffffffu, all) && lane == 0) S.bad = 1;
        if (lane == 0) {
            S.tot[q] = s;
            if (WHAT == kAlpha) S.alpha[q] = S.rz[q] / s;
            if (WHAT == kBeta && q < NR) {
                S.beta[q] = s * S.rz_inv[q];
                S.rz_prev[q] = S.rz[q];
                S.rz[q] = s;
                S.flag_z[q] = isfinite(s) ? 0 : kNonfinite;
            }
            if (WHAT == kBeta && q >= NR) {
                const int k = q - NR;
                S.rr[k] = s;
                S.flag_r[k] = (isfinite(s) ? 0 : kNonfinite) | (s <= S.target[k] ? kConverged : 0) |
                              (DROP && s < 1e-4 * S.rr_true[k] ? kDropped : 0);
            }
        }
    }
    __syncthreads();
    return S.bad == 0;
}

// Sums of y over the T lanes of each row (see row_product).
template <typename TV, int NR, bool CP>
__device__ __forceinline__ void sum_row_lanes(int T, int t, TV (&y)[NR][3]) {
    if constexpr (CP) {
        const bool up2 = t & (T >> 1), up1 = t & (T >> 2);
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            // lanes of the upper half keep component 2, those of the lower half 0 and 1
            const TV g0 = __shfl_xor_sync(0xffffffffu, up2 ? y[k][0] : y[k][2], T >> 1);
            const TV g1 = __shfl_xor_sync(0xffffffffu, y[k][1], T >> 1);
            TV k0 = (up2 ? y[k][2] : y[k][0]) + g0;
            const TV k1 = y[k][1] + g1;
            const TV got = __shfl_xor_sync(0xffffffffu, up1 ? k0 : (up2 ? k0 : k1), T >> 2);
            k0 = (up2 ? k0 : (up1 ? k1 : k0)) + got;
            for (int o = T >> 3; o > 0; o >>= 1) k0 += __shfl_xor_sync(0xffffffffu, k0, o);
            y[k][0] = k0;
        }
    } else {
        for (int o = T >> 1; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < NR; ++k)
#pragma unroll
                for (int a = 0; a < 3; ++a) y[k][a] += __shfl_xor_sync(0xffffffffu, y[k][a], o);
    }
}

// One row's block products against the ext vectors in shared memory, T lanes
// a row.  CP: component a is summed into the lanes t with t / (T / 4) == a (two
// halving steps, then plain ones: 4 additions for T = 8 instead of 9); otherwise
// every lane of the row gets the three sums.
template <typename TV, int NR, bool CP>
__device__ __forceinline__ void row_product(const ResArgs& A, const TV* sv, const uint16_t* sc, const TV* pe, int vt,
                                            int t, int lane32, int64_t g0, int len, TV (&y)[NR][3]) {
#pragma unroll
    for (int k = 0; k < NR; ++k) y[k][0] = y[k][1] = y[k][2] = (TV)0;
    auto term = [&](const TV (&m)[9], int c) {
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            const TV* p = pe + 3 * ((size_t)k * A.next + c);
            const TV p0 = p[0], p1 = p[1], p2 = p[2];
#pragma unroll
            for (int a = 0; a < 3; ++a)
                y[k][a] = fma(m[3 * a], p0, fma(m[3 * a + 1], p1, fma(m[3 * a + 2], p2, y[k][a])));
        }
    };
#pragma unroll 2
    for (int k = 0; k < A.KR; ++k) {
        const int c = sc[k * A.VT + vt];
        TV m[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) m[q] = sv[(size_t)(k * 9 + q) * A.VT + vt];
        term(m, c);
    }
    const TV* vals;
    if constexpr (sizeof(TV) == 8) vals = A.v64;
    else vals = A.v32;
#pragma unroll 2
    for (int k = A.KR; k < A.K; ++k) {
        const int j = k * A.T + t;
        if (j >= len) break;
        const int c = sc[k * A.VT + vt];
        TV m[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) m[q] = vals[((g0 + j) * 9 + q) * 32 + lane32];
        term(m, c);
    }
    sum_row_lanes<TV, NR, CP>(A.T, t, y);
}

// TV: value and direction type of the recurrence's product (double: the FP64
// method, float: the mixed one, whose true residuals read the FP64 values).
// CP: see row_product (T >= 4).  The threads play two parts: T lanes of a row
// form its product, and thread o < 3 x rows keeps x, r and the preconditioner
// of DOF o of the CTA, so that the vector work and the sums fill few warps
// instead of a few lanes of every warp.  DYN: all time steps of a Newmark run;
// a step's right-hand side and the residual of its start share one pass over
// the operator (resident where it fits) and the mass.
template <typename TV, int NR, bool CP, bool DYN>
__global__ void __launch_bounds__(res_threads(NR), 1) k_resident_pcg(ResArgs A, DynArgs D) {
    static_assert(!DYN || NR == 1, "the Newmark loop solves one right-hand side a step");
    constexpr bool MIXED = sizeof(TV) == 4;
    extern __shared__ __align__(16) unsigned char smem[];
    TV* pe = reinterpret_cast<TV*>(smem);
    double* zs = reinterpret_cast<double*>(smem + A.off_z);
    double* ys = reinterpret_cast<double*>(smem + A.off_y);  // row products of the CTA's DOF
    TV* sv = reinterpret_cast<TV*>(smem + A.off_v);
    uint16_t* sc = reinterpret_cast<uint16_t*>(smem + A.off_c);
    ResShared& S = *reinterpret_cast<ResShared*>(smem + A.off_s);
    const int tid = threadIdx.x, warp = tid >> 5;
    const int row0 = A.row0[blockIdx.x], nrow = A.row0[blockIdx.x + 1] - row0;
    // lane of a row
    const int rl = tid / A.T, t = tid - rl * A.T;
    const bool valid = rl < nrow;
    const int row = row0 + (valid ? rl : 0);
    const int vt = valid ? tid : 0;
    const int lane32 = row & 31;
    const int64_t g0 = A.slice_off[row >> 5];
    const int len = valid ? A.row_len[row] : 0;
    const int quarter = CP ? A.T >> 2 : 1;  // lanes that hold the same component
    const int n_lane_warps = (A.VT + 31) >> 5;
    // owner of a DOF
    const int nown = 3 * nrow;
    const bool owner = tid < nown;
    const size_t dof = 3 * (size_t)row0 + (owner ? tid : 0);
    const int ndw = (3 * A.rows + 31) >> 5;  // warps that hold owners
    const int next = A.ext_ptr[blockIdx.x + 1] - A.ext_ptr[blockIdx.x];
    const int32_t* ext = A.ext + A.ext_ptr[blockIdx.x];
    const uint16_t* gl = A.lcol + (size_t)blockIdx.x * A.K * A.VT;
    const TV* vals;
    if constexpr (MIXED) vals = A.v32;
    else vals = A.v64;
    for (int q = tid; q < A.K * A.VT; q += blockDim.x) sc[q] = gl[q];
    if (tid < A.VT)
        for (int k = 0; k < A.KR; ++k) {
            const int j = k * A.T + t;
#pragma unroll
            for (int q = 0; q < 9; ++q)
                sv[(size_t)(k * 9 + q) * A.VT + tid] = j < len ? vals[((g0 + j) * 9 + q) * 32 + lane32] : (TV)0;
        }
    for (int q = tid; q < NR * A.next * 3; q += blockDim.x) pe[q] = (TV)0;
    if (tid == 0) S.bad = 0;
    if (DYN && blockIdx.x == 0 && tid == 0) D.out->next_step = D.n_steps;
    double x[NR], r[NR], di = 0.0;
    float bi[3] = {0.f, 0.f, 0.f};
    if (A.pc == ASEND_PC_JACOBI) {
        di = A.dinv[dof];
    } else {  // row of the node's block
#pragma unroll
        for (int b = 0; b < 3; ++b) bi[b] = A.binv[3 * dof + b];
    }
#pragma unroll
    for (int k = 0; k < NR; ++k) {
        x[k] = A.zero_x ? 0.0 : A.x[(size_t)k * A.n_dof + dof];
        r[k] = 0.0;
    }
    double f[NR] = {};
    unsigned long long epoch = A.epoch0;
    unsigned long long zep[NR];  // epoch of each right-hand side's last published z
    // z = M r of the owners' DOF, published; their shares of r.z and r.r.
    // Called by all threads (the block preconditioner passes r through ys).
    auto publish_z = [&](int k, double& rz, double& rr) {
        double z = di * r[k];
        if (A.pc != ASEND_PC_JACOBI) {
            __syncthreads();
            if (owner) ys[tid] = r[k];
            __syncthreads();
            const int o = owner ? tid / 3 * 3 : 0;
            z = (double)fmaf(bi[0], (float)ys[o], fmaf(bi[1], (float)ys[o + 1], bi[2] * (float)ys[o + 2]));
        }
        zep[k] = epoch + 1;
        rz = rr = 0.0;
        if (owner) {
            st_word(A.z + (size_t)k * A.n_dof + dof, z, epoch + 1);
            rz = r[k] * z;
            rr = r[k] * r[k];
        }
    };
    // put(q, z) for the ext items q (3 x node + component) of right-hand side
    // k from q0 in steps of step, four words in flight, each waited for
    auto fetch_z = [&](int k, int q0, int step, auto&& put) {
        const ulonglong2* zk = A.z + (size_t)k * A.n_dof;
        for (int q = q0; q < 3 * next; q += 4 * step) {
            const ulonglong2* w[4];
            unsigned long long v[4], e[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int qu = min(q + u * step, 3 * next - 1), i = qu / 3;
                w[u] = zk + 3 * (size_t)ext[i] + (qu - 3 * i);
            }
            int spin = 0;
            bool all;
            do {
                all = true;
#pragma unroll
                for (int u = 0; u < 4; ++u) ld_word(w[u], v[u], e[u]);
#pragma unroll
                for (int u = 0; u < 4; ++u) all &= e[u] == zep[k];
            } while (!all && ++spin < kPollLimit);
            if (!all) S.bad = 1;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (q + u * step < 3 * next) put(q + u * step, __longlong_as_double((long long)v[u]));
        }
    };
    // row sums of the lanes to ys
    auto put_rows = [&](int k, const auto (&y)[NR][3]) {
        if (!valid) return;
        double* yk = ys + (size_t)k * 3 * A.rows + 3 * rl;
        if constexpr (CP) {
            if (t % quarter == 0 && t < 3 * quarter) yk[t / quarter] = (double)y[k][0];
        } else if (t == 0) {
#pragma unroll
            for (int a = 0; a < 3; ++a) yk[a] = (double)y[k][a];
        }
    };
    // r_k = f_k - A64 x_k from the published x (FP64 values, FP64 sums)
    auto true_residual = [&](int k, bool zero) {
        if (!zero) {
            double y[1][3] = {{0.0, 0.0, 0.0}};
            for (int j = t; j < len; j += A.T) {
                const int64_t g = g0 + j;
                const double* xk = A.x + (size_t)k * A.n_dof + 3 * (size_t)A.col[g * 32 + lane32];
                const double x0 = __ldcg(xk), x1 = __ldcg(xk + 1), x2 = __ldcg(xk + 2);
                const double* m = A.v64 + (g * 9) * 32 + lane32;
#pragma unroll
                for (int a = 0; a < 3; ++a)
                    y[0][a] = fma(m[(3 * a) * 32], x0,
                                  fma(m[(3 * a + 1) * 32], x1, fma(m[(3 * a + 2) * 32], x2, y[0][a])));
            }
            __syncwarp();
            sum_row_lanes<double, 1, CP>(A.T, t, y);
            __syncthreads();  // ys is free
            if (valid) {
                if constexpr (CP) {
                    if (t % quarter == 0 && t < 3 * quarter) ys[3 * rl + t / quarter] = y[0][0];
                } else if (t == 0) {
#pragma unroll
                    for (int a = 0; a < 3; ++a) ys[3 * rl + a] = y[0][a];
                }
            }
            __syncthreads();
        }
        r[k] = f[k] - (zero || !owner ? 0.0 : ys[tid]);
    };
    // DYN: ys[0 ..] = A u + M (a - cM u) [+ D (v - cD u)], ys[3 rows ..] = A x
    // of the published state and start x
    auto step_products = [&]() {
        double y[2][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
        for (int j = t, k = 0; j < len; j += A.T, ++k) {
            const int64_t g = g0 + j;
            const size_t cn = 3 * (size_t)A.col[g * 32 + lane32];
            double un[3], wn[3], xn[3], zn[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                un[b] = __ldcg(D.u + cn + b);
                wn[b] = __ldcg(D.a + cn + b) - D.cM * un[b];
                xn[b] = __ldcg(A.x + cn + b);
                if (D.d64) zn[b] = __ldcg(D.v + cn + b) - D.cD * un[b];
            }
#pragma unroll
            for (int q = 0; q < 9; ++q) {
                double kv;
                if (!MIXED && k < A.KR) kv = (double)sv[(size_t)(k * 9 + q) * A.VT + vt];
                else kv = A.v64[(g * 9 + q) * 32 + lane32];
                const double mv = D.m64[(g * 9 + q) * 32 + lane32];
                y[0][q / 3] = fma(kv, un[q % 3], fma(mv, wn[q % 3], y[0][q / 3]));
                y[1][q / 3] = fma(kv, xn[q % 3], y[1][q / 3]);
                if (D.d64) y[0][q / 3] = fma(D.d64[(g * 9 + q) * 32 + lane32], zn[q % 3], y[0][q / 3]);
            }
        }
        __syncwarp();
        sum_row_lanes<double, 2, CP>(A.T, t, y);
        __syncthreads();  // ys is free
        if (valid) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                double* yh = ys + (size_t)h * 3 * A.rows + 3 * rl;
                if constexpr (CP) {
                    if (t % quarter == 0 && t < 3 * quarter) yh[t / quarter] = y[h][0];
                } else if (t == 0) {
#pragma unroll
                    for (int a = 0; a < 3; ++a) yh[a] = y[h][a];
                }
            }
        }
        __syncthreads();
    };
    auto store = [&](double* out, const double (&v)[NR]) {
        if (!owner) return;
#pragma unroll
        for (int k = 0; k < NR; ++k) out[(size_t)k * A.n_dof + dof] = v[k];
    };
    auto nothing = []() {};

    int iter[NR], n_repl = 0, since = 0;
    bool fin[NR], nonfinite = false, timed_out = false;  // the same in every thread
    int run_iters = 0, run_capped = 0;                   // DYN: over the launch's steps
    double run_rel2 = 0.0;
    for (int step = DYN ? D.step0 : 0; step < (DYN ? D.n_steps : 1); ++step) {
    // ---- right-hand side and initial residual
    since = 0;
    {
        double v[3 * NR];
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            if constexpr (DYN) {
                f[0] = r[0] = 0.0;
                if (step > 0) step_products();
                if (owner) {
                    f[0] = D.amp[step] * D.f0[dof] + D.pen[dof] - (step > 0 ? ys[tid] : 0.0);
                    r[0] = f[0] - (step > 0 ? ys[3 * A.rows + tid] : 0.0);
                }
            } else {
                f[k] = A.f[(size_t)k * A.n_dof + dof];
                true_residual(k, A.zero_x != 0);
            }
            publish_z(k, v[k], v[NR + k]);
            v[2 * NR + k] = owner ? f[k] * f[k] : 0.0;
            iter[k] = 0;
        }
        timed_out = !exchange<3 * NR, NR, kSum, false, false>(A, S, ndw, v, ++epoch, nothing);
        if (tid < NR) {
            const double rz = S.tot[tid], rr = S.tot[NR + tid];
            S.rz[tid] = rz;
            S.beta[tid] = 0.0;
            S.rr[tid] = S.rr_true[tid] = rr;
            S.bb[tid] = S.tot[2 * NR + tid];
            S.target[tid] = A.tol2 * S.bb[tid];
            S.flag_r[tid] = (isfinite(rr) && isfinite(rz) ? 0 : kNonfinite) | (rr <= S.target[tid] ? kConverged : 0);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            nonfinite |= (S.flag_r[k] & kNonfinite) != 0;
            fin[k] = S.flag_r[k] != 0;
        }
    }
    int it = 0;
    bool have_z = false;  // zs holds the last published z of every unfinished right-hand side
    for (;;) {
        bool all = true;
#pragma unroll
        for (int k = 0; k < NR; ++k) all &= fin[k];
        if (all || nonfinite || timed_out || it >= A.cap) break;
        // p = z + beta p on every ext node (a finished right-hand side keeps its p)
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            if (fin[k]) continue;
            const double beta = S.beta[k];
            TV* pk = pe + (size_t)k * A.next * 3;
            auto put = [&](int q, double z) { pk[q] = (TV)(z + beta * (double)pk[q]); };
            if (have_z) {
                const double* zk = zs + (size_t)k * A.next * 3;
                for (int q = tid; q < 3 * next; q += blockDim.x) put(q, zk[q]);
            } else {
                fetch_z(k, tid, blockDim.x, put);
            }
        }
        __syncthreads();
        if (warp < n_lane_warps) {
            TV y[NR][3];
            row_product<TV, NR, CP>(A, sv, sc, pe, vt, t, lane32, g0, len, y);
#pragma unroll
            for (int k = 0; k < NR; ++k) put_rows(k, y);
        }
        __syncthreads();
        double p_own[NR], y_own[NR], va[NR];
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            va[k] = 0.0;
            if (warp >= ndw) continue;
            p_own[k] = owner ? (double)pe[(size_t)k * A.next * 3 + tid] : 0.0;
            y_own[k] = owner ? ys[(size_t)k * 3 * A.rows + tid] : 0.0;
            va[k] = p_own[k] * y_own[k];
        }
        timed_out = !exchange<NR, NR, kAlpha, false, false>(A, S, ndw, va, ++epoch, nothing);
        if (timed_out) break;
        double v[2 * NR];
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            v[k] = v[NR + k] = 0.0;
            if (fin[k]) continue;
            if (warp < ndw) {
                const double alpha = S.alpha[k];
                x[k] += alpha * p_own[k];
                r[k] -= alpha * y_own[k];
            }
            zep[k] = epoch + 1;
            if (warp < ndw || A.pc != ASEND_PC_JACOBI) publish_z(k, v[k], v[NR + k]);
        }
        // warps that carry no sum fetch the new z meanwhile, where they are many
        have_z = (int)(blockDim.x >> 5) >= 4 * NR;
        timed_out = !exchange<2 * NR, NR, kBeta, false, MIXED>(A, S, ndw, v, ++epoch, [&]() {
            if (!have_z) return;
#pragma unroll
            for (int k = 0; k < NR; ++k) {
                double* zk = zs + (size_t)k * A.next * 3;
                if (!fin[k])
                    fetch_z(k, tid - 64 * NR, blockDim.x - 64 * NR, [&](int q, double z) { zk[q] = z; });
            }
        });
        if (timed_out) break;
        ++it;
        ++since;
        bool repl[NR], any = false, conv[NR];
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            repl[k] = conv[k] = false;
            if (fin[k]) continue;
            iter[k] += 1;
            const int flags = S.flag_z[k] | S.flag_r[k];
            if (flags & kNonfinite) {
                nonfinite = true;
                continue;
            }
            conv[k] = (flags & kConverged) != 0;
            // kDropped (mixed): the FP32-operator recurrence has dropped 1e4
            // below the last true residual: replace it before the two drift apart
            repl[k] = flags != 0 || (A.replace_every > 0 && since >= A.replace_every);
            any |= repl[k];
        }
        if (!any || nonfinite) continue;
        // true residuals: publish x, then f - A64 x; a converged recurrence
        // that the true residual does not confirm restarts its direction (p =
        // z), the others keep theirs
        since = 0;
        have_z = false;
        store(A.x, x);
        const double none[1] = {0.0};
        timed_out = !exchange<1, 1, kSum, true, false>(A, S, ndw, none, ++epoch, nothing);
        if (timed_out) break;
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            v[k] = v[NR + k] = 0.0;
            if (!repl[k]) continue;
            true_residual(k, false);
            publish_z(k, v[k], v[NR + k]);
            ++n_repl;
        }
        timed_out = !exchange<2 * NR, NR, kSum, false, false>(A, S, ndw, v, ++epoch, nothing);
        if (timed_out) break;
        if (tid < NR) {
            bool rp = false, cv = false;
#pragma unroll
            for (int k = 0; k < NR; ++k)
                if (k == tid) rp = repl[k], cv = conv[k];
            if (rp) {
                const double rz = S.tot[tid], rr = S.tot[NR + tid];
                S.rr[tid] = S.rr_true[tid] = rr;
                S.rz[tid] = rz;
                S.beta[tid] = cv ? 0.0 : rz / S.rz_prev[tid];
                S.flag_r[tid] =
                    (isfinite(rr) && isfinite(rz) ? 0 : kNonfinite) | (rr <= S.target[tid] ? kConverged : 0);
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            if (!repl[k]) continue;
            nonfinite |= (S.flag_r[k] & kNonfinite) != 0;
            fin[k] = S.flag_r[k] != 0;
        }
    }
    if constexpr (DYN) {
        if (nonfinite || timed_out) break;  // the state stays that of the last good step
        if (blockIdx.x == 0 && tid == 0) {
            run_iters += iter[0];
            run_capped |= !fin[0];
            if (S.bb[0] > 0.0) run_rel2 = fmax(run_rel2, S.rr_true[0] / S.bb[0]);
        }
        if (owner) {  // corrector, history shift, next predictor (k_newmark_update)
            const double upi = D.up[dof], vpi = D.vp[dof], api = D.ap[dof];
            const double un = D.u[dof] + x[0];
            const double an = D.c1 * (upi - un + D.dt * vpi + D.c2 * api);
            const double vn = vpi + D.dt * ((1.0 - D.gamma) * api + D.gamma * an);
            const double a2 = D.c1 * (D.dt * vn + D.c2 * an);
            D.up[dof] = un;
            D.vp[dof] = vn;
            D.ap[dof] = an;
            D.u[dof] = un;
            D.a[dof] = a2;
            D.v[dof] = vn + D.dt * ((1.0 - D.gamma) * an + D.gamma * a2);
            if (D.hist_fields > 0) {
                double* h = D.hist + (size_t)step * D.hist_fields * A.n_dof + dof;
                h[0] = un;
                if (D.hist_fields == 3) {
                    h[(size_t)A.n_dof] = vn;
                    h[2 * (size_t)A.n_dof] = an;
                }
            }
            if ((int)dof == D.probe) D.probe_hist[step] = un;
            if (D.extrapolate) {  // next start: 2 du - du_prev (the increment itself after the first step)
                const double d = x[0];
                if (step > 0) x[0] = 2.0 * d - D.du_prev[dof];
                D.du_prev[dof] = d;
            }
            A.x[dof] = x[0];
        }
        if (step + 1 < D.n_steps) {
            if (epoch - A.epoch0 >= kLaunchExchanges) {  // the state is stored: the next launch goes on from it
                if (blockIdx.x == 0 && tid == 0) D.out->next_step = step + 1;
                break;
            }
            const double none[1] = {0.0};
            timed_out = !exchange<1, 1, kSum, true, false>(A, S, ndw, none, ++epoch, nothing);
            if (timed_out) break;
        }
    }
    }
    if (timed_out && tid == 0) *A.err = 1;
    if constexpr (DYN) {
        if (blockIdx.x == 0 && tid == 0) {
            D.out->iterations += run_iters;
            D.out->capped |= run_capped;
            D.out->nonfinite = nonfinite || timed_out;
            D.out->rel_residual = fmax(D.out->rel_residual, sqrt(run_rel2));
        }
        return;
    }
    store(A.x, x);
    store(A.r, r);
    if (blockIdx.x == 0 && tid == 0) {
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            RhsScalars& s = A.sc[k];
            s.rr = S.rr[k];
            s.rr_last_true = S.rr_true[k];
            s.bb = S.bb[k];
            s.target = S.target[k];
            s.iter = iter[k];
            s.finished = fin[k] && !nonfinite;
            s.done = fin[k];
            s.nonfinite = nonfinite || timed_out;
            s.n_repl = k == 0 ? n_repl : 0;
        }
    }
}

template <typename TV, int NR, bool DYN>
const void* kernel_cp(bool cp) {
    return cp ? (const void*)k_resident_pcg<TV, NR, true, DYN> : (const void*)k_resident_pcg<TV, NR, false, DYN>;
}
template <typename TV>
const void* kernel_nr(int nr, bool cp, bool dyn) {
    if (dyn) return kernel_cp<TV, 1, true>(cp);
    switch (nr) {
        case 1: return kernel_cp<TV, 1, false>(cp);
        case 2: return kernel_cp<TV, 2, false>(cp);
        case 3: return kernel_cp<TV, 3, false>(cp);
        default: return kernel_cp<TV, 4, false>(cp);
    }
}
const void* resident_kernel(bool mixed, int nr, bool cp, bool dyn) {
    return mixed ? kernel_nr<float>(nr, cp, dyn) : kernel_nr<double>(nr, cp, dyn);
}

struct Layout {
    int off_z, off_y, off_v, off_c, off_s, KR;
    size_t bytes;
};
// Shared memory of a plan for values of vs bytes and nr right-hand sides: as
// many column steps of values as fit; bytes > limit when not even none do.
Layout layout_of(const ResidentPlan& P, size_t vs, int nr, bool dyn, size_t limit) {
    auto up = [](size_t v) { return (v + 15) & ~(size_t)15; };
    Layout L{};
    const size_t p = up((size_t)nr * P.next * 3 * vs), z = up((size_t)nr * P.next * 3 * sizeof(double));
    const size_t c = up((size_t)P.K * P.VT * sizeof(uint16_t));
    const size_t y = up((size_t)(dyn ? 2 : nr) * 3 * P.rows * sizeof(double));
    const size_t fixed = p + z + y + c + up(sizeof(ResShared)), step = (size_t)9 * P.VT * vs;
    L.KR = fixed > limit ? 0 : (int)std::min<size_t>(P.K, (limit - fixed) / step);
    L.off_z = (int)p;
    L.off_y = (int)(p + z);
    L.off_v = (int)(p + z + y);
    L.off_c = (int)(p + z + y + up(step * L.KR));
    L.off_s = (int)(L.off_c + c);
    L.bytes = fixed + up(step * L.KR);
    return L;
}

// Rows, ext nodes and local column ids of every CTA.
void build_plan(Ctx& c, ResidentPlan& P) {
    const Sbell& A = c.A;
    const int n = A.n_rows;
    P.rows = std::max((n + P.sms - 1) / P.sms, kResMinRows);
    P.grid = (n + P.rows - 1) / P.rows;
    P.T = 1;
    while (P.T < kResMaxLanes && P.rows * P.T * 2 <= kResLanes) P.T *= 2;
    P.VT = P.rows * P.T;
    int maxlen = 1;
    for (int r = 0; r < n; ++r) maxlen = std::max(maxlen, (int)A.h_row_len[r]);
    P.K = (maxlen + P.T - 1) / P.T;
    std::vector<int32_t> row0(P.grid + 1), ep(P.grid + 1, 0), ext, place(n, -1), seen(n, -1);
    std::vector<uint16_t> lcol((size_t)P.grid * P.K * P.VT, 0);
    P.next = 0;
    bool ok = true;
    for (int b = 0; b <= P.grid; ++b) row0[b] = std::min(n, b * P.rows);
    for (int b = 0; b < P.grid; ++b) {
        const int e0 = (int)ext.size();
        for (int r = row0[b]; r < row0[b + 1]; ++r) {
            seen[r] = b;
            place[r] = (int)ext.size() - e0;
            ext.push_back(r);
        }
        for (int r = row0[b]; r < row0[b + 1]; ++r) {
            const int rl = r - row0[b];
            const int64_t g0 = A.h_slice_off[r / kSlice];
            for (int j = 0; j < A.h_row_len[r]; ++j) {
                const int cn = A.h_col[(size_t)(g0 + j) * kSlice + r % kSlice];
                if (seen[cn] != b) {
                    seen[cn] = b;
                    place[cn] = (int)ext.size() - e0;
                    ext.push_back(cn);
                }
                lcol[((size_t)b * P.K + j / P.T) * P.VT + rl * P.T + j % P.T] = (uint16_t)place[cn];
            }
        }
        ep[b + 1] = (int)ext.size();
        P.next = std::max(P.next, ep[b + 1] - e0);
        ok &= ep[b + 1] - e0 <= 65535;
    }
    P.fits = ok;
    P.row0.upload(row0, c.stream);
    P.ext_ptr.upload(ep, c.stream);
    P.ext.upload(ext, c.stream);
    P.lcol.upload(lcol, c.stream);
    ASEND_CUDA(cudaStreamSynchronize(c.stream));  // the host vectors go out of scope
    P.words.alloc((size_t)2 * kMaxRhs * 3 * P.grid * P.grid);
    P.words.zero(c.stream);
    P.flags.alloc(2);
    P.flags.zero(c.stream);
}

}  // namespace

bool resident_timed_out(Ctx& c) {
    int flag = 0;
    if (!c.resident || !c.resident->flags.n) return false;
    ASEND_CUDA(cudaMemcpyAsync(&flag, c.resident->flags.p, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    ASEND_CUDA(cudaMemsetAsync(c.resident->flags.p, 0, sizeof(int), c.stream));
    ASEND_CUDA(cudaStreamSynchronize(c.stream));
    return flag != 0;
}

// The line lies where the kernel's layout ends: one DOF of a CTA a thread,
// which is 341 node rows an SM with one right-hand side (51,800 rows on 152
// SMs) and 213 with more (32,400).  Up to there the resident kernel was the
// faster one at every size measured (FP64 unless said): 525 rows 19.4 -> 3.5
// ms (two solves), 4,960 rows x 6 mixed 159 -> 48 ms, 20,402 shell rows 47.5
// -> 20.9 ms (60 time steps), 45,602 shell rows with a third of the values on
// chip 16.2 -> 10.7 ms (20 steps), 44,541 hex8 rows with 4 of 14 column steps
// on chip 74.5 -> 38.2 ms, mixed 106 -> 52 ms.
bool resident_usable(Ctx& c, const asend_solve_opts& o, int nr) {
    if (o.method != ASEND_METHOD_FP64 && o.method != ASEND_METHOD_MIXED) return false;
    if (c.n_inst > 1) return false;
    if (!c.resident || c.resident->pattern != c.pattern_serial) {
        auto P = std::make_shared<ResidentPlan>();
        P->pattern = c.pattern_serial;
        int coop = 0, sms = 0, smem = 0;
        ASEND_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c.device));
        ASEND_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device));
        ASEND_CUDA(cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, c.device));
        P->sms = std::min(sms, kMaxCtas);
        P->smem = (size_t)smem;
        P->fits = coop != 0 && c.A.n_rows <= P->sms * (res_threads(1) / 3);
        if (P->fits) build_plan(c, *P);
        c.resident = P;
    }
    const ResidentPlan& P = *c.resident;
    if (!P.fits || 3 * P.rows > res_threads(nr)) return false;
    const size_t vs = o.method == ASEND_METHOD_MIXED ? 4 : 8;
    const Layout L = layout_of(P, vs, nr, nr == 1, P.smem);  // (one right-hand side: room for a Newmark run)
    return L.bytes <= P.smem;
}

namespace {

// Launch over the plan of the current pattern, without synchronisation.
void launch_resident(Ctx& c, const asend_solve_opts& o, ResArgs a, const DynArgs* D, int nr) {
    ResidentPlan& P = *c.resident;
    const bool mixed = o.method == ASEND_METHOD_MIXED;
    const Layout L = layout_of(P, mixed ? 4 : 8, nr, D != nullptr, P.smem);
    if (P.z.n < (size_t)nr * c.n_dof) {  // words of epoch 0: older than every solve's
        P.z.alloc((size_t)nr * c.n_dof);
        P.z.zero(c.stream);
    }
    if (P.epoch >= 1ull << 63) {  // after 8.4 million launches: no word of the first ones may match again
        P.words.zero(c.stream);
        P.z.zero(c.stream);
        P.epoch = 0;
    }
    const int G = o.graph_iters > 0 ? o.graph_iters : 16, max_it = o.max_iter > 0 ? o.max_iter : c.n_dof;
    a.n_rows = c.A.n_rows;
    a.n_dof = c.n_dof;
    a.rows = P.rows;
    a.T = P.T;
    a.K = P.K;
    a.KR = L.KR;
    a.VT = P.VT;
    a.next = P.next;
    // the cap is looked at once a chunk of graph_iters iterations, as by the graphs
    a.cap = (int)std::min<int64_t>(((int64_t)max_it + G - 1) / G * G, INT32_MAX);
    a.replace_every = o.replace_every;
    a.off_z = L.off_z;
    a.off_y = L.off_y;
    a.off_v = L.off_v;
    a.off_c = L.off_c;
    a.off_s = L.off_s;
    a.n_words = kMaxRhs * 3;
    a.slice_off = c.A.slice_off.p;
    a.row_len = c.A.row_len.p;
    a.col = c.A.col.p;
    a.v64 = c.A.v64.p;
    a.v32 = c.A.v32.p;
    a.row0 = P.row0.p;
    a.ext_ptr = P.ext_ptr.p;
    a.ext = P.ext.p;
    a.lcol = P.lcol.p;
    a.z = P.z.p;
    a.dinv = c.d_dinv.p;
    a.binv = c.d_binv.p;
    a.words = P.words.p;
    a.epoch0 = P.epoch;
    P.epoch += 1ull << 40;  // more exchanges than one launch can make
    a.tol2 = o.rel_tol * o.rel_tol;
    a.err = P.flags.p;
    DynArgs none;
    std::memset(&none, 0, sizeof(none));
    const void* k = resident_kernel(mixed, nr, P.T >= 4, D != nullptr);
    const int threads = std::max({kResMinThreads, (P.VT + 31) / 32 * 32, (3 * P.rows + 31) / 32 * 32});
    // not this launch's size: the attribute is the kernel's, whichever context's thread sets it
    ASEND_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P.smem));
    void* args[] = {&a, D ? const_cast<DynArgs*>(D) : &none};
    ASEND_CUDA(cudaLaunchCooperativeKernel(k, dim3(P.grid), dim3(threads), args, L.bytes, c.stream));
    ++c.launches;
}

}  // namespace

void resident_enqueue(Ctx& c, const asend_solve_opts& o, int pc, bool warm, const double* d_f, double* d_x, double* d_r,
                      int nr, void* d_sc) {
    ResArgs a;
    std::memset(&a, 0, sizeof(a));
    a.pc = pc;
    a.zero_x = warm ? 0 : 1;
    a.f = d_f;
    a.x = d_x;
    a.r = d_r;
    a.sc = static_cast<RhsScalars*>(d_sc);
    launch_resident(c, o, a, nullptr, nr);
}

ResidentRun resident_newmark(Ctx& c, const asend_solve_opts& o, const NewmarkState& N) {
    ResArgs a;
    std::memset(&a, 0, sizeof(a));
    a.pc = o.precond;
    a.zero_x = 1;
    a.x = N.du;
    DArr<ResidentRun> out;
    out.alloc(1);
    out.zero(c.stream);
    DynArgs D;
    std::memset(&D, 0, sizeof(D));
    D.n_steps = N.n_steps;
    D.extrapolate = o.warm_start == 2;
    D.probe = N.probe;
    D.hist_fields = N.hist_fields;
    D.m64 = c.A.m64.p;
    D.d64 = c.A.d64.n ? c.A.d64.p : nullptr;
    D.f0 = N.f0;
    D.pen = N.pen;
    D.amp = N.amp;
    D.cM = c.cM;
    D.cD = c.cD;
    D.dt = c.dt;
    D.gamma = c.gamma;
    D.c1 = N.c1;
    D.c2 = N.c2;
    D.u = N.u;
    D.v = N.v;
    D.a = N.a;
    D.up = N.up;
    D.vp = N.vp;
    D.ap = N.ap;
    D.du_prev = N.du_prev;
    D.probe_hist = N.probe_hist;
    D.hist = N.hist;
    D.out = out.p;
    for (;;) {
        launch_resident(c, o, a, &D, 1);
        ResidentRun r;
        ASEND_CUDA(cudaMemcpyAsync(&r, out.p, sizeof(r), cudaMemcpyDeviceToHost, c.stream));
        ASEND_CUDA(cudaStreamSynchronize(c.stream));
        if (r.nonfinite && resident_timed_out(c)) throw CudaError("a grid-wide wait of the resident PCG ran out");
        if (r.nonfinite || r.next_step >= N.n_steps) return r;
        D.step0 = r.next_step;
        a.zero_x = 0;
    }
}

}  // namespace asend
