// k_box.cu -- matrix-free operator products on structured blocks of equal box
// elements: the finest level of the multigrid CG without its assembled values.
//
// The reference multiplies an assembled row-list matrix
// (SparseMat::vector_multiply, solverSrc/asend_run_job/src/list_ent_meth.rs:64-79).
// On the assembled operator the finest products are bound by its bytes (200 x
// 40 x 40 hex8: 688 MB for the CG product's FP32 pairs, 118 us; 365 MB for a
// smoothing product, 60 us).  With one element class per block the operator is
// sum_e E_e K^ + diagonal penalty, and everything a product has to read -- the
// vector and one modulus an element -- stays in L2: the time is arithmetic.
//
// Arithmetic.  A box has three reflections, so K^ falls apart in the basis of
// corner sign patterns: with p = (px, py, pz) the parities of a pattern,
// component c of pattern p only meets the components d of patterns q with p
// xor e_c = q xor e_d.  Eight blocks L = p xor e_c remain, five 3 x 3 and
// (the constant pattern p = 0 being a translation, which K^ annihilates) three
// 2 x 2: 57 products an element instead of 576, plus the sums and differences
// that form the patterns and undo them.
//
// Rounded entries annihilate a translation only to rounding, and the net force
// that leaves, although 1e-16 to 1e-15 of an entry, adds up over a slender
// model to an elastic foundation that moves its solution by 1e-9.  So that the
// product is that of the assembled operator in this respect too, the patterns
// come from the entries the assembly uses (FP64, or their FP32 pairs) and the
// pair product keeps the 3 x 3 block of the net force of a translation (FP32:
// it is itself of rounding size).  What else the patterns leave out is of that
// size and balanced within the element.
//
// Layout.  A thread owns one position m = j (nz + 1) + k of the node planes i =
// const and marches along i: at layer l it holds element (l, j, k), whose
// corners are the positions m, m + 1, m + nz + 1, m + nz + 2 of planes l and l +
// 1.  The in-plane half of the patterns is formed once a plane and used by the
// layers on both sides; the contributions of the two layers to a plane meet in
// the pattern basis, so the in-plane half is also undone once a plane.  A CTA
// covers a run of positions (with nz + 2 more on either side: the neighbours'
// contributions and corners) and a run of planes (with one layer more); the
// corner sums pass through shared memory, one barrier a layer.  Runs are sized
// so that one wave of CTAs covers the blocks.
//
// Two arithmetics: FP32 (the V-cycle's residual, post-smoothing and power
// steps) and FP32 pairs (the CG product), whose sums are TwoSum with the errors
// carried in the low parts: its error against 64 bits is 0.5 to 1.4e-15 of |K|
// |u| (the assembled pair product's 2.7 to 9.5e-15).  Measured, product /
// residual, against the assembled ones: 200 x 40 x 40: 36.8 / 12.3 us (118 /
// 60); 128 x 64 x 64: 57 / 18.4 us (200 / 98); 100 x 20 x 20: 16.5 / 6.2 us (21
// / 10).  FP32 issue bounds the pair product (12 warps an SM at the registers
// it needs; 62 % of the issue slots of the busy SMs), latency the FP32 ones.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>

#include "box.cuh"

namespace asend {

// One CTA's share: positions t0 .. t0 + blockDim - 1 (the first nz + 2 only
// contribute) of node planes i0 .. i1 - 1 of a block; or, n_pad > 0, the rows
// node0 .. node0 + n_pad - 1 of nodes without elements (unit diagonal).
struct BoxItem {
    int node0, el0, nx, ny, nz, cls, t0, i0, i1, n_pad;
};

struct BoxPlan {
    int64_t pattern = -1, epoch = -1;
    bool ok = false;
    int threads = 0, halo = 0, n_items = 0, pairs = 0, n_rows = 0;
    DArr<BoxItem> items;
    DArr<float2> B[2];                       // [n_cls][kBoxB] pattern blocks (hi, lo) of K^ in FP64, as pairs
    DArr<int32_t> cta_inst, inst_cta0, inst_ncta;  // batched stacks: CTAs by instance
    DArr<int32_t> pen_dof;                   // constrained DOF, coefficient^2, instance
    DArr<double> pen_coef, pen_sf;
    DArr<int32_t> pen_inst;
    DArr<float2> pen;                        // [n_dof] penalty of each DOF (pairs)
    DArr<uint8_t> pen_node;                  // nodes with a penalty
    DArr<float2> E;                          // element moduli as pairs
};

namespace {
using namespace pcg;

constexpr int kBoxThreads = 384;  // threads of a CTA at most (168 registers each fill an SM)
constexpr int kBoxB = 48;         // 39 entries of the symmetric pattern blocks, 9 of the net force

struct BoxArgs {
    const BoxItem* items;
    const float2* B;
    const float2* E;
    const float2* pen;
    const uint8_t* pen_node;
    int halo;
    int n_rows;
};

struct P2 {  // value h + l, not renormalised: |l| stays near 2^-24 of the operands
    float h, l;
};
__device__ __forceinline__ float add(float a, float b) { return a + b; }
__device__ __forceinline__ float sub(float a, float b) { return a - b; }
__device__ __forceinline__ P2 add(P2 a, P2 b) {
    const F2 s = two_sum(a.h, b.h);
    return {s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l))};
}
__device__ __forceinline__ P2 sub(P2 a, P2 b) { return add(a, P2{-b.h, -b.l}); }
__device__ __forceinline__ void zero(float& a) { a = 0.f; }
__device__ __forceinline__ void zero(P2& a) { a = {0.f, 0.f}; }

// net force per modulus of the translation of the patterns 0
__device__ __forceinline__ void net_force(const float2* B, const float (&)[3][4], const float (&)[3][4], float,
                                          float (&o)[3]) {
    o[0] = o[1] = o[2] = 0.f;  // below the FP32 products' rounding
}
__device__ __forceinline__ void net_force(const float2* B, const P2 (&hi)[3][4], const P2 (&low)[3][4], float e,
                                          P2 (&o)[3]) {
    const float t[3] = {hi[0][0].h + low[0][0].h, hi[1][0].h + low[1][0].h, hi[2][0].h + low[2][0].h};
#pragma unroll
    for (int c = 0; c < 3; ++c)
        o[c] = {e * fmaf(B[3 * c].x, t[0], fmaf(B[3 * c + 1].x, t[1], B[3 * c + 2].x * t[2])), 0.f};
}

// b0 x0 + b1 x1 (+ b2 x2), scaled by the modulus e
template <int N>
__device__ __forceinline__ float dot_scaled(const float2 (&b)[N], const float (&x)[N], float2 e) {
    float s = b[0].x * x[0];
#pragma unroll
    for (int q = 1; q < N; ++q) s = fmaf(b[q].x, x[q], s);
    return s * e.x;
}
template <int N>
__device__ __forceinline__ P2 dot_scaled(const float2 (&b)[N], const P2 (&x)[N], float2 e) {
    float S = __fmul_rn(b[0].x, x[0].h);
    float C = __fmaf_rn(b[0].x, x[0].h, -S);
    C = __fmaf_rn(b[0].x, x[0].l, C);
    C = __fmaf_rn(b[0].y, x[0].h, C);
#pragma unroll
    for (int q = 1; q < N; ++q) split_term(b[q].x, b[q].y, x[q].h, x[q].l, S, C);
    const float p = __fmul_rn(S, e.x);
    const float r = __fmaf_rn(S, e.x, -p);
    return {p, __fmaf_rn(S, e.y, __fmaf_rn(C, e.x, r))};
}

template <typename T>
struct Parts;  // float4 words of a node
template <>
struct Parts<float> {
    static constexpr int N = 1;
    __device__ static void split(const float4 (&w)[1], float (&v)[3]) { v[0] = w[0].x, v[1] = w[0].y, v[2] = w[0].z; }
    __device__ static void join(const float (&v)[3], float4 (&w)[1]) { w[0] = make_float4(v[0], v[1], v[2], 0.f); }
};
template <>
struct Parts<P2> {
    static constexpr int N = 2;
    __device__ static void split(const float4 (&w)[2], P2 (&v)[3]) {
        v[0] = {w[0].x, w[1].x}, v[1] = {w[0].y, w[1].y}, v[2] = {w[0].z, w[1].z};
    }
    __device__ static void join(const P2 (&v)[3], float4 (&w)[2]) {
        w[0] = make_float4(v[0].h, v[1].h, v[2].h, 0.f);
        w[1] = make_float4(v[0].l, v[1].l, v[2].l, 0.f);
    }
};

template <typename T>
constexpr size_t box_smem(int threads, int halo) {
    return sizeof(float2) * kBoxB + sizeof(float4) * Parts<T>::N * (2 * (size_t)(threads + halo) + 6 * (size_t)threads);
}

// epi(row, y, x) for every node row of the CTA's share: y = (A x)_row, x its own
// entries.  All threads of the CTA call it.
template <typename T, typename Epi>
__device__ __forceinline__ void box_march(const BoxArgs& A, const float4* __restrict__ x, unsigned char* smem, Epi&& epi) {
    constexpr int NW = Parts<T>::N;
    const int NT = blockDim.x, tau = threadIdx.x;
    const BoxItem it = A.items[blockIdx.x];
    if (it.n_pad > 0) {
        for (int r = it.node0 + tau; r < it.node0 + it.n_pad; r += NT) {
            float4 w[NW];
#pragma unroll
            for (int q = 0; q < NW; ++q) w[q] = x[(size_t)NW * r + q];
            T v[3];
            Parts<T>::split(w, v);
            epi(r, v, v);
        }
        return;
    }
    const int H = A.halo, stride = it.nz + 1, halo = it.nz + 2, plane = (it.ny + 1) * stride;
    float2* sB = reinterpret_cast<float2*>(smem);
    float4* su = reinterpret_cast<float4*>(smem + sizeof(float2) * kBoxB);  // [2][NW][NT + H]
    float4* sc = su + 2 * NW * (NT + H);                                    // [2][3][NW][NT]
    if (tau < kBoxB) sB[tau] = A.B[(size_t)it.cls * kBoxB + tau];
    const int m = it.t0 + tau, m2 = it.t0 + NT + tau;
    const bool in_plane = m >= 0 && m < plane;
    const bool more = tau < halo, in_plane2 = more && m2 >= 0 && m2 < plane;
    const int j = in_plane ? m / stride : 0, k = in_plane ? m - j * stride : 0;
    const bool has_el = in_plane && j < it.ny && k < it.nz;
    const size_t el = (size_t)it.el0 + (size_t)j * it.nz + k;
    const int el_step = it.ny * it.nz;
    const bool out = in_plane && tau >= halo;
    auto load = [&](int l, bool in, int pos, float4 (&w)[NW]) {
        const bool on = in && l <= it.nx;
        const float4* p = x + (size_t)NW * (it.node0 + (size_t)(on ? l : 0) * plane + (on ? pos : 0));
#pragma unroll
        for (int q = 0; q < NW; ++q) w[q] = on ? p[q] : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto keep = [&](int l, const float4 (&w)[NW], const float4 (&w2)[NW]) {
        float4* b = su + (l & 1) * NW * (NT + H);
#pragma unroll
        for (int q = 0; q < NW; ++q) {
            b[q * (NT + H) + tau] = w[q];
            if (more) b[q * (NT + H) + NT + tau] = w2[q];
        }
    };
    // in-plane patterns (py, pz) -> [2 py + pz] of the element's four corners in plane l
    auto patterns = [&](int l, const T (&own)[3], T (&o)[3][4]) {
        const float4* b = su + (l & 1) * NW * (NT + H) + tau;
        T n01[3], n10[3], n11[3];
        float4 w[NW];
#pragma unroll
        for (int q = 0; q < NW; ++q) w[q] = b[q * (NT + H) + 1];
        Parts<T>::split(w, n01);
#pragma unroll
        for (int q = 0; q < NW; ++q) w[q] = b[q * (NT + H) + stride];
        Parts<T>::split(w, n10);
#pragma unroll
        for (int q = 0; q < NW; ++q) w[q] = b[q * (NT + H) + stride + 1];
        Parts<T>::split(w, n11);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const T s0 = add(own[c], n01[c]), d0 = sub(n01[c], own[c]);
            const T s1 = add(n10[c], n11[c]), d1 = sub(n11[c], n10[c]);
            o[c][0] = add(s0, s1);
            o[c][1] = add(d0, d1);
            o[c][2] = sub(s1, s0);
            o[c][3] = sub(d1, d0);
        }
    };
    const int first = max(it.i0 - 1, 0);  // first layer: a whole one below i0, whose upper half is used
    T own[3], own_next[3], low[3][4], up[3][4];
    float4 w[NW], w2[NW];
    load(first, in_plane, m, w);
    load(first, in_plane2, m2, w2);
    keep(first, w, w2);
    Parts<T>::split(w, own);
    load(first + 1, in_plane, m, w);
    load(first + 1, in_plane2, m2, w2);
    keep(first + 1, w, w2);
    Parts<T>::split(w, own_next);
    float2 e = has_el && first < it.nx ? A.E[el + (size_t)first * el_step] : make_float2(0.f, 0.f);
    __syncthreads();
    patterns(first, own, low);
    __syncthreads();  // plane first is read: the first layer stores plane first + 2 over it
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int q = 0; q < 4; ++q) zero(up[c][q]);
    for (int l = first; l < it.i1; ++l) {
        const bool give = l >= it.i0;                   // plane l is this CTA's
        const bool another = l + 1 < it.i1;             // a further layer follows
        if (another) {
            load(l + 2, in_plane, m, w);
            load(l + 2, in_plane2, m2, w2);
        }
        const float2 e_next = has_el && another && l + 1 < it.nx ? A.E[el + (size_t)(l + 1) * el_step]
                                                                 : make_float2(0.f, 0.f);
        T V[3][4];
        {
            T hi[3][4];
            patterns(l + 1, own_next, hi);
            // u[c][p], p = px + 2 py + 4 pz; then the block outputs in place
            T u[3][8], net[3];
            net_force(sB + 39, hi, low, e.x, net);
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int p = (q >> 1) * 2 + (q & 1) * 4;
                    if (q) u[c][p] = add(hi[c][q], low[c][q]);
                    u[c][p + 1] = sub(hi[c][q], low[c][q]);
                    low[c][q] = hi[c][q];
                }
            auto block3 = [&](int L, int at) {
                const int px = L ^ 1, py = L ^ 2, pz = L ^ 4;
                const T v[3] = {u[0][px], u[1][py], u[2][pz]};
                const float2 b00 = sB[at], b01 = sB[at + 1], b02 = sB[at + 2], b11 = sB[at + 3], b12 = sB[at + 4],
                             b22 = sB[at + 5];
                const float2 r0[3] = {b00, b01, b02}, r1[3] = {b01, b11, b12}, r2[3] = {b02, b12, b22};
                u[0][px] = dot_scaled(r0, v, e);
                u[1][py] = dot_scaled(r1, v, e);
                u[2][pz] = dot_scaled(r2, v, e);
            };
            auto block2 = [&](int ca, int pa, int cb, int pb, int at) {
                const T v[2] = {u[ca][pa], u[cb][pb]};
                const float2 b00 = sB[at], b01 = sB[at + 1], b11 = sB[at + 2];
                const float2 r0[2] = {b00, b01}, r1[2] = {b01, b11};
                u[ca][pa] = dot_scaled(r0, v, e);
                u[cb][pb] = dot_scaled(r1, v, e);
            };
            block3(0, 0);
            block3(3, 6);
            block3(5, 12);
            block3(6, 18);
            block3(7, 24);
            block2(1, 3, 2, 5, 30);  // L = 1: y of pattern xy, z of xz
            block2(0, 3, 2, 6, 33);  // L = 2: x of xy, z of yz
            block2(0, 5, 1, 6, 36);  // L = 4: x of xz, y of yz
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int p = (q >> 1) * 2 + (q & 1) * 4;
                    if (q) {
                        V[c][q] = add(up[c][q], sub(u[c][p], u[c][p + 1]));
                        up[c][q] = add(u[c][p], u[c][p + 1]);
                    } else if constexpr (sizeof(T) == 4) {
                        V[c][0] = sub(up[c][0], u[c][1]);
                        up[c][0] = u[c][1];
                    } else {
                        V[c][0] = add(up[c][0], sub(net[c], u[c][1]));
                        up[c][0] = add(net[c], u[c][1]);
                    }
                }
        }
        T y[3];
        if (give) {
            T c01[3], c10[3], c11[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const T a = sub(V[c][0], V[c][1]), b = add(V[c][0], V[c][1]);
                const T a1 = sub(V[c][2], V[c][3]), b1 = add(V[c][2], V[c][3]);
                y[c] = sub(a, a1);
                c01[c] = sub(b, b1);
                c10[c] = add(a, a1);
                c11[c] = add(b, b1);
            }
            float4* o = sc + (l & 1) * 3 * NW * NT + tau;
            float4 t[NW];
            Parts<T>::join(c01, t);
#pragma unroll
            for (int q = 0; q < NW; ++q) o[q * NT] = t[q];
            Parts<T>::join(c10, t);
#pragma unroll
            for (int q = 0; q < NW; ++q) o[(NW + q) * NT] = t[q];
            Parts<T>::join(c11, t);
#pragma unroll
            for (int q = 0; q < NW; ++q) o[(2 * NW + q) * NT] = t[q];
        }
        if (another) keep(l + 2, w, w2);
        __syncthreads();
        if (give && out) {
            const float4* o = sc + (l & 1) * 3 * NW * NT + tau;
            const int from[3] = {1, stride, stride + 1};
#pragma unroll
            for (int h = 0; h < 3; ++h) {
                T v[3];
                float4 t[NW];
#pragma unroll
                for (int q = 0; q < NW; ++q) t[q] = o[(h * NW + q) * NT - from[h]];
                Parts<T>::split(t, v);
#pragma unroll
                for (int c = 0; c < 3; ++c) y[c] = add(y[c], v[c]);
            }
            const int row = it.node0 + l * plane + m;
            if (A.pen_node[row]) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float2 one[1] = {make_float2(1.f, 0.f)};
                    const T v[1] = {own[c]};
                    y[c] = add(y[c], dot_scaled(one, v, A.pen[3 * (size_t)row + c]));
                }
            }
            epi(row, y, own);
        }
        e = e_next;
#pragma unroll
        for (int c = 0; c < 3; ++c) own[c] = own_next[c];
        if (another) Parts<T>::split(w, own_next);
    }
}

__global__ void __launch_bounds__(kBoxThreads, 1) k_box_product(BoxArgs X, PcgArgs A, int n_inst,
                                                                int part_stride) {
    pdl_begin();
    extern __shared__ __align__(16) unsigned char smem[];
    const size_t rhs = blockIdx.y;  // this right-hand side's vectors, scalars, partials and tickets
    A.sc += rhs;
    RhsScalars* S = A.sc + cta_instance(A) * kMaxRhs;
    if (A.ctl->active[rhs] == 0 || S[0].done) return;
    A.p = reinterpret_cast<float4*>(A.p) + rhs * 2 * A.n_rows;
    A.ap = reinterpret_cast<float2*>(A.ap) + rhs * A.n_dof;
    A.partials += rhs * part_stride * (kMaxRhs * 3);
    A.tickets += rhs * n_inst * 4;
    F2 acc{0.f, 0.f};
    float2* ap = reinterpret_cast<float2*>(A.ap);
    box_march<P2>(X, reinterpret_cast<const float4*>(A.p), smem, [&](int row, const P2 (&y)[3], const P2 (&p)[3]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const F2 v = two_sum(y[c].h, y[c].l);
            ap[3 * (size_t)row + c] = make_float2(v.h, v.l);
            acc = f2_add(acc, f2_mul(F2{p[c].h, p[c].l}, v));
        }
    });
    double d[1][1] = {{f2_dbl(acc)}};
    double tot[1][1];
    if (last_block_reduce<1, 1>(A, d, 0, tot) && threadIdx.x == 0) set_alpha(S[0], tot[0][0]);
}

__global__ void __launch_bounds__(kBoxThreads, 1) k_box_resid(BoxArgs X, const float* b, const float4* x, float* r,
                                                              const Control* ctl) {
    pdl_begin();
    if (ctl && ctl->active[blockIdx.y] == 0) return;
    b += (size_t)blockIdx.y * 3 * X.n_rows;
    x += (size_t)blockIdx.y * X.n_rows;
    r += (size_t)blockIdx.y * 3 * X.n_rows;
    extern __shared__ __align__(16) unsigned char smem[];
    box_march<float>(X, x, smem, [&](int row, const float (&y)[3], const float (&)[3]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) r[3 * (size_t)row + c] = b[3 * (size_t)row + c] - y[c];
    });
}

__global__ void __launch_bounds__(kBoxThreads, 1) k_box_post(BoxArgs X, const float* __restrict__ binv, const float* b,
                                                             const float4* x, float4* y4, const Control* ctl) {
    pdl_begin();
    if (ctl && ctl->active[blockIdx.y] == 0) return;
    b += (size_t)blockIdx.y * 3 * X.n_rows;
    x += (size_t)blockIdx.y * X.n_rows;
    y4 += (size_t)blockIdx.y * X.n_rows;
    extern __shared__ __align__(16) unsigned char smem[];
    box_march<float>(X, x, smem, [&](int row, const float (&y)[3], const float (&xv)[3]) {
        const float* B = binv + 9 * (size_t)row;
        const float d0 = b[3 * (size_t)row] - y[0], d1 = b[3 * (size_t)row + 1] - y[1], d2 = b[3 * (size_t)row + 2] - y[2];
        y4[row] = make_float4(xv[0] + B[0] * d0 + B[1] * d1 + B[2] * d2, xv[1] + B[3] * d0 + B[4] * d1 + B[5] * d2,
                              xv[2] + B[6] * d0 + B[7] * d1 + B[8] * d2, 0.f);
    });
}

__global__ void __launch_bounds__(kBoxThreads, 1) k_box_power(BoxArgs X, const float* __restrict__ dinv,
                                                              const float4* __restrict__ x, float4* __restrict__ y4,
                                                              float* __restrict__ nrm, int k, double* __restrict__ part,
                                                              uint32_t* __restrict__ ticket) {
    pdl_begin();
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double sm[32];
    __shared__ bool last;
    const float inv = 1.f / nrm[k];
    double acc = 0.0;
    box_march<float>(X, x, smem, [&](int row, const float (&y)[3], const float (&)[3]) {
        const float* B = dinv + 9 * (size_t)row;
        const float z0 = inv * (B[0] * y[0] + B[1] * y[1] + B[2] * y[2]);
        const float z1 = inv * (B[3] * y[0] + B[4] * y[1] + B[5] * y[2]);
        const float z2 = inv * (B[6] * y[0] + B[7] * y[1] + B[8] * y[2]);
        y4[row] = make_float4(z0, z1, z2, 0.f);
        acc += (double)z0 * z0 + (double)z1 * z1 + (double)z2 * z2;
    });
    double a[1] = {acc};
    block_sum<1>(a, sm);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = a[0];
        last = take_ticket(ticket + k) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    double s[1] = {0.0};
#pragma unroll 4
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) s[0] += __ldcg(part + b);
    block_sum<1>(s, sm);
    if (threadIdx.x == 0) nrm[k + 1] = (float)sqrt(s[0]);
}

__global__ void k_box_penalty(int n, const int32_t* __restrict__ dof, const double* __restrict__ coef,
                              const int32_t* __restrict__ inst, const double* __restrict__ sf,
                              float2* __restrict__ pen) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const F2 v = f2_of(sf[inst[i]] * coef[i]);
    pen[dof[i]] = make_float2(v.h, v.l);
}

__global__ void k_box_moduli(int n, const double* __restrict__ E, float2* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const F2 v = f2_of(E[i]);
    out[i] = make_float2(v.h, v.l);
}

// The symmetric pattern blocks of K^ (576, reference corner order), in the
// order box_march reads them: B = Phi^T K^ Phi / 64 on the patterns of each L.
void pattern_blocks(const double* K, float2* out) {
    const int corner[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0}, {0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}};
    auto phi = [&](int p, int a) {
        double s = 1.0;
        for (int ax = 0; ax < 3; ++ax)
            if (p >> ax & 1) s *= corner[a][ax] ? 1.0 : -1.0;
        return s;
    };
    auto entry = [&](int L, int c, int d) {
        const int p = L ^ (1 << c), q = L ^ (1 << d);
        double s = 0.0;
        for (int a = 0; a < 8; ++a)
            for (int b = 0; b < 8; ++b) s += phi(p, a) * phi(q, b) * K[(3 * a + c) * 24 + 3 * b + d];
        return s / 64.0;
    };
    int at = 0;
    auto put = [&](double v) {
        const float h = (float)v;
        out[at++] = make_float2(h, (float)(v - (double)h));
    };
    for (int L : {0, 3, 5, 6, 7})
        for (int c = 0; c < 3; ++c)
            for (int d = c; d < 3; ++d) put(entry(L, c, d));
    for (int L : {1, 2, 4}) {
        const int skip = L == 1 ? 0 : (L == 2 ? 1 : 2);  // the translation
        const int a = skip == 0 ? 1 : 0, b = skip == 2 ? 1 : 2;
        put(entry(L, a, a));
        put(entry(L, a, b));
        put(entry(L, b, b));
    }
    for (int c = 0; c < 3; ++c)
        for (int d = 0; d < 3; ++d) {
            double s = 0.0;
            for (int a = 0; a < 8; ++a)
                for (int b = 0; b < 8; ++b) s += K[(3 * a + c) * 24 + 3 * b + d];
            put(s / 64.0);
        }
}

// Shares of the blocks: the CTA size and the planes a CTA takes that finish
// first.  A CTA's layers come one after the other (a layer below its first plane
// is computed twice: + 1, and the first loads: + 0.5); a layer takes longer the
// more warps share the SM: the pair product of ten planes 26.7 us with 64 to 128
// threads an SM, 35 to 36.5 with 192 to 256, 47.2 with 384 (one CTA or three), which
// 0.45 + 0.55 of the full SM's threads follows within 0.07.  What it picks was
// the fastest of the shares tried: 100 x 20 x 20 elements 96 threads x 1 plane 16.5 us
// (384 x 3 22.6, 96 x 12 28.7), 200 x 40 x 40 384 x 7 36.9 us (384 x 8 40.6, 192 x 25
// 71.2, 256 x 25 71.8).
void make_items(BoxPlan& P, const std::vector<std::array<int, 5>>& blocks, const std::vector<int>& cls, int n_nodes,
                int sms, std::vector<BoxItem>& items, std::vector<int32_t>& blk_of) {
    P.halo = 0;
    for (auto& b : blocks) P.halo = std::max(P.halo, b[2] + 2);
    auto segs = [&](const std::array<int, 5>& b, int nt) {
        const int plane = (b[1] + 1) * (b[2] + 1), useful = nt - (b[2] + 2);
        return (plane + useful - 1) / useful;
    };
    double best = 1e300;
    int best_nt = 0, best_len = 0, longest = 0;
    for (auto& b : blocks) longest = std::max(longest, b[0] + 1);
    for (int nt : {64, 96, 128, 192, 256, 384}) {
        if (nt < 2 * P.halo && nt < kBoxThreads) continue;
        const int slots = sms * (kBoxThreads / nt);
        for (int len = 1; len <= longest; ++len) {
            int64_t n = 0;
            for (auto& b : blocks) n += (int64_t)segs(b, nt) * ((b[0] + len) / len);
            const int64_t per_sm = std::min<int64_t>(kBoxThreads / nt, (n + sms - 1) / sms);
            const double layer = 0.45 + 0.55 * (double)(per_sm * nt) / kBoxThreads;
            const double t = (double)((n + slots - 1) / slots) * (len + 1.5) * layer;
            if (t < best) {
                best = t;
                best_nt = nt;
                best_len = len;
            }
        }
    }
    P.threads = best_nt;
    for (size_t q = 0; q < blocks.size(); ++q) {
        const auto& b = blocks[q];
        const int halo = b[2] + 2, useful = best_nt - halo, n_seg = segs(b, best_nt);
        for (int i0 = 0; i0 <= b[0]; i0 += best_len)
            for (int s = 0; s < n_seg; ++s) {
                items.push_back(BoxItem{b[3], b[4], b[0], b[1], b[2], cls[q], s * useful - halo, i0,
                                        std::min(i0 + best_len, b[0] + 1), 0});
                blk_of.push_back((int32_t)q);
            }
        const int end = b[3] + (b[0] + 1) * (b[1] + 1) * (b[2] + 1);
        const int stop = q + 1 < blocks.size() ? blocks[q + 1][3] : n_nodes;
        if (stop > end) {
            items.push_back(BoxItem{end, 0, 0, 0, 0, 0, 0, 0, 0, stop - end});
            blk_of.push_back((int32_t)q);
        }
    }
    P.n_items = (int)items.size();
}

BoxArgs args_of(const BoxPlan& P) { return BoxArgs{P.items.p, P.B[P.pairs].p, P.E.p, P.pen.p, P.pen_node.p, P.halo, P.n_rows}; }

template <typename T, typename... K, typename... Args>
void launch(Ctx& c, const BoxPlan& P, int nr, void (*k)(K...), Args... args) {
    const size_t smem = box_smem<T>(P.threads, P.halo);
    // the attribute is the kernel's, not the context's: the largest launch's, so that
    // threads with contexts of their own do not lower it under each other's launches
    ASEND_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)box_smem<T>(kBoxThreads, kBoxThreads / 2)));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)P.n_items, (unsigned)nr);
    cfg.blockDim = dim3((unsigned)P.threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = c.pdl ? 1 : 0;
    ASEND_CUDA(cudaLaunchKernelEx(&cfg, k, K(args)...));
}

}  // namespace

BoxPlan* box_plan(Ctx& c, const std::vector<std::array<int, 5>>& blocks) {
    if (!c.class_sum || c.cls_box.empty() || blocks.empty()) return nullptr;
    if (!c.box || c.box->pattern != c.pattern_serial) {
        auto P = std::make_shared<BoxPlan>();
        P->pattern = c.pattern_serial;
        P->ok = true;
        std::vector<int> cls;
        for (auto& b : blocks) {
            const int64_t n = (int64_t)b[0] * b[1] * b[2];
            const int k = c.h_cls_of[b[4]];
            for (int64_t e = 0; P->ok && e < n; ++e) P->ok = c.h_cls_of[b[4] + e] == k;
            P->ok = P->ok && c.cls_box[k] && 2 * (b[2] + 2) <= kBoxThreads;
            cls.push_back(k);
        }
        // diagonal penalties on the blocks' nodes only
        std::vector<uint8_t> in_block(c.n_nodes, 0);
        for (auto& b : blocks)
            std::fill_n(in_block.begin() + b[3], (size_t)(b[0] + 1) * (b[1] + 1) * (b[2] + 1), (uint8_t)1);
        for (size_t r = 0; P->ok && r + 1 < c.c_ptr.size(); ++r)
            P->ok = c.c_ptr[r + 1] - c.c_ptr[r] == 1 && in_block[c.c_dof[c.c_ptr[r]] / 3];
        c.box = P;
        if (!P->ok) return nullptr;
        int sms = 0;
        ASEND_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device));
        std::vector<BoxItem> items;
        std::vector<int32_t> blk_of;
        make_items(*P, blocks, cls, c.n_nodes, sms, items, blk_of);
        std::vector<double> k64((size_t)c.n_cls * 576);
        ASEND_CUDA(cudaMemcpyAsync(k64.data(), c.cls_ke.p, sizeof(double) * k64.size(), cudaMemcpyDeviceToHost, c.stream));
        ASEND_CUDA(cudaStreamSynchronize(c.stream));
        for (int pairs = 0; pairs < 2; ++pairs) {
            std::vector<float2> B((size_t)c.n_cls * kBoxB, make_float2(0.f, 0.f));
            if (pairs)
                for (double& v : k64) {
                    const float h = (float)v;
                    v = (double)h + (double)(float)(v - (double)h);
                }
            for (int k : cls) pattern_blocks(&k64[(size_t)k * 576], &B[(size_t)k * kBoxB]);
            P->B[pairs].upload(B, c.stream);
            ASEND_CUDA(cudaStreamSynchronize(c.stream));
        }
        std::vector<int32_t> first(blocks.size(), 0), count(blocks.size(), 0), pd, pi;
        for (size_t i = 0; i < blk_of.size(); ++i)
            if (count[blk_of[i]]++ == 0) first[blk_of[i]] = (int32_t)i;
        std::vector<double> sum(c.n_dof, 0.0), pc;
        std::vector<uint8_t> pn(c.n_nodes, 0);
        for (size_t r = 0; r + 1 < c.c_ptr.size(); ++r) {
            const int k = c.c_ptr[r], d = c.c_dof[k];
            sum[d] += c.c_coef[k] * c.c_coef[k];
            pn[d / 3] = 1;
        }
        for (int d = 0; d < c.n_dof; ++d)
            if (sum[d] != 0.0) {
                pd.push_back(d);
                pc.push_back(sum[d]);
                pi.push_back(c.n_inst > 1 ? instance_of_node(c, d / 3) : 0);
            }
        P->items.upload(items, c.stream);
        if (c.n_inst > 1) {
            P->cta_inst.upload(blk_of, c.stream);
            P->inst_cta0.upload(first, c.stream);
            P->inst_ncta.upload(count, c.stream);
        }
        P->pen_dof.upload(pd, c.stream);
        P->pen_coef.upload(pc, c.stream);
        P->pen_inst.upload(pi, c.stream);
        P->pen_node.upload(pn, c.stream);
        P->pen.alloc(c.n_dof);
        P->pen.zero(c.stream);
        P->E.alloc(c.n_el);
        P->n_rows = c.n_nodes;
        ASEND_CUDA(cudaStreamSynchronize(c.stream));  // the host vectors go out of scope
    }
    BoxPlan& P = *c.box;
    if (!P.ok) return nullptr;
    if (P.epoch != c.assembly_epoch) {  // this assembly's moduli and penalty scales
        k_box_moduli<<<(c.n_el + 255) / 256, 256, 0, c.stream>>>(c.n_el, c.d_E.p, P.E.p);
        const int n = (int)P.pen_dof.n;
        std::vector<double> sf(1, c.sf);
        if (c.n_inst > 1) sf = c.sf_inst;
        P.pen_sf.upload(sf, c.stream);
        if (n > 0)
            k_box_penalty<<<(n + 255) / 256, 256, 0, c.stream>>>(n, P.pen_dof.p, P.pen_coef.p, P.pen_inst.p, P.pen_sf.p,
                                                                 P.pen.p);
        c.launches += 1 + (n > 0);
        ASEND_CUDA(cudaGetLastError());
        P.epoch = c.assembly_epoch;
        P.pairs = c.class_pairs ? 1 : 0;
    }
    return &P;
}

const void* box_patterns(const BoxPlan& P) { return P.B[P.pairs].p; }
int box_ctas(const BoxPlan& P) { return P.n_items; }

void box_product(Ctx& c, const BoxPlan& P, PcgArgs a, int nr, int part_stride) {
    if (c.n_inst > 1) {  // this launch's own map of CTAs to instances
        a.cta_inst = P.cta_inst.p;
        a.inst_cta0 = P.inst_cta0.p;
        a.inst_ncta = P.inst_ncta.p;
    }
    launch<P2>(c, P, nr, k_box_product, args_of(P), a, std::max(1, c.n_inst), part_stride);
}
void box_resid(Ctx& c, const BoxPlan& P, const float* b, const float4* x, float* r, const Control* ctl, int nr) {
    launch<float>(c, P, nr, k_box_resid, args_of(P), b, x, r, ctl);
}
void box_post(Ctx& c, const BoxPlan& P, const float* binv, const float* b, const float4* x, float4* y4,
              const Control* ctl, int nr) {
    launch<float>(c, P, nr, k_box_post, args_of(P), binv, b, x, y4, ctl);
}
void box_power(Ctx& c, const BoxPlan& P, const float* dinv, const float4* x, float4* y4, float* nrm, int k,
               double* part, uint32_t* ticket) {
    launch<float>(c, P, 1, k_box_power, args_of(P), dinv, x, y4, nrm, k, part, ticket);
}

// moduli, direction and A p, each once
double box_product_bytes(const Ctx& c) { return 8.0 * c.n_el + 32.0 * c.n_nodes + 8.0 * c.n_dof; }

}  // namespace asend
