// k_mg.cu -- geometric multigrid preconditioner for structured hex8 blocks and
// the multigrid-preconditioned (flexible) CG driver.
//
// The reference preconditions its CG with LDL^T factors of diagonal blocks of
// the stiffness matrix (lower_tri_mat_meth.rs:15-241, block size from
// model_prep.rs:888-902) and otherwise follows conj_grad_sparse
// (matrix_functions.rs:285-362).  A block factorization has no efficient GPU
// form; this module replaces it by a V-cycle whose cost per application is a
// few SpMVs and whose iteration count is nearly independent of the mesh size.
//
// Hierarchy (structured block nx x ny x nz, node (i,j,k) = (i*(ny+1)+j)*(nz+1)+k):
//  * each level halves the element count per axis (an odd count leaves one
//    coarse element spanning a single fine element), down to <= 256 DOFs;
//  * prolongation is trilinear interpolation in index space, per component;
//  * coarse operators are Galerkin, formed element by element:
//        K_C = sum_{e child of C} Q_e^T K_e Q_e,
//    Q_e the 24x24 trilinear map from C's corners to e's corners.  For nested
//    grids this equals P^T A P exactly (without the penalty rows), and unlike
//    rediscretised coarse hex8 grids it does not lock in bending;
//  * penalty constraints enter coarse levels lumped: pen_c = P^T pen_f row sums;
//  * smoothing: one pre- and one post-sweep of damped nodal block Jacobi;
//  * coarsest level: explicit inverse (Gauss-Jordan, one cluster a block);
//  * all level arithmetic in FP32; the outer CG keeps the FP64 operator,
//    FP64 vectors and dots, and uses the Polak-Ribiere (flexible) beta
//    beta = -alpha (z . Ap) / (r_old . z_old), which tolerates the FP32
//    preconditioner's rounding asymmetry.
#include <algorithm>
#include <array>
#include <cstring>
#include <cmath>
#include <memory>
#include <utility>

#include <cooperative_groups.h>

#include "box.cuh"
#include "pcg_common.cuh"

namespace asend {

struct MgAxis {
    int n_f = 0, n_c = 0;         // fine / coarse element counts
    std::vector<int32_t> xs;      // coarse node -> fine node index (n_c + 1)
    std::vector<int32_t> lo;      // fine node -> lower coarse node (n_f + 1)
    std::vector<float> w;         // fine node -> weight of lo + 1
};

// One structured block of a level: a single model's grid, or one instance of
// a batched stack.  Block b of every level belongs to instance b; blocks are
// coarsened independently, and a block that needs no further coarsening is
// carried down unchanged (identity maps) until every block is coarse enough.
struct MgBlk {
    int nx = 0, ny = 0, nz = 0;   // cells
    int node0 = 0, el0 = 0;       // first node / element in the level numbering
    MgAxis ax[3];                 // maps from the finer level's block (levels >= 1)
    int ox[3] = {0, 0, 0};        // offsets into the level's packed xs
    double h[3] = {0, 0, 0};      // cell spacing per axis
    bool done = false;            // coarse enough: identity maps below this level
    int n_nodes() const { return (nx + 1) * (ny + 1) * (nz + 1); }
    int n_el() const { return nx * ny * nz; }
};

// Device descriptor of block b of a level; levels >= 1 also describe the
// finer level's block b (f*) and the block's axis maps.
struct BlkDev {
    int nx, ny, nz, node0, el0;
    int fnx, fny, fnz, fnode0, fel0;
    int ox0, ox1, ox2;
    int dense0;
};

struct MgLevel {
    int n_nodes = 0, n_el = 0, n_dof = 0;  // totals (level 0 of a batch includes padding nodes)
    std::vector<MgBlk> blk;
    DArr<BlkDev> d_blk;
    DArr<int32_t> pre_node, pre_el;  // per-block starts (+ total)
    DArr<int32_t> row_blk;        // block of each row (stacks of blocks)
    BlkDev one;                   // the descriptor of a lone block
    DArr<int32_t> d_xs;           // packed per block and axis
    Sbell own;                    // pattern + FP32 values (levels >= 1)
    Sbell* A = nullptr;
    DArr<float> Ke;               // Galerkin element matrices [n_el][24][24]
    std::vector<float> h_pen;     // lumped penalty per DOF (in units of sf)
    DArr<float> pen;
    DArr<float> binv, b, r, x4, y4;
    DArr<float> pow_vec;          // last power-iteration vector (warm start)
    bool pow_warm = false;
    int pow_steps = 0;            // steps of the last estimate
};

// Levels of the V-cycle's fused tail (k_vc_tail)
constexpr int kTailLevels = 6, kTailThreads = 1024, kTailCtas = 16, kTailSmem = 224 * 1024, kTailRows = 1024;
constexpr int kTailLd = 249;    // values of a row, 243: 16 lanes x 2 rows on different banks
constexpr int kTailCols = 28;   // columns of a row and their number
struct TailView {
    int n;  // levels, the last one the coarsest
    struct Level {
        BlkDev d;
        const float* v;
        const float* binv;
        int n_rows, own;  // rows, rows a CTA
        // shared memory, in floats
        int xo, ro;  // the vectors' copies (float4): iterate; residual, then result (the coarsest's xo: b)
        int so;      // own rows: [own][12] b and smoother block
        int co;      // own rows' columns, uint16 [own][kTailCols]
        int po;      // per node, uint16: 8 x first coarse node of its prolongation + axes between two
        int to;      // own rows' restriction: fine node + 65536 x axis sides that contribute
        int vo;      // own rows' values [own][kTailLd], or -1: in global memory
    } L[kTailLevels];
    const float* b;
    const float4* x4;
    float4* y4;
};

struct MgHierarchy {
    std::vector<std::unique_ptr<MgLevel>> L;
    DArr<float> dense, ainv;      // coarsest operators, one dense block per instance, inverted in place
    int n_coarse = 0;             // largest coarsest block (DOF)
    int n_blk = 1;
    int tail0 = 0;                // first level of the V-cycle's fused tail (0: no tail)
    TailView tail;                // its levels
    int tail_smem = 0;            // bytes
    std::vector<int32_t> h_dense0;  // offset of each block's dense matrix (floats)
    DArr<double> blk_sf;          // penalty scale per block (instance)
    DArr<float> child;            // projected class matrices of the first coarsening [n_cls][27][576]
    bool child_ready = false;
    // stacks: CTAs of the pair method's vector kernels (instance, rows; first
    // CTA and their number per instance)
    DArr<int32_t> cg_inst, cg_cta0, cg_ncta;
    DArr<int2> cg_rows;
    // captured outer iterations, reused while the launch arguments match
    std::vector<std::pair<std::vector<uint8_t>, cudaGraphExec_t>> graphs;
    ~MgHierarchy() {
        for (auto& g : graphs) cudaGraphExecDestroy(g.second);
    }
    int64_t epoch = -1;
    float omega = 0.6f;           // damping used when the eigenvalue estimate fails
    bool l0_learned = false;      // finest-level smoother blocks come from the learned model
    bool l0_damped = false;       // finest-level eigenvalue-damped blocks are current
    DArr<float> pow_nrm;          // power-iteration norms per level [levels][kPowSteps + 1]
    DArr<uint32_t> pow_ticket;    // last-CTA tickets per level and step
    DArr<double> pow_part;        // per-CTA partial sums
    DArr<unsigned int> pow_bound; // ||D^-1 A||_inf per level (float bits)
    DArr<float> pow_omega;        // damping in use per level
    bool safe_damping = false;    // omega from the guaranteed bound (after a failed solve)
    BoxPlan* box = nullptr;       // matrix-free finest products of the current operator (or none)
    bool box_cycle = false;       // V-cycles take them, too (inside the CG; a V-cycle that a caller sees
                                  // keeps the assembled values)
    DArr<float> vl_q, vl_mw, vl_t4, vl_r2, vl_w;  // learned-smoother training vectors
};

// Matrix-free finest products in the V-cycles of a scope.
struct BoxCycle {
    MgHierarchy& H;
    explicit BoxCycle(MgHierarchy& h) : H(h) { H.box_cycle = true; }
    ~BoxCycle() { H.box_cycle = false; }
};

constexpr int kPowSteps = 10;      // from a hashed start vector
constexpr int kPowWarmSteps = 4;   // from the previous assembly's vector

namespace {
using namespace pcg;

constexpr int kT = 128;
inline int grid_of(int n) { return (n + kT - 1) / kT; }
// Grid of the split method's CG kernels on a single instance: grid-stride
// loops over 4 CTAs per SM (152 SMs) instead of one CTA per 128 rows, so the
// last-CTA reductions sum 608 partials, not thousands.
constexpr int kPersistCtas = 152 * 4;

// Launch on the context's stream, with programmatic dependent launch when the
// context allows it (the kernel then starts while its predecessor drains and
// waits for it in pdl_begin(); every kernel launched here calls it first).
template <typename... KArgs, typename... Args>
void launch_k(const Ctx& c, void (*k)(KArgs...), dim3 grid, int block, size_t smem, Args&&... args) {
    if (!c.pdl) {
        k<<<grid, block, smem, c.stream>>>(std::forward<Args>(args)...);
        return;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    ASEND_CUDA(cudaLaunchKernelEx(&cfg, k, std::forward<Args>(args)...));
}
// Levels with at least this many node rows run the staged (bulk-copy) row
// products, one row per lane; smaller ones split each row over 16 lanes (with
// fewer, 8,192 rows leave SMs idle).
constexpr int kStagedRows = 8192;
// classes up to which the first coarsening uses projected class matrices
// (27 x 576 floats each, 62 KB)
constexpr int kMaxChildClasses = 512;

__device__ __forceinline__ int nid(int i, int j, int k, int ny, int nz) { return (i * (ny + 1) + j) * (nz + 1) + k; }

// hex8 corner offsets in the reference's corner order
__constant__ int c_corner[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0},
                                   {0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}};

struct LevelView {  // kernel-side view of a coarse level's blocks and maps from the finer level
    int n_blk;
    const BlkDev* blk;
    const int32_t* xs;
};

// Block of index idx: the largest b with pre[b] <= idx (pre ascending).
__device__ __forceinline__ int find_blk(const int32_t* __restrict__ pre, int n_blk, int idx) {
    int lo = 0, hi = n_blk - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pre[mid] <= idx) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// ---------------------------------------------------------------------------
// Galerkin coarsening by elements
// ---------------------------------------------------------------------------
// One CTA per coarse element C of level l.  Its <= 8 children (elements of level
// l-1) are processed together: each child's FP32 stiffness comes from the
// stored Galerkin matrices of level l-1, or for l = 1 is integrated here from
// the fine geometry (2x2x2 Gauss points, closed-form isotropic blocks as in
// the assembly kernel); then T_e = K_e (Q_e x I3) and
// K_C = sum_e (Q_e x I3)^T T_e.  A thread holds the eight entries of K_e that
// share its (child, row, component) in registers and forms their eight columns of
// T_e, then four rows of a column of K_C, so that an operand in shared
// memory serves 4 to 8 FMAs; one entry a thread (two loads an FMA) was bound by
// those loads: 750 us over the levels of 128 x 64 x 64 elements, now 304.
constexpr int kCoarsenThreads = 576;
constexpr int kTLd = 27;  // row stride of T (24 columns): lanes of 11 rows on different banks
__global__ void __launch_bounds__(kCoarsenThreads)
k_coarsen(LevelView cv, const int32_t* __restrict__ pre_el, const float* __restrict__ fine_ke,
          const float* __restrict__ cls_ke, const int32_t* __restrict__ cls_of, const double* __restrict__ xyz,
          const int32_t* __restrict__ conn0, const double* __restrict__ E, const double* __restrict__ nu,
          float* __restrict__ coarse_ke) {
    __shared__ float Ke[8][24 * kTLd];  // the integrated K_e, then T_e
    __shared__ __align__(16) float Q[8][8][8];
    __shared__ float g[8][8][8][3];
    __shared__ float wdet[8][8];
    __shared__ float xl[8][8][3];
    __shared__ int fe[8];
    const int t = threadIdx.x;
    const int C = blockIdx.x;
    const BlkDev& d = cv.blk[find_blk(pre_el, cv.n_blk, C)];
    const int Cl = C - d.el0;
    const int ci = Cl / (d.ny * d.nz), cj = (Cl / d.nz) % d.ny, ck = Cl % d.nz;
    const int s0 = cv.xs[d.ox0 + ci], w0 = cv.xs[d.ox0 + ci + 1] - s0;
    const int s1 = cv.xs[d.ox1 + cj], w1 = cv.xs[d.ox1 + cj + 1] - s1;
    const int s2 = cv.xs[d.ox2 + ck], w2 = cv.xs[d.ox2 + ck + 1] - s2;
    const int nch = w0 * w1 * w2;
    if (t < nch * 64) {  // interpolation weights of child ch: fine corner a <- coarse corner b
        const int ch = t >> 6, a = (t >> 3) & 7, b = t & 7;
        const int o0 = ch / (w1 * w2), o1 = (ch / w2) % w1, o2 = ch % w2;
        const float xi0 = (float)(o0 + c_corner[a][0]) / w0;
        const float xi1 = (float)(o1 + c_corner[a][1]) / w1;
        const float xi2 = (float)(o2 + c_corner[a][2]) / w2;
        Q[ch][a][b] = (c_corner[b][0] ? xi0 : 1.f - xi0) * (c_corner[b][1] ? xi1 : 1.f - xi1) *
                      (c_corner[b][2] ? xi2 : 1.f - xi2);
        if (a == 0 && b == 0) fe[ch] = d.fel0 + ((s0 + o0) * d.fny + (s1 + o1)) * d.fnz + (s2 + o2);
    }
    __syncthreads();
    if (!cls_ke && !fine_ke) {
        if (t < nch * 24) {
            const int ch = t / 24, a = (t / 3) % 8, j = t % 3;
            const int e = fe[ch];
            const int n0 = conn0[(size_t)e * 8], na = conn0[(size_t)e * 8 + a];
            xl[ch][a][j] = (float)(xyz[3 * (size_t)na + j] - xyz[3 * (size_t)n0 + j]);
        }
        __syncthreads();
        if (t < nch * 8) {  // Gauss-point data of child ch, point gp
            const int ch = t >> 3, gp = t & 7;
            const float gq = 0.5773502691896257f;
            const float s[3] = {(gp & 1) ? gq : -gq, (gp & 2) ? gq : -gq, (gp & 4) ? gq : -gq};
            float dn[8][3];
            float J[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
            for (int a = 0; a < 8; ++a) {
                const float sg0 = c_corner[a][0] ? 1.f : -1.f, sg1 = c_corner[a][1] ? 1.f : -1.f,
                            sg2 = c_corner[a][2] ? 1.f : -1.f;
                const float f0 = 1 + sg0 * s[0], f1 = 1 + sg1 * s[1], f2 = 1 + sg2 * s[2];
                dn[a][0] = 0.125f * sg0 * f1 * f2;
                dn[a][1] = 0.125f * sg1 * f0 * f2;
                dn[a][2] = 0.125f * sg2 * f0 * f1;
                for (int i = 0; i < 3; ++i)
                    for (int j = 0; j < 3; ++j) J[i][j] += xl[ch][a][i] * dn[a][j];
            }
            const float c00 = J[1][1] * J[2][2] - J[1][2] * J[2][1];
            const float c01 = J[1][2] * J[2][0] - J[1][0] * J[2][2];
            const float c02 = J[1][0] * J[2][1] - J[1][1] * J[2][0];
            const float det = J[0][0] * c00 + J[0][1] * c01 + J[0][2] * c02;
            const float id = 1.f / det;
            float Ji[3][3];
            Ji[0][0] = c00 * id;
            Ji[1][0] = c01 * id;
            Ji[2][0] = c02 * id;
            Ji[0][1] = (J[0][2] * J[2][1] - J[0][1] * J[2][2]) * id;
            Ji[1][1] = (J[0][0] * J[2][2] - J[0][2] * J[2][0]) * id;
            Ji[2][1] = (J[0][1] * J[2][0] - J[0][0] * J[2][1]) * id;
            Ji[0][2] = (J[0][1] * J[1][2] - J[0][2] * J[1][1]) * id;
            Ji[1][2] = (J[0][2] * J[1][0] - J[0][0] * J[1][2]) * id;
            Ji[2][2] = (J[0][0] * J[1][1] - J[0][1] * J[1][0]) * id;
            for (int a = 0; a < 8; ++a)
                for (int j = 0; j < 3; ++j)
                    g[ch][gp][a][j] = dn[a][0] * Ji[0][j] + dn[a][1] * Ji[1][j] + dn[a][2] * Ji[2][j];
            wdet[ch][gp] = det;
        }
        __syncthreads();
        if (t < nch * 64) {  // node-pair block (a, b) of child ch
            const int ch = t >> 6, a = (t >> 3) & 7, b = t & 7;
            const double Ee = E[fe[ch]], ne = nu[fe[ch]];
            const float lam = (float)(Ee * ne / ((1.0 + ne) * (1.0 - 2.0 * ne)));
            const float mu = (float)(Ee / (2.0 * (1.0 + ne)));
            float S[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
            for (int gp = 0; gp < 8; ++gp)
                for (int i = 0; i < 3; ++i)
                    for (int j = 0; j < 3; ++j) S[i][j] += wdet[ch][gp] * g[ch][gp][a][i] * g[ch][gp][b][j];
            const float tr = mu * (S[0][0] + S[1][1] + S[2][2]);
            for (int i = 0; i < 3; ++i)
                for (int j = 0; j < 3; ++j)
                    Ke[ch][(3 * a + i) * kTLd + 3 * b + j] = lam * S[i][j] + mu * S[j][i] + ((i == j) ? tr : 0.f);
        }
    }
    __syncthreads();
    // T_ch = K_ch (Q_ch x I3): this thread's entries (row, 3 a2 + c2) of child ch
    const int ch = t / 72, row = t % 72 / 3, c2 = t % 3;
    float kv[8];
    if (ch < nch) {
        if (cls_ke) {  // K_e = E_e * (unit-modulus matrix of the element's geometry class)
            const float Ee = (float)E[fe[ch]];
            const float* src = cls_ke + (size_t)cls_of[fe[ch]] * 576 + row * 24 + c2;
#pragma unroll
            for (int a2 = 0; a2 < 8; ++a2) kv[a2] = Ee * src[3 * a2];
        } else if (fine_ke) {
            const float* src = fine_ke + (size_t)fe[ch] * 576 + row * 24 + c2;
#pragma unroll
            for (int a2 = 0; a2 < 8; ++a2) kv[a2] = src[3 * a2];
        } else {
#pragma unroll
            for (int a2 = 0; a2 < 8; ++a2) kv[a2] = Ke[ch][row * kTLd + 3 * a2 + c2];
        }
    }
    __syncthreads();  // K_e is read
    if (ch < nch) {
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int a2 = 0; a2 < 8; ++a2) {
            const float4 q0 = *reinterpret_cast<const float4*>(Q[ch][a2]);
            const float4 q1 = *reinterpret_cast<const float4*>(Q[ch][a2] + 4);
            const float qv[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
            for (int b = 0; b < 8; ++b) acc[b] = fmaf(kv[a2], qv[b], acc[b]);
        }
#pragma unroll
        for (int b = 0; b < 8; ++b) Ke[ch][row * kTLd + 3 * b + c2] = acc[b];
    }
    __syncthreads();
    // K_C = sum_ch (Q_ch x I3)^T T_ch: rows 3 b + c1, b = b0 .. b0 + 3, of column col
    if (t >= 144) return;
    const int b0 = t / 72 * 4, c1 = t % 72 / 24, col = t % 24;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int h = 0; h < nch; ++h)
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const float4 qv = *reinterpret_cast<const float4*>(Q[h][a] + b0);
            const float tv = Ke[h][(3 * a + c1) * kTLd + col];
            acc[0] = fmaf(qv.x, tv, acc[0]);
            acc[1] = fmaf(qv.y, tv, acc[1]);
            acc[2] = fmaf(qv.z, tv, acc[2]);
            acc[3] = fmaf(qv.w, tv, acc[3]);
        }
#pragma unroll
    for (int b = 0; b < 4; ++b) coarse_ke[(size_t)C * 576 + (3 * (b0 + b) + c1) * 24 + col] = acc[b];
}

// First coarsening of a level-0 block made of geometry classes: with
// K_e = E_e K^_cls, the coarse matrix K_C = sum_ch E_ch (Q_ch x I3)^T K^ (Q_ch x I3)
// is linear in the children's moduli, and the projected class matrix depends
// only on the child's place in its coarse element.  Per axis a child is one
// of three cases (coarse cell of width 1; width 2, first or second half), so
// 27 projected matrices per class, built once per hierarchy in FP64 from the
// FP64 class matrices (CTA = (case, class)).
__global__ void __launch_bounds__(256) k_child_mats(const double* __restrict__ cls_ke, float* __restrict__ out) {
    __shared__ double K[576];
    __shared__ double T[576];
    __shared__ double Q[8][8];
    const int tc = blockIdx.x, cls = blockIdx.y, t = threadIdx.x;
    int w[3], o[3];
    for (int ax = 0, v = tc; ax < 3; ++ax, v /= 3) {
        const int s = v % 3;
        w[ax] = s == 0 ? 1 : 2;
        o[ax] = s == 2 ? 1 : 0;
    }
    for (int q = t; q < 576; q += blockDim.x) K[q] = cls_ke[(size_t)cls * 576 + q];
    if (t < 64) {
        const int a = t >> 3, b = t & 7;
        double q = 1.0;
        for (int ax = 0; ax < 3; ++ax) {
            const double xi = (double)(o[ax] + c_corner[a][ax]) / w[ax];
            q *= c_corner[b][ax] ? xi : 1.0 - xi;
        }
        Q[a][b] = q;
    }
    __syncthreads();
    for (int q = t; q < 576; q += blockDim.x) {  // T = K (Q x I3)
        const int row = q / 24, col = q % 24, b = col / 3, c2 = col % 3;
        double acc = 0.0;
        for (int a = 0; a < 8; ++a) acc += K[row * 24 + 3 * a + c2] * Q[a][b];
        T[q] = acc;
    }
    __syncthreads();
    for (int q = t; q < 576; q += blockDim.x) {  // (Q x I3)^T T
        const int row = q / 24, col = q % 24, b = row / 3, c1 = row % 3;
        double acc = 0.0;
        for (int a = 0; a < 8; ++a) acc += Q[a][b] * T[(3 * a + c1) * 24 + col];
        out[((size_t)cls * 27 + tc) * 576 + q] = (float)acc;
    }
}

// K_C = sum_ch E_ch B[cls_ch][case_ch]: one CTA of 144 threads per coarse
// element, four consecutive entries per thread.
__global__ void __launch_bounds__(144) k_coarsen_lin(LevelView cv, const int32_t* __restrict__ pre_el,
                                                     const double* __restrict__ E, const int32_t* __restrict__ cls_of,
                                                     const float* __restrict__ child, float* __restrict__ coarse_ke) {
    __shared__ float ew[8];
    __shared__ int bi[8];
    __shared__ int nch_s;
    const int t = threadIdx.x, C = blockIdx.x;
    if (t < 8) {
        const BlkDev& d = cv.blk[find_blk(pre_el, cv.n_blk, C)];
        const int Cl = C - d.el0;
        const int ci = Cl / (d.ny * d.nz), cj = (Cl / d.nz) % d.ny, ck = Cl % d.nz;
        const int s0 = cv.xs[d.ox0 + ci], w0 = cv.xs[d.ox0 + ci + 1] - s0;
        const int s1 = cv.xs[d.ox1 + cj], w1 = cv.xs[d.ox1 + cj + 1] - s1;
        const int s2 = cv.xs[d.ox2 + ck], w2 = cv.xs[d.ox2 + ck + 1] - s2;
        const int nch = w0 * w1 * w2;
        if (t == 0) nch_s = nch;
        if (t < nch) {
            const int o0 = t / (w1 * w2), o1 = (t / w2) % w1, o2 = t % w2;
            const int e = d.fel0 + ((s0 + o0) * d.fny + (s1 + o1)) * d.fnz + (s2 + o2);
            const int tc = (w0 == 1 ? 0 : 1 + o0) + 3 * (w1 == 1 ? 0 : 1 + o1) + 9 * (w2 == 1 ? 0 : 1 + o2);
            ew[t] = (float)E[e];
            bi[t] = cls_of[e] * 27 + tc;
        }
    }
    __syncthreads();
    const int nch = nch_s;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int ch = 0; ch < nch; ++ch) {
        const float4 b = reinterpret_cast<const float4*>(child + (size_t)bi[ch] * 576)[t];
        const float e = ew[ch];
        acc.x = fmaf(e, b.x, acc.x);
        acc.y = fmaf(e, b.y, acc.y);
        acc.z = fmaf(e, b.z, acc.z);
        acc.w = fmaf(e, b.w, acc.w);
    }
    reinterpret_cast<float4*>(coarse_ke + (size_t)C * 576)[t] = acc;
}

// binv := omega m^-1 (cofactors in FP64)
__device__ __forceinline__ void smoother_block(const double (&m)[9], float omega, float* B) {
    const double c00 = m[4] * m[8] - m[5] * m[7], c01 = m[5] * m[6] - m[3] * m[8], c02 = m[3] * m[7] - m[4] * m[6];
    const double id = omega / (m[0] * c00 + m[1] * c01 + m[2] * c02);
    B[0] = (float)(c00 * id);
    B[1] = (float)((m[2] * m[7] - m[1] * m[8]) * id);
    B[2] = (float)((m[1] * m[5] - m[2] * m[4]) * id);
    B[3] = (float)(c01 * id);
    B[4] = (float)((m[0] * m[8] - m[2] * m[6]) * id);
    B[5] = (float)((m[2] * m[3] - m[0] * m[5]) * id);
    B[6] = (float)(c02 * id);
    B[7] = (float)((m[1] * m[6] - m[0] * m[7]) * id);
    B[8] = (float)((m[0] * m[4] - m[1] * m[3]) * id);
}

// lo: a split-only assembly whose FP64 diagonal blocks were asked for (nullptr:
// the values as they are)
template <typename TV>
__global__ void k_smoother_blocks(int n_rows, const int64_t* __restrict__ slice_off, const uint8_t* __restrict__ diag,
                                  const TV* __restrict__ vals, const float* __restrict__ lo, float* __restrict__ binv) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= n_rows) return;
    const int64_t g = slice_off[row >> 5] + diag[row];
    const int lane = row & 31;
    double m[9];
#pragma unroll
    for (int q = 0; q < 9; ++q)
        m[q] = (double)vals[(g * 9 + q) * 32 + lane] + (lo ? (double)lo[(g * 9 + q) * 32 + lane] : 0.0);
    smoother_block(m, 1.f, binv + 9 * (size_t)row);
}

// A coarse level's values from its element matrices, one CTA per slice of 32
// rows: every row sums its <= 8 elements' three matrix rows (72 consecutive
// floats each, one warp a row, all of a row's loads in flight) in shared memory
// in the order of the elements' parities, adds the lumped penalty (scaled by
// the block's penalty scale), and the slice is written once, with its smoother
// blocks D^-1 and the bound ||D^-1 A||_inf >= lambda_max (float bits under
// atomicMax).  Each element matrix is read once and each value written once, so
// the kernel is bound by those bytes; eight coloured scatters, the clearing, the
// penalty, the blocks and the bound as kernels of their own took 1.4 ms over the levels of
// 128 x 64 x 64 elements, this one 245 us.
constexpr int kValThreads = 256;
constexpr int kValLd = 33;
constexpr size_t kValSmem = sizeof(float) * (27 * 9 * kValLd + 9 * kValLd);

__global__ void __launch_bounds__(kValThreads)
k_level_values(int n_rows, const BlkDev* __restrict__ blk, const int32_t* __restrict__ row_blk, BlkDev one,
               const float* __restrict__ ke, const float* __restrict__ pen, const double* __restrict__ blk_sf,
               float* __restrict__ vals, float* __restrict__ binv, unsigned int* __restrict__ bound_bits) {
    extern __shared__ __align__(16) float vsm[];
    float* Bs = vsm + 27 * 9 * kValLd;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int q = threadIdx.x; q < 27 * 9 * kValLd; q += kValThreads) vsm[q] = 0.f;
    __syncthreads();
    // this lane's entries of an element's three rows: (i, column corner b, j)
    int vo[3], co[3][3];
#pragma unroll
    for (int w = 0; w < 3; ++w) {
        const int s = min(lane + 32 * w, 71), b = s % 24 / 3;
        vo[w] = s / 24 * 3 + s % 3;
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) co[w][ax] = c_corner[b][ax];
    }
    for (int q = warp; q < 32; q += kValThreads / 32) {
        const int row = blockIdx.x * 32 + q;
        if (row >= n_rows) break;
        const int b = row_blk ? row_blk[row] : 0;
        const BlkDev d = row_blk ? blk[b] : one;
        const int l = row - d.node0, sj = d.nz + 1, si = (d.ny + 1) * sj;
        if (l >= (d.nx + 1) * si) continue;  // padding node between instances
        const int i = l / si, j = (l - i * si) / sj, k = l - i * si - j * sj;
        const int i0 = max(i - 1, 0), j0 = max(j - 1, 0), k0 = max(k - 1, 0);
        const int nj = min(j + 1, d.ny) - j0 + 1, nk = min(k + 1, d.nz) - k0 + 1;
        float v[8][3];
#pragma unroll
        for (int c = 0; c < 8; ++c) {  // the adjacent element of parity c
            const int ei = ((i & 1) == (c >> 2)) ? i : i - 1, ej = ((j & 1) == ((c >> 1) & 1)) ? j : j - 1,
                      ek = ((k & 1) == (c & 1)) ? k : k - 1;
            const bool in = ei >= 0 && ej >= 0 && ek >= 0 && ei < d.nx && ej < d.ny && ek < d.nz;
            const int di = i - ei, dj = j - ej, a = 4 * (k - ek) + (dj ? 3 - di : di);
            const float* K = ke + ((size_t)d.el0 + (ei * d.ny + ej) * d.nz + ek) * 576 + 72 * a;
#pragma unroll
            for (int w = 0; w < 3; ++w) v[c][w] = in && lane + 32 * w < 72 ? __ldcs(K + lane + 32 * w) : 0.f;
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int ei = ((i & 1) == (c >> 2)) ? i : i - 1, ej = ((j & 1) == ((c >> 1) & 1)) ? j : j - 1,
                      ek = ((k & 1) == (c & 1)) ? k : k - 1;
            if (ei >= 0 && ej >= 0 && ek >= 0 && ei < d.nx && ej < d.ny && ek < d.nz) {  // uniform over the warp
#pragma unroll
                for (int w = 0; w < 3; ++w)
                    if (lane + 32 * w < 72) {
                        const int at = ((ei + co[w][0] - i0) * nj + (ej + co[w][1] - j0)) * nk + (ek + co[w][2] - k0);
                        vsm[(at * 9 + vo[w]) * kValLd + q] += v[c][w];
                    }
            }
            __syncwarp();
        }
        if (lane < 3) {
            const int at = ((i - i0) * nj + (j - j0)) * nk + (k - k0);
            const float sf = (float)blk_sf[b];
            vsm[(at * 9 + 4 * lane) * kValLd + q] += sf * pen[3 * row + lane];
        }
        __syncwarp();
        if (lane < 9) {  // the diagonal block, for the smoother
            const int at = ((i - i0) * nj + (j - j0)) * nk + (k - k0);
            Bs[lane * kValLd + q] = vsm[(at * 9 + lane) * kValLd + q];
        }
    }
    __syncthreads();
    const int row = blockIdx.x * 32 + lane;
    float* out = vals + (size_t)blockIdx.x * (27 * 9 * 32);
    for (int x = warp; x < 27 * 9; x += kValThreads / 32) out[(size_t)x * 32 + lane] = vsm[x * kValLd + lane];
    bool real = row < n_rows;
    if (real) {
        const BlkDev d = row_blk ? blk[row_blk[row]] : one;
        real = row - d.node0 < (d.nx + 1) * (d.ny + 1) * (d.nz + 1);
    }
    if (warp == 0 && row < n_rows) {
        double m[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) m[q] = real ? (double)Bs[q * kValLd + lane] : 0.0;
        float B[9];
        smoother_block(m, 1.f, B);
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            Bs[q * kValLd + lane] = B[q];
            binv[9 * (size_t)row + q] = B[q];
        }
    }
    if (!bound_bits) return;
    __syncthreads();
    if (warp >= 3) return;
    float sum = 0.f;  // component `warp` of the row's sum
    if (real) {
        float B[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) B[q] = Bs[(3 * warp + q) * kValLd + lane];
#pragma unroll 3
        for (int j = 0; j < 27; ++j) {
            const float* m = vsm + j * 9 * kValLd + lane;
#pragma unroll
            for (int b = 0; b < 3; ++b)
                sum += fabsf(B[0] * m[b * kValLd] + B[1] * m[(3 + b) * kValLd] + B[2] * m[(6 + b) * kValLd]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum = fmaxf(sum, __shfl_xor_sync(0xffffffffu, sum, o));
    if (lane == 0 && sum > 0.f) atomicMax(bound_bits, __float_as_uint(sum));
}

// Coarsest level: one dense matrix per block (n_b = 3 x the block's nodes,
// at offset dense0), filled row by row (one CTA per node row), then inverted
// in place by Gauss-Jordan (SPD, no pivoting), one cluster per block.
__global__ void k_dense_build(int n_rows, const int64_t* __restrict__ slice_off, const uint8_t* __restrict__ row_len,
                              const int32_t* __restrict__ col, const float* __restrict__ vals, LevelView cv,
                              const int32_t* __restrict__ pre_node, float* __restrict__ D) {
    const int row = blockIdx.x;
    const BlkDev& d = cv.blk[find_blk(pre_node, cv.n_blk, row)];
    const int n = 3 * (d.nx + 1) * (d.ny + 1) * (d.nz + 1);
    const int lr = row - d.node0;
    if (lr >= n / 3) return;  // padding node between instances
    float* Db = D + d.dense0;
    for (int q = threadIdx.x; q < 3 * n; q += blockDim.x) Db[(size_t)(3 * lr) * n + q] = 0.f;
    __syncthreads();
    const int lane = row & 31, len = row_len[row];
    const int64_t g0 = slice_off[row >> 5];
    for (int q = threadIdx.x; q < len * 9; q += blockDim.x) {
        const int j = q / 9, v = q % 9, a = v / 3, c = v % 3;
        const int64_t g = g0 + j;
        const int cn = col[g * 32 + lane] - d.node0;
        Db[(size_t)(3 * lr + a) * n + 3 * cn + c] = vals[(g * 9 + v) * 32 + lane];
    }
}

// Coarsest inverse: in-place Gauss-Jordan of one block's matrix (n <= 256, which
// the coarsening rule guarantees) by a cluster of 8 CTAs, CTA r holding rows
// 32 r .. 32 r + 31 in registers (warp w rows 4 w .. 4 w + 3, lane columns lane +
// 32 j).  For panel P (rows / columns k0 .. k0 + 31) its owner forms the 32 rows
// R that eliminate it and writes them to the panel's rows of the matrix in
// global memory (L2: 8 readers of one SM's shared memory took three times as
// long); after a cluster barrier the others read them and apply A_i = A_i - A_iP R
// with the panel columns of A_i cleared first.  No pivoting: the coarse
// operators are SPD.  Up to 234 DOF R = D A_P with D = A_PP^-1 (the elimination
// regrouped by panels), above it the owner eliminates column by column and the
// others follow its steps, each size keeping the rounding of its V-cycles.
// Bound by the serial panels, 32 pivots of one CTA barrier each; rows in
// registers and one pass over memory a panel instead of shared memory with
// 8-way conflicts: n = 216 170 -> 99 us, n = 243 636 -> 126 us.
constexpr int kGjCtas = 8, kGjN = 256, kGjThreads = 256, kGjBlocked = 234;
constexpr int kGjLd = 33;  // transposed copy: 256 columns of 32 rows
constexpr size_t kGjSmem = sizeof(float) * (32 * kGjN + kGjN * kGjLd);

__global__ void __cluster_dims__(kGjCtas, 1, 1) __launch_bounds__(kGjThreads)
k_gauss_jordan(LevelView cv, float* Dall) {
    extern __shared__ __align__(16) float gj[];
    float* R = gj;               // the panel's eliminating rows [32][256]
    float* S = gj + 32 * kGjN;   // the owner's rows / the transposed copy
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int r = (int)cl.block_rank(), t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const BlkDev& dv = cv.blk[blockIdx.x / kGjCtas];
    const int n = 3 * (dv.nx + 1) * (dv.ny + 1) * (dv.nz + 1);
    const bool blocked = n <= kGjBlocked;
    float* Ag = Dall + dv.dense0;
    const int row0 = 32 * r + 4 * warp;
    float a[4][8];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int i = row0 + u, q = lane + 32 * j;
            a[u][j] = (i < n && q < n) ? Ag[(size_t)i * n + q] : 0.f;
        }
    cl.sync();  // loaded: the panels' rows in global memory may be written
    for (int P = 0; 32 * P < n; ++P) {
        const int k0 = 32 * P, kb = min(32, n - k0);
        float pc[4];  // the panel's columns of the own rows
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            pc[u] = 0.f;
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (j == P) pc[u] = a[u][j];
        }
        if (r == P) {
            if (blocked) {
                // A_PP (its padding the identity) inverted in pc; rows exchanged
                // through R
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (4 * warp + u >= kb || lane >= kb) pc[u] = 4 * warp + u == lane ? 1.f : 0.f;
            }
            for (int w = 0; 4 * w < kb; ++w) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int p = 4 * w + u;
                    if (p >= kb) break;
                    float* row = R + p * kGjN;
                    if (warp == w) {
                        const float inv = 1.f / __shfl_sync(0xffffffffu, pc[u], p);
                        const float pm = lane == p ? inv : pc[u] * inv;
                        if (!blocked) {
#pragma unroll
                            for (int j = 0; j < 8; ++j) row[lane + 32 * j] = j == P ? pm : a[u][j] * inv;
                        } else {
                            row[lane] = pm;
                        }
                    }
                    __syncthreads();
                    const float pm = row[blocked ? lane : k0 + lane];
                    float ci[4];
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        ci[v] = __shfl_sync(0xffffffffu, pc[v], p);
                        pc[v] = fmaf(-ci[v], pm, lane == p ? 0.f : pc[v]);
                        if (v == u && warp == w) pc[v] = pm;
                    }
                    if (!blocked) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float m = row[lane + 32 * j];
#pragma unroll
                            for (int v = 0; v < 4; ++v)
                                a[v][j] = (v == u && warp == w) ? m : fmaf(-ci[v], m, a[v][j]);
                        }
                    }
                }
            }
            if (blocked) {  // R = D A_P, R_PP = D
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int j = 0; j < 8; ++j) S[(4 * warp + u) * kGjN + lane + 32 * j] = a[u][j], a[u][j] = 0.f;
                __syncthreads();
#pragma unroll 4
                for (int q = 0; q < 32; ++q) {
                    float d[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) d[u] = __shfl_sync(0xffffffffu, pc[u], q);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float m = S[q * kGjN + lane + 32 * j];
#pragma unroll
                        for (int u = 0; u < 4; ++u) a[u][j] = fmaf(d[u], m, a[u][j]);
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (j == P) a[u][j] = pc[u];
                    const int i = row0 + u, q = lane + 32 * j;
                    // unblocked: the rows as they eliminated, not as they ended
                    if (i < n && q < n) Ag[(size_t)i * n + q] = blocked ? a[u][j] : R[(4 * warp + u) * kGjN + q];
                }
        }
        cl.sync();  // R is in global memory
        if (r == P) continue;
        if (t < n) {
#pragma unroll 16
            for (int q = 0; q < 32; ++q) R[q * kGjN + t] = q < kb ? __ldcg(Ag + (size_t)(k0 + q) * n + t) : 0.f;
        } else {
#pragma unroll 16
            for (int q = 0; q < 32; ++q) R[q * kGjN + t] = 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (j == P) a[u][j] = 0.f;
#pragma unroll 4
        for (int q = 0; q < 32; ++q) {
            if (!blocked && q >= kb) break;
            float ci[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) ci[u] = __shfl_sync(0xffffffffu, pc[u], q);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float m = R[q * kGjN + lane + 32 * j];
#pragma unroll
                for (int u = 0; u < 4; ++u) a[u][j] = fmaf(-ci[u], m, a[u][j]);
            }
            if (!blocked) {
                const float m = R[q * kGjN + k0 + lane];
#pragma unroll
                for (int u = 0; u < 4; ++u) pc[u] = fmaf(-ci[u], m, lane == q ? 0.f : pc[u]);
            }
        }
        if (!blocked) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (j == P) a[u][j] = pc[u];
        }
        __syncthreads();  // R is read
    }
    // the exact inverse is symmetric: average the FP32 rounding asymmetry out,
    // so the coarse solve (and with it the V-cycle) is a symmetric operator
    cl.sync();  // every panel's rows are read
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int i = row0 + u, q = lane + 32 * j;
            if (i < n && q < n) Ag[(size_t)i * n + q] = a[u][j];
        }
    cl.sync();
    if (32 * r + lane < n) {
#pragma unroll 16
        for (int q = warp; q < n; q += 8) S[q * kGjLd + lane] = __ldcg(Ag + (size_t)q * n + 32 * r + lane);
    }
    cl.sync();  // the transposed columns are read
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int i = row0 + u, q = lane + 32 * j;
            if (i < n && q < n) Ag[(size_t)i * n + q] = 0.5f * (a[u][j] + S[q * kGjLd + 4 * warp + u]);
        }
}

// ---------------------------------------------------------------------------
// V-cycle kernels (all FP32; x4/y4 node-padded float4)
// ---------------------------------------------------------------------------
struct SbView {
    int n_rows;
    const int64_t* slice_off;
    const uint8_t* row_len;
    const int32_t* col;
    const float* v;
};

// The V-cycle runs for several right-hand sides at once: blockIdx.y picks one,
// whose level vectors follow each other.  A right-hand side none of whose
// instances iterates any more is left alone.
__device__ __forceinline__ bool vc_idle(const Control* ctl) { return ctl && ctl->active[blockIdx.y] == 0; }
template <typename T>
__device__ __forceinline__ T* rhs_of(T* v, size_t n) {
    return v + blockIdx.y * n;
}

// Row product with three block columns in flight per step: the column
// indices, 27 values and three gathers of a step are independent loads, so
// their latencies overlap instead of forming one 27-long dependent chain.
__device__ __forceinline__ void sb_row(const SbView& A, int row, const float4* __restrict__ x, float (&y)[3]) {
    y[0] = y[1] = y[2] = 0.f;
    const int lane = row & 31;
    const int64_t g0 = A.slice_off[row >> 5];
    const int len = A.row_len[row];
    int j = 0;
    for (; j + 3 <= len; j += 3) {
        const int64_t g = g0 + j;
        int c[3];
        float m[3][9];
#pragma unroll
        for (int u = 0; u < 3; ++u) c[u] = A.col[(g + u) * 32 + lane];
#pragma unroll
        for (int u = 0; u < 3; ++u)
#pragma unroll
            for (int q = 0; q < 9; ++q) m[u][q] = A.v[((g + u) * 9 + q) * 32 + lane];
        float4 p[3];
#pragma unroll
        for (int u = 0; u < 3; ++u) p[u] = x[c[u]];
#pragma unroll
        for (int u = 0; u < 3; ++u)
#pragma unroll
            for (int a = 0; a < 3; ++a)
                y[a] = fmaf(m[u][a * 3], p[u].x, fmaf(m[u][a * 3 + 1], p[u].y, fmaf(m[u][a * 3 + 2], p[u].z, y[a])));
    }
    for (; j < len; ++j) {
        const int64_t g = g0 + j;
        const int c = A.col[g * 32 + lane];
        const float* v = A.v + (g * 9) * 32 + lane;
        const float4 p = x[c];
#pragma unroll
        for (int a = 0; a < 3; ++a)
            y[a] = fmaf(v[(a * 3) * 32], p.x, fmaf(v[(a * 3 + 1) * 32], p.y, fmaf(v[(a * 3 + 2) * 32], p.z, y[a])));
    }
}

// The share of row `row`'s product held by lane t of its T lanes (block
// columns t, t + T, ...); the T lanes of a row are consecutive threads of one
// warp and are summed by xor shuffles, which every lane of the warp executes.
template <int T>
__device__ __forceinline__ void sb_row_part(const SbView& A, int row, int t, const float4* __restrict__ x,
                                            float (&y)[3]) {
    y[0] = y[1] = y[2] = 0.f;
    const int lane = row & 31;
    const int64_t g0 = A.slice_off[row >> 5];
    const int len = A.row_len[row];
    for (int j = t; j < len; j += T) {
        const int64_t g = g0 + j;
        const int c = A.col[g * 32 + lane];
        const float* v = A.v + (g * 9) * 32 + lane;
        float m[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) m[q] = v[q * 32];
        const float4 p = x[c];
#pragma unroll
        for (int a = 0; a < 3; ++a) y[a] = fmaf(m[a * 3], p.x, fmaf(m[a * 3 + 1], p.y, fmaf(m[a * 3 + 2], p.z, y[a])));
    }
}

template <int T>
__device__ __forceinline__ void sum_lanes(float (&y)[3]) {
#pragma unroll
    for (int o = T / 2; o >= 1; o >>= 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) y[a] += __shfl_xor_sync(0xffffffffu, y[a], o);
}

__global__ void k_vc_smooth0(int n, const float* __restrict__ binv, const float* b, float4* x,
                             const Control* ctl) {
    pdl_begin();
    if (vc_idle(ctl)) return;
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= n) return;
    b = rhs_of(b, 3 * (size_t)n);
    x = rhs_of(x, n);
    const float* B = binv + 9 * (size_t)row;
    const float b0 = b[3 * row], b1 = b[3 * row + 1], b2 = b[3 * row + 2];
    x[row] = make_float4(B[0] * b0 + B[1] * b1 + B[2] * b2, B[3] * b0 + B[4] * b1 + B[5] * b2,
                         B[6] * b0 + B[7] * b1 + B[8] * b2, 0.f);
}

__global__ void __launch_bounds__(kT) k_vc_resid(SbView A, const float* __restrict__ b, const float4* __restrict__ x,
                                                 float* __restrict__ r, const Control* ctl) {
    pdl_begin();
    if (vc_idle(ctl)) return;
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= A.n_rows) return;
    float y[3];
    sb_row(A, row, x, y);
#pragma unroll
    for (int a = 0; a < 3; ++a) r[3 * row + a] = b[3 * row + a] - y[a];
}

// ---------------------------------------------------------------------------
// Staged FP32 level products (the finest level's residual and post-smoothing
// sweep).  As the split outer product: warp w of CTA b owns the slices
// b * W + w + j * gridDim.x * W, and the slices' FP32 values and column
// indices stream through a per-warp ring of shared-memory stages filled by
// cp.async.bulk and completed on mbarriers; the gathered x stays a plain
// load.  Per row the products are summed in the order of sb_row.
// ---------------------------------------------------------------------------
template <int G, int S>
struct F32Stage {
    static constexpr int kVal = 9 * 32;                      // floats per group
    static constexpr int kStage = G * (kVal * 4 + 32 * 4);   // bytes per stage
    static constexpr int kWarp = S * kStage;
    static constexpr int kBar = 128;
    static constexpr int smem(int threads) { return kBar + (threads / 32) * kWarp; }
    static_assert((kT / 32) * S <= kBar / 8, "one mbarrier per warp and stage must fit the barrier area");
    static_assert(kStage % 16 == 0 && (G * kVal * 4) % 16 == 0, "bulk copies need 16-byte aligned stages");
};
constexpr int kVcG = 4, kVcS = 2;  // stage shape of the finest level's products

// y_k = A x_k for the right-hand sides k of the mask `on` (NR at most), whose
// vectors are n_rows apart: a slice's values are staged once for all of them.
template <int G, int S, int NR, typename Epi>
__device__ __forceinline__ bool f32_staged_slices(const SbView& A, const float4* x, unsigned on, unsigned char* smem,
                                                  Epi&& epi) {
    using St = F32Stage<G, S>;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wpc = blockDim.x >> 5;
    const int n_sl = (A.n_rows + 31) >> 5;
    const int sl0 = blockIdx.x * wpc + warp, sl_step = gridDim.x * wpc;
    if (sl0 >= n_sl) return true;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem) + warp * S;
    unsigned char* ring = smem + St::kBar + warp * St::kWarp;
    int psl = sl0, pk = 0, issued = 0;
    int64_t pg0 = 0;
    int png = 0;
    auto load_slice = [&](int sl) {
        pg0 = A.slice_off[sl];
        png = (int)(A.slice_off[sl + 1] - pg0);
    };
    auto issue_next = [&]() {  // lane 0
        if (psl >= n_sl) return;
        const int s = issued % S;
        const int cnt = min(G, png - pk * G);
        const int64_t gk = pg0 + (int64_t)pk * G;
        unsigned char* st = ring + s * St::kStage;
        mbar_expect_tx(bars + s, (uint32_t)cnt * (St::kVal * 4 + 32 * 4));
        bulk_g2s(st, A.v + gk * St::kVal, cnt * St::kVal * 4, bars + s);
        bulk_g2s(st + G * St::kVal * 4, A.col + gk * 32, cnt * 32 * 4, bars + s);
        ++issued;
        if (++pk * G >= png) {
            pk = 0;
            psl += sl_step;
            if (psl < n_sl) load_slice(psl);
        }
    };
    if (lane == 0) {
#pragma unroll
        for (int s = 0; s < S; ++s) mbar_init(bars + s, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_shared();
        load_slice(psl);
        for (int s = 0; s < S; ++s) issue_next();
    }
    __syncwarp();
    int used = 0;
    bool ok = true;
    for (int sl = sl0; sl < n_sl && ok; sl += sl_step) {
        const int row = sl * 32 + lane;
        const int64_t g0 = A.slice_off[sl];
        const int ng = (int)(A.slice_off[sl + 1] - g0);
        const int len = row < A.n_rows ? A.row_len[row] : 0;
        const int nst = (ng + G - 1) / G;
        float y[NR][3];
#pragma unroll
        for (int k = 0; k < NR; ++k) y[k][0] = y[k][1] = y[k][2] = 0.f;
        for (int k = 0; k < nst; ++k) {
            const int s = used % S;
            if (!__all_sync(0xffffffffu, mbar_wait(bars + s, (uint32_t)((used / S) & 1)))) {
                ok = false;
                break;
            }
            const float* hv = reinterpret_cast<const float*>(ring + s * St::kStage);
            const int* cv = reinterpret_cast<const int*>(hv + G * St::kVal);
            const int cnt = min(G, ng - k * G);
            float4 p[G][NR];
#pragma unroll
            for (int u = 0; u < G; ++u)
                if (u < cnt && k * G + u < len) {
                    const float4* xc = x + cv[u * 32 + lane];
#pragma unroll
                    for (int h = 0; h < NR; ++h)
                        if (NR == 1 || (on >> h & 1)) p[u][h] = xc[(size_t)h * A.n_rows];
                }
#pragma unroll
            for (int u = 0; u < G; ++u) {
                if (u < cnt && k * G + u < len) {
                    const float* m = hv + u * St::kVal + lane;
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        const float m0 = m[(a * 3) * 32], m1 = m[(a * 3 + 1) * 32], m2 = m[(a * 3 + 2) * 32];
#pragma unroll
                        for (int h = 0; h < NR; ++h)
                            if (NR == 1 || (on >> h & 1))
                                y[h][a] = fmaf(m0, p[u][h].x, fmaf(m1, p[u][h].y, fmaf(m2, p[u][h].z, y[h][a])));
                    }
                }
            }
            ++used;
            __syncwarp();
            if (lane == 0) {
                fence_async_shared();
                issue_next();
            }
        }
        if (!ok) break;
        if (row < A.n_rows)
#pragma unroll
            for (int h = 0; h < NR; ++h)
                if (NR == 1 || (on >> h & 1)) epi(row, h, y[h]);
    }
    if (!ok) {
        const int upto = __shfl_sync(0xffffffffu, issued, 0);
        if (lane == 0)
            for (int q = used; q < upto; ++q) mbar_wait(bars + q % S, (uint32_t)((q / S) & 1));
        __syncwarp();
        // poison this warp's first row: the V-cycle output turns non-finite
        // and the solve reports it
        const int row = sl0 * 32 + lane;
        const float nan[3] = {__int_as_float(0x7fc00000), 0.f, 0.f};
        for (int h = 0; row < A.n_rows && h < NR; ++h)
            if (NR == 1 || (on >> h & 1)) epi(row, h, nan);
    }
    return ok;
}

// right-hand sides with an instance that still iterates, of nr (NR == 1: this one's)
template <int NR>
__device__ __forceinline__ unsigned vc_on(const Control* ctl, int nr) {
    if constexpr (NR == 1) return !vc_idle(ctl);
    unsigned on = 0;
    for (int k = 0; k < nr; ++k) on |= (!ctl || ctl->active[k] != 0) << k;
    return on;
}

// r = b - A x over the level's rows (staged)
template <int NR>
__global__ void __launch_bounds__(kT) k_vc_resid_staged(SbView A, const float* b, const float4* x, float* r,
                                                        const Control* ctl, int nr) {
    pdl_begin();
    const unsigned on = vc_on<NR>(ctl, nr);
    if (!on) return;
    if constexpr (NR == 1) {
        b = rhs_of(b, 3 * (size_t)A.n_rows);
        x = rhs_of(x, A.n_rows);
        r = rhs_of(r, 3 * (size_t)A.n_rows);
    }
    extern __shared__ __align__(128) unsigned char vc_smem[];
    f32_staged_slices<kVcG, kVcS, NR>(A, x, on, vc_smem, [&](int row, int h, const float (&y)[3]) {
        const size_t at = 3 * ((size_t)h * A.n_rows + row);
#pragma unroll
        for (int a = 0; a < 3; ++a) r[at + a] = b[at + a] - y[a];
    });
}

// y4 = x + B^-1 (b - A x) over the level's rows (staged)
template <int NR>
__global__ void __launch_bounds__(kT) k_vc_post_staged(SbView A, const float* __restrict__ binv, const float* b,
                                                       const float4* x, float4* y4, const Control* ctl, int nr) {
    pdl_begin();
    const unsigned on = vc_on<NR>(ctl, nr);
    if (!on) return;
    if constexpr (NR == 1) {
        b = rhs_of(b, 3 * (size_t)A.n_rows);
        x = rhs_of(x, A.n_rows);
        y4 = rhs_of(y4, A.n_rows);
    }
    extern __shared__ __align__(128) unsigned char vc_smem[];
    f32_staged_slices<kVcG, kVcS, NR>(A, x, on, vc_smem, [&](int row, int h, const float (&y)[3]) {
        const size_t at = (size_t)h * A.n_rows + row;
        const float d0 = b[3 * at] - y[0], d1 = b[3 * at + 1] - y[1], d2 = b[3 * at + 2] - y[2];
        const float* B = binv + 9 * (size_t)row;
        const float4 xv = x[at];
        y4[at] = make_float4(xv.x + B[0] * d0 + B[1] * d1 + B[2] * d2, xv.y + B[3] * d0 + B[4] * d1 + B[5] * d2,
                             xv.z + B[6] * d0 + B[7] * d1 + B[8] * d2, 0.f);
    });
}

// r = b - A x (POST = false) or y4 = x + B^-1 (b - A x) on any pattern, T lanes a
// row (a small finest level).
template <int T, bool POST>
__global__ void __launch_bounds__(kT) k_vc_rows_any(SbView A, const float* __restrict__ binv, const float* b,
                                                    const float4* x, float* r, float4* y4, const Control* ctl) {
    pdl_begin();
    if (vc_idle(ctl)) return;
    b = rhs_of(b, 3 * (size_t)A.n_rows);
    x = rhs_of(x, A.n_rows);
    const int gt = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = gt / T, t = gt % T;
    const bool ok = row < A.n_rows;
    float y[3] = {0.f, 0.f, 0.f};
    if (ok) sb_row_part<T>(A, row, t, x, y);
    sum_lanes<T>(y);
    if (!ok || t != 0) return;
    const float d0 = b[3 * row] - y[0], d1 = b[3 * row + 1] - y[1], d2 = b[3 * row + 2] - y[2];
    if constexpr (!POST) {
        r = rhs_of(r, 3 * (size_t)A.n_rows);
        r[3 * row] = d0, r[3 * row + 1] = d1, r[3 * row + 2] = d2;
    } else {
        const float* B = binv + 9 * (size_t)row;
        const float4 xv = x[row];
        rhs_of(y4, A.n_rows)[row] =
            make_float4(xv.x + B[0] * d0 + B[1] * d1 + B[2] * d2, xv.y + B[3] * d0 + B[4] * d1 + B[5] * d2,
                        xv.z + B[6] * d0 + B[7] * d1 + B[8] * d2, 0.f);
    }
}

// Coarse-level variants with T lanes per row: a coarse level has too few
// rows to fill the GPU with one thread each, and a row's 27 block columns
// then form a long chain of dependent loads; T lanes split the chain.  These
// kernels are a handful of L2 round trips long, so the level's structure is
// computed instead of loaded (the columns of a row are its neighbours in the
// block, in node order; coarse levels keep 27 column groups a slice): for one
// block its description comes with the launch, in a stack with one load through
// the row's block.  Values, gathers, right-hand side and smoother block are
// then one round trip (caches cold, 6,171 rows of 100 x 20 x 20: a product 6.5 ->
// 5.1 us, a restriction 5.0 -> 4.0 us, a prolongation 4.1 -> 3.7 us, the coarsest
// solve 8.8 -> 3.2 us).  The sums and their order are sb_row_part's.
struct GeoView {
    int n_rows;
    const BlkDev* blk;       // descriptors; row_blk == nullptr: one block, `one`
    const int32_t* row_blk;  // block of each row
    BlkDev one;
    const float* v;
};

__device__ __forceinline__ BlkDev blk_of(const GeoView& G, int row) {
    return G.row_blk ? G.blk[G.row_blk[row]] : G.one;
}

// The share of lane t of T in row `row`'s product: v(9 q + w) entry w of its q-th
// block, x(c) the entry of a column.
template <int T, typename V, typename X>
__device__ __forceinline__ void geo_row_part(const BlkDev& d, int row, int t, V&& v, X&& x, float (&y)[3]) {
    const int l = row - d.node0;
    const int sj = d.nz + 1, si = (d.ny + 1) * sj;
    const int i = l / si, j = (l - i * si) / sj, k = l - i * si - j * sj;
    const int i0 = max(i - 1, 0), j0 = max(j - 1, 0), k0 = max(k - 1, 0);
    const int nj = min(j + 1, d.ny) - j0 + 1, nk = min(k + 1, d.nz) - k0 + 1;
    const int len = (min(i + 1, d.nx) - i0 + 1) * nj * nk;
    const int first = d.node0 + i0 * si + j0 * sj + k0;
    constexpr int U = (27 + T - 1) / T;
    constexpr int STEP = U < 4 ? U : 4;  // columns in flight
    y[0] = y[1] = y[2] = 0.f;
#pragma unroll
    for (int u0 = 0; u0 < U; u0 += STEP) {
        float m[STEP][9];
        float4 p[STEP];
#pragma unroll
        for (int u = 0; u < STEP; ++u) {
            const int q = t + (u0 + u) * T;
            if (q < len) {
                const int qk = q / nk, c = first + (qk / nj) * si + (qk % nj) * sj + (q - qk * nk);
                p[u] = x(c);
#pragma unroll
                for (int w = 0; w < 9; ++w) m[u][w] = v(q * 9 + w);
            }
        }
#pragma unroll
        for (int u = 0; u < STEP; ++u) {
            const int q = t + (u0 + u) * T;
            if (q < len) {
#pragma unroll
                for (int a = 0; a < 3; ++a)
                    y[a] = fmaf(m[u][a * 3], p[u].x, fmaf(m[u][a * 3 + 1], p[u].y, fmaf(m[u][a * 3 + 2], p[u].z, y[a])));
            }
        }
    }
}

// r = b - A x (POST = false) or y4 = x + B^-1 (b - A x)
template <int T, bool POST>
__global__ void __launch_bounds__(kT) k_vc_rows(GeoView G, const float* __restrict__ binv, const float* b,
                                                const float4* x, float* r, float4* y4, const Control* ctl) {
    pdl_begin();
    if (vc_idle(ctl)) return;
    b = rhs_of(b, 3 * (size_t)G.n_rows);
    x = rhs_of(x, G.n_rows);
    const int gt = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = gt / T, t = gt % T;
    const bool ok = row < G.n_rows, lead = ok && t == 0;
    float y[3] = {0.f, 0.f, 0.f}, bv[3] = {0.f, 0.f, 0.f}, B[9];
    float4 xv = make_float4(0.f, 0.f, 0.f, 0.f);
    if (lead) {
#pragma unroll
        for (int a = 0; a < 3; ++a) bv[a] = b[3 * row + a];
        if constexpr (POST) {
            xv = x[row];
#pragma unroll
            for (int q = 0; q < 9; ++q) B[q] = binv[9 * (size_t)row + q];
        }
    }
    if (ok) {
        const float* v = G.v + (size_t)(row >> 5) * (27 * 9 * 32) + (row & 31);
        geo_row_part<T>(blk_of(G, row), row, t, [v](int e) { return v[(size_t)e * 32]; }, [x](int c) { return x[c]; }, y);
    }
    sum_lanes<T>(y);
    if (!lead) return;
    if constexpr (!POST) {
        r = rhs_of(r, 3 * (size_t)G.n_rows);
#pragma unroll
        for (int a = 0; a < 3; ++a) r[3 * row + a] = bv[a] - y[a];
    } else {
        y4 = rhs_of(y4, G.n_rows);
        const float d0 = bv[0] - y[0], d1 = bv[1] - y[1], d2 = bv[2] - y[2];
        y4[row] = make_float4(xv.x + B[0] * d0 + B[1] * d1 + B[2] * d2, xv.y + B[3] * d0 + B[4] * d1 + B[5] * d2,
                              xv.z + B[6] * d0 + B[7] * d1 + B[8] * d2, 0.f);
    }
}

__global__ void __launch_bounds__(kT) k_vc_post(SbView A, const float* __restrict__ binv, const float* __restrict__ b,
                                                const float4* __restrict__ x, float4* __restrict__ y4,
                                                const Control* ctl) {
    pdl_begin();
    if (vc_idle(ctl)) return;
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= A.n_rows) return;
    float y[3];
    sb_row(A, row, x, y);
    const float d0 = b[3 * row] - y[0], d1 = b[3 * row + 1] - y[1], d2 = b[3 * row + 2] - y[2];
    const float* B = binv + 9 * (size_t)row;
    const float4 xv = x[row];
    y4[row] = make_float4(xv.x + B[0] * d0 + B[1] * d1 + B[2] * d2, xv.y + B[3] * d0 + B[4] * d1 + B[5] * d2,
                          xv.z + B[6] * d0 + B[7] * d1 + B[8] * d2, 0.f);
}

// ---------------------------------------------------------------------------
// Gradient of the V-cycle residual loss with respect to the finest-level
// smoother blocks M (learned smoother training).  With z = V(b), x2 the
// level-0 iterate before post-smoothing, q = b - A z, r2 = b - A x2,
// w = A q, t = w - A M w and v = t - A P C R t (C: coarse V-cycle,
// R = P^T), the loss ||q||^2 has dL/dM_n = -2 (v_n b_n^T + w_n r2_n^T).
// ---------------------------------------------------------------------------
// q = b - A z, r2 = b - A x2; loss += ||q||^2
__global__ void __launch_bounds__(kT) k_vl_resid(SbView A, const float* __restrict__ b, const float4* __restrict__ z,
                                                 const float4* __restrict__ x2, float4* __restrict__ q,
                                                 float* __restrict__ r2, double* __restrict__ loss) {
    __shared__ double sm[32];
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    double acc[1] = {0.0};
    if (row < A.n_rows) {
        float y[3], u[3];
        sb_row(A, row, z, y);
        sb_row(A, row, x2, u);
        const float q0 = b[3 * row] - y[0], q1 = b[3 * row + 1] - y[1], q2 = b[3 * row + 2] - y[2];
        q[row] = make_float4(q0, q1, q2, 0.f);
#pragma unroll
        for (int a = 0; a < 3; ++a) r2[3 * row + a] = b[3 * row + a] - u[a];
        acc[0] = (double)q0 * q0 + (double)q1 * q1 + (double)q2 * q2;
    }
    block_sum<1>(acc, sm);
    if (threadIdx.x == 0 && acc[0] != 0.0) atomicAdd(loss, acc[0]);
}

// w = A q (stored as float[3n]); mw = M w (float4)
__global__ void __launch_bounds__(kT) k_vl_w(SbView A, const float* __restrict__ M, const float4* __restrict__ q,
                                             float* __restrict__ w, float4* __restrict__ mw) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= A.n_rows) return;
    float y[3];
    sb_row(A, row, q, y);
#pragma unroll
    for (int a = 0; a < 3; ++a) w[3 * row + a] = y[a];
    const float* B = M + 9 * (size_t)row;
    mw[row] = make_float4(B[0] * y[0] + B[1] * y[1] + B[2] * y[2], B[3] * y[0] + B[4] * y[1] + B[5] * y[2],
                          B[6] * y[0] + B[7] * y[1] + B[8] * y[2], 0.f);
}

// t = w - A mw (float[3n] and float4 copies)
__global__ void __launch_bounds__(kT) k_vl_t(SbView A, const float* __restrict__ w, const float4* __restrict__ mw,
                                             float* __restrict__ t, float4* __restrict__ t4) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= A.n_rows) return;
    float y[3];
    sb_row(A, row, mw, y);
    const float t0 = w[3 * row] - y[0], t1 = w[3 * row + 1] - y[1], t2 = w[3 * row + 2] - y[2];
    t[3 * row] = t0;
    t[3 * row + 1] = t1;
    t[3 * row + 2] = t2;
    t4[row] = make_float4(t0, t1, t2, 0.f);
}

// r := r - A z (stationary multigrid iteration on residuals)
__global__ void __launch_bounds__(kT) k_vl_rstep(SbView A, const float4* __restrict__ z, float* __restrict__ r) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= A.n_rows) return;
    float y[3];
    sb_row(A, row, z, y);
#pragma unroll
    for (int a = 0; a < 3; ++a) r[3 * row + a] -= y[a];
}

// v = t - A cc (cc = P C R t); G_n += -sym(2 (v b^T + w r2^T)), G stored g00 g11 g22 g01 g02 g12
__global__ void __launch_bounds__(kT) k_vl_grad(SbView A, const float4* __restrict__ t4, const float4* __restrict__ cc,
                                                const float* __restrict__ b, const float* __restrict__ w,
                                                const float* __restrict__ r2, float* __restrict__ G) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= A.n_rows) return;
    float y[3];
    sb_row(A, row, cc, y);
    const float4 tv = t4[row];
    const float v[3] = {tv.x - y[0], tv.y - y[1], tv.z - y[2]};
    const float bb[3] = {b[3 * row], b[3 * row + 1], b[3 * row + 2]};
    const float ww[3] = {w[3 * row], w[3 * row + 1], w[3 * row + 2]};
    const float rr[3] = {r2[3 * row], r2[3 * row + 1], r2[3 * row + 2]};
    auto gij = [&](int i, int j) { return -(v[i] * bb[j] + v[j] * bb[i] + ww[i] * rr[j] + ww[j] * rr[i]); };
    float* g = G + 6 * (size_t)row;
    g[0] += gij(0, 0);
    g[1] += gij(1, 1);
    g[2] += gij(2, 2);
    g[3] += gij(0, 1);
    g[4] += gij(0, 2);
    g[5] += gij(1, 2);
}

// ---------------------------------------------------------------------------
// Smoother damping: omega = 4 / (3 lambda), lambda an estimate of the largest
// eigenvalue of D^-1 A by power iteration (D = nodal diagonal blocks), so the
// damped block-Jacobi sweep stays a contraction on elongated or strongly
// heterogeneous elements.  All on the device: step k computes
// y = D^-1 A (x / nrm[k]) and nrm[k+1] = ||y||; the last CTA of a step sums
// the per-CTA partials in CTA order (deterministic).
// ---------------------------------------------------------------------------
__global__ void k_pow_init(int n, float4* __restrict__ x, float* __restrict__ nrm, int fill) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row == 0) nrm[0] = 1.f;
    if (row >= n || !fill) return;
    auto h = [](uint32_t v) {  // integer hash -> [-1, 1)
        v ^= v >> 16; v *= 0x7feb352du; v ^= v >> 15; v *= 0x846ca68bu; v ^= v >> 16;
        return (float)(v >> 8) * (2.f / 16777216.f) - 1.f;
    };
    x[row] = make_float4(h(3u * row + 1u), h(3u * row + 2u), h(3u * row + 3u), 0.f);
}

__global__ void __launch_bounds__(kT) k_pow_step(SbView A, const float* __restrict__ dinv, const float4* __restrict__ x,
                                                 float4* __restrict__ y4, float* __restrict__ nrm, int k,
                                                 double* __restrict__ part, uint32_t* __restrict__ ticket) {
    __shared__ double sm[32];
    __shared__ bool last;
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    const float inv = 1.f / nrm[k];
    double acc[1] = {0.0};
    if (row < A.n_rows) {
        float y[3];
        sb_row(A, row, x, y);
        const float* B = dinv + 9 * (size_t)row;
        const float z0 = inv * (B[0] * y[0] + B[1] * y[1] + B[2] * y[2]);
        const float z1 = inv * (B[3] * y[0] + B[4] * y[1] + B[5] * y[2]);
        const float z2 = inv * (B[6] * y[0] + B[7] * y[1] + B[8] * y[2]);
        y4[row] = make_float4(z0, z1, z2, 0.f);
        acc[0] = (double)z0 * z0 + (double)z1 * z1 + (double)z2 * z2;
    }
    block_sum<1>(acc, sm);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = acc[0];
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

// The same step on a coarse level, four lanes a row (a component of the product
// each, nine columns in flight; the fourth repeats the third's loads): one
// thread a row left a level of 6,171 rows on 49 CTAs with nine dependent rounds
// of loads, 13.8 us; now 8.3 (of
// which the sums in FP64 and the last CTA's part are the most).  Each component's sum is k_pow_step's.
__global__ void __launch_bounds__(kT) k_pow_rows(GeoView G, const float* __restrict__ dinv, const float4* __restrict__ x,
                                                 float4* __restrict__ y4, float* __restrict__ nrm, int k,
                                                 double* __restrict__ part, uint32_t* __restrict__ ticket) {
    __shared__ double sm[32];
    __shared__ bool last;
    const int gt = blockIdx.x * blockDim.x + threadIdx.x;
    const bool ok = (gt >> 2) < G.n_rows;
    const int row = ok ? gt >> 2 : 0, comp = min(gt & 3, 2);
    const float inv = 1.f / nrm[k];
    const BlkDev d = blk_of(G, row);
    const int l = row - d.node0, sj = d.nz + 1, si = (d.ny + 1) * sj;
    const int i = l / si, j = (l - i * si) / sj, kk = l - i * si - j * sj;
    const int i0 = max(i - 1, 0), j0 = max(j - 1, 0), k0 = max(kk - 1, 0);
    // padding between instances (i > nx): no columns
    const int ni = i <= d.nx ? min(i + 1, d.nx) - i0 + 1 : 0;
    const int nj = min(j + 1, d.ny) - j0 + 1, nk = min(kk + 1, d.nz) - k0 + 1;
    x += d.node0 + i0 * si + j0 * sj + k0;
    const float* v = G.v + (size_t)(row >> 5) * (27 * 9 * 32) + comp * 96 + (row & 31);
    const float B[3] = {dinv[9 * (size_t)row + 3 * comp], dinv[9 * (size_t)row + 3 * comp + 1],
                        dinv[9 * (size_t)row + 3 * comp + 2]};
    float y = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float m[9][3];
        float4 p[9];
#pragma unroll
        for (int u = 0; u < 9; ++u)
            if (a < ni && u / 3 < nj && u % 3 < nk) {
                p[u] = x[a * si + (u / 3) * sj + u % 3];
#pragma unroll
                for (int w = 0; w < 3; ++w) m[u][w] = v[((a * nj + u / 3) * nk + u % 3) * 288 + w * 32];
            }
#pragma unroll
        for (int u = 0; u < 9; ++u)
            if (a < ni && u / 3 < nj && u % 3 < nk)
                y = fmaf(m[u][0], p[u].x, fmaf(m[u][1], p[u].y, fmaf(m[u][2], p[u].z, y)));
    }
    const int quad = threadIdx.x & 28;
    const float a0 = __shfl_sync(0xffffffffu, y, quad), a1 = __shfl_sync(0xffffffffu, y, quad + 1),
                a2 = __shfl_sync(0xffffffffu, y, quad + 2);
    const float z = inv * (B[0] * a0 + B[1] * a1 + B[2] * a2);
    const float z1 = __shfl_sync(0xffffffffu, z, quad + 1), z2 = __shfl_sync(0xffffffffu, z, quad + 2);
    double acc[1] = {0.0};
    if (ok) {
        reinterpret_cast<float*>(y4 + row)[gt & 3] = (gt & 3) == 3 ? 0.f : z;
        if ((gt & 3) == 0) acc[0] = (double)z * z + (double)z1 * z1 + (double)z2 * z2;
    }
    block_sum<1>(acc, sm);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = acc[0];
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

// Guaranteed bound ||D^-1 A||_inf >= lambda_max(D^-1 A): the largest absolute
// row sum of D_n^-1 A_nm over the row's blocks (binv holds D^-1), as the
// float bits of a non-negative value under atomicMax.
__global__ void __launch_bounds__(kT) k_inf_bound(SbView A, const float* __restrict__ dinv,
                                                  unsigned int* __restrict__ bound_bits) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    float best = 0.f;
    if (row < A.n_rows) {
        const float* B = dinv + 9 * (size_t)row;
        const int lane = row & 31;
        const int64_t g0 = A.slice_off[row >> 5];
        const int len = A.row_len[row];
        float sum[3] = {0.f, 0.f, 0.f};
        for (int j = 0; j < len; ++j) {
            const float* v = A.v + ((g0 + j) * 9) * 32 + lane;
            float m[9];
#pragma unroll
            for (int q = 0; q < 9; ++q) m[q] = v[q * 32];
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b)
                    sum[a] += fabsf(B[3 * a] * m[b] + B[3 * a + 1] * m[3 + b] + B[3 * a + 2] * m[6 + b]);
        }
        best = fmaxf(sum[0], fmaxf(sum[1], sum[2]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
    if ((threadIdx.x & 31) == 0 && best > 0.f) atomicMax(bound_bits, __float_as_uint(best));
}

// binv := omega * binv (binv held D^-1) with omega = scale / lambda, lambda =
// the power estimate nrm[k], or the guaranteed bound when safe is set
__global__ void k_scale_blocks(int n, float* __restrict__ binv, const float* __restrict__ nrm, int k,
                               const unsigned int* __restrict__ bound_bits, int safe, float scale,
                               float* __restrict__ omega_out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 9 * n) return;
    const float est = nrm[k], bound = __uint_as_float(*bound_bits);
    float lam = safe ? bound : est;
    if (!(lam > 0.f) || !isfinite(lam)) lam = bound;
    const float omega = (lam > 0.f && isfinite(lam)) ? scale / lam : 0.5f;
    binv[i] *= omega;
    if (i == 0) *omega_out = omega;
}

// Transfers.  Along an axis a coarse node m lies on the fine node 2 m (the last
// one on the fine end), or on m where the axis is not coarsened, so positions
// and weights (1/2 from the neighbours across a cell of two) are computed.
__device__ __forceinline__ int fine_of(int m, int nc, int nf) { return nc == nf ? m : min(2 * m, nf); }

// acc += sum_I w_I y_c[I] at node fl of the fine block of coarse block d; y(c) the
// coarse vector's entry.  false: outside the block.
template <typename Y>
__device__ __forceinline__ bool prolong_at(const BlkDev& d, int fl, Y&& yc, float4& acc) {
    const int sj = d.fnz + 1, si = (d.fny + 1) * sj;
    if (fl >= (d.fnx + 1) * si) return false;
    const int at[3] = {fl / si, (fl % si) / sj, fl % sj};
    const int nf[3] = {d.fnx, d.fny, d.fnz}, nc[3] = {d.nx, d.ny, d.nz};
    int lo[3];
    bool mid[3];  // between two coarse nodes
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const bool co = nc[ax] != nf[ax];
        lo[ax] = !co ? at[ax] : (at[ax] == nf[ax] ? nc[ax] : at[ax] >> 1);
        mid[ax] = co && (at[ax] & 1) && at[ax] < nf[ax];
    }
    const int base = d.node0 + nid(lo[0], lo[1], lo[2], d.ny, d.nz);
    float4 y[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int di = q >> 2, dj = (q >> 1) & 1, dk = q & 1;
        if ((!di || mid[0]) && (!dj || mid[1]) && (!dk || mid[2]))
            y[q] = yc(base + (di * (d.ny + 1) + dj) * (d.nz + 1) + dk);
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int di = q >> 2, dj = (q >> 1) & 1, dk = q & 1;
        if ((!di || mid[0]) && (!dj || mid[1]) && (!dk || mid[2])) {
            const float ww = (mid[0] ? 0.5f : 1.f) * (mid[1] ? 0.5f : 1.f) * (mid[2] ? 0.5f : 1.f);
            acc.x += ww * y[q].x;
            acc.y += ww * y[q].y;
            acc.z += ww * y[q].z;
        }
    }
    return true;
}

// x_f[i] += sum_I w_iI y_c[I] over the fine level's nodes (a fine node outside
// every block -- padding between instances -- is left alone); G describes the
// coarse level's blocks (with their finer blocks), row_blk the fine rows'.
__global__ void k_vc_prolong(GeoView G, int n_fine, const float4* yc, float4* xf, const Control* ctl) {
    pdl_begin();
    if (vc_idle(ctl)) return;
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n_fine) return;
    yc = rhs_of(yc, G.n_rows);
    xf = rhs_of(xf, n_fine);
    float4 acc = xf[f];
    const BlkDev d = blk_of(G, f);
    if (prolong_at(d, f - d.fnode0, [yc](int c) { return yc[c]; }, acc)) xf[f] = acc;
}

// Coarsest solve y = A_b^-1 b per block: one warp per row (eight loads a lane
// in flight: a 256-wide row in one pass), kDenseRows rows a CTA.  y is
// node-padded.
constexpr int kDenseRows = 8;
template <typename B>
__device__ __forceinline__ float dense_row(const float* ar, int n, B&& b) {
    const int lane = threadIdx.x & 31;
    float a[8], bv[8], acc = 0.f;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const int j = lane + 32 * t;
        a[t] = j < n ? ar[j] : 0.f;
        bv[t] = j < n ? b(j) : 0.f;
    }
#pragma unroll
    for (int t = 0; t < 8; ++t)
        if (lane + 32 * t < n) acc = fmaf(a[t], bv[t], acc);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    return acc;
}

__global__ void __launch_bounds__(32 * kDenseRows) k_vc_dense(GeoView G, const float* __restrict__ ainv, const float* b,
                                                              float* y4, const Control* ctl) {
    pdl_begin();
    if (vc_idle(ctl)) return;
    const int row = blockIdx.z * kDenseRows + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const BlkDev d = G.row_blk ? G.blk[blockIdx.x] : G.one;
    const int n = 3 * (d.nx + 1) * (d.ny + 1) * (d.nz + 1);
    if (row >= n) return;
    const float* bb = rhs_of(b, 3 * (size_t)G.n_rows) + 3 * (size_t)d.node0;
    const float acc = dense_row(ainv + d.dense0 + (size_t)row * n, n, [bb](int j) { return bb[j]; });
    if (lane == 0) rhs_of(y4, 4 * (size_t)G.n_rows)[4 * ((size_t)d.node0 + row / 3) + row % 3] = acc;
}

// sum over the fine nodes f of w_x w_y w_z r(f) at node ol of coarse block d
// LARGE: plane by plane, skipping the planes of an axis that is not coarsened
// (there are enough nodes to hide the rounds of loads; the first coarsenings of a
// stretched grid leave an axis as it is: 9 taps of 27; 140,000 nodes 12.8 -> 9.1 us).
template <bool LARGE, typename R>
__device__ __forceinline__ float restrict_at(const BlkDev& d, int ol, R&& r) {
    const int sj = d.nz + 1, si = (d.ny + 1) * sj;
    const int m[3] = {ol / si, (ol % si) / sj, ol % sj};
    const int nf[3] = {d.fnx, d.fny, d.fnz}, nc[3] = {d.nx, d.ny, d.nz};
    int x[3];
    bool on[3][3];  // axis, tap x - 1, x, x + 1
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        x[ax] = fine_of(m[ax], nc[ax], nf[ax]);
        on[ax][0] = m[ax] > 0 && x[ax] - fine_of(m[ax] - 1, nc[ax], nf[ax]) == 2;
        on[ax][1] = true;
        on[ax][2] = m[ax] < nc[ax] && fine_of(m[ax] + 1, nc[ax], nf[ax]) - x[ax] == 2;
    }
    if constexpr (LARGE) {
        float s = 0.f;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (!on[0][a]) continue;
            float v[9];
#pragma unroll
            for (int q = 0; q < 9; ++q) {
                const int b = q / 3, c = q % 3;
                const size_t src = d.fnode0 + ((size_t)(x[0] + a - 1) * (d.fny + 1) + (x[1] + b - 1)) * (d.fnz + 1) + (x[2] + c - 1);
                v[q] = on[1][b] && on[2][c] ? r(src) : 0.f;
            }
#pragma unroll
            for (int q = 0; q < 9; ++q) {
                const int b = q / 3, c = q % 3;
                if (on[1][b] && on[2][c]) s = fmaf((a == 1 ? 1.f : 0.5f) * (b == 1 ? 1.f : 0.5f) * (c == 1 ? 1.f : 0.5f), v[q], s);
            }
        }
        return s;
    }
    float v[27];
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        const int a = q / 9, b = q / 3 % 3, c = q % 3;
        const size_t src = d.fnode0 + ((size_t)(x[0] + a - 1) * (d.fny + 1) + (x[1] + b - 1)) * (d.fnz + 1) + (x[2] + c - 1);
        v[q] = on[0][a] && on[1][b] && on[2][c] ? r(src) : 0.f;
    }
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        const int a = q / 9, b = q / 3 % 3, c = q % 3;
        const float ww = (a == 1 ? 1.f : 0.5f) * (b == 1 ? 1.f : 0.5f) * (c == 1 ? 1.f : 0.5f);
        if (on[0][a] && on[1][b] && on[2][c]) s = fmaf(ww, v[q], s);
    }
    return s;
}

// Trilinear restriction R = P^T over every block at once, four lanes per coarse
// node (a component each, the fourth idle): b_c[m] = sum over the fine nodes f
// of w_x w_y w_z r_f, where along each axis the fine nodes next to 2 m
// contribute with 1/2 when they lie across a cell of two.  Fixed slots let the
// 27 loads of a lane issue together.  The coarse level's first smoothing sweep
// x4 = B^-1 b is fused in (binv non-null).
template <bool LARGE>
__global__ void __launch_bounds__(kT) k_vc_restrict(GeoView G, int n_fine, const float* in, float* out,
                                                    const float* __restrict__ binv, float4* x4, const Control* ctl) {
    pdl_begin();
    if (vc_idle(ctl)) return;
    const int gt = blockIdx.x * blockDim.x + threadIdx.x;
    const bool ok = (gt >> 2) < G.n_rows;
    const int o = ok ? gt >> 2 : 0, comp = min(gt & 3, 2);
    in = rhs_of(in, 3 * (size_t)n_fine) + comp;
    float B[3] = {0.f, 0.f, 0.f};
    if (binv) {
#pragma unroll
        for (int q = 0; q < 3; ++q) B[q] = binv[9 * (size_t)o + 3 * comp + q];
    }
    const BlkDev d = blk_of(G, o);
    const float s = restrict_at<LARGE>(d, o - d.node0, [in](size_t f) { return in[3 * f]; });
    const int lane0 = (threadIdx.x & 31) & ~3;
    const float s0 = __shfl_sync(0xffffffffu, s, lane0), s1 = __shfl_sync(0xffffffffu, s, lane0 + 1),
                s2 = __shfl_sync(0xffffffffu, s, lane0 + 2);
    if (!ok || (gt & 3) == 3) return;
    rhs_of(out, 3 * (size_t)G.n_rows)[3 * (size_t)o + comp] = s;
    if (binv)
        reinterpret_cast<float*>(rhs_of(x4, G.n_rows) + o)[comp] = B[0] * s0 + B[1] * s1 + B[2] * s2;
}

// The V-cycle's smallest levels (down to the coarsest and back) of a lone block as
// one launch, a cluster of 16 CTAs per right-hand side.  A step on these levels is
// a few hundred cycles of work that a launch of its own turns into 3 us (and
// a step through global memory with a cluster barrier into 2.5, most of it the
// fence), so the vectors live in every CTA's shared memory: a CTA stores its rows'
// results into the other copies, and a cluster barrier ends the step.  Each CTA owns
// a run of rows of every level.  What does not change between V-cycles -- the own
// rows' values, columns and smoother blocks, the rows of the coarsest inverse, the
// transfers' indices -- is laid out before the wait for the kernel that restricts
// to the first level (nothing in between writes any of it); that hides these loads
// with launch overlap only, which is off by default (a 100 x 20 x 20 solve 3.10 ms,
// with overlap 3.17).  The prolongation is made by every CTA for its whole copy.  The
// sums and their order are those of the separate kernels.  Bound by the barriers (1,500
// cycles with the stores before them) and short dependent chains: 100 x 20 x 20
// elements (nine launches of 28 us) 19.5 us launched alone, 23.9 among a step's
// kernels; 57 x 13 x 11 (16 us) 11.2 alone.
__device__ __forceinline__ void tail_tables(const TailView& V, int l, float* tsm, int r0, int mine) {
    const TailView::Level& L = V.L[l];
    const BlkDev& d = L.d;
    const int tid = threadIdx.x, sj = d.nz + 1, si = (d.ny + 1) * sj;
    if (l < V.n - 1) {
        uint16_t* col = reinterpret_cast<uint16_t*>(tsm + L.co);
        for (int q = tid; q < mine * kTailCols; q += kTailThreads) {
            const int lr = q / kTailCols, e = q % kTailCols, row = r0 + lr;
            const int i = row / si, j = (row - i * si) / sj, k = row - i * si - j * sj;
            const int i0 = max(i - 1, 0), j0 = max(j - 1, 0), k0 = max(k - 1, 0);
            const int nj = min(j + 1, d.ny) - j0 + 1, nk = min(k + 1, d.nz) - k0 + 1;
            const int len = (min(i + 1, d.nx) - i0 + 1) * nj * nk;
            const int ek = e / nk;
            col[q] = (uint16_t)(e == 27 ? len : e < len ? (i0 + ek / nj) * si + (j0 + ek % nj) * sj + k0 + e - ek * nk : row);
            if (e < 9) tsm[L.so + 12 * lr + 3 + e] = L.binv[9 * (size_t)row + e];
        }
        const BlkDev& c = V.L[l + 1].d;
        uint16_t* pro = reinterpret_cast<uint16_t*>(tsm + L.po);
        for (int f = tid; f < L.n_rows; f += kTailThreads) {
            const int at[3] = {f / si, (f % si) / sj, f % sj};
            const int nf[3] = {c.fnx, c.fny, c.fnz}, nc[3] = {c.nx, c.ny, c.nz};
            int lo[3], mid = 0;
#pragma unroll
            for (int ax = 0; ax < 3; ++ax) {
                const bool two = nc[ax] != nf[ax];
                lo[ax] = !two ? at[ax] : (at[ax] == nf[ax] ? nc[ax] : at[ax] >> 1);
                mid |= (two && (at[ax] & 1) && at[ax] < nf[ax]) << ax;
            }
            pro[f] = (uint16_t)(8 * nid(lo[0], lo[1], lo[2], c.ny, c.nz) + mid);
        }
    }
    if (l > 0) {
        int* res = reinterpret_cast<int*>(tsm + L.to);
        for (int q = tid; q < mine; q += kTailThreads) {
            const int o = r0 + q, m[3] = {o / si, (o % si) / sj, o % sj};
            const int nf[3] = {d.fnx, d.fny, d.fnz}, nc[3] = {d.nx, d.ny, d.nz};
            int x[3], on = 0;
#pragma unroll
            for (int ax = 0; ax < 3; ++ax) {
                x[ax] = fine_of(m[ax], nc[ax], nf[ax]);
                on |= (m[ax] > 0 && x[ax] - fine_of(m[ax] - 1, nc[ax], nf[ax]) == 2) << (2 * ax);
                on |= (m[ax] < nc[ax] && fine_of(m[ax] + 1, nc[ax], nf[ax]) - x[ax] == 2) << (2 * ax + 1);
            }
            res[q] = nid(x[0], x[1], x[2], d.fny, d.fnz) + (on << 16);
        }
    }
}

__global__ void __launch_bounds__(kTailThreads) k_vc_tail(const __grid_constant__ TailView V,
                                                          const float* __restrict__ ainv, const Control* ctl) {
    extern __shared__ __align__(16) float tsm[];
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int rank = (int)cl.block_rank(), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int last = V.n - 1;
    auto vec = [&](int off) { return reinterpret_cast<float4*>(tsm + off); };
    for (int l = 0; l <= last; ++l) {
        const TailView::Level& L = V.L[l];
        const int r0 = rank * L.own, mine = max(0, min(L.own, L.n_rows - r0));
        if (l < last && L.vo >= 0)  // a warp reads an entry of 32 rows at a time
            for (int p = 0; p < mine; p += 32) {
                const int lr = min(p + lane, mine - 1), row = r0 + lr;
                const float* src = L.v + (size_t)(row >> 5) * (27 * 9 * 32) + (row & 31);
                float* dst = tsm + L.vo + lr * kTailLd;
#pragma unroll 8
                for (int e = warp; e < 27 * 9; e += kTailThreads / 32) dst[e] = src[(size_t)e * 32];
            }
        tail_tables(V, l, tsm, r0, mine);
    }
    // the coarsest inverse: one warp a row
    const int nd = 3 * V.L[last].n_rows, drow = warp * kTailCtas + rank;
    float ai[8];
#pragma unroll
    for (int t = 0; t < 8; ++t)
        ai[t] = drow < nd && lane + 32 * t < nd ? ainv[(size_t)drow * nd + lane + 32 * t] : 0.f;
    cl.sync();  // every CTA runs: its shared memory may be written
    pdl_begin();
    if (vc_idle(ctl)) return;  // the same for the whole cluster
    {
        const TailView::Level& L = V.L[0];
        const int r0 = rank * L.own, mine = max(0, min(L.own, L.n_rows - r0));
        const float4* x = rhs_of(V.x4, L.n_rows);
        const float* b = rhs_of(V.b, 3 * (size_t)L.n_rows) + 3 * r0;
        for (int q = tid; q < L.n_rows; q += kTailThreads) vec(L.xo)[q] = x[q];
        for (int q = tid; q < 3 * mine; q += kTailThreads) tsm[L.so + q / 3 * 12 + q % 3] = b[q];
    }
    __syncthreads();
    // residuals b - A x of the own rows of level l, 16 lanes a row (all get the sums)
    auto rows = [&](int l, auto&& epi) {
        const TailView::Level& L = V.L[l];
        const float4* x = vec(L.xo);
        const int t = tid & 15, r0 = rank * L.own, mine = min(L.own, L.n_rows - r0);
        for (int p = 0; p < L.own; p += kTailThreads / 16) {
            const int lr = p + (tid >> 4), row = r0 + lr;
            const bool ok = lr < mine;
            const float* own = tsm + L.so + lr * 12;
            float y[3] = {0.f, 0.f, 0.f};
            if (ok) {
                const uint16_t* col = reinterpret_cast<const uint16_t*>(tsm + L.co) + lr * kTailCols;
                const int len = col[27];
                auto part = [&](auto&& v) {
                    float m[2][9];
                    float4 xv[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        if (t + 16 * u < len) {
                            xv[u] = x[col[t + 16 * u]];
#pragma unroll
                            for (int w = 0; w < 9; ++w) m[u][w] = v((t + 16 * u) * 9 + w);
                        }
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        if (t + 16 * u < len)
#pragma unroll
                            for (int a = 0; a < 3; ++a)
                                y[a] = fmaf(m[u][a * 3], xv[u].x,
                                            fmaf(m[u][a * 3 + 1], xv[u].y, fmaf(m[u][a * 3 + 2], xv[u].z, y[a])));
                };
                if (L.vo >= 0) {
                    const float* v = tsm + L.vo + lr * kTailLd;
                    part([v](int e) { return v[e]; });
                } else {
                    const float* v = L.v + (size_t)(row >> 5) * (27 * 9 * 32) + (row & 31);
                    part([v](int e) { return v[e * 32]; });
                }
            }
            sum_lanes<16>(y);
            if (ok) {
                const float r[3] = {own[0] - y[0], own[1] - y[1], own[2] - y[2]};
                epi(row, t, own + 3, r);
            }
        }
    };
    // own rows of a vector to the other CTAs' copies: two warps a CTA, 512 bytes a store
    auto publish = [&](int off, int own, int n) {
        __syncthreads();
        const int r0 = rank * own, mine = min(own, n - r0), to = warp & (kTailCtas - 1);
        const float4* src = vec(off) + r0;
        float4* dst = cl.map_shared_rank(vec(off), to) + r0;
        if (to != rank)
            for (int q = lane + 32 * (warp / kTailCtas); q < mine; q += 32 * (kTailThreads / 32 / kTailCtas)) dst[q] = src[q];
        cl.sync();
    };
    for (int l = 0; l < last; ++l) {
        const TailView::Level &L = V.L[l], &C = V.L[l + 1];
        rows(l, [&](int row, int t, const float*, const float (&r)[3]) {
            if (t == 0) vec(L.ro)[row] = make_float4(r[0], r[1], r[2], 0.f);
        });
        publish(L.ro, L.own, L.n_rows);
        // restriction and the coarse level's first sweep, four lanes a node
        const float* r = reinterpret_cast<const float*>(vec(L.ro));
        const int sj = C.d.fnz + 1, si = (C.d.fny + 1) * sj;
        const int comp = min(tid & 3, 2), quad = lane & ~3, r0 = rank * C.own, mine = min(C.own, C.n_rows - r0);
        for (int p = 0; p < C.own; p += kTailThreads / 4) {
            if (p + 8 * warp >= mine) continue;  // the warp's nodes
            const int lo = p + (tid >> 2);
            const bool ok = lo < mine;
            const int at = reinterpret_cast<const int*>(tsm + C.to)[min(lo, mine - 1)], on = at >> 16;
            const float* rc = r + 4 * (at & 0xffff) + comp;
            float v[27], s = 0.f;
#pragma unroll
            for (int q = 0; q < 27; ++q) {  // all in flight; the sides that do not contribute add 0
                const int i = q / 9, j = q / 3 % 3, k = q % 3;
                const int need = (i == 1 ? 0 : 1 << (i / 2)) | (j == 1 ? 0 : 4 << (j / 2)) | (k == 1 ? 0 : 16 << (k / 2));
                const bool in = (on & need) == need;
                v[q] = rc[in ? 4 * ((i - 1) * si + (j - 1) * sj + k - 1) : 0];
                v[q] = in ? v[q] : 0.f;
            }
#pragma unroll
            for (int q = 0; q < 27; ++q)
                s = fmaf((q / 9 == 1 ? 1.f : 0.5f) * (q / 3 % 3 == 1 ? 1.f : 0.5f) * (q % 3 == 1 ? 1.f : 0.5f), v[q], s);
            const float s0 = __shfl_sync(0xffffffffu, s, quad), s1 = __shfl_sync(0xffffffffu, s, quad + 1),
                        s2 = __shfl_sync(0xffffffffu, s, quad + 2);
            float4 out = make_float4(s0, s1, s2, 0.f);
            if (l + 1 < last) {
                float* own = tsm + C.so + min(lo, mine - 1) * 12;
                const float* B = own + 3 + 3 * comp;
                const float x = B[0] * s0 + B[1] * s1 + B[2] * s2;
                if (ok && (tid & 3) != 3) own[comp] = s;
                out.x = __shfl_sync(0xffffffffu, x, quad);
                out.y = __shfl_sync(0xffffffffu, x, quad + 1);
                out.z = __shfl_sync(0xffffffffu, x, quad + 2);
            }
            if (ok && (tid & 3) == 0) vec(C.xo)[r0 + lo] = out;
        }
        publish(C.xo, C.own, C.n_rows);
    }
    {
        const TailView::Level& L = V.L[last];
        const float* b = reinterpret_cast<const float*>(vec(L.xo));
        if (drow < nd) {
            float bv[8], acc = 0.f;
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const int j = lane + 32 * t;
                bv[t] = j < nd ? b[4 * (j / 3) + j % 3] : 0.f;
            }
#pragma unroll
            for (int t = 0; t < 8; ++t)
                if (lane + 32 * t < nd) acc = fmaf(ai[t], bv[t], acc);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane < kTailCtas)
                reinterpret_cast<float*>(cl.map_shared_rank(vec(L.ro), lane) + drow / 3)[drow % 3] = acc;
        }
        cl.sync();
    }
    for (int l = last - 1; l >= 0; --l) {
        const TailView::Level &L = V.L[l], &C = V.L[l + 1];
        float4* x = vec(L.xo);
        const float4* yc = vec(C.ro);
        const int sj = C.d.nz + 1, si = (C.d.ny + 1) * sj;
        for (int f = tid; f < L.n_rows; f += kTailThreads) {
            const int at = reinterpret_cast<const uint16_t*>(tsm + L.po)[f], mid = at & 7;
            const float ww = (mid & 1 ? 0.5f : 1.f) * (mid & 2 ? 0.5f : 1.f) * (mid & 4 ? 0.5f : 1.f);
            const float4* y = yc + (at >> 3);
            float4 acc = x[f];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int need = (q >> 2) | (q & 2) | (q & 1) << 2;  // q = 4 di + 2 dj + dk
                if ((mid & need) == need) {
                    const float4 v = y[(q >> 2) * si + (q >> 1 & 1) * sj + (q & 1)];
                    acc.x += ww * v.x;
                    acc.y += ww * v.y;
                    acc.z += ww * v.z;
                }
            }
            x[f] = acc;
        }
        __syncthreads();
        float4* y4 = rhs_of(V.y4, L.n_rows);
        rows(l, [&](int row, int t, const float* B, const float (&e)[3]) {
            const float4 xv = x[row];
            const float4 y = make_float4(xv.x + B[0] * e[0] + B[1] * e[1] + B[2] * e[2],
                                         xv.y + B[3] * e[0] + B[4] * e[1] + B[5] * e[2],
                                         xv.z + B[6] * e[0] + B[7] * e[1] + B[8] * e[2], 0.f);
            if (t == 0) (l > 0 ? vec(L.ro) : y4)[row] = y;
        });
        if (l > 0) publish(L.ro, L.own, L.n_rows);
    }
}

// ---------------------------------------------------------------------------
// multigrid-preconditioned flexible CG kernels (up to 4 right-hand sides; every
// instance of a batched stack at once, with its own scalars and tickets)
// ---------------------------------------------------------------------------
struct MgPcg {
    PcgArgs a;            // outer operator, x, r, p, ap, partials, sc, ctl (nrhs = 1)
    float4* xp;           // split method: the correction e of x since its last true residual,
                          // node-padded FP32 pairs (hi float4, lo float4)
    float4* xt;           // split method on a split-only operator: x as three node-padded FP32
                          // parts (hi, lo, remainder) for the true residual (else nullptr)
    float* b0;            // V-cycle input (level-0 rhs, FP32 r)
    const float4* z;      // V-cycle output (level-0 y4)
    const float* binv0;   // level-0 smoother blocks: the first sweep
    float4* x40;          // x4 = B^-1 r is fused into the kernels writing b0
    int n_inst;           // instances (1: a single model)
    int part_stride;      // CTAs of the partials array per right-hand side
    const int2* cg_rows;  // stacks: rows of each CTA of the vector kernels (else nullptr)
};

// The rows of a thread of the pair method's vector kernels.
struct RowRange {
    int begin, end, step;
};
__device__ __forceinline__ RowRange cg_range(const MgPcg& M) {
    if (M.cg_rows) {
        const int2 q = M.cg_rows[blockIdx.x];
        return {q.x + (int)threadIdx.x, q.y, (int)blockDim.x};
    }
    return {(int)(blockIdx.x * blockDim.x + threadIdx.x), M.a.n_rows, (int)(gridDim.x * blockDim.x)};
}

// The kernels' second grid dimension is the right-hand side: its slice of every
// vector, scalar set, ticket and partials array (F32: the mixed method's FP32
// direction and A p).
template <bool F32>
__device__ __forceinline__ MgPcg rhs_view(MgPcg M) {
    const size_t k = blockIdx.y, n = M.a.n_rows, nd = M.a.n_dof;
    PcgArgs& A = M.a;
    A.f += k * nd;
    A.x += k * nd;
    A.r += k * nd;
    A.p = reinterpret_cast<char*>(A.p) + k * n * (F32 ? 16 : 32);
    A.ap = reinterpret_cast<char*>(A.ap) + k * nd * (F32 ? 4 : 8);
    A.partials += k * M.part_stride * (kMaxRhs * 3);
    A.tickets += k * M.n_inst * 4;
    A.sc += k;
    M.xp += 2 * k * n;
    if (M.xt) M.xt += 3 * k * n;
    M.b0 += k * nd;
    M.z += k * n;
    M.x40 += k * n;
    return M;
}

// Nothing left to do for this CTA's instance and right-hand side.
__device__ __forceinline__ bool mg_done(const PcgArgs& A, const RhsScalars* S) {
    return A.ctl->active[blockIdx.y] == 0 || S[0].done;
}

// The instances still iterating are counted per right-hand side; with the last
// one whose recurrence converges every remaining captured kernel of that
// right-hand side ends at once.
__device__ __forceinline__ void retire_instance(const PcgArgs& A) { atomicSub(&A.ctl->active[blockIdx.y], 1); }

// First kernel of a captured chunk of iterations: count the instances not done
// (grid: right-hand sides).
__global__ void k_mg_count_active(MgPcg M) {
    pdl_begin();
    const PcgArgs& A = M.a;
    int n = 0;
    for (int i = threadIdx.x; i < M.n_inst; i += blockDim.x) n += A.sc[(size_t)i * kMaxRhs + blockIdx.x].done ? 0 : 1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if (threadIdx.x == 0) A.ctl->active[blockIdx.x] = n;
}

__device__ __forceinline__ void fused_smooth0(const MgPcg& M, int row, const double (&r)[3]) {
    const float* B = M.binv0 + 9 * (size_t)row;
    const float r0 = (float)r[0], r1 = (float)r[1], r2 = (float)r[2];
    M.x40[row] = make_float4(B[0] * r0 + B[1] * r1 + B[2] * r2, B[3] * r0 + B[4] * r1 + B[5] * r2,
                             B[6] * r0 + B[7] * r1 + B[8] * r2, 0.f);
}

template <typename TV, typename TP>
__global__ void __launch_bounds__(kThreads) k_mg_spmv_dot(MgPcg M) {
    pdl_begin();
    using PV = typename ApOf<TP>::T;
    M = rhs_view<sizeof(TV) == 4 && std::is_same<TP, float>::value>(M);
    const PcgArgs& A = M.a;
    RhsScalars* S = A.sc + cta_instance(A) * kMaxRhs;
    if (mg_done(A, S)) return;
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    double d[1][1] = {{0.0}};
    if (row < A.n_rows) {
        PV y[1][3];
        const TV* vals;
        if constexpr (sizeof(TV) == 4) vals = A.v32; else vals = A.v64;
        spmv_row<TV, TP, 1>(row, A, vals, A.p, y);
        PV pv[3];
        PadVec<TP>::load(A.p, row, pv);
        PV* ap = reinterpret_cast<PV*>(A.ap) + 3 * (size_t)row;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            ap[q] = y[0][q];
            d[0][0] += (double)pv[q] * (double)y[0][q];
        }
    }
    double tot[1][1];
    if (last_block_reduce<1, 1>(A, d, 0, tot) && threadIdx.x == 0) {
        RhsScalars& s = S[0];
        s.pAp = tot[0][0];
        s.alpha = s.rz / s.pAp;
    }
}

// The FP64 product with four lanes a row, for single models whose rows alone leave
// SMs idle: one thread a row walked 27 columns one step after the other (7,930
// rows: 52.6 us).  FP64 issue (64 cycles a warp instruction) bounds it from there:
// the lanes' sums are exchanged so that each lane ends with one component (3
// additions, where eight lanes with the whole sum each took 9 for half the rows)
// and makes that component's share of p.Ap; 7,930
// rows, two right-hand sides: eight lanes 19.7 us, now 13.4.
constexpr int kLaneRows = 152 * 1024 / 4;  // rows whose lanes fill the GPU
__global__ void __launch_bounds__(kThreads) k_mg_spmv_dot_lanes(MgPcg M) {
    pdl_begin();
    M = rhs_view<false>(M);
    const PcgArgs& A = M.a;
    RhsScalars* S = A.sc;
    if (mg_done(A, S)) return;
    const int gt = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = gt / 4, t = gt % 4;
    const bool ok = row < A.n_rows;
    double y[3] = {0.0, 0.0, 0.0}, d[1][1] = {{0.0}};
    if (ok) {
        const int lane = row & 31, len = A.row_len[row];
        const int64_t g0 = A.slice_off[row >> 5];
#pragma unroll 2
        for (int j = t; j < len; j += 4) {
            const int64_t g = g0 + j;
            double m[9], p[3];
            PadVec<double>::load(A.p, (size_t)A.col[g * 32 + lane], p);
#pragma unroll
            for (int q = 0; q < 9; ++q) m[q] = A.v64[(g * 9 + q) * 32 + lane];
#pragma unroll
            for (int a = 0; a < 3; ++a) y[a] = fma(m[3 * a], p[0], fma(m[3 * a + 1], p[1], fma(m[3 * a + 2], p[2], y[a])));
        }
    }
    const bool up = t & 2, odd = t & 1;
    double lo = (up ? y[2] : y[0]) + __shfl_xor_sync(0xffffffffu, up ? y[0] : y[2], 2);
    const double hi = (up ? 0.0 : y[1]) + __shfl_xor_sync(0xffffffffu, up ? y[1] : 0.0, 2);
    lo = (odd ? hi : lo) + __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 1);  // component t
    if (ok && t < 3) {
        double pv[3];
        PadVec<double>::load(A.p, row, pv);
        reinterpret_cast<double*>(A.ap)[3 * (size_t)row + t] = lo;
        d[0][0] = (t == 0 ? pv[0] : t == 1 ? pv[1] : pv[2]) * lo;
    }
    double tot[1][1];
    if (last_block_reduce<1, 1>(A, d, 0, tot) && threadIdx.x == 0) {
        S[0].pAp = tot[0][0];
        S[0].alpha = S[0].rz / S[0].pAp;
    }
}

// ---------------------------------------------------------------------------
// Split method, vector side: the correction e of x (node-padded), r and A p
// (natural layout) are FP32 pairs and every per-row update and dot product is
// pair arithmetic on the FP32 pipes; FP64 is left to the per-CTA reductions
// (one value per thread), the scalars, and the true residuals (x64 += e, then
// r = f - A64 x64), formed two or three times per solve.
// ---------------------------------------------------------------------------
__device__ __forceinline__ F2 ld_pair(const float2* v, size_t i) {
    const float2 q = v[i];
    return {q.x, q.y};
}
__device__ __forceinline__ void st_pair(float2* v, size_t i, F2 a) { v[i] = make_float2(a.h, a.l); }
__device__ __forceinline__ void ld_pad_pair(const void* p, size_t node, F2 (&v)[3]) {
    const float4 h = reinterpret_cast<const float4*>(p)[2 * node];
    const float4 l = reinterpret_cast<const float4*>(p)[2 * node + 1];
    v[0] = {h.x, l.x};
    v[1] = {h.y, l.y};
    v[2] = {h.z, l.z};
}
__device__ __forceinline__ void st_pad_pair(void* p, size_t node, const F2 (&v)[3]) {
    reinterpret_cast<float4*>(p)[2 * node] = make_float4(v[0].h, v[1].h, v[2].h, 0.f);
    reinterpret_cast<float4*>(p)[2 * node + 1] = make_float4(v[0].l, v[1].l, v[2].l, 0.f);
}

// Store A p of this row (pairs) and return p . A p over the row's 3 DOF (a
// pair: a thread sums its rows in pairs and converts to FP64 once).
__device__ __forceinline__ F2 pair_ap_dot(const PcgArgs& A, int row, const F2 (&y)[3]) {
    F2 pv[3];
    ld_pad_pair(A.p, row, pv);
    float2* ap = reinterpret_cast<float2*>(A.ap);
    F2 acc{0.f, 0.f};
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        st_pair(ap, 3 * (size_t)row + q, y[q]);
        acc = f2_add(acc, f2_mul(pv[q], y[q]));
    }
    return acc;
}

// The register-fed split product with the pair epilogue.
__global__ void __launch_bounds__(kThreads) k_mg_spmv_dot_pair(MgPcg M) {
    pdl_begin();
    M = rhs_view<false>(M);
    const PcgArgs& A = M.a;
    RhsScalars* Sc = A.sc + cta_instance(A) * kMaxRhs;
    if (mg_done(A, Sc)) return;
    F2 acc{0.f, 0.f};
    for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < A.n_rows; row += gridDim.x * blockDim.x) {
        float Sm[1][3], Cc[1][3];
        spmv_row_split_sc<1>(row, A, A.p, Sm, Cc);
        const F2 y[3] = {two_sum(Sm[0][0], Cc[0][0]), two_sum(Sm[0][1], Cc[0][1]), two_sum(Sm[0][2], Cc[0][2])};
        acc = f2_add(acc, pair_ap_dot(A, row, y));
    }
    double d[1][1] = {{f2_dbl(acc)}};
    double tot[1][1];
    if (last_block_reduce<1, 1>(A, d, 0, tot) && threadIdx.x == 0) set_alpha(Sc[0], tot[0][0]);
}

// The split method iterates on x = x64 + e: x64 (FP64) changes only when a
// true residual is formed, and the correction e gathered since then is an
// FP32 pair.  Folding e into x64 there (and at the end) keeps the stored
// solution in FP64, so the pairs' 48-bit rounding of e stays far below the
// solve's tolerance (x itself as a pair left a noise floor near 1e-9).
// x64 += e, e = 0 for the instances whose true residual is formed next (all
// rows when all is set)
__global__ void __launch_bounds__(kThreads) k_fold_pairs(MgPcg M, int all) {
    pdl_begin();
    M = rhs_view<false>(M);
    const PcgArgs& A = M.a;
    const RhsScalars* S = A.sc + cta_instance(A) * kMaxRhs;
    if (!all && !S[0].replace) return;
    const RowRange rows = cg_range(M);
    for (int row = rows.begin; row < rows.end; row += rows.step) {
        F2 e[3];
        ld_pad_pair(M.xp, row, e);
        float t[3][3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const double xv = A.x[3 * (size_t)row + q] + f2_dbl(e[q]);
            A.x[3 * (size_t)row + q] = xv;
            if (M.xt) {  // x = hi + lo + remainder, each FP32
                const float h = (float)xv;
                const double r1 = xv - (double)h;
                const float l = (float)r1;
                t[0][q] = h;
                t[1][q] = l;
                t[2][q] = (float)(r1 - (double)l);
            }
        }
        const F2 z[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
        st_pad_pair(M.xp, row, z);
        if (M.xt)
#pragma unroll
            for (int k = 0; k < 3; ++k) M.xt[3 * (size_t)row + k] = make_float4(t[k][0], t[k][1], t[k][2], 0.f);
    }
}

// One term (h + l)(xh + xl + xr) of a true residual, added to a three-level
// sum (S, C, D): S the leading sum, C the next order, D the rest.  The
// products h xh, h xl and l xh are split exactly (FMA) and every rounding
// error of S and C goes one level down, so only D rounds, at 2^-24 of a
// 2^-48-sized quantity: the sum keeps about 70 bits, where the CG product's
// two levels keep 48 (enough for a search direction, not for f - A x, whose
// terms are 10^4 times |f| on a point-loaded cantilever).
__device__ __forceinline__ void res_term(float h, float l, float xh, float xl, float xr, float& S, float& C,
                                         float& D) {
    const float p1 = __fmul_rn(h, xh), e1 = __fmaf_rn(h, xh, -p1);
    const float p2 = __fmul_rn(h, xl), e2 = __fmaf_rn(h, xl, -p2);
    const float p3 = __fmul_rn(l, xh), e3 = __fmaf_rn(l, xh, -p3);
    const F2 s0 = two_sum(S, p1);
    S = s0.h;
    const F2 c1 = two_sum(C, s0.l);
    const F2 c2 = two_sum(c1.h, e1);
    const F2 c3 = two_sum(c2.h, p2);
    const F2 c4 = two_sum(c3.h, p3);
    C = c4.h;
    D = __fadd_rn(D, __fadd_rn(__fadd_rn(c1.l, c2.l), __fadd_rn(c3.l, c4.l)));
    D = __fadd_rn(D, __fadd_rn(e2, e3));
    D = __fmaf_rn(h, xr, __fmaf_rn(l, xl, D));
}

constexpr int kZeroStart = 2;  // init: the start is x = 0, so r = f

// True residual r = f - A x from the operator's hi / lo values (split-only
// assembly: no FP64 values) and the three FP32 parts of x written by the
// fold, each term by res_term.  Three threads a row, a component each, in warps
// of 32 rows (coalesced as one thread a row would be): with one thread a row a model
// of 44,541 rows had 21 KB of loads in flight an SM (a solve's three evaluations 186 us,
// now 106).  The first 128 threads then sum their rows' squares in the components'
// order and make the reduction.
constexpr int kResThreads = 3 * kThreads;
__global__ void __launch_bounds__(kResThreads) k_mg_residual_split(MgPcg M, int init, double tol2) {
    __shared__ F2 sq[3][kThreads];
    pdl_begin();
    M = rhs_view<false>(M);
    const PcgArgs& A = M.a;
    RhsScalars* S = A.sc + cta_instance(A) * kMaxRhs;
    if (!init && !S[0].replace) return;
    const int a = threadIdx.x / kThreads, rl = threadIdx.x % kThreads, row = blockIdx.x * kThreads + rl;
    F2 q{0.f, 0.f};
    if (row < A.n_rows) {
        const int lane = row & 31;
        float Sm = 0.f, Cc = 0.f, Dd = 0.f;
        const int64_t g0 = A.slice_off[row >> 5];
        const int len = init == kZeroStart ? 0 : A.row_len[row];
#pragma unroll 2
        for (int j = 0; j < len; ++j) {
            const int64_t g = g0 + j;
            const int c = A.col[g * 32 + lane];
            const float4 xh = M.xt[3 * (size_t)c], xl = M.xt[3 * (size_t)c + 1], xr = M.xt[3 * (size_t)c + 2];
            const float* hv = A.v32 + (g * 9 + 3 * a) * 32 + lane;
            const float* lv = A.v32lo + (g * 9 + 3 * a) * 32 + lane;
            res_term(hv[0], lv[0], xh.x, xl.x, xr.x, Sm, Cc, Dd);
            res_term(hv[32], lv[32], xh.y, xl.y, xr.y, Sm, Cc, Dd);
            res_term(hv[64], lv[64], xh.z, xl.z, xr.z, Sm, Cc, Dd);
        }
        const size_t o = 3 * (size_t)row + a;
        // f - (S + C + D): the leading cancellation against f is exact in
        // the pairs' TwoSum; C and D enter below it
        const F2 y = f2_add(two_sum(Sm, Cc), F2{Dd, 0.f});
        const F2 rv = f2_add(f2_of(A.f[o]), f2_neg(y));
        st_pair(reinterpret_cast<float2*>(A.r), o, rv);
        M.b0[o] = rv.h;
        q = f2_mul(rv, rv);
    }
    sq[a][rl] = q;
    __syncthreads();
    if (a > 0) return;
    F2 rr{0.f, 0.f};
    double ff = 0.0;
    if (row < A.n_rows)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            rr = f2_add(rr, sq[k][rl]);
            if (init) {
                const double f = A.f[3 * (size_t)row + k];
                ff += f * f;
            }
        }
    double d[1][2] = {{f2_dbl(rr), ff}};
    double tot[1][2];
    if (last_block_reduce<1, 2>(A, d, 3, tot, kThreads) && threadIdx.x == 0) {
        RhsScalars& s = S[0];
        s.rr = tot[0][0];
        s.rr_last_true = tot[0][0];
        if (init) {
            s.bb = tot[0][1];
            s.target = tol2 * s.bb;
            s.iter = 0;
            s.beta = 0.0;
            s.restart = 1;
        }
        s.replace = 0;
        s.refresh = 1;
        s.nonfinite = isfinite(s.rr) ? 0 : 1;
        s.finished = (s.rr <= s.target) || s.nonfinite;
        s.done = s.finished;
    }
}

// e += alpha p, r -= alpha A p, b0 = r (FP32), |r|^2, and the level-0 first
// smoothing sweep.
__global__ void __launch_bounds__(kThreads) k_mg_update_xr_pair(MgPcg M) {
    pdl_begin();
    M = rhs_view<false>(M);
    const PcgArgs& A = M.a;
    RhsScalars* S = A.sc + cta_instance(A) * kMaxRhs;
    if (mg_done(A, S)) return;
    F2 rr{0.f, 0.f};
    const F2 alpha{S[0].alpha2[0], S[0].alpha2[1]};
    const RowRange rows = cg_range(M);
    for (int row = rows.begin; row < rows.end; row += rows.step) {
        F2 pv[3], xv[3];
        ld_pad_pair(A.p, row, pv);
        ld_pad_pair(M.xp, row, xv);
        const float2* ap = reinterpret_cast<const float2*>(A.ap);
        float2* r = reinterpret_cast<float2*>(A.r);
        float rf[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const size_t o = 3 * (size_t)row + q;
            xv[q] = f2_add(xv[q], f2_mul(alpha, pv[q]));
            const F2 rv = f2_add(ld_pair(r, o), f2_neg(f2_mul(alpha, ld_pair(ap, o))));
            st_pair(r, o, rv);
            M.b0[o] = rv.h;
            rf[q] = rv.h;
            rr = f2_add(rr, f2_mul(rv, rv));
        }
        st_pad_pair(M.xp, row, xv);
        const float* B = M.binv0 + 9 * (size_t)row;
        M.x40[row] = make_float4(B[0] * rf[0] + B[1] * rf[1] + B[2] * rf[2], B[3] * rf[0] + B[4] * rf[1] + B[5] * rf[2],
                                 B[6] * rf[0] + B[7] * rf[1] + B[8] * rf[2], 0.f);
    }
    double d[1][1] = {{f2_dbl(rr)}};
    double tot[1][1];
    if (last_block_reduce<1, 1>(A, d, 1, tot) && threadIdx.x == 0) {
        RhsScalars& s = S[0];
        s.rr = tot[0][0];
        s.iter += 1;
        if (!isfinite(s.rr)) {
            s.nonfinite = 1;
            s.done = 1;
        } else if (s.rr <= s.target) {
            s.done = 1;
            s.restart = 1;  // this iteration's p update is skipped
        }
        if (s.done) retire_instance(A);
    }
}

// r . z and (mode 0) A p . z in pairs, beta (Polak-Ribiere); mode 1: rz
// after a true-residual evaluation, and p = z on a restart.
__global__ void __launch_bounds__(kThreads) k_mg_rz_pair(MgPcg M, int mode) {
    pdl_begin();
    M = rhs_view<false>(M);
    const PcgArgs& A = M.a;
    RhsScalars* S = A.sc + cta_instance(A) * kMaxRhs;
    if (mode == 0 && mg_done(A, S)) return;
    if (mode == 1 && !S[0].refresh) return;
    const bool restart = mode == 1 && S[0].restart;
    F2 a0{0.f, 0.f}, a1{0.f, 0.f};
    const RowRange rows = cg_range(M);
    for (int row = rows.begin; row < rows.end; row += rows.step) {
        const float4 z = M.z[row];
        const float zz[3] = {z.x, z.y, z.z};
        const float2* r = reinterpret_cast<const float2*>(A.r);
        const float2* ap = reinterpret_cast<const float2*>(A.ap);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const size_t o = 3 * (size_t)row + q;
            a0 = f2_add(a0, f2_mul_f(ld_pair(r, o), zz[q]));
            if (mode == 0) a1 = f2_add(a1, f2_mul_f(ld_pair(ap, o), zz[q]));
        }
        if (restart) {
            const F2 pz[3] = {{zz[0], 0.f}, {zz[1], 0.f}, {zz[2], 0.f}};
            st_pad_pair(A.p, row, pz);
        }
    }
    double d[1][2] = {{f2_dbl(a0), f2_dbl(a1)}};
    double tot[1][2];
    if (last_block_reduce<1, 2>(A, d, 2, tot) && threadIdx.x == 0) {
        RhsScalars& s = S[0];
        if (mode == 0) {
            s.beta = -s.alpha * tot[0][1] / s.rz;
            const F2 b = f2_of(s.beta);
            s.beta2[0] = b.h;
            s.beta2[1] = b.l;
        }
        s.rz = tot[0][0];
        if (mode == 1) {
            s.refresh = 0;
            s.restart = 0;
        }
        if (!isfinite(s.rz)) {
            s.nonfinite = 1;
            if (!s.done) {
                s.done = 1;
                if (mode == 0) retire_instance(A);
            }
            s.finished = 1;
        }
    }
}

// p = z + beta p in pairs
__global__ void __launch_bounds__(kThreads) k_mg_update_p_pair(MgPcg M) {
    pdl_begin();
    M = rhs_view<false>(M);
    const PcgArgs& A = M.a;
    RhsScalars* S = A.sc + cta_instance(A) * kMaxRhs;
    if (mg_done(A, S)) return;
    const F2 beta{S[0].beta2[0], S[0].beta2[1]};
    const RowRange rows = cg_range(M);
    for (int row = rows.begin; row < rows.end; row += rows.step) {
        const float4 z = M.z[row];
        F2 pv[3];
        ld_pad_pair(A.p, row, pv);
        pv[0] = f2_add(f2_mul(beta, pv[0]), F2{z.x, 0.f});
        pv[1] = f2_add(f2_mul(beta, pv[1]), F2{z.y, 0.f});
        pv[2] = f2_add(f2_mul(beta, pv[2]), F2{z.z, 0.f});
        st_pad_pair(A.p, row, pv);
    }
}

// The split product with its values and columns staged through shared memory
// by bulk copies (spmv_row_split_staged): same rows per CTA, same results and
// the same pair epilogue and p.Ap reduction as k_mg_spmv_dot_pair.  A warp whose
// copies time out makes its rows' contribution NaN, which the solve reports
// as a non-finite breakdown.
template <int G, int S>
__global__ void __launch_bounds__(kThreads) k_mg_spmv_dot_staged(MgPcg M) {
    pdl_begin();
    extern __shared__ __align__(128) unsigned char st_smem[];
    M = rhs_view<false>(M);
    const PcgArgs& A = M.a;
    RhsScalars* Sc = A.sc + cta_instance(A) * kMaxRhs;
    if (mg_done(A, Sc)) return;
    F2 acc{0.f, 0.f};
    const bool ok = split_staged_slices<G, S>(
        A, A.p, st_smem, [&](int row, const F2 (&y)[3]) { acc = f2_add(acc, pair_ap_dot(A, row, y)); });
    double d[1][1] = {{f2_dbl(acc)}};
    if (!ok) d[0][0] = __longlong_as_double(0x7ff8000000000000ll);
    double tot[1][1];
    if (last_block_reduce<1, 1>(A, d, 0, tot) && threadIdx.x == 0) set_alpha(Sc[0], tot[0][0]);
}

// Launch of the split outer product: by default matrix-free where the blocks
// allow it; in one of its shapes on the assembled values (ASEND_PRODUCT_*)
// otherwise or when one is asked for: register-fed, or staged with G groups per
// stage and S stages per warp.
template <int G, int S>
void launch_staged(const Ctx& c, const MgPcg& M, dim3 grid) {
    launch_k(c, k_mg_spmv_dot_staged<G, S>, grid, kThreads, SplitStage<G, S>::smem(kThreads), M);
}

// Opt the staged shapes into their dynamic shared memory (above the 48 KB
// default) on the current device; called outside stream capture.
template <int G, int S>
void staged_attr() {
    ASEND_CUDA(cudaFuncSetAttribute(k_mg_spmv_dot_staged<G, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    SplitStage<G, S>::smem(kThreads)));
}
void product_attrs() {
    static bool done[64] = {};
    int dev = 0;
    ASEND_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && done[dev]) return;
    staged_attr<2, 3>();
    staged_attr<3, 2>();
    staged_attr<2, 2>();
    staged_attr<4, 2>();
    if (dev >= 0 && dev < 64) done[dev] = true;
}

void launch_split_product(Ctx& c, const MgPcg& M, dim3 grid) {
    if (c.product_variant == ASEND_PRODUCT_DEFAULT && c.mg->box) {  // 36.8 against 118 us (200 x 40 x 40)
        box_product(c, *c.mg->box, M.a, (int)grid.y, M.part_stride);
        return;
    }
    switch (c.product_variant) {
        case ASEND_PRODUCT_REGISTERS: launch_k(c, k_mg_spmv_dot_pair, grid, kThreads, 0, M); break;
        case ASEND_PRODUCT_STAGED_3x2: launch_staged<3, 2>(c, M, grid); break;
        case ASEND_PRODUCT_STAGED_2x2: launch_staged<2, 2>(c, M, grid); break;
        case ASEND_PRODUCT_STAGED_4x2: launch_staged<4, 2>(c, M, grid); break;
        default: launch_staged<2, 3>(c, M, grid); break;  // ASEND_PRODUCT_DEFAULT, ASEND_PRODUCT_STAGED_2x3
    }
}

template <typename TP>
__global__ void __launch_bounds__(kThreads) k_mg_update_xr(MgPcg M) {
    pdl_begin();
    using PV = typename ApOf<TP>::T;
    M = rhs_view<std::is_same<TP, float>::value>(M);
    const PcgArgs& A = M.a;
    RhsScalars* S = A.sc + cta_instance(A) * kMaxRhs;
    if (mg_done(A, S)) return;
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    double d[1][1] = {{0.0}};
    if (row < A.n_rows) {
        const double alpha = S[0].alpha;
        PV pv[3];
        PadVec<TP>::load(A.p, row, pv);
        const PV* ap = reinterpret_cast<const PV*>(A.ap) + 3 * (size_t)row;
        double rr[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const size_t o = 3 * (size_t)row + q;
            A.x[o] += alpha * (double)pv[q];
            const double rv = A.r[o] - alpha * (double)ap[q];
            A.r[o] = rv;
            M.b0[o] = (float)rv;
            rr[q] = rv;
            d[0][0] += rv * rv;
        }
        fused_smooth0(M, row, rr);
    }
    double tot[1][1];
    if (last_block_reduce<1, 1>(A, d, 1, tot) && threadIdx.x == 0) {
        RhsScalars& s = S[0];
        s.rr = tot[0][0];
        s.iter += 1;
        if (!isfinite(s.rr)) {
            s.nonfinite = 1;
            s.done = 1;
        } else if (s.rr <= s.target) {
            s.done = 1;
            s.restart = 1;  // this iteration's p update is skipped
        }
        if (s.done) retire_instance(A);
    }
}

// mode 0: after an iteration's V-cycle -> beta (Polak-Ribiere), rz
// mode 1: start of the solve, or after a true-residual evaluation: for every
//         instance whose refresh flag is set, rz, and p = z when its restart
//         flag is set (initialisation, or convergence of the recurrence)
template <typename TP>
__global__ void __launch_bounds__(kThreads) k_mg_rz(MgPcg M, int mode) {
    pdl_begin();
    using PV = typename ApOf<TP>::T;
    M = rhs_view<std::is_same<TP, float>::value>(M);
    const PcgArgs& A = M.a;
    RhsScalars* S = A.sc + cta_instance(A) * kMaxRhs;
    if (mode == 0 && mg_done(A, S)) return;
    if (mode == 1 && !S[0].refresh) return;
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    double d[1][2] = {{0.0, 0.0}};
    if (row < A.n_rows) {
        const float4 z = M.z[row];
        const double zz[3] = {z.x, z.y, z.z};
        const PV* ap = reinterpret_cast<const PV*>(A.ap) + 3 * (size_t)row;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            d[0][0] += zz[q] * A.r[3 * (size_t)row + q];
            if (mode == 0) d[0][1] += zz[q] * (double)ap[q];
        }
        if (mode == 1 && S[0].restart) PadVec<TP>::store(A.p, row, zz);
    }
    double tot[1][2];
    if (last_block_reduce<1, 2>(A, d, 2, tot) && threadIdx.x == 0) {
        RhsScalars& s = S[0];
        if (mode == 0) s.beta = -s.alpha * tot[0][1] / s.rz;
        s.rz = tot[0][0];
        if (mode == 1) {
            s.refresh = 0;
            s.restart = 0;
        }
        if (!isfinite(s.rz)) {
            s.nonfinite = 1;
            if (!s.done) {
                s.done = 1;
                if (mode == 0) retire_instance(A);
            }
            s.finished = 1;
        }
    }
}

template <typename TP>
__global__ void __launch_bounds__(kThreads) k_mg_update_p(MgPcg M) {
    pdl_begin();
    using PV = typename ApOf<TP>::T;
    M = rhs_view<std::is_same<TP, float>::value>(M);
    const PcgArgs& A = M.a;
    RhsScalars* S = A.sc + cta_instance(A) * kMaxRhs;
    if (mg_done(A, S)) return;
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= A.n_rows) return;
    const double beta = S[0].beta;
    const float4 z = M.z[row];
    PV pv[3];
    PadVec<TP>::load(A.p, row, pv);
    const double pn[3] = {z.x + beta * (double)pv[0], z.y + beta * (double)pv[1], z.z + beta * (double)pv[2]};
    PadVec<TP>::store(A.p, row, pn);
}

// FP64 true residual r = f - A64 x, b0 = float(r) for every instance
// (init = 1: also |f|^2, the target and fresh recurrence state) or for the
// instances whose replace flag is set (init = 0).  Marks them for the rz /
// direction refresh that follows the next V-cycle.
template <bool PAIR_R>
__global__ void __launch_bounds__(kThreads) k_mg_residual(MgPcg M, int init, double tol2) {
    pdl_begin();
    M = rhs_view<false>(M);
    const PcgArgs& A = M.a;
    RhsScalars* S = A.sc + cta_instance(A) * kMaxRhs;
    if (!init && !S[0].replace) return;
    double d[1][2] = {{0.0, 0.0}};
    for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < A.n_rows; row += gridDim.x * blockDim.x) {
        const int lane = row & 31;
        double y[3] = {0, 0, 0};
        const int64_t g0 = A.slice_off[row >> 5];
        const int len = init == kZeroStart ? 0 : A.row_len[row];
        for (int j = 0; j < len; ++j) {
            const int64_t g = g0 + j;
            const int c = A.col[g * 32 + lane];
            const double* v = A.v64 + (g * 9) * 32 + lane;
            const double x0 = A.x[3 * (size_t)c], x1 = A.x[3 * (size_t)c + 1], x2 = A.x[3 * (size_t)c + 2];
#pragma unroll
            for (int a = 0; a < 3; ++a) y[a] = fma(v[(a * 3) * 32], x0, fma(v[(a * 3 + 1) * 32], x1, fma(v[(a * 3 + 2) * 32], x2, y[a])));
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const size_t o = 3 * (size_t)row + a;
            const double rv = A.f[o] - y[a];
            if constexpr (PAIR_R) st_pair(reinterpret_cast<float2*>(A.r), o, f2_of(rv));  // split method
            else A.r[o] = rv;
            M.b0[o] = (float)rv;
            d[0][0] += rv * rv;
            d[0][1] += A.f[o] * A.f[o];
        }
    }
    double tot[1][2];
    if (last_block_reduce<1, 2>(A, d, 3, tot) && threadIdx.x == 0) {
        RhsScalars& s = S[0];
        s.rr = tot[0][0];
        s.rr_last_true = tot[0][0];
        if (init) {
            s.bb = tot[0][1];
            s.target = tol2 * s.bb;
            s.iter = 0;
            s.beta = 0.0;
            s.restart = 1;
        }
        s.replace = 0;
        s.refresh = 1;
        s.nonfinite = isfinite(s.rr) ? 0 : 1;
        s.finished = (s.rr <= s.target) || s.nonfinite;
        s.done = s.finished;
    }
}

// ---------------------------------------------------------------------------
// host: hierarchy construction
// ---------------------------------------------------------------------------
// Coarse-node positions on one axis: every second fine node (the last cell
// of an odd count is merged into its neighbour), or all of them when the axis
// is not coarsened at this level (semi-coarsening).
MgAxis make_axis(int n_f, bool coarsen) {
    MgAxis a;
    a.n_f = n_f;
    const int step = coarsen ? 2 : 1;
    for (int i = 0; i <= n_f; i += step) a.xs.push_back(i);
    if (a.xs.back() != n_f) a.xs.push_back(n_f);
    a.n_c = (int)a.xs.size() - 1;
    a.lo.assign(n_f + 1, 0);
    a.w.assign(n_f + 1, 0.f);
    for (int i = 0; i <= n_f; ++i) {
        const int m = (int)(std::upper_bound(a.xs.begin(), a.xs.end(), i) - a.xs.begin()) - 1;
        a.lo[i] = m;  // i == xs[m] gives weight 0 for m + 1 (never read)
        a.w[i] = (m < a.n_c) ? (float)(i - a.xs[m]) / (float)(a.xs[m + 1] - a.xs[m]) : 0.f;
    }
    return a;
}

// SBELL pattern, element connectivity, slot map and parity colouring of a
// level made of the blocks L.blk (nodes and elements numbered block by block;
// elements of different blocks share no node).
void level_pattern(Ctx& c, MgLevel& L) {
    const int N = L.n_nodes;
    std::vector<std::vector<int32_t>> adj(N);
    for (const MgBlk& B : L.blk) {
        auto id = [&](int i, int j, int k) { return B.node0 + (i * (B.ny + 1) + j) * (B.nz + 1) + k; };
        for (int i = 0; i <= B.nx; ++i)
            for (int j = 0; j <= B.ny; ++j)
                for (int k = 0; k <= B.nz; ++k) {
                    auto& v = adj[id(i, j, k)];
                    for (int di = -1; di <= 1; ++di)
                        for (int dj = -1; dj <= 1; ++dj)
                            for (int dk = -1; dk <= 1; ++dk) {
                                const int a = i + di, b = j + dj, q = k + dk;
                                if (a < 0 || b < 0 || q < 0 || a > B.nx || b > B.ny || q > B.nz) continue;
                                v.push_back(id(a, b, q));
                            }
                    std::sort(v.begin(), v.end());
                }
    }
    Sbell& A = L.own;
    A.b = 3;
    A.n_rows = N;
    A.n_slices = (N + kSlice - 1) / kSlice;
    A.h_slice_off.assign(A.n_slices + 1, 0);
    A.h_row_len.assign(N, 0);
    A.h_diag.assign(N, 0);
    for (int s = 0; s < A.n_slices; ++s) {
        A.h_slice_off[s + 1] = A.h_slice_off[s] + 27;  // known without the table (GeoView)
    }
    A.n_groups = A.h_slice_off[A.n_slices];
    A.h_col.assign((size_t)A.n_groups * kSlice, 0);
    for (int r = 0; r < N; ++r) {
        const int s = r / kSlice, lane = r % kSlice;
        const int64_t w = A.h_slice_off[s + 1] - A.h_slice_off[s];
        A.h_row_len[r] = (uint8_t)adj[r].size();
        for (int64_t j = 0; j < w; ++j) {
            const int col = (j < (int64_t)adj[r].size()) ? adj[r][j] : r;
            A.h_col[(size_t)(A.h_slice_off[s] + j) * kSlice + lane] = col;
            if (j < (int64_t)adj[r].size() && adj[r][j] == r) A.h_diag[r] = (uint8_t)j;
        }
    }
    A.slice_off.upload(A.h_slice_off, c.stream);
    A.col.upload(A.h_col, c.stream);
    A.row_len.upload(A.h_row_len, c.stream);
    A.diag.upload(A.h_diag, c.stream);
    A.v32.alloc((size_t)A.n_groups * 9 * kSlice);
    L.A = &L.own;
}

// Device block descriptors and per-block start tables of level l (levels
// >= 1 also describe the finer level's blocks).
void level_tables(Ctx& c, MgHierarchy& H, int l) {
    MgLevel& L = *H.L[l];
    const MgLevel* F = l > 0 ? H.L[l - 1].get() : nullptr;
    const int nb = (int)L.blk.size();
    std::vector<BlkDev> dv(nb);
    std::vector<int32_t> pn(nb + 1), pe(nb + 1);
    for (int b = 0; b < nb; ++b) {
        const MgBlk& B = L.blk[b];
        BlkDev& d = dv[b];
        std::memset(&d, 0, sizeof(d));
        d.nx = B.nx;
        d.ny = B.ny;
        d.nz = B.nz;
        d.node0 = B.node0;
        d.el0 = B.el0;
        if (F) {
            const MgBlk& P = F->blk[b];
            d.fnx = P.nx;
            d.fny = P.ny;
            d.fnz = P.nz;
            d.fnode0 = P.node0;
            d.fel0 = P.el0;
        }
        d.ox0 = B.ox[0];
        d.ox1 = B.ox[1];
        d.ox2 = B.ox[2];
        d.dense0 = (l + 1 == (int)H.L.size() && !H.h_dense0.empty()) ? H.h_dense0[b] : 0;
        pn[b] = B.node0;
        pe[b] = B.el0;
    }
    pn[nb] = L.n_nodes;
    pe[nb] = L.n_el;
    L.d_blk.upload(dv, c.stream);
    L.one = dv[0];
    if (nb > 1) {
        std::vector<int32_t> rb(L.n_nodes);
        for (int b = 0; b < nb; ++b) std::fill(rb.begin() + pn[b], rb.begin() + pn[b + 1], b);
        L.row_blk.upload(rb, c.stream);
    }
    L.pre_node.upload(pn, c.stream);
    L.pre_el.upload(pe, c.stream);
    ASEND_CUDA(cudaStreamSynchronize(c.stream));  // the host tables go out of scope
}

// The blocks of level C (with their finer blocks), found from the rows of R.
GeoView geo_of(const MgLevel& C, const MgLevel& R) {
    GeoView g{};
    g.n_rows = C.n_nodes;
    g.blk = C.d_blk.p;
    g.row_blk = C.blk.size() > 1 ? R.row_blk.p : nullptr;
    g.one = C.one;
    g.v = C.own.v32.p;
    return g;
}

LevelView view_of(const MgLevel& L) {
    LevelView v{};
    v.n_blk = (int)L.blk.size();
    v.blk = L.d_blk.p;
    v.xs = L.d_xs.p;
    return v;
}

SbView sbview(const MgLevel& L) {
    return SbView{L.A->n_rows, L.A->slice_off.p, L.A->row_len.p, L.A->col.p, L.A->v32.p};
}

// Level-0 blocks: the declared structured block, or one block per instance
// of a batched stack (asend_set_instance_blocks).
std::vector<MgBlk> level0_blocks(const Ctx& c) {
    std::vector<MgBlk> out;
    auto spacing = [&](MgBlk& B) {
        const int n100 = (B.ny + 1) * (B.nz + 1), n010 = B.nz + 1, n001 = 1;
        const int nb[3] = {n100, n010, n001};
        for (int ax = 0; ax < 3; ++ax) {
            double d2 = 0.0;
            for (int j = 0; j < 3; ++j) {
                const double d = c.xyz[3 * (size_t)(B.node0 + nb[ax]) + j] - c.xyz[3 * (size_t)B.node0 + j];
                d2 += d * d;
            }
            B.h[ax] = std::sqrt(d2);
        }
    };
    if (!c.inst_dims.empty()) {
        int el0 = 0;
        for (int i = 0; i < c.n_inst; ++i) {
            MgBlk B;
            B.nx = c.inst_dims[3 * i];
            B.ny = c.inst_dims[3 * i + 1];
            B.nz = c.inst_dims[3 * i + 2];
            B.node0 = c.inst_node_ptr[i];
            B.el0 = el0;
            el0 += B.n_el();
            spacing(B);
            out.push_back(B);
        }
    } else if (c.bx > 0) {
        MgBlk B;
        B.nx = c.bx;
        B.ny = c.by;
        B.nz = c.bz;
        spacing(B);
        out.push_back(B);
    }
    return out;
}

// The fused tail takes the levels below the finest of at most kTailRows rows whose
// vectors fit in a CTA's shared memory; values go there from the coarsest level up
// while they fit.  1,024 rows are one pass of the cluster's CTAs (64 rows of 16
// lanes each); a level that needs a second one is slower there than as launches:
// solves with a level of 595, 684, 882, 1,008 rows in the tail 1.17, 1.39, 1.39, 1.52
// ms (as launches 1.23, 1.46, 1.45, 1.57), of 1,056, 1,176, 1,392, 1,512, 1,680 rows
// 1.58, 1.51, 1.75, 1.52, 2.31 ms (1.58, 1.49, 1.72, 1.48, 2.18).
// Stacks keep one launch per level and step: a cluster per block needs more
// SMs than there are, and the blocks' rows fill them as it is.
void plan_tail(MgHierarchy& H) {
    const int nl = (int)H.L.size();
    if (H.n_blk != 1 || nl < 3) return;
    constexpr int kFloats = kTailSmem / 4;
    auto own = [&](int l) { return (H.L[l]->n_nodes + kTailCtas - 1) / kTailCtas; };
    auto up4 = [](int n) { return (n + 3) / 4 * 4; };
    int at = 0;
    TailView& V = H.tail;
    V = TailView{};
    std::vector<TailView::Level> lv;  // from the coarsest up
    for (int l = nl - 1; l >= 1 && nl - l <= kTailLevels; --l) {
        MgLevel& M = *H.L[l];
        const int n = M.n_nodes, o = own(l);
        TailView::Level L{M.one, M.own.v32.p, M.binv.p, n, o, 0, 0, 0, 0, 0, 0, -1};
        int off = at;
        auto take = [&](int floats) { const int p = off; off += up4(floats); return p; };
        L.xo = take(4 * n);
        L.ro = take(4 * n);
        L.to = take(o);
        if (l + 1 < nl) {
            L.so = take(12 * o);
            L.co = take((kTailCols * o + 1) / 2);
            L.po = take((n + 1) / 2);
        }
        if (off > kFloats || n > kTailRows) break;
        at = off;
        lv.push_back(L);
    }
    V.n = (int)lv.size();
    if (V.n < 2) return;
    for (int q = 0; q < V.n; ++q) {
        TailView::Level& L = V.L[V.n - 1 - q];
        L = lv[q];
        const int need = up4(L.own * kTailLd);
        if (q > 0 && at + need <= kFloats) {
            L.vo = at;
            at += need;
        }
    }
    H.tail0 = nl - V.n;
    H.tail_smem = 4 * at;
    ASEND_CUDA(cudaFuncSetAttribute(k_vc_tail, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    ASEND_CUDA(cudaFuncSetAttribute(k_vc_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailSmem));
}

// CTAs of the pair method's vector kernels on a stack: whole tiles of 128 rows of
// one instance, up to eight once that leaves two CTAs an SM.  A CTA's FP64
// sums hold the FP64 pipe for some 50 x 64 cycles whatever its rows: with a tile
// each, 1,606 tiles x 4 right-hand sides, they were two thirds of the kernels
// (r.z 28.1 us, now 16.3; x, r update 30.7, now 25.3).  Not a function of the number
// of right-hand sides: the sums' order is a case's own.
void vector_ctas(Ctx& c, MgHierarchy& H) {
    const int tiles = (c.n_nodes + kThreads - 1) / kThreads;
    const int per = std::max(1, std::min(8, tiles / (2 * 152))) * kThreads;
    std::vector<int32_t> inst, first, count;
    std::vector<int2> rows;
    for (int i = 0; i < c.n_inst; ++i) {
        const int end = i + 1 < c.n_inst ? c.inst_node_ptr[i + 1] : c.n_nodes;
        first.push_back((int32_t)rows.size());
        for (int r = c.inst_node_ptr[i]; r < end; r += per) {
            inst.push_back(i);
            rows.push_back(make_int2(r, std::min(r + per, end)));
        }
        count.push_back((int32_t)rows.size() - first.back());
    }
    H.cg_inst.upload(inst, c.stream);
    H.cg_cta0.upload(first, c.stream);
    H.cg_ncta.upload(count, c.stream);
    H.cg_rows.upload(rows, c.stream);
    ASEND_CUDA(cudaStreamSynchronize(c.stream));  // the host tables go out of scope
}

void build_hierarchy(Ctx& c) {
    if (c.type != 8 && c.type != 81)
        throw InputError("multigrid needs structured hex8 / brickIM blocks (asend_set_block_structure or "
                         "asend_set_instance_blocks)");
    std::vector<MgBlk> b0 = level0_blocks(c);
    if (b0.empty())
        throw InputError("multigrid needs structured hex8 / brickIM blocks (asend_set_block_structure or "
                         "asend_set_instance_blocks)");
    c.box.reset();  // (the blocks may be others than the last plan's)
    auto H = std::make_shared<MgHierarchy>();
    H->n_blk = (int)b0.size();
    auto L0 = std::make_unique<MgLevel>();
    L0->n_nodes = c.n_nodes;
    L0->n_el = c.n_el;
    L0->n_dof = c.n_dof;
    L0->blk = b0;
    L0->A = &c.A;
    // level-0 lumped penalty (coef^2 per constrained DOF, in units of the instance's scale)
    L0->h_pen.assign(c.n_dof, 0.f);
    for (size_t r = 0; r + 1 < c.c_ptr.size(); ++r)
        for (int k = c.c_ptr[r]; k < c.c_ptr[r + 1]; ++k) L0->h_pen[c.c_dof[k]] += (float)(c.c_coef[k] * c.c_coef[k]);
    H->L.push_back(std::move(L0));
    for (;;) {
        MgLevel& F = *H->L.back();
        // Per block: the coarsest grid is solved directly (<= 256 DOF);
        // semi-coarsening coarsens only the axes whose spacing is within a
        // factor sqrt(2) of the smallest (the strongly coupled directions of
        // stretched elements), the others wait until the cells are
        // isotropic.  An axis two cells thick is coarsened to one cell only
        // once every axis is that thin: a one-cell-thick coarse grid of a
        // deep bar is a poor coarse space.  A block that is done is carried
        // down unchanged while other blocks still coarsen.
        const int nb = (int)F.blk.size();
        std::vector<std::array<bool, 3>> co(nb);
        bool any_block = false;
        for (int b = 0; b < nb; ++b) {
            const MgBlk& P = F.blk[b];
            co[b] = {false, false, false};
            if (P.done || 3 * P.n_nodes() <= 256 || (P.nx <= 1 && P.ny <= 1 && P.nz <= 1)) continue;
            const int nf[3] = {P.nx, P.ny, P.nz};
            const bool all_thin = nf[0] <= 2 && nf[1] <= 2 && nf[2] <= 2;
            auto eligible = [&](int ax) { return nf[ax] >= 2 && (nf[ax] > 2 || all_thin); };
            double hmin = 1e300;
            for (int ax = 0; ax < 3; ++ax)
                if (eligible(ax)) hmin = std::min(hmin, P.h[ax]);
            for (int ax = 0; ax < 3; ++ax) {
                co[b][ax] = eligible(ax) && P.h[ax] <= 1.4142135623730951 * hmin;
                any_block |= co[b][ax];
            }
        }
        if (!any_block) break;
        auto L = std::make_unique<MgLevel>();
        std::vector<int32_t> xs;
        int node0 = 0, el0 = 0;
        for (int b = 0; b < nb; ++b) {
            const MgBlk& P = F.blk[b];
            MgBlk B;
            const int nf[3] = {P.nx, P.ny, P.nz};
            bool any = false;
            for (int ax = 0; ax < 3; ++ax) {
                B.ax[ax] = make_axis(nf[ax], co[b][ax]);
                B.h[ax] = P.h[ax] * (double)nf[ax] / (double)B.ax[ax].n_c;
                any |= co[b][ax];
            }
            B.done = !any;
            B.nx = B.ax[0].n_c;
            B.ny = B.ax[1].n_c;
            B.nz = B.ax[2].n_c;
            B.node0 = node0;
            B.el0 = el0;
            node0 += B.n_nodes();
            el0 += B.n_el();
            for (int ax = 0; ax < 3; ++ax) {
                B.ox[ax] = (int)xs.size();
                xs.insert(xs.end(), B.ax[ax].xs.begin(), B.ax[ax].xs.end());
            }
            L->blk.push_back(B);
        }
        L->n_nodes = node0;
        L->n_el = el0;
        L->n_dof = 3 * node0;
        L->d_xs.upload(xs, c.stream);
        // lumped Galerkin penalty: pen_c[I] = sum_i w_iI pen_f[i]
        L->h_pen.assign(L->n_dof, 0.f);
        for (int b = 0; b < nb; ++b) {
            const MgBlk& P = F.blk[b];
            const MgBlk& B = L->blk[b];
            for (int i = 0; i <= P.nx; ++i)
                for (int j = 0; j <= P.ny; ++j)
                    for (int k = 0; k <= P.nz; ++k) {
                        const int f = P.node0 + (i * (P.ny + 1) + j) * (P.nz + 1) + k;
                        const float p0 = F.h_pen[3 * f], p1 = F.h_pen[3 * f + 1], p2 = F.h_pen[3 * f + 2];
                        if (p0 == 0.f && p1 == 0.f && p2 == 0.f) continue;
                        const int li[3] = {B.ax[0].lo[i], B.ax[1].lo[j], B.ax[2].lo[k]};
                        const float wi[3] = {B.ax[0].w[i], B.ax[1].w[j], B.ax[2].w[k]};
                        for (int d0 = 0; d0 < 2; ++d0)
                            for (int d1 = 0; d1 < 2; ++d1)
                                for (int d2 = 0; d2 < 2; ++d2) {
                                    const float ww = (d0 ? wi[0] : 1 - wi[0]) * (d1 ? wi[1] : 1 - wi[1]) *
                                                     (d2 ? wi[2] : 1 - wi[2]);
                                    if (ww == 0.f) continue;
                                    const int I = B.node0 +
                                                  ((li[0] + d0) * (B.ny + 1) + (li[1] + d1)) * (B.nz + 1) + (li[2] + d2);
                                    L->h_pen[3 * I] += ww * p0;
                                    L->h_pen[3 * I + 1] += ww * p1;
                                    L->h_pen[3 * I + 2] += ww * p2;
                                }
                    }
        }
        level_pattern(c, *L);
        L->Ke.alloc((size_t)L->n_el * 576);
        H->L.push_back(std::move(L));
    }
    for (auto& Lp : H->L) {
        MgLevel& L = *Lp;
        L.pen.upload(L.h_pen, c.stream);
        L.binv.alloc((size_t)9 * L.n_nodes);
        L.b.alloc(L.n_dof);
        L.r.alloc(L.n_dof);
        L.x4.alloc((size_t)4 * L.n_nodes);
        L.y4.alloc((size_t)4 * L.n_nodes);
    }
    // coarsest level: one dense block per instance
    MgLevel& Lc = *H->L.back();
    H->h_dense0.assign(H->n_blk, 0);
    size_t dense_tot = 0;
    H->n_coarse = 0;
    for (int b = 0; b < H->n_blk; ++b) {
        const int nd = 3 * Lc.blk[b].n_nodes();
        H->h_dense0[b] = (int32_t)dense_tot;
        dense_tot += (size_t)nd * nd;
        H->n_coarse = std::max(H->n_coarse, nd);
    }
    if (H->n_coarse > kGjN) throw InputError("multigrid coarsest level too large");  // not by the rule above
    if (dense_tot > (size_t)INT32_MAX) throw InputError("multigrid coarsest blocks too large");
    H->dense.alloc(dense_tot);
    for (int l = 0; l < (int)H->L.size(); ++l) level_tables(c, *H, l);
    plan_tail(*H);
    if (c.n_inst > 1) vector_ctas(c, *H);
    ASEND_CUDA(cudaStreamSynchronize(c.stream));
    c.mg = H;
}

void damp_smoother(Ctx& c, int l) {
    MgHierarchy& H = *c.mg;
    MgLevel& L = *H.L[l];
    float* nrm = H.pow_nrm.p + (size_t)l * (kPowSteps + 1);
    uint32_t* tk = H.pow_ticket.p + (size_t)l * kPowSteps;
    float4* xa = reinterpret_cast<float4*>(L.x4.p);
    float4* xb = reinterpret_cast<float4*>(L.y4.p);
    const int g = grid_of(L.n_nodes);
    // later assemblies start from the previous dominant vector (the operator
    // changes little between assemblies of one hierarchy): fewer steps
    const bool warm = L.pow_warm;
    const int steps = warm ? kPowWarmSteps : kPowSteps;
    if (L.pow_vec.n != (size_t)4 * L.n_nodes) L.pow_vec.alloc((size_t)4 * L.n_nodes);
    ASEND_CUDA(cudaMemsetAsync(tk, 0, sizeof(uint32_t) * kPowSteps, c.stream));
    if (l == 0) ASEND_CUDA(cudaMemsetAsync(H.pow_bound.p, 0, sizeof(unsigned int), c.stream));
    if (warm)
        ASEND_CUDA(cudaMemcpyAsync(xa, L.pow_vec.p, sizeof(float) * 4 * L.n_nodes, cudaMemcpyDeviceToDevice,
                                   c.stream));
    k_pow_init<<<g, kT, 0, c.stream>>>(L.n_nodes, xa, nrm, warm ? 0 : 1);
    BoxPlan* box = l == 0 ? H.box : nullptr;
    for (int k = 0; k < steps; ++k) {
        if (box) box_power(c, *box, L.binv.p, xa, xb, nrm, k, H.pow_part.p, tk);
        else if (l > 0 && L.n_nodes < kStagedRows)
            k_pow_rows<<<grid_of(4 * L.n_nodes), kT, 0, c.stream>>>(geo_of(L, L), L.binv.p, xa, xb, nrm, k,
                                                                    H.pow_part.p, tk);
        else k_pow_step<<<g, kT, 0, c.stream>>>(sbview(L), L.binv.p, xa, xb, nrm, k, H.pow_part.p, tk);
        std::swap(xa, xb);
    }
    ASEND_CUDA(cudaMemcpyAsync(L.pow_vec.p, xa, sizeof(float) * 4 * L.n_nodes, cudaMemcpyDeviceToDevice, c.stream));
    L.pow_warm = true;
    L.pow_steps = steps;
    unsigned int* bound = H.pow_bound.p + l;
    if (l == 0) k_inf_bound<<<g, kT, 0, c.stream>>>(sbview(L), L.binv.p, bound);  // else with the values
    k_scale_blocks<<<(9 * L.n_nodes + 255) / 256, 256, 0, c.stream>>>(L.n_nodes, L.binv.p, nrm, steps, bound,
                                                                       H.safe_damping ? 1 : 0, c.mg_damping,
                                                                       H.pow_omega.p + l);
    c.launches += steps + 2 + (l == 0);
}

// per-assembly values: Galerkin element matrices, level operators, penalty,
// smoother blocks, coarsest inverses
// Level-0 smoother blocks (undamped D_n^-1) from the FP64 values, or from the
// FP32 values after a split-only assembly (the smoother is FP32 either way).
void level0_smoother_blocks(Ctx& c, MgLevel& L0) {
    if (c.v64_valid)
        k_smoother_blocks<double><<<grid_of(L0.n_nodes), kT, 0, c.stream>>>(L0.n_nodes, c.A.slice_off.p, c.A.diag.p,
                                                                            c.A.v64.p, nullptr, L0.binv.p);
    else
        k_smoother_blocks<float><<<grid_of(L0.n_nodes), kT, 0, c.stream>>>(L0.n_nodes, c.A.slice_off.p, c.A.diag.p,
                                                                           c.A.v32.p, c.diag64 ? c.A.v32lo.p : nullptr,
                                                                           L0.binv.p);
}

// Per-assembly multigrid values.  skip_l0: the solve takes its finest-level
// smoother blocks from the learned model, so the finest level's eigenvalue
// estimate (its power iteration, the largest of the set-up) is not made.
void setup_values(Ctx& c, bool skip_l0) {
    MgHierarchy& H = *c.mg;
    const int n_lev = (int)H.L.size();
    H.pow_nrm.alloc((size_t)n_lev * (kPowSteps + 1));
    H.pow_bound.alloc((size_t)n_lev);
    H.pow_omega.alloc((size_t)n_lev);
    H.pow_bound.zero(c.stream);
    H.pow_omega.zero(c.stream);
    H.pow_ticket.alloc((size_t)n_lev * kPowSteps);
    int pow_ctas = std::max(grid_of(H.L[0]->n_nodes), H.box ? box_ctas(*H.box) : 0);
    for (int l = 1; l < n_lev; ++l)
        pow_ctas = std::max(pow_ctas, grid_of((H.L[l]->n_nodes < kStagedRows ? 4 : 1) * H.L[l]->n_nodes));
    H.pow_part.alloc((size_t)pow_ctas);
    {
        std::vector<double> sf(H.n_blk, c.sf);
        if (c.n_inst > 1 && (int)c.sf_inst.size() == H.n_blk) sf = c.sf_inst;
        H.blk_sf.upload(sf, c.stream);
    }
    if (!skip_l0) {
        MgLevel& L0 = *H.L[0];
        level0_smoother_blocks(c, L0);
        ++c.launches;
        if (n_lev > 1) damp_smoother(c, 0);
    }
    H.l0_damped = !skip_l0;
    for (size_t l = 1; l < H.L.size(); ++l) {
        MgLevel& L = *H.L[l];
        MgLevel& F = *H.L[l - 1];
        const float* fine_ke = F.Ke.p;
        const float* cls_ke = nullptr;
        const int32_t* cls_of = nullptr;
        if (l == 1) {
            // level 0: K_e = E_e * (unit-modulus matrix of its geometry class)
            // when the assembly keeps classes; otherwise hex8 matrices are
            // integrated inside k_coarsen and brickIM ones (condensed
            // incompatible modes) are computed first
            fine_ke = nullptr;
            if (c.cls_ke32.n && c.cls_type == c.type && c.ortho.empty()) {
                cls_ke = c.cls_ke32.p;
                cls_of = c.d_cls_of.p;
            } else if (c.type == 81) {
                F.Ke.alloc((size_t)c.n_el * 576);
                brickim_element_ke32(c, F.Ke.p);
                fine_ke = F.Ke.p;
            }
        }
        if (l == 1 && cls_ke && c.n_cls <= kMaxChildClasses) {
            if (!H.child_ready) {
                H.child.alloc((size_t)c.n_cls * 27 * 576);
                k_child_mats<<<dim3(27, c.n_cls), 256, 0, c.stream>>>(c.cls_ke.p, H.child.p);
                ++c.launches;
                H.child_ready = true;
            }
            k_coarsen_lin<<<L.n_el, 144, 0, c.stream>>>(view_of(L), L.pre_el.p, c.d_E.p, cls_of, H.child.p, L.Ke.p);
        } else {
            k_coarsen<<<L.n_el, kCoarsenThreads, 0, c.stream>>>(view_of(L), L.pre_el.p, fine_ke, cls_ke, cls_of, c.d_xyz.p,
                                                    c.d_conn.p, c.d_E.p, c.d_nu.p, L.Ke.p);
        }
        const bool lone = L.blk.size() == 1;
        k_level_values<<<L.own.n_slices, kValThreads, kValSmem, c.stream>>>(
            L.n_nodes, L.d_blk.p, lone ? nullptr : L.row_blk.p, L.one, L.Ke.p, L.pen.p, H.blk_sf.p, L.own.v32.p,
            L.binv.p, l + 1 < H.L.size() ? H.pow_bound.p + l : nullptr);
        c.launches += 2;
        if (l + 1 < H.L.size()) damp_smoother(c, (int)l);  // the coarsest level is solved directly
    }
    MgLevel& Lc = *H.L.back();
    k_dense_build<<<Lc.n_nodes, 128, 0, c.stream>>>(Lc.n_nodes, Lc.A->slice_off.p, Lc.A->row_len.p, Lc.A->col.p,
                                                    Lc.A->v32.p, view_of(Lc), Lc.pre_node.p, H.dense.p);
    ASEND_CUDA(cudaFuncSetAttribute(k_gauss_jordan, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGjSmem));
    k_gauss_jordan<<<H.n_blk * kGjCtas, kGjThreads, kGjSmem, c.stream>>>(view_of(Lc), H.dense.p);
    c.launches += 2;
    ASEND_CUDA(cudaGetLastError());
    H.epoch = c.assembly_epoch;
}

// Restriction of level l's residual r to level l + 1's right-hand side b (and
// its first smoothing sweep, unless l + 1 is the coarsest level).
void restrict_to(Ctx& c, int l, const Control* ctl, int nr = 1) {
    MgHierarchy& H = *c.mg;
    MgLevel& L = *H.L[l];
    MgLevel& C = *H.L[l + 1];
    const bool last = (l + 2 == (int)H.L.size());  // the coarsest level is solved directly: no sweep
    launch_k(c, C.n_nodes >= kStagedRows ? k_vc_restrict<true> : k_vc_restrict<false>, dim3(grid_of(4 * C.n_nodes), nr), kT,
             0, geo_of(C, C), L.n_nodes, L.r.p, C.b.p, last ? nullptr : C.binv.p, reinterpret_cast<float4*>(C.x4.p), ctl);
}

void coarsest_solve(Ctx& c, const Control* ctl, int nr = 1) {
    MgHierarchy& H = *c.mg;
    MgLevel& Lc = *H.L.back();
    launch_k(c, k_vc_dense, dim3(H.n_blk, nr, (H.n_coarse + kDenseRows - 1) / kDenseRows), 32 * kDenseRows, 0,
             geo_of(Lc, Lc), H.dense.p, Lc.b.p, Lc.y4.p, ctl);
}

void prolong_from(Ctx& c, int l, const Control* ctl, int nr = 1) {
    MgHierarchy& H = *c.mg;
    MgLevel& L = *H.L[l];
    MgLevel& C = *H.L[l + 1];
    launch_k(c, k_vc_prolong, dim3(grid_of(L.n_nodes), nr), kT, 0, geo_of(C, L), L.n_nodes,
             reinterpret_cast<const float4*>(C.y4.p), reinterpret_cast<float4*>(L.x4.p), ctl);
}

// One V(1,1) cycle on level 0's b.  With fused0, the caller has already
// written level 0's first sweep x4 = B^-1 b (fused into the PCG update).
// Residual r = b - A x (post = false) or post-smoothing y4 = x + B^-1 (b - A x) of
// level l for nr right-hand sides: matrix-free on the finest level of a box
// model inside the CG, staged for many rows, several lanes a row for few.
void level_rows(Ctx& c, int l, bool post, const Control* ctl, int nr = 1) {
    MgHierarchy& H = *c.mg;
    MgLevel& L = *H.L[l];
    const float4* x = reinterpret_cast<const float4*>(L.x4.p);
    float4* y = reinterpret_cast<float4*>(L.y4.p);
    if (l == 0 && H.box && H.box_cycle) {
        if (post) box_post(c, *H.box, L.binv.p, L.b.p, x, y, ctl, nr);
        else box_resid(c, *H.box, L.b.p, x, L.r.p, ctl, nr);
        return;
    }
    if (L.n_nodes < kStagedRows) {  // 16 lanes a row
        const dim3 g((unsigned)grid_of(16 * L.n_nodes), nr);
        if (l > 0) {
            const GeoView G = geo_of(L, L);
            if (post) launch_k(c, k_vc_rows<16, true>, g, kT, 0, G, L.binv.p, L.b.p, x, L.r.p, y, ctl);
            else launch_k(c, k_vc_rows<16, false>, g, kT, 0, G, L.binv.p, L.b.p, x, L.r.p, y, ctl);
        } else {  // a small finest level: any pattern
            const SbView A = sbview(L);
            if (post) launch_k(c, k_vc_rows_any<16, true>, g, kT, 0, A, L.binv.p, L.b.p, x, L.r.p, y, ctl);
            else launch_k(c, k_vc_rows_any<16, false>, g, kT, 0, A, L.binv.p, L.b.p, x, L.r.p, y, ctl);
        }
        return;
    }
    // four right-hand sides by one reading of the values once every warp of the
    // persistent grid has a slice (91,000 rows: a residual 44 -> 35 us, a
    // post-smoothing 39 -> 32), else by a grid each (16,500 rows: 9.8 us, by one
    // reading 14.9: a quarter of the warps)
    const bool together = nr > 1 && L.n_nodes >= kPersistCtas * kT;
    const dim3 grid(std::min(grid_of(L.n_nodes), kPersistCtas), together ? 1 : nr);
    const size_t smem = (size_t)F32Stage<kVcG, kVcS>::smem(kT);
    if (post)
        launch_k(c, together ? k_vc_post_staged<kMaxRhs> : k_vc_post_staged<1>, grid, kT, smem, sbview(L), L.binv.p, L.b.p, x, y,
                 ctl, nr);
    else
        launch_k(c, together ? k_vc_resid_staged<kMaxRhs> : k_vc_resid_staged<1>, grid, kT, smem, sbview(L), L.b.p, x, L.r.p, ctl,
                 nr);
}

void fused_tail(Ctx& c, const Control* ctl, int nr) {
    MgHierarchy& H = *c.mg;
    TailView V = H.tail;
    MgLevel& T = *H.L[H.tail0];
    V.b = T.b.p;
    V.x4 = reinterpret_cast<const float4*>(T.x4.p);
    V.y4 = reinterpret_cast<float4*>(T.y4.p);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kTailCtas, (unsigned)nr);
    cfg.blockDim = dim3(kTailThreads);
    cfg.dynamicSmemBytes = (size_t)H.tail_smem;
    cfg.stream = c.stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {kTailCtas, 1, 1};
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = c.pdl ? 2 : 1;
    ASEND_CUDA(cudaLaunchKernelEx(&cfg, k_vc_tail, V, (const float*)H.dense.p, ctl));
}

void vcycle(Ctx& c, const Control* ctl, bool fused0, int nr = 1) {
    MgHierarchy& H = *c.mg;
    const int nl = (int)H.L.size();
    if (!fused0 && nl > 1) {
        MgLevel& L = *H.L[0];
        launch_k(c, k_vc_smooth0, dim3(grid_of(L.n_nodes), nr), kT, 0, L.n_nodes, L.binv.p, L.b.p,
                 reinterpret_cast<float4*>(L.x4.p), ctl);
    }
    const int top = c.mg_tail && H.tail0 ? H.tail0 : nl - 1;
    for (int l = 0; l < top; ++l) {
        level_rows(c, l, false, ctl, nr);
        restrict_to(c, l, ctl, nr);
    }
    if (top < nl - 1) fused_tail(c, ctl, nr);
    else coarsest_solve(c, ctl, nr);
    for (int l = top - 1; l >= 0; --l) {
        prolong_from(c, l, ctl, nr);
        level_rows(c, l, true, ctl, nr);
    }
}

int vcycle_launches(const Ctx& c) {
    return 4 * (c.mg_tail && c.mg->tail0 ? c.mg->tail0 : (int)c.mg->L.size() - 1) + 1;
}

// Level vectors for nr right-hand sides (grow only; the captured graphs hold
// their addresses).
void level_vectors(MgHierarchy& H, int nr) {
    for (auto& Lp : H.L) {
        MgLevel& L = *Lp;
        if (L.b.n >= (size_t)nr * L.n_dof) continue;
        for (auto& g : H.graphs) cudaGraphExecDestroy(g.second);
        H.graphs.clear();
        L.b.alloc((size_t)nr * L.n_dof);
        L.r.alloc((size_t)nr * L.n_dof);
        L.x4.alloc((size_t)nr * 4 * L.n_nodes);
        L.y4.alloc((size_t)nr * 4 * L.n_nodes);
    }
}

// L0.x4 = P C R (L0.r): the coarse-grid correction of one V-cycle alone
// (restriction of level 0's r, the V-cycle of the coarser levels, and the
// prolongation into a zeroed level-0 vector; no level-0 smoothing).
void coarse_correction(Ctx& c) {
    MgHierarchy& H = *c.mg;
    const int nl = (int)H.L.size();
    MgLevel& L0 = *H.L[0];
    for (int l = 0; l < nl - 1; ++l) {
        MgLevel& L = *H.L[l];
        if (l > 0)
            launch_k(c, k_vc_resid, grid_of(L.n_nodes), kT, 0, sbview(L), L.b.p, reinterpret_cast<float4*>(L.x4.p),
                                                                L.r.p, nullptr);
        restrict_to(c, l, nullptr);
    }
    coarsest_solve(c, nullptr);
    ASEND_CUDA(cudaMemsetAsync(L0.x4.p, 0, sizeof(float) * 4 * L0.n_nodes, c.stream));
    for (int l = nl - 2; l >= 0; --l) {
        MgLevel& L = *H.L[l];
        prolong_from(c, l, nullptr);
        if (l > 0)
            launch_k(c, k_vc_post, grid_of(L.n_nodes), kT, 0, sbview(L), L.binv.p, L.b.p,
                                                               reinterpret_cast<const float4*>(L.x4.p),
                                                               reinterpret_cast<float4*>(L.y4.p), nullptr);
    }
    c.launches += 6 * (nl - 1) - 1;
}


}  // namespace

void mg_invalidate_values(Ctx& c) {
    if (c.mg) c.mg->epoch = -1;
}

void mg_prepare(Ctx& c, bool learned) {
    product_attrs();
    if (!c.mg) build_hierarchy(c);
    {
        std::vector<std::array<int, 5>> blocks;
        for (const MgBlk& b : c.mg->L[0]->blk) blocks.push_back({b.nx, b.ny, b.nz, b.node0, b.el0});
        c.mg->box = box_plan(c, blocks);
    }
    if (c.mg->epoch != c.assembly_epoch) {
        setup_values(c, learned);
        c.mg->l0_learned = false;
    }
}

// Finest-level smoother blocks: damped block Jacobi (omega D_n^-1, omega from
// the eigenvalue estimate), or the
// learned nodal blocks M_n (recomputed on every request, since the weights
// may have changed since the last one).
void mg_select_smoother(Ctx& c, bool learned) {
    MgHierarchy& H = *c.mg;
    MgLevel& L0 = *H.L[0];
    if (learned) {
        learned_blocks(c, L0.binv.p, true);
        H.l0_learned = true;
    } else if (H.l0_learned || !H.l0_damped) {
        level0_smoother_blocks(c, L0);
        ++c.launches;
        if (H.L.size() > 1) damp_smoother(c, 0);
        H.l0_learned = false;
        H.l0_damped = true;
    }
}

void mg_apply(Ctx& c, const float* d_b, float* d_z4) {
    mg_prepare(c);
    mg_select_smoother(c, false);
    MgLevel& L0 = *c.mg->L[0];
    ASEND_CUDA(cudaMemcpyAsync(L0.b.p, d_b, sizeof(float) * c.n_dof, cudaMemcpyDeviceToDevice, c.stream));
    vcycle(c, nullptr, false);
    ASEND_CUDA(cudaMemcpyAsync(d_z4, L0.y4.p, sizeof(float) * 4 * c.n_nodes, cudaMemcpyDeviceToDevice, c.stream));
    c.launches += vcycle_launches(c);
}

int mg_levels(const Ctx& c) { return c.mg ? (int)c.mg->L.size() : 0; }

// Mean device time of n_launch back-to-back launches of one kernel of the
// multigrid CG (0: outer product + p.Ap in the method's value format; 1:
// level-0 V-cycle residual; 2: level-0 post-smoothing) and its algorithmic
// bytes per launch.  Scratch scalars keep the kernels from exiting early.
double mg_time_kernel(Ctx& c, int kernel, int method, int n_launch, double* bytes) {
    ensure_v64(c);
    mg_prepare(c);
    mg_select_smoother(c, false);
    MgHierarchy& H = *c.mg;
    const BoxCycle box_cycle(H);
    MgLevel& L0 = *H.L[0];
    const int n = c.A.n_rows, nd = c.n_dof;
    const int grid = (method == ASEND_METHOD_SPLIT && kernel == 0) ? std::min(grid_of(n), kPersistCtas) : grid_of(n);
    const double blocks = (double)(c.A.nnz_scalar() / 9);
    if (kernel != 0 && H.L.size() < 2) throw InputError("multigrid hierarchy has a single level");
    DArr<RhsScalars> sc;
    DArr<Control> ctl;
    DArr<double> part, p, ap;
    const int NI = std::max(1, c.n_inst);
    DArr<uint32_t> tk;
    sc.alloc((size_t)NI * kMaxRhs);
    ctl.alloc(1);
    tk.alloc((size_t)NI * 4);
    sc.zero(c.stream);
    Control on;
    std::memset(&on, 0, sizeof(on));
    on.active[0] = 1;  // or the kernels would have nothing to do
    ctl.upload(&on, 1, c.stream);
    tk.zero(c.stream);
    part.alloc((size_t)std::max(grid, H.box ? box_ctas(*H.box) : 0) * kMaxRhs * 3);
    p.alloc((size_t)4 * n);
    ap.alloc(nd);
    MgPcg M;
    std::memset(&M, 0, sizeof(M));
    PcgArgs& a = M.a;
    a.n_rows = n;
    a.nrhs = 1;
    a.n_dof = nd;
    a.slice_off = c.A.slice_off.p;
    a.row_len = c.A.row_len.p;
    a.col = c.A.col.p;
    a.v32 = c.A.v32.p;
    a.v32lo = c.A.v32lo.p;
    a.v64 = c.A.v64.p;
    a.p = p.p;
    a.ap = ap.p;
    a.partials = part.p;
    a.sc = sc.p;
    a.ctl = ctl.p;
    a.tickets = tk.p;
    M.n_inst = 1;
    M.part_stride = 0;
    // the direction's values do not change the kernels' work: zeros
    ASEND_CUDA(cudaMemsetAsync(p.p, 0, sizeof(double) * 4 * n, c.stream));
    auto launch = [&]() {
        if (kernel == 0) {
            if (method == ASEND_METHOD_MIXED) k_mg_spmv_dot<float, float><<<grid, kThreads, 0, c.stream>>>(M);
            else if (method == ASEND_METHOD_SPLIT) launch_split_product(c, M, grid);
            else k_mg_spmv_dot<double, double><<<grid, kThreads, 0, c.stream>>>(M);
        } else {  // the finest level's products as the V-cycle runs them
            level_rows(c, 0, kernel == 2, nullptr);
        }
    };
    const double ps = (method == ASEND_METHOD_MIXED) ? 4.0 : 8.0;  // bytes per value / direction entry
    if (kernel == 0) *bytes = blocks * (9.0 * ps + 4.0) + (double)n * 4.0 * ps + (double)nd * ps;
    else if (kernel == 1) *bytes = blocks * 40.0 + (double)n * 16.0 + (double)nd * 8.0;
    else *bytes = blocks * 40.0 + (double)n * (16.0 + 36.0 + 16.0) + (double)nd * 4.0;
    if (H.box && (kernel > 0 || (method == ASEND_METHOD_SPLIT && c.product_variant == ASEND_PRODUCT_DEFAULT)))
        *bytes = kernel == 0 ? box_product_bytes(c)
                             : 8.0 * c.n_el + (double)n * (kernel == 1 ? 16.0 : 68.0) + (double)nd * (kernel == 1 ? 8.0 : 4.0);
    for (int w = 0; w < 3; ++w) launch();
    ASEND_CUDA(cudaEventRecord(c.ev0, c.stream));
    for (int i = 0; i < n_launch; ++i) launch();
    ASEND_CUDA(cudaEventRecord(c.ev1, c.stream));
    ASEND_CUDA(cudaEventSynchronize(c.ev1));
    ASEND_CUDA(cudaGetLastError());
    float ms = 0.f;
    ASEND_CUDA(cudaEventElapsedTime(&ms, c.ev0, c.ev1));
    c.launches += n_launch + 3;
    return ms / n_launch;
}

// per-level diagnostics: dims (nx, ny, nz), power estimate and guaranteed
// bound of lambda_max(D^-1 A), damping in use (the coarsest level: zeros)
void mg_level_info(Ctx& c, int level, int32_t* dims, double* lam_est, double* lam_bound, double* omega) {
    if (!c.mg || level < 0 || level >= (int)c.mg->L.size()) throw InputError("no such multigrid level");
    MgHierarchy& H = *c.mg;
    MgLevel& L = *H.L[level];
    if (dims) {  // the first block (instance 0)
        dims[0] = L.blk[0].nx;
        dims[1] = L.blk[0].ny;
        dims[2] = L.blk[0].nz;
    }
    float nrm = 0.f, om = 0.f;
    unsigned int bb = 0;
    if (H.pow_nrm.n) {
        ASEND_CUDA(cudaMemcpyAsync(&nrm, H.pow_nrm.p + (size_t)level * (kPowSteps + 1) + L.pow_steps, sizeof(float),
                                   cudaMemcpyDeviceToHost, c.stream));
        ASEND_CUDA(cudaMemcpyAsync(&bb, H.pow_bound.p + level, sizeof(unsigned int), cudaMemcpyDeviceToHost, c.stream));
        ASEND_CUDA(cudaMemcpyAsync(&om, H.pow_omega.p + level, sizeof(float), cudaMemcpyDeviceToHost, c.stream));
        ASEND_CUDA(cudaStreamSynchronize(c.stream));
    }
    float bf;
    std::memcpy(&bf, &bb, sizeof(float));
    if (lam_est) *lam_est = nrm;
    if (lam_bound) *lam_bound = bf;
    if (omega) *omega = om;
}

// z = V(b) with the current finest-level smoother, host FP32 vectors [n_dof]
void mg_vcycle_host(Ctx& c, const float* b, float* z) {
    mg_prepare(c);
    MgHierarchy& H = *c.mg;
    MgLevel& L0 = *H.L[0];
    if (H.L.size() < 2) throw InputError("multigrid hierarchy has a single level");
    ASEND_CUDA(cudaMemcpyAsync(L0.b.p, b, sizeof(float) * c.n_dof, cudaMemcpyHostToDevice, c.stream));
    vcycle(c, nullptr, false);
    c.launches += vcycle_launches(c);
    std::vector<float> y4((size_t)4 * c.n_nodes);
    ASEND_CUDA(cudaMemcpyAsync(y4.data(), L0.y4.p, sizeof(float) * y4.size(), cudaMemcpyDeviceToHost, c.stream));
    ASEND_CUDA(cudaStreamSynchronize(c.stream));
    for (int i = 0; i < c.n_nodes; ++i)
        for (int a = 0; a < 3; ++a) z[3 * (size_t)i + a] = y4[4 * (size_t)i + a];
}

// r := (I - A V)^k r on a host FP32 vector [n_dof] with the finest-level
// smoother in force (learned or damped): the residual after k stationary
// V-cycle iterations, dominated by the modes the V-cycle reduces slowest.
void mg_stationary_residual(Ctx& c, float* r_host, int k, bool learned_smoother) {
    mg_prepare(c);
    mg_select_smoother(c, learned_smoother);
    MgHierarchy& H = *c.mg;
    MgLevel& L0 = *H.L[0];
    if (H.L.size() < 2) throw InputError("multigrid hierarchy has a single level");
    if (H.vl_w.n != (size_t)c.n_dof) H.vl_w.alloc(c.n_dof);
    ASEND_CUDA(cudaMemcpyAsync(H.vl_w.p, r_host, sizeof(float) * c.n_dof, cudaMemcpyHostToDevice, c.stream));
    const int g = grid_of(L0.n_nodes);
    for (int i = 0; i < k; ++i) {
        ASEND_CUDA(cudaMemcpyAsync(L0.b.p, H.vl_w.p, sizeof(float) * c.n_dof, cudaMemcpyDeviceToDevice, c.stream));
        vcycle(c, nullptr, false);
        k_vl_rstep<<<g, kT, 0, c.stream>>>(sbview(L0), reinterpret_cast<const float4*>(L0.y4.p), H.vl_w.p);
        c.launches += vcycle_launches(c) + 1;
    }
    ASEND_CUDA(cudaMemcpyAsync(r_host, H.vl_w.p, sizeof(float) * c.n_dof, cudaMemcpyDeviceToHost, c.stream));
    ASEND_CUDA(cudaStreamSynchronize(c.stream));
}

// Loss sum_s ||b_s - A V(b_s)||^2 over the samples (FP32, unit-norm b_s) with
// the learned finest-level smoother blocks, added to *d_loss; the block
// gradient (summed over samples) is added to gblk [n_nodes][6].  The caller
// has installed the learned blocks (mg_select_smoother(c, true)).
void mg_learned_loss_grad(Ctx& c, const float* samples, int n_samples, float* gblk, double* d_loss) {
    MgHierarchy& H = *c.mg;
    MgLevel& L0 = *H.L[0];
    const int n = L0.n_nodes, nd = 3 * n;
    if (H.L.size() < 2) throw InputError("multigrid hierarchy has a single level");
    if (H.vl_q.n != (size_t)4 * n) {
        H.vl_q.alloc((size_t)4 * n);
        H.vl_mw.alloc((size_t)4 * n);
        H.vl_t4.alloc((size_t)4 * n);
        H.vl_r2.alloc(nd);
        H.vl_w.alloc(nd);
    }
    float4* q = reinterpret_cast<float4*>(H.vl_q.p);
    float4* mw = reinterpret_cast<float4*>(H.vl_mw.p);
    float4* t4 = reinterpret_cast<float4*>(H.vl_t4.p);
    const int g = grid_of(n);
    for (int s = 0; s < n_samples; ++s) {
        const float* b = samples + (size_t)s * nd;
        ASEND_CUDA(cudaMemcpyAsync(L0.b.p, b, sizeof(float) * nd, cudaMemcpyDeviceToDevice, c.stream));
        vcycle(c, nullptr, false);  // z in L0.y4, x2 in L0.x4
        k_vl_resid<<<g, kT, 0, c.stream>>>(sbview(L0), b, reinterpret_cast<const float4*>(L0.y4.p),
                                          reinterpret_cast<const float4*>(L0.x4.p), q, H.vl_r2.p, d_loss);
        k_vl_w<<<g, kT, 0, c.stream>>>(sbview(L0), L0.binv.p, q, H.vl_w.p, mw);
        k_vl_t<<<g, kT, 0, c.stream>>>(sbview(L0), H.vl_w.p, mw, L0.r.p, t4);
        coarse_correction(c);  // L0.x4 = P C R t
        k_vl_grad<<<g, kT, 0, c.stream>>>(sbview(L0), t4, reinterpret_cast<const float4*>(L0.x4.p), b, H.vl_w.p,
                                         H.vl_r2.p, gblk);
        c.launches += vcycle_launches(c) + 4;
    }
    ASEND_CUDA(cudaGetLastError());
}


namespace {
int pcg_solve_mg_once(Ctx& c, const asend_solve_opts& o, asend_solve_stats* st, bool warm, const double* d_f,
                      double* d_x, int nrhs_all);
}

// Multigrid-preconditioned flexible CG, up to four right-hand sides at a time.  A
// solve that turns non-finite (a smoother damped from an eigenvalue estimate
// that fell short of a localised top mode) is repeated from zero with every
// level's damping taken from the guaranteed bound ||D^-1 A||_inf, which then
// stays in force for this hierarchy.
int pcg_solve_mg(Ctx& c, const asend_solve_opts& o, asend_solve_stats* st, bool warm, const double* d_f, double* d_x,
                 int nrhs_all) {
    const int rc = pcg_solve_mg_once(c, o, st, warm, d_f, d_x, nrhs_all);
    if (rc != ASEND_NONFINITE || !c.mg || c.mg->safe_damping) return rc;
    c.mg->safe_damping = true;
    mg_invalidate_values(c);
    return pcg_solve_mg_once(c, o, st, false, d_f, d_x, nrhs_all);
}

namespace {
int pcg_solve_mg_once(Ctx& c, const asend_solve_opts& o, asend_solve_stats* st, bool warm, const double* d_f,
                      double* d_x, int nrhs_all) {
    const bool mixed = o.method == ASEND_METHOD_MIXED;
    const bool split = o.method == ASEND_METHOD_SPLIT;
    if (!split) ensure_v64(c);  // the split method runs on the hi / lo values alone
    const bool split_only = split && !c.v64_valid;  // the true residual from the pairs too
    mg_prepare(c, o.precond == ASEND_PC_MG_LEARNED);
    mg_select_smoother(c, o.precond == ASEND_PC_MG_LEARNED);
    MgHierarchy& H = *c.mg;
    const BoxCycle box_cycle(H);
    const int n = c.A.n_rows, nd = c.n_dof;
    const int max_it = o.max_iter > 0 ? o.max_iter : nd;
    const int G = o.graph_iters > 0 ? o.graph_iters : 8;
    if (!warm) ASEND_CUDA(cudaMemsetAsync(d_x, 0, (size_t)nrhs_all * nd * sizeof(double), c.stream));
    c.d_r.alloc(std::max(c.d_r.n, (size_t)nrhs_all * nd));
    const int grid = grid_of(n);
    // four lanes a row where one thread a row leaves SMs idle
    const bool fp64_lanes = !mixed && !split && c.n_inst <= 1 && n <= kLaneRows;
    const size_t n_part = (size_t)std::max({grid, H.box ? box_ctas(*H.box) : 0, fp64_lanes ? grid_of(4 * n) : 0});
    const int nr_max = std::min(nrhs_all, kMaxRhs);
    c.d_partials.alloc(std::max(c.d_partials.n, nr_max * n_part * kMaxRhs * 3));
    if (mixed) {
        c.d_p32.alloc(std::max(c.d_p32.n, (size_t)kMaxRhs * 4 * n));
        c.d_ap32.alloc(std::max(c.d_ap32.n, (size_t)kMaxRhs * nd));
    } else {  // FP64: 2 x double2 per node; split: hi + lo float4 per node (same bytes)
        c.d_p64.alloc(std::max(c.d_p64.n, (size_t)kMaxRhs * 4 * n));
        c.d_ap64.alloc(std::max(c.d_ap64.n, (size_t)kMaxRhs * nd));
    }
    if (split) c.d_xpair.alloc(std::max(c.d_xpair.n, (size_t)nr_max * 2 * n));
    if (split_only) c.d_xtrip.alloc(std::max(c.d_xtrip.n, (size_t)nr_max * 3 * n));
    level_vectors(H, nr_max);
    // one scalar set per instance and right-hand side, persistent so the
    // captured iteration graphs stay valid across solves
    const int NI = c.n_inst > 1 ? c.n_inst : 1;
    // a batched stack's reductions are per instance: its own row ranges
    const int grid_cg = (split && NI == 1) ? std::min(grid, kPersistCtas) : grid;
    const int grid_v = (split && NI > 1) ? (int)H.cg_rows.n : grid_cg;
    const size_t sc_need = sizeof(RhsScalars) * NI * kMaxRhs, tk_need = sizeof(uint32_t) * NI * 4 * kMaxRhs;
    if (c.pcg_sc.n < sc_need) c.pcg_sc.alloc(sc_need);
    if (c.pcg_ctl.n < sizeof(Control)) c.pcg_ctl.alloc(sizeof(Control));
    if (c.pcg_tk.n < tk_need) c.pcg_tk.alloc(tk_need);
    RhsScalars* d_sc = reinterpret_cast<RhsScalars*>(c.pcg_sc.p);
    Control* d_ctl = reinterpret_cast<Control*>(c.pcg_ctl.p);
    ensure_pinned_scalars(c, sc_need);
    RhsScalars* h = reinterpret_cast<RhsScalars*>(c.h_sc);
    int iters_max = 0, repl = 0, status = 0;
    double relmax = 0.0;
    MgLevel& L0 = *H.L[0];
    ASEND_CUDA(cudaEventRecord(c.ev0, c.stream));
    for (int r0 = 0; r0 < nrhs_all; r0 += kMaxRhs) {
        const int nr = std::min(kMaxRhs, nrhs_all - r0);
        MgPcg M;
        std::memset(&M, 0, sizeof(M));  // padding too: the bytes key the cached graph
        PcgArgs& a = M.a;
        a.n_rows = n;
        a.nrhs = nr;
        a.n_dof = nd;
        a.slice_off = c.A.slice_off.p;
        a.row_len = c.A.row_len.p;
        a.col = c.A.col.p;
        a.v32 = c.A.v32.p;
        a.v32lo = c.A.v32lo.p;
        a.v64 = c.A.v64.p;
        a.f = d_f + (size_t)r0 * nd;
        a.x = d_x + (size_t)r0 * nd;
        a.r = c.d_r.p + (size_t)r0 * nd;
        a.p = mixed ? (void*)c.d_p32.p : (void*)c.d_p64.p;
        a.ap = mixed ? (void*)c.d_ap32.p : (void*)c.d_ap64.p;
        a.partials = c.d_partials.p;
        a.sc = d_sc;
        a.ctl = d_ctl;
        if (NI > 1) {
            a.cta_inst = c.d_cta_inst.p;
            a.inst_cta0 = c.d_inst_cta0.p;
            a.inst_ncta = c.d_inst_ncta.p;
        }
        a.tickets = reinterpret_cast<uint32_t*>(c.pcg_tk.p);
        ASEND_CUDA(cudaMemsetAsync(c.pcg_tk.p, 0, tk_need, c.stream));
        M.b0 = L0.b.p;
        M.z = reinterpret_cast<const float4*>(L0.y4.p);
        M.binv0 = L0.binv.p;
        M.x40 = reinterpret_cast<float4*>(L0.x4.p);
        M.n_inst = NI;
        M.part_stride = (int)n_part;
        if (split) {  // the split method's correction e (FP32 pairs) starts at zero
            M.xp = c.d_xpair.p;
            M.xt = split_only ? c.d_xtrip.p : nullptr;
            ASEND_CUDA(cudaMemsetAsync(M.xp, 0, sizeof(float4) * 2 * n * nr, c.stream));
        }
        ASEND_CUDA(cudaMemsetAsync(d_sc, 0, sc_need, c.stream));
        ASEND_CUDA(cudaMemsetAsync(d_ctl, 0, sizeof(Control), c.stream));
        MgPcg V = M;  // the pair method's vector kernels
        if (split && NI > 1) {
            V.cg_rows = H.cg_rows.p;
            V.a.cta_inst = H.cg_inst.p;
            V.a.inst_cta0 = H.cg_cta0.p;
            V.a.inst_ncta = H.cg_ncta.p;
        }
        auto launch_residual = [&](int init) {
            if (split) {  // x64 += e first (the instances being replaced), then r = f - A64 x64
                launch_k(c, k_fold_pairs, dim3(grid_v, nr), kThreads, 0, V, init);
                if (split_only)
                    launch_k(c, k_mg_residual_split, dim3(grid, nr), kResThreads, 0, M, init, o.rel_tol * o.rel_tol);
                else  // FP64-pipe bound: all 4 warps of every row tile in flight
                    launch_k(c, k_mg_residual<true>, dim3(grid, nr), kThreads, 0, M, init, o.rel_tol * o.rel_tol);
                c.launches += 2;
            } else {
                launch_k(c, k_mg_residual<false>, dim3(grid, nr), kThreads, 0, M, init, o.rel_tol * o.rel_tol);
                ++c.launches;
            }
        };
        auto launch_iteration = [&]() {
            if (mixed) {
                launch_k(c, k_mg_spmv_dot<float, float>, dim3(grid, nr), kThreads, 0, M);
                launch_k(c, k_mg_update_xr<float>, dim3(grid, nr), kThreads, 0, M);
            } else if (split) {
                launch_split_product(c, M, dim3(grid_cg, nr));
                launch_k(c, k_mg_update_xr_pair, dim3(grid_v, nr), kThreads, 0, V);
            } else {
                if (fp64_lanes) launch_k(c, k_mg_spmv_dot_lanes, dim3(grid_of(4 * n), nr), kThreads, 0, M);
                else launch_k(c, k_mg_spmv_dot<double, double>, dim3(grid, nr), kThreads, 0, M);
                launch_k(c, k_mg_update_xr<double>, dim3(grid, nr), kThreads, 0, M);
            }
            vcycle(c, a.ctl, true, nr);
            if (mixed) {
                launch_k(c, k_mg_rz<float>, dim3(grid, nr), kThreads, 0, M, 0);
                launch_k(c, k_mg_update_p<float>, dim3(grid, nr), kThreads, 0, M);
            } else if (split) {
                launch_k(c, k_mg_rz_pair, dim3(grid_v, nr), kThreads, 0, V, 0);
                launch_k(c, k_mg_update_p_pair, dim3(grid_v, nr), kThreads, 0, V);
            } else {
                launch_k(c, k_mg_rz<double>, dim3(grid, nr), kThreads, 0, M, 0);
                launch_k(c, k_mg_update_p<double>, dim3(grid, nr), kThreads, 0, M);
            }
        };
        // V-cycle of every instance's current b0, then rz (and p = z on a
        // restart) for the instances the residual kernel marked
        auto launch_start = [&]() {
            vcycle(c, nullptr, false, nr);
            if (mixed) launch_k(c, k_mg_rz<float>, dim3(grid, nr), kThreads, 0, M, 1);
            else if (split) launch_k(c, k_mg_rz_pair, dim3(grid_v, nr), kThreads, 0, V, 1);
            else launch_k(c, k_mg_rz<double>, dim3(grid, nr), kThreads, 0, M, 1);
            c.launches += vcycle_launches(c) + 2;
        };
        launch_residual(warm ? 1 : kZeroStart);
        launch_start();
        ASEND_CUDA(cudaGetLastError());
        // A chunk of iterations as one graph, kept with the hierarchy and reused
        // while the launch arguments are the same (they fully define the graph)
        // (with everything else that changes the captured sequence: the
        // method, the chunk length, the product shape, the launch overlap, the
        // fused tail, the matrix-free plan and which of its pattern blocks)
        auto chunk = [&](int iterations) {
            const void* box[2] = {H.box, H.box ? box_patterns(*H.box) : nullptr};
            std::vector<uint8_t> key(sizeof(MgPcg) + 4 * sizeof(int) + sizeof(box));
            std::memcpy(key.data(), &M, sizeof(MgPcg));
            std::memcpy(key.data() + sizeof(MgPcg) + 4 * sizeof(int), box, sizeof(box));
            const int extra[4] = {o.method, iterations, c.product_variant,
                                  (H.box_cycle ? 1 : 0) | (c.pdl ? 2 : 0) | (c.mg_tail ? 4 : 0)};
            std::memcpy(key.data() + sizeof(MgPcg), extra, sizeof(extra));
            for (auto& g : H.graphs)
                if (g.first == key) return g.second;
            cudaGraph_t graph;
            cudaGraphExec_t exec = nullptr;
            ASEND_CUDA(cudaStreamBeginCapture(c.stream, cudaStreamCaptureModeThreadLocal));
            launch_k(c, k_mg_count_active, nr, 32, 0, M);
            for (int i = 0; i < iterations; ++i) launch_iteration();
            ASEND_CUDA(cudaStreamEndCapture(c.stream, &graph));
            ASEND_CUDA(cudaGraphInstantiate(&exec, graph, 0));
            ASEND_CUDA(cudaGraphDestroy(graph));
            if (H.graphs.size() >= 16) {
                ASEND_CUDA(cudaGraphExecDestroy(H.graphs.front().second));
                H.graphs.erase(H.graphs.begin());
            }
            H.graphs.emplace_back(key, exec);
            return exec;
        };
        const int per_iter = 4 + vcycle_launches(c);
        const size_t sc_bytes = sizeof(RhsScalars) * NI * kMaxRhs;
        int since_repl[kMaxRhs] = {};
        // Expected number of iterations left, from each case's rate between two
        // reads of its residual (0: not known).  A chunk runs to its end whatever
        // converges in it, at some 13 empty launches an iteration, and the last one
        // or two iterations after a true residual would be a chunk of their own:
        // a short last stretch is launched as chunks of kShort (100 x 20 x 20 elements, 30
        // iterations: 40 launched, now 32; the step 4.21 -> 4.06 ms.  Launched without a graph
        // the stretch was slower, 4.37 ms: 13 launches an iteration are host-bound).
        // Not where the chunks' ends decide more than the stop (mixed: the drop that
        // asks for a true residual; replace_every).
        constexpr int kShort = 2;
        std::vector<double> rr_prev((size_t)NI * kMaxRhs, 0.0), log_rate((size_t)NI * kMaxRhs, 0.0);
        int since_read = 0;
        // A load case ends by itself, as if it were alone: converged, non-finite in one
        // of its instances, or at the cap.  From there its kernels have nothing to do.
        bool ended[kMaxRhs] = {};
        for (;;) {
            double left = 0.0;
            bool known = !mixed && o.replace_every == 0;
            ASEND_CUDA(cudaMemcpyAsync(h, d_sc, sc_bytes, cudaMemcpyDeviceToHost, c.stream));
            ASEND_CUDA(cudaStreamSynchronize(c.stream));
            bool any_replace = false, stopped = false, all_ended = true;
            int it_now = 0;  // of the cases that go on
            for (int k = 0; k < nr; ++k) {
                if (ended[k]) continue;
                bool open = false, bad = false;
                int it_k = 0;
                for (int q = k; q < NI * kMaxRhs; q += kMaxRhs) {
                    it_k = std::max(it_k, (int)h[q].iter);
                    bad |= h[q].nonfinite != 0;
                    open |= !h[q].finished;
                }
                if (bad) status = std::max(status, (int)ASEND_NONFINITE);
                else if (open && it_k >= max_it) status = std::max(status, (int)ASEND_MAX_ITER);
                else if (open) {
                    all_ended = false;
                    it_now = std::max(it_now, it_k);
                    continue;
                }
                ended[k] = true;
                for (int q = k; q < NI * kMaxRhs; q += kMaxRhs) {
                    stopped |= !h[q].done;
                    h[q].done = 1;
                }
            }
            if (all_ended) break;
            for (int k = 0; k < nr; ++k) {
                if (ended[k]) continue;
                const bool periodic = o.replace_every > 0 && since_repl[k] >= o.replace_every;
                bool replace = false;
                for (int q = k; q < NI * kMaxRhs; q += kMaxRhs) {
                    RhsScalars& s = h[q];
                    if (s.finished) continue;
                    if (since_read > 0 && rr_prev[q] > 0.0 && s.rr > 0.0)
                        log_rate[q] = std::log(s.rr / rr_prev[q]) / since_read;
                    rr_prev[q] = s.done ? 0.0 : s.rr;
                    if (log_rate[q] < 0.0 && s.rr > s.target) left = std::max(left, std::log(s.target / s.rr) / log_rate[q]);
                    else known = false;
                    const bool drop = mixed && s.rr < 1e-4 * s.rr_last_true;
                    if (s.done || drop || periodic) {
                        s.replace = 1;
                        replace = true;
                    }
                }
                if (replace) since_repl[k] = 0;
                any_replace |= replace;
            }
            if (any_replace || stopped) ASEND_CUDA(cudaMemcpyAsync(d_sc, h, sc_bytes, cudaMemcpyHostToDevice, c.stream));
            if (any_replace) {
                // after convergence of the recurrence the last p update was
                // skipped: the instance restarts its direction (p = z);
                // otherwise p is kept
                launch_residual(0);
                launch_start();
                ++repl;
                since_read = 0;
                continue;
            }
            const int rest = known && left < G ? ((int)std::ceil(left) + kShort) / kShort * kShort : G;
            const bool some = rest + kShort <= G && it_now + rest < max_it;
            since_read = some ? rest : G;
            for (int i = 0; i < since_read; i += some ? kShort : G) {
                ASEND_CUDA(cudaGraphLaunch(chunk(some ? kShort : G), c.stream));
                c.launches += (int64_t)per_iter * (some ? kShort : G) + 1;
            }
            for (int& n : since_repl) n += since_read;
        }
        if (split) {  // the solution: x64 + e
            launch_k(c, k_fold_pairs, dim3(grid_v, nr), kThreads, 0, V, 1);
            ++c.launches;
        }
        ASEND_CUDA(cudaMemcpyAsync(h, d_sc, sc_bytes, cudaMemcpyDeviceToHost, c.stream));
        ASEND_CUDA(cudaStreamSynchronize(c.stream));
        for (int q = 0; q < NI * kMaxRhs; ++q) {
            if (q % kMaxRhs >= nr) continue;
            const RhsScalars& s = h[q];
            iters_max = std::max(iters_max, (int)s.iter);
            if (s.nonfinite) status = ASEND_NONFINITE;
            else if (!s.finished) status = std::max(status, (int)ASEND_MAX_ITER);
            if (s.bb == 0.0) continue;  // empty load case of this instance
            relmax = std::max(relmax, std::sqrt(s.rr_last_true / s.bb));
        }
    }
    ASEND_CUDA(cudaEventRecord(c.ev1, c.stream));
    ASEND_CUDA(cudaEventSynchronize(c.ev1));
    ASEND_CUDA(cudaGetLastError());
    float ms = 0.f;
    ASEND_CUDA(cudaEventElapsedTime(&ms, c.ev0, c.ev1));
    c.last_method = o.method;
    if (st) {
        st->iterations = iters_max;
        st->status = status;
        st->replacements = repl;
        st->n_rhs = nrhs_all;
        st->rel_residual = relmax;
        st->ms_solve = ms;
        st->ms_assemble = c.last_assemble_ms;
        st->penalty_scale = c.sf;
    }
    return status;
}

}  // namespace

}  // namespace asend
