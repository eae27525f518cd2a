// The device code of k_box.cu on the CPU (test infrastructure): box_kernels.inc
// is cut from the sources by test_box_host.py.  The threads of a CTA are
// fibers that run one after the other from barrier to barrier, upwards or
// downwards, so accesses to shared memory that no barrier orders give
// different results in the two orders.
#include <ucontext.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <functional>
#include <memory>
#include <vector>

#define __device__
#define __global__
#define __forceinline__ inline
#define __launch_bounds__(...)

struct dim3 {
    unsigned x = 0, y = 0, z = 0;
};
struct float2 {
    float x, y;
};
struct alignas(16) float4 {
    float x, y, z, w;
};
inline float2 make_float2(float x, float y) { return {x, y}; }
inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline float fmaf(float a, float b, float c) { return std::fma(a, b, c); }
template <typename T>
T __ldcg(const T* p) {
    return *p;
}
using std::max;
using std::min;

static dim3 threadIdx, blockIdx, blockDim, gridDim;

// ---- fibers
static ucontext_t g_main;
static ucontext_t* g_self;
static std::function<void()> g_body;
static std::vector<uint8_t> g_done;
static void fiber_entry(int t) {
    g_body();
    g_done[t] = 1;
}
static void __syncthreads() { swapcontext(g_self, &g_main); }
static unsigned char* smem;
constexpr size_t kSmem = 227 * 1024, kStack = 128 * 1024;

static void run_cta(int threads, bool down, const std::function<void()>& body) {
    static std::vector<unsigned char> stacks, shared(kSmem + 16);
    stacks.resize(kStack * threads);
    smem = shared.data() + (16 - (uintptr_t)shared.data() % 16) % 16;
    std::memset(smem, 0xff, kSmem);  // NaN: nothing may be read before it is written
    std::vector<ucontext_t> ctx(threads);
    g_body = body;
    g_done.assign(threads, 0);
    for (int t = 0; t < threads; ++t) {
        getcontext(&ctx[t]);
        ctx[t].uc_stack.ss_sp = &stacks[kStack * t];
        ctx[t].uc_stack.ss_size = kStack;
        ctx[t].uc_link = &g_main;
        makecontext(&ctx[t], (void (*)())fiber_entry, 1, t);
    }
    for (bool any = true; any;) {  // one barrier interval a pass
        any = false;
        for (int q = 0; q < threads; ++q) {
            const int t = down ? threads - 1 - q : q;
            if (g_done[t]) continue;
            any = true;
            threadIdx.x = (unsigned)t;
            g_self = &ctx[t];
            swapcontext(&g_main, &ctx[t]);
        }
    }
}

// ---- what the kernels use from elsewhere
constexpr int kMaxRhs = 4;
struct RhsScalars {
    int done = 0;
};
struct Control {
    int32_t active[kMaxRhs];
};
struct PcgArgs {
    int n_rows, n_dof;
    RhsScalars* sc;
    Control* ctl;
    void *p, *ap;
    double* partials;
    uint32_t* tickets;
};
static int cta_instance(const PcgArgs&) { return 0; }
static void pdl_begin() {}
static double g_dot, g_sum;
template <int NR, int NV>
bool last_block_reduce(const PcgArgs&, double (&v)[NR][NV], int, double (&)[NR][NV]) {
    g_dot += v[0][0];
    return false;
}
static void set_alpha(RhsScalars&, double) {}
template <int K>
void block_sum(double (&v)[K], double*) {
    g_sum += v[0];
    __syncthreads();
    v[0] = g_sum;
    __syncthreads();
    g_sum = 0.0;
    __syncthreads();
}
static uint32_t take_ticket(uint32_t* t) { return (*t)++; }

struct BoxPlan {
    int threads = 0, halo = 0, n_items = 0;
};

#include "box_kernels.inc"

// One launch of a kernel (0: pair product, 1: FP32 residual, 2: post-smoothing, 3:
// power step) on n_blk blocks (nx ny nz node0 el0) of class 0, moduli and
// penalties as pairs.  x: [n_nodes][8] pairs (hi of 3 and a pad, lo of 3 and a
// pad) or [n_nodes][4].  out: as the kernel writes it.  part: the power step's
// sum of every CTA, or the product's p.Ap.  Returns the number of CTAs.
extern "C" int box_launch(int kind, int n_blk, const int32_t* blk, int n_nodes, int sms, const double* K, const float* E,
                          const float* pen, const float* x, const float* b, const float* binv, int down, float* out,
                          double* part, int32_t* shape) {
    std::vector<std::array<int, 5>> blocks(n_blk);
    for (int q = 0; q < n_blk; ++q)
        for (int k = 0; k < 5; ++k) blocks[q][k] = blk[5 * q + k];
    BoxPlan P;
    std::vector<BoxItem> items;
    std::vector<int32_t> blk_of;
    make_items(P, blocks, std::vector<int>(n_blk, 0), n_nodes, sms, items, blk_of);
    std::vector<float2> B(kBoxB);
    pattern_blocks(K, B.data());
    const float2* pen2 = reinterpret_cast<const float2*>(pen);
    std::vector<uint8_t> pn(n_nodes, 0);
    for (int d = 0; d < 3 * n_nodes; ++d) pn[d / 3] |= pen2[d].x != 0.f;
    const BoxArgs X{items.data(), B.data(), reinterpret_cast<const float2*>(E), pen2, pn.data(), P.halo, n_nodes};
    shape[0] = P.threads;
    for (const BoxItem& it : items) shape[1] = std::max(shape[1], it.i1 - it.i0);
    std::vector<float4> xv(2 * (size_t)n_nodes), yv(n_nodes);
    std::memcpy(xv.data(), x, sizeof(float4) * (kind == 0 ? 2 : 1) * n_nodes);
    RhsScalars sc;
    Control ctl{{1, 1, 1, 1}};
    PcgArgs A{n_nodes, 3 * n_nodes, &sc, &ctl, xv.data(), out, nullptr, nullptr};
    float nrm[2] = {1.5f, 0.f};
    uint32_t ticket = 0;
    g_dot = g_sum = 0.0;
    blockDim.x = (unsigned)P.threads;
    gridDim.x = (unsigned)P.n_items;
    for (int c = 0; c < P.n_items; ++c) {
        blockIdx.x = (unsigned)c;
        run_cta(P.threads, down != 0, [&]() {
            if (kind == 0) k_box_product(X, A, 1, 0);
            else if (kind == 1) k_box_resid(X, b, xv.data(), out, &ctl);
            else if (kind == 2) k_box_post(X, binv, b, xv.data(), yv.data(), &ctl);
            else k_box_power(X, binv, xv.data(), yv.data(), nrm, 0, part, &ticket);
        });
    }
    if (kind == 0) part[0] = g_dot;
    if (kind >= 2) std::memcpy(out, yv.data(), sizeof(float4) * n_nodes);
    return P.n_items;
}
