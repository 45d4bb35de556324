// The velocity-field MLP (3 -> W -> W -> W -> 3, softplus) on the 5th-generation
// tensor cores: evaluation with its RK4 stage update, vector-Jacobian product
// and weight gradients (the same operations as mo_mlp.cu's FP32 kernels, for
// W = 64, 128 or 256; a narrower hidden layer is zero-padded to the next W).
//
// FP32 accuracy from FP16 products.  Every operand x of a contraction is
// scaled by a power of two so that a bound of its magnitude lies in [2^14, 2^15):
// the largest magnitude of a weight matrix; for a row of activations or their
// gradients what its inputs and the weights' norms allow, up to a few binades above
// its values; for the weight gradients the largest such bound that any call on the
// packed parameters has seen.  It is split into hi = fp16(x) and lo = fp16(x - hi):
// 22 bits down to 2^-17 of the bound, a bit less for every binade below, nothing
// below 2^-39.  A product is hi*hi + hi*lo + lo*hi (lo*lo is below 2^-24 of it), accumulated
// in FP32 in tensor memory.  That accumulation truncates toward zero: of a
// 256-long sum of positive activations times weights of both signs, chains of
// 16 / 8 / 4 / 2 / 1 steps (K = 16 each) lose 2.8 / 1.5 / 0.9 / 0.6 / 0.4 e-7
// on average and are 3.2 / 1.9 / 1.2 / 0.9 / 0.9 e-7 off (rms; an FP32 FMA
// chain: 2.6e-7, unbiased).  A bias does not average out over rows, so the
// small cross terms come first, the hi*hi chains are kept short (four
// accumulators of W/64 steps, of 4 for the weight gradients), the accumulators are added in FP32 registers
// with rounding to nearest, and the mean loss that is left is given back: the
// split weights are those of W * (1 + loss), the weight gradients are scaled at
// the end (constants fitted to FP64 gradients; they are right on average for sums of
// positive activations and a bias of their size, 2e-8 to 6e-8, for others).
// Against FP64 and beside the FP32 kernels of mo_mlp.cu (relative L2 errors of
// states and gradients, widths 64 and 256, two steps): Xavier weights 0.4e-7 to
// 1.5e-7 (0.7e-7 to 2.2e-7); weights of lognormal size, one weight 1e3 times the
// others: 0.3 to 1.3 of theirs; weights of 1e-3 and 1e-6 of Xavier's: states 1.9e-7
// and 2.7e-7 (1.4e-7 and 1.6e-7), gradients 0.4 to 1.0 of theirs; rows or columns that
// differ tenfold either way: below 3e-7.  Beyond that the bounds leave fewer bits:
// with one weight 1e5 times the others states are 2e-6 to 3e-6 off (0.5e-6 to 2e-6)
// and weight gradients up to 2e-3, more where the flow itself grows to 1e9.
//
//   k_tc_pack   parameters -> operand images (the exact shared-memory layout:
//               K-major rows of 64 halves, 128-byte swizzle), in the order
//               the kernels stream them
//   k_tc_fwd    evaluations of 128-vertex tiles and the RK4 update: one, or a flow's
//   k_tc_bwd    vector-Jacobian products of 128-vertex tiles: one, or a step's four
//   k_tc_wgrad  dW += G^T H over the rows of a step's four evaluations
//   k_tc_reduce partial sums -> gradients, once per backward pass
//
// Activations and gradients between kernels are FP32 in blocks of 8 columns:
// element (row, c) of a 128-row tile at ((tile*(W/8) + c/8)*128 + row)*8 + c%8,
// so a warp whose lanes are rows moves 1 KB of consecutive bytes per access.
// Every wait is bounded in time; one that runs out leaves NaN in the outputs of
// its call and in the packed weights' scales, and so in whatever later calls make
// with them and from what it left.
#include <cuda_fp16.h>

#include <type_traits>

#include "mo_common.cuh"
#include "mo_wait.cuh"

namespace mo {
namespace tc {

constexpr int TILE = 128;             // rows of a tile = lanes of the tensor memory
constexpr int EPI = 512;              // epilogue threads: 4 column groups x 128 rows
constexpr int THREADS = EPI + 128;    // + a warpgroup: one warp copies, one issues the MMAs
constexpr int STAGES = 5;             // weight stages in flight

template <int W>
struct Cfg {
    static constexpr int KB = W / 64;                  // 64-column blocks of the contraction
    static constexpr int NH = W == 256 ? 2 : 1;        // halves of the output columns
    static constexpr int NS = W / NH;                  // columns of a half = rows of a weight stage
    static constexpr int HC = NS / 4;                  // columns of an epilogue thread in a half
    static constexpr int GROUPS = KB == 4 ? 2 : 1;     // weight stages come group by group: lo images, hi images
    static constexpr int KBH = KB / GROUPS;            // blocks of a group
    static constexpr int IMG_STAGES = NH * 2 * KB;     // weight stages of a layer
    static constexpr int STAGE = NS * 128;             // bytes: NS rows x 64 halves
    static constexpr int A_PIECE = KB * TILE * 128;    // bytes of the activations' hi (or lo) image
    static constexpr int TMEM = 4 * NS;                // tensor memory columns: four accumulators of a half
    // column sums: 8-column blocks of a warp, and row ranges where there are more warps than blocks
    static constexpr int SUM_BLOCKS = W == 256 ? 2 : 1, SUM_PARTS = W == 64 ? 2 : 1;
    // shared memory: activation images, weight stages, parameter vectors, rows, barriers
    static constexpr int VECS = 2 * A_PIECE + STAGES * STAGE;
    static constexpr int ROWS = VECS + 9 * 4 * W;
    static constexpr int BARS = ROWS + 3 * 2048;
    static constexpr int SMEM = BARS + 160;           // see Block::init
    // mean relative truncation of a layer's sums (see the top)
    static constexpr float TRUNCATED = W == 256 ? 4e-8f : 0.f;
    // packed parameters (bytes)
    static constexpr int IMAGE = 4 * W * W;            // hi and lo of one matrix
    static constexpr int P_VEC = 4 * IMAGE;            // [9][W]: W1 x, y, z, b1, W4 x, y, z, b2, b3
    static constexpr int P_MISC = P_VEC + 36 * W;      // floats: see enum Misc
    static constexpr int P_MAX = P_MISC + 64;          // uint: bits of bounds of |H1|, |H2|, |G2|, |G3| seen
    static constexpr int PACK = P_MAX + 32;
};
static_assert(Cfg<256>::SMEM <= 227 * 1024, "shared memory of one block");

enum Vec { V_W1X, V_W1Y, V_W1Z, V_B1, V_W4X, V_W4Y, V_W4Z, V_B2, V_B3 };
// 1/scale of W2 and W3, b4[3], and the norms that bound a row's activations and
// gradients: max_c |W1[c,:]|_1, max b1, max_c sum_k max(W2[c,k], 0), max b2,
// max |W4|, max_k sum_n |W3[n,k]|
enum Misc { M_INV2, M_INV3, M_B4, M_N1 = 5, M_MB1, M_N2, M_MB2, M_M4, M_N3 };

// ---- small pieces ----------------------------------------------------------
__device__ __forceinline__ uint32_t s32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// The power of two that brings a magnitude mx into [2^14, 2^15), up to the largest
// finite one, and its inverse.  Small ones stay smaller, so that the product of a
// row's and a matrix's inverse is a normal float: rows keep full precision down to
// 2e-25 (HI = 96), matrices down to 2^-16 (HI = 30).
template <int HI = 96>
__device__ __forceinline__ float pow2_scale(float mx, float* inv) {
    const int e = min(max(141 - ((__float_as_int(mx) >> 23) & 255), 141 - 254), HI);
    *inv = __int_as_float((127 - e) << 23);
    return __int_as_float((127 + e) << 23);
}

// a, b (scaled) -> halves hi and lo with hi + lo = value * (1 + more) to 22 bits
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo, float more = 0.f) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = more == 0.f ? __floats2half2_rn(a - f.x, b - f.y)
                                  : __floats2half2_rn(fmaf(a, more, a - f.x), fmaf(b, more, b - f.y));
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

__device__ __forceinline__ float2 f2(float s) { return make_float2(s, s); }

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// ex2.approx is 4e-8 to 5e-8 low on average (measured); this, added to its
// argument, gives 4e-8 back.
constexpr float EX2_LOW = 6e-8f;

__device__ __forceinline__ float max_nan(float a, float b) {  // NaN if either is
    float y;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
    return y;
}

// softplus(z) = max(z, 0) + log1p(exp(-|z|)); log1p(t) = t + t^2 q(t) on [0, 1],
// q a degree-8 minimax fit (5e-9).  NaN and infinities pass through.
__device__ __forceinline__ float2 softplus2(float2 z) {
    const float2 p = __ffma2_rn(make_float2(fmaxf(-fabsf(z.x), -126.f), fmaxf(-fabsf(z.y), -126.f)), f2(1.44269504f),
                                f2(EX2_LOW));
    const float2 t = make_float2(ex2(p.x), ex2(p.y));
    float2 q = f2(-0.0032440139912068844f);
    q = __ffma2_rn(q, t, f2(0.019851412624120712f));
    q = __ffma2_rn(q, t, f2(-0.05695943906903267f));
    q = __ffma2_rn(q, t, f2(0.10603645443916321f));
    q = __ffma2_rn(q, t, f2(-0.15305587649345398f));
    q = __ffma2_rn(q, t, f2(0.19675937294960022f));
    q = __ffma2_rn(q, t, f2(-0.24954132735729218f));
    q = __ffma2_rn(q, t, f2(0.3332996368408203f));
    q = __ffma2_rn(q, t, f2(-0.4999990165233612f));
    const float2 l = __ffma2_rn(__fmul2_rn(q, t), t, t);
    return __fadd2_rn(make_float2(max_nan(z.x, 0.f), max_nan(z.y, 0.f)), l);
}

// softplus'(z) = 1 - exp(-h) from h = softplus(z); below 0.5 by the series
// h (1 - h/2 + ...) (a degree-5 minimax fit, 1e-9), where the subtraction cancels.
__device__ __forceinline__ float2 sigmoid_of_h2(float2 h) {
    const float2 p = __ffma2_rn(make_float2(fminf(h.x, 126.f), fminf(h.y, 126.f)), f2(-1.44269504f), f2(EX2_LOW));
    const float2 t = make_float2(ex2(p.x), ex2(p.y));
    float2 q = f2(-0.0011216348502784967f);
    q = __ffma2_rn(q, h, f2(0.008187386207282543f));
    q = __ffma2_rn(q, h, f2(-0.041629090905189514f));
    q = __ffma2_rn(q, h, f2(0.16666224598884583f));
    q = __ffma2_rn(q, h, f2(-0.4999998211860657f));
    q = __ffma2_rn(__fmul2_rn(q, h), h, h);
    const float2 o = __fadd2_rn(f2(1.0f), make_float2(-t.x, -t.y));
    return make_float2(h.x > 0.5f ? o.x : q.x, h.y > 0.5f ? o.y : q.y);  // NaN: the series
}

__device__ __forceinline__ void stg8(float* p, const float (&v)[8]) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
                 "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}
__device__ __forceinline__ void ldg8(const float* p, float* v) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p));
}

// The packed weights' scales after a wait that ran out.
__device__ __forceinline__ void spoil(float* misc) {
    reinterpret_cast<volatile float*>(misc)[M_INV2] = NAN;
    reinterpret_cast<volatile float*>(misc)[M_INV3] = NAN;
}

// ---- barriers, copies, MMA -------------------------------------------------
__device__ __forceinline__ void bar_init(uint32_t bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok != 0;
}
// Waits for the phase; after two seconds of polling (or once another wait of the block
// ran out) it sets *late and returns: the block then runs to its end without
// waiting and its outputs are overwritten with NaN.  OWN: for what this thread
// itself has in flight, which is waited for (two seconds) whatever ran out.
// False: the wait ran out.
template <bool OWN = false>
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, volatile int* late) {
    if (bar_try(bar, parity)) return true;
    WaitLimit limit(wait_clock());
    while (!bar_try(bar, parity)) {
        if (limit.over(wait_clock()) || (!OWN && *late)) {
            *late = 1;
            return false;
        }
    }
    return true;
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, int bytes, uint32_t bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// Shared-memory operand descriptor, 128-byte swizzle.  K-major: lbo unused, sbo
// 1024 (8 rows of 128 bytes).  MN-major: lbo the distance of 64-element column
// blocks, sbo 1024 (8 rows along K).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo) {
    return (uint64_t)((addr & 0x3ffffu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(1024u >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// Instruction descriptor: FP32 accumulator, FP16 operands, M x N; mn: both operands MN-major.
__host__ __device__ constexpr uint32_t inst_desc(int m, int n, bool mn) {
    return (1u << 4) | (mn ? (3u << 15) : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// Both are called by a whole warp and executed by its elected lane (the same one
// each time): the operands stay in uniform registers, which the instructions
// want; a lane's own registers cost a move each, more than an MMA takes.
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t inst, bool add) {
    asm volatile(
        "{\n.reg .pred p, q;\nelect.sync _|q, 0xffffffff;\nsetp.ne.b32 p, %4, 0;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(inst), "r"((uint32_t)add)
        : "memory");
}
__device__ __forceinline__ void commit(uint32_t bar) {
    asm volatile(
        "{\n.reg .pred q;\nelect.sync _|q, 0xffffffff;\n"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar)
        : "memory");
}
// ... if the elected lane says so
__device__ __forceinline__ void commit_if(uint32_t bar, bool ok) {
    asm volatile(
        "{\n.reg .pred p, q;\nelect.sync _|q, 0xffffffff;\nsetp.ne.and.b32 p, %1, 0, q;\n"
        "@p tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar),
        "r"((uint32_t)ok)
        : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

#define MO_TC_R8(v)                                                                                              \
    "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])

// 8 columns of this thread's tensor-memory lane
__device__ __forceinline__ void tmem_ld8(uint32_t a, float (&v)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
        "tcgen05.wait::ld.sync.aligned;"
        : MO_TC_R8(v)
        : "r"(a)
        : "memory");
}
// ... of two accumulators, added (all four in flight held 32 results, which k_tc_bwd
// paid for: 95.6 us against 93.2)
__device__ __forceinline__ void tmem_sum2(uint32_t a, uint32_t b, float (&v)[8]) {
    float p[8], q[8];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%16];\n"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%17];\n"
        "tcgen05.wait::ld.sync.aligned;"
        : MO_TC_R8(p), MO_TC_R8(q)
        : "r"(a), "r"(b)
        : "memory");
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = p[j] + q[j];
}
// ... of four accumulators at distance d, added
__device__ __forceinline__ void tmem_sum4(uint32_t a, uint32_t d, float* v) {
    float s[8], t[8];
    tmem_sum2(a, a + d, s);
    tmem_sum2(a + 2 * d, a + 3 * d, t);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = s[j] + t[j];
}

// A block starts with 640 x 96 registers; the epilogue's four warpgroups take
// 104 each, the fifth keeps 64: 512*104 + 128*64 = 61,440 of 61,440.  (With 112
// and 32 the MMA thread spilled its descriptors, and a spill goes to L2: an MMA
// every 400 clocks instead of 65.)
__device__ __forceinline__ void regs_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 104;"); }
__device__ __forceinline__ void regs_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 64;"); }

__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, 512;" ::: "memory"); }

// Programmatic dependent launch: an adjoint (and a flow whose blocks have one or
// two tiles) is a chain of launches, and at a few thousand vertices a launch's
// start (tensor memory, barriers, the first weights) is a third of its time.  A launch that says so
// starts beside the one before it and waits here for its results; everything
// but the packed weights, which no evaluation changes, is read and written
// after the wait, and with plain loads (a non-coherent one may not see what
// another running kernel wrote).
__device__ __forceinline__ void chain_start() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---- parameters ------------------------------------------------------------
struct Params {
    const float *W1, *b1, *W2, *b2, *W3, *b3, *W4, *b4;
    int m;
};

// Block (i, s): slice s of image i (0: W2, 1: W3 rows = output units, for the
// evaluation; 2: W2^T, 3: W3^T for the gradient); the first blocks also the
// vectors and norms (the maxima and the norms' words were zeroed before).
template <int W>
__global__ void __launch_bounds__(256) k_tc_pack(Params p, unsigned char* __restrict__ out) {
    using C = Cfg<W>;
    __shared__ float sh[8];
    const int tid = threadIdx.x, img = blockIdx.x, m = p.m, lane = tid & 31;
    const float* Wm = (img & 1) ? p.W3 : p.W2;
    float* misc = reinterpret_cast<float*>(out + C::P_MISC);
    uint32_t* norm = reinterpret_cast<uint32_t*>(misc);
    float mx = 0.f;
#pragma unroll 8
    for (int i = tid; i < m * m; i += 256) mx = fmaxf(mx, fabsf(__ldg(Wm + i)));
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) sh[tid >> 5] = mx;
    __syncthreads();
    for (int k = 0; k < 8; ++k) mx = fmaxf(mx, sh[k]);
    float inv;
    const float sc = pow2_scale<30>(mx, &inv);
    unsigned char* base = out + (size_t)img * C::IMAGE;
    for (int it = blockIdx.y * 256 + tid; it < W * W / 8; it += gridDim.y * 256) {
        const int n = it / (W / 8), k8 = it % (W / 8);
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float x[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int k = 8 * k8 + 2 * j + e;
                x[e] = (n < m && k < m) ? sc * __ldg(img < 2 ? Wm + n * m + k : Wm + k * m + n) : 0.f;
            }
            split2(x[0], x[1], hi[j], lo[j], C::TRUNCATED);
        }
        // stages: column half by half, group by group, lo images of its blocks, then their hi images
        const int kb = k8 >> 3, half = n / C::NS, nn = n % C::NS, group = kb / C::KBH, in = kb % C::KBH;
        const int at = nn * 128 + (((k8 & 7) ^ (nn & 7)) << 4), first = half * 2 * C::KB + group * 2 * C::KBH + in;
        *reinterpret_cast<uint4*>(base + (size_t)first * C::STAGE + at) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        *reinterpret_cast<uint4*>(base + (size_t)(first + C::KBH) * C::STAGE + at) =
            make_uint4(hi[0], hi[1], hi[2], hi[3]);
    }
    if (img == 0) {  // sum of the positive weights of every unit, a warp per row
        for (int n = blockIdx.y * 8 + (tid >> 5); n < m; n += gridDim.y * 8) {
            float s = 0.f;
            for (int k = lane; k < m; k += 32) s += fmaxf(__ldg(p.W2 + n * m + k), 0.f);
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) atomicMax(norm + M_N2, __float_as_uint(s));
        }
    }
    if (blockIdx.y != 0) return;
    if (img < 2 && tid == 0) misc[img] = inv;
    float* vec = reinterpret_cast<float*>(out + C::P_VEC);
    for (int c = tid; c < W; c += 256) {
        const bool in = c < m;
        if (img == 0) {
            const float x = in ? p.W1[3 * c] : 0.f, y = in ? p.W1[3 * c + 1] : 0.f, z = in ? p.W1[3 * c + 2] : 0.f;
            const float b = in ? p.b1[c] : 0.f;
            vec[V_W1X * W + c] = x; vec[V_W1Y * W + c] = y; vec[V_W1Z * W + c] = z; vec[V_B1 * W + c] = b;
            atomicMax(norm + M_N1, __float_as_uint(fabsf(x) + fabsf(y) + fabsf(z)));
            atomicMax(norm + M_MB1, __float_as_uint(fmaxf(b, 0.f)));
        } else if (img == 1) {
            const float x = in ? p.W4[c] : 0.f, y = in ? p.W4[m + c] : 0.f, z = in ? p.W4[2 * m + c] : 0.f;
            vec[V_W4X * W + c] = x; vec[V_W4Y * W + c] = y; vec[V_W4Z * W + c] = z;
            atomicMax(norm + M_M4, __float_as_uint(fmaxf(fmaxf(fabsf(x), fabsf(y)), fabsf(z))));
            if (c < 3) misc[M_B4 + c] = p.b4[c];
        } else if (img == 2) {
            vec[V_B2 * W + c] = in ? p.b2[c] : 0.f;
            vec[V_B3 * W + c] = in ? p.b3[c] : 0.f;
            atomicMax(norm + M_MB2, __float_as_uint(in ? fmaxf(p.b2[c], 0.f) : 0.f));
        } else if (in) {
            float s = 0.f;
#pragma unroll 8
            for (int n = 0; n < m; ++n) s += fabsf(__ldg(p.W3 + n * m + c));
            atomicMax(norm + M_N3, __float_as_uint(s));
        }
    }
}

// ---- what the evaluation and the gradient share ------------------------------
// A layer's product runs in halves of 128 output columns (W = 256), each into
// four accumulators that the epilogue empties before the next half.
template <int W>
struct Block {
    using C = Cfg<W>;
    unsigned char* sm;
    uint32_t a, stage0, full, empty, a_ready, d_ready, drained, idle, tmem;  // shared-memory addresses; tensor memory base
    volatile int* late;
    int done = 0;  // results waited for (epilogue)

    __device__ void init(unsigned char* smem, const unsigned char* pack) {
        sm = smem;
        a = s32(smem);
        stage0 = a + 2 * C::A_PIECE;
        full = a + C::BARS;
        empty = full + 8 * STAGES;
        a_ready = empty + 8 * STAGES;
        d_ready = a_ready + 8;
        drained = d_ready + 8;
        idle = drained + 8;
        const int slot = C::BARS + 8 * (2 * STAGES + 4);
        static_assert(8 * (2 * STAGES + 4) + 16 <= 160, "barriers, tensor memory address, late");
        late = reinterpret_cast<volatile int*>(smem + slot + 8);
        if (threadIdx.x >> 5 == EPI / 32 + 1) {  // the MMA warp
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(a + slot),
                         "n"(C::TMEM)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
        }
        if (threadIdx.x == 0) {
            for (int i = 0; i < STAGES; ++i) {
                bar_init(full + 8 * i, 1);
                bar_init(empty + 8 * i, 1);
            }
            bar_init(a_ready, EPI);
            bar_init(d_ready, 1);
            bar_init(drained, EPI);
            bar_init(idle, 1);
            *late = (a & 1023u) ? 1 : 0;  // the operand images need 1 KB alignment
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        for (int i = threadIdx.x; i < 9 * W; i += THREADS)
            reinterpret_cast<float*>(smem + C::VECS)[i] = __ldg(reinterpret_cast<const float*>(pack + C::P_VEC) + i);
        fence_before();
        __syncthreads();
        fence_after();
        tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(smem + slot), 0);  // uniform
    }

    __device__ void finish() {
        fence_before();
        __syncthreads();
        if (threadIdx.x >> 5 == EPI / 32 + 1)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(C::TMEM));
    }

    // If a wait ran out, the calls after this one make NaN (one thread, when all
    // others' waits are behind them).
    __device__ __forceinline__ void hand_on(unsigned char* pack) const {
        if (*late) spoil(reinterpret_cast<float*>(pack + C::P_MISC));
    }

    __device__ __forceinline__ const float* vec(int v, int c) const {
        return reinterpret_cast<const float*>(sm + C::VECS) + v * W + c;
    }

    // Copies the weight stages of images img0, img1 for `tiles` tiles (one thread).
    __device__ void produce(const unsigned char* img0, const unsigned char* img1, int tiles) {
        int it = 0;
        for (int t = 0; t < tiles; ++t)
            for (int l = 0; l < 2; ++l)
                for (int s = 0; s < C::IMG_STAGES; ++s, ++it) {
                    const int st = it % STAGES;
                    if (it >= STAGES && !bar_wait(empty + 8 * st, (it / STAGES - 1) & 1, late)) goto end;
                    bulk_load(stage0 + st * C::STAGE, (l ? img1 : img0) + (size_t)s * C::STAGE, C::STAGE, full + 8 * st);
                }
    end:
        // none of its copies is in flight when the block ends
        for (int k = max(0, it - STAGES); k < it; ++k) bar_wait<true>(full + 8 * (k % STAGES), (k / STAGES) & 1, late);
    }

    // Issues the MMAs of two layers for `tiles` tiles (one warp).  An MMA takes 65
    // clocks, and the warp has to issue the next one in that time.
    __device__ void issue(int tiles) {
        const uint64_t bd = smem_desc(stage0, 16);
        int st = 0, emptied = 0;
        uint32_t parity = 0;  // of stage st's current use
        bool filled = true;   // a stage whose copy was not waited for is not handed back
        for (int t = 0; t < 2 * tiles; ++t) {
            bar_wait(a_ready, t & 1, late);
            fence_after();
#pragma unroll 1
            for (int h = 0; h < C::NH; ++h) {
                if (h > 0) {  // the first half's accumulators are read
                    bar_wait(drained, emptied++ & 1, late);
                    fence_after();
                }
                uint64_t ad = smem_desc(a, 16);
                uint32_t d = tmem;
#pragma unroll 1
                for (int g = 0; g < C::GROUPS; ++g) {
                    constexpr int DB = 4 / C::KB * C::NS;  // a block's accumulators
                    // hi * lo: the weights' lo stages are done with
#pragma unroll
                    for (int i = 0; i < C::KBH; ++i) {
                        filled &= bar_wait(full + 8 * st, parity, late);
                        block(ad + i * (TILE * 128 >> 4), bd + st * (C::STAGE >> 4), d + i * DB, true);
                        commit_if(empty + 8 * st, filled);
                        if (++st == STAGES) {
                            st = 0;
                            parity ^= 1;
                        }
                    }
                    // lo * hi, then hi * hi
                    int hs[C::KBH];
#pragma unroll
                    for (int i = 0; i < C::KBH; ++i) {
                        hs[i] = st;
                        filled &= bar_wait(full + 8 * st, parity, late);
                        block(ad + i * (TILE * 128 >> 4) + (C::A_PIECE >> 4), bd + st * (C::STAGE >> 4), d + i * DB,
                              false);
                        if (++st == STAGES) {
                            st = 0;
                            parity ^= 1;
                        }
                    }
#pragma unroll
                    for (int i = 0; i < C::KBH; ++i) {
                        block(ad + i * (TILE * 128 >> 4), bd + hs[i] * (C::STAGE >> 4), d + i * DB, false);
                        commit_if(empty + 8 * hs[i], filled);
                    }
                    ad += C::KBH * (TILE * 128 >> 4);
                    d += C::KBH * DB;
                }
                commit(d_ready);
            }
        }
        if (__any_sync(0xffffffffu, *late)) {  // nobody else has waited for the last MMAs then
            commit(idle);
            bar_wait<true>(idle, 0, late);
        }
    }

    // The four steps of a block of an activation image times a weight stage,
    // KB steps to an accumulator; first: the accumulators start there.
    __device__ __forceinline__ void block(uint64_t ad, uint64_t bd, uint32_t d, bool first) {
        constexpr uint32_t inst = inst_desc(TILE, C::NS, false);
#pragma unroll
        for (int k = 0; k < 4; ++k)
            mma(d + k / C::KB * C::NS, ad + (uint64_t)(2 * k), bd + (uint64_t)(2 * k), inst,
                !(first && k % C::KB == 0));
    }

    // Waits for the next result (epilogue).
    __device__ __forceinline__ void wait_result() {
        bar_wait(d_ready, done++ & 1, late);
        fence_after();
    }

    // Sums of the four column groups' values (group order), in group 0 or in ALL.
    template <bool ALL = false>
    __device__ __forceinline__ void row_sums(float& v0, float& v1, float& v2, int g, int r) {
        float* x = reinterpret_cast<float*>(sm + C::ROWS);
        x[g * TILE + r] = v0;
        x[(4 + g) * TILE + r] = v1;
        x[(8 + g) * TILE + r] = v2;
        epi_sync();
        if (ALL || g == 0) {
            v0 = ((x[r] + x[TILE + r]) + x[2 * TILE + r]) + x[3 * TILE + r];
            v1 = ((x[4 * TILE + r] + x[5 * TILE + r]) + x[6 * TILE + r]) + x[7 * TILE + r];
            v2 = ((x[8 * TILE + r] + x[9 * TILE + r]) + x[10 * TILE + r]) + x[11 * TILE + r];
        }
        epi_sync();
    }

    // 8 halves (columns c..c+7 of row r) into the hi and lo images of the activations.
    __device__ __forceinline__ void put8(int r, int c, const uint32_t* hi, const uint32_t* lo) {
        const uint32_t at = a + (c >> 6) * (TILE * 128) + r * 128 + ((((c >> 3) & 7) ^ (r & 7)) << 4);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(hi[0]), "r"(hi[1]), "r"(hi[2]),
                     "r"(hi[3])
                     : "memory");
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + C::A_PIECE), "r"(lo[0]), "r"(lo[1]),
                     "r"(lo[2]), "r"(lo[3])
                     : "memory");
    }

    // The images are written: hand them to the MMA warp.
    __device__ __forceinline__ void publish() {
        fence_async();
        fence_before();
        bar_arrive(a_ready);
    }
    // A half's accumulators are read.
    __device__ __forceinline__ void release_half() {
        fence_before();
        bar_arrive(drained);
    }
};

__device__ __forceinline__ float2 xy(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 zw(float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// 8 values -> the halves of their images
__device__ __forceinline__ void split8(const float* v, float sc, uint32_t* hi, uint32_t* lo) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 x = __fmul2_rn(make_float2(v[2 * j], v[2 * j + 1]), f2(sc));
        split2(x.x, x.y, hi[j], lo[j]);
    }
}

// ---- evaluation ------------------------------------------------------------
// One evaluation, or the 4 * steps of a flow.  A step's first evaluation reads the
// state x + s*3n (u for the first of all), the others the one before's unext +
// s*ustep + (k-1)*3n; the state after step s goes to next + s*3n, the last to accum.
struct FwdArgs {
    const float *u, *x;
    int64_t n;
    unsigned char* pack;
    float a, a2, wgt, wgt1;  // of evaluations 0 and 1, 2; 0 and 3, 1 and 2
    int init_acc;
    float *unext, *accum, *store;
    int64_t astride;
    int chained;  // the launch before it wrote none of the packed weights
    int evals;
    int64_t ustep;
    float* next;
};

// k = f(u) of the tile's rows; unext = x + a*k, accum = (init ? x : accum) + wgt*k;
// STORE: H1, H2, H3 (blocks of 8 columns) at store + l*astride.
//
// 16 epilogue warps: a thread owns one row and W/4 columns.  They, not the
// tensor cores, bound the kernel (three softplus layers of ~14 issue slots a
// value against 6,200 clocks of MMA a layer), so every MMA runs beside them:
// a layer's first half beside the work of the layer around it (layer 1 of
// the next tile, the last layer of the previous one), its second half
// beside the first half's epilogue.  No more than 32 results are held in
// registers at a time (64 spilled, and a spill goes to L2: shared memory leaves
// 20 KB of L1).
//
// A row's flow needs no other row, so a flow is one launch: a block takes its
// tiles through evaluation after evaluation, and the next one's layer 1 runs
// beside the last layers of this one across the evaluations too.  SERIAL: one
// tile a block, whose next evaluation can only begin when this one's k is there;
// the row's state stays in registers.  (A launch an evaluation before: 20 steps of
// 200,003 vertices, W = 256: 14.1 ms, 13.6 here; 10 steps of 2,563 with their
// gradient, W = 64: 869 us, 758 here; of 49,688, 20 steps with the adjoint: 22.4 and
// 21.4 ms.)
template <int W, bool STORE, bool SERIAL>
__global__ void __launch_bounds__(THREADS, 1) k_tc_fwd(FwdArgs A) {
    using C = Cfg<W>;
    extern __shared__ __align__(1024) unsigned char smem[];
    Block<W> B;
    chain_start();
    if (!A.chained) chain_wait();  // the packed weights may be what is waited for
    B.init(smem, A.pack);
    const int tiles_all = (int)((A.n + TILE - 1) / TILE);
    const int tiles = SERIAL ? 1 : (tiles_all - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    const int items = tiles * A.evals;  // evaluation by evaluation
    const int w = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    if (w >= EPI / 32) {
        regs_down();
        if (w == EPI / 32 && lane == 0) B.produce(A.pack, A.pack + C::IMAGE, items);
        if (w == EPI / 32 + 1) B.issue(items);
        __syncwarp();
    } else {
        regs_up();
        chain_wait();
        constexpr int HC = C::HC, NH = C::NH, G8 = HC / 8;
        const int g = w >> 2, r = 32 * (w & 3) + lane, c0 = g * HC;
        const uint32_t lane_base = B.tmem + ((uint32_t)(32 * (w & 3)) << 16) + c0;
        const float* misc = reinterpret_cast<const float*>(A.pack + C::P_MISC);
        const float inv2 = __ldg(misc + M_INV2), inv3 = __ldg(misc + M_INV3);
        float hm1 = 0.f, hm2 = 0.f;  // bounds of the activations seen (for the weight gradients' scales)

        uint32_t hi[G8][4], lo[G8][4];  // the first half of layer 1 of the next tile
        float inv1 = 0.f, hb1 = 0.f, sc1 = 0.f, ux = 0.f, uy = 0.f, uz = 0.f;
        float sx[3] = {0.f, 0.f, 0.f}, sa[3] = {0.f, 0.f, 0.f};  // SERIAL: the row's state, its next one
        // an item's evaluation and tile; its place in the store (a step's three
        // layers have four evaluations each)
        auto eval_of = [&](int i) { return SERIAL ? i : i / tiles; };
        auto tile_of = [&](int i, int e) { return (int)blockIdx.x + (i - e * tiles) * (int)gridDim.x; };
        auto place = [&](int i) {
            if (!STORE) return 0;
            const int e = eval_of(i);
            return (12 * (e >> 2) + (e & 3)) * tiles_all + tile_of(i, e);
        };
        auto at8 = [&](int tile, int c) { return (((int64_t)tile * (W / 8) + c / 8) * TILE + r) * 8; };
        auto keep = [&](int l, int tile, int c, const float* v) {  // the training pass keeps every layer
            if (STORE) {
                const float o[8] = {v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]};
                stg8(A.store + l * A.astride + at8(tile, c), o);
            }
        };
        // A row's layer-1 activations are below |W1|_1 |u|_inf + max b1 + ln 2.
        auto begin1 = [&](int item) {
            if (!SERIAL || item == 0) {
                const int e = eval_of(item), k = e & 3;
                const int64_t row = (int64_t)tile_of(item, e) * TILE + r, s3n = (int64_t)(e >> 2) * 3 * A.n;
                const float* u = e == 0   ? A.u
                                 : k == 0 ? A.x + s3n
                                          : A.unext + (e >> 2) * A.ustep + (k - 1) * 3 * A.n;
                ux = uy = uz = 0.f;
                if (row < A.n) {
                    ux = u[3 * row];
                    uy = u[3 * row + 1];
                    uz = u[3 * row + 2];
                }
                if (SERIAL) {
                    sx[0] = ux;
                    sx[1] = uy;
                    sx[2] = uz;
                }
            }
            hb1 = fmaf(__ldg(misc + M_N1), fmaxf(fmaxf(fabsf(ux), fabsf(uy)), fabsf(uz)), __ldg(misc + M_MB1)) + 0.7f;
            hm1 = fmaxf(hm1, hb1);
            sc1 = pow2_scale(hb1, &inv1);
        };
        // 8 columns of layer 1: softplus(W1 u + b1)
        auto layer1 = [&](int tile, int c, uint32_t* h4, uint32_t* l4) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; j += 4) {
                const float4 x = ld4(B.vec(V_W1X, c + j)), y = ld4(B.vec(V_W1Y, c + j));
                const float4 z = ld4(B.vec(V_W1Z, c + j)), b = ld4(B.vec(V_B1, c + j));
                const float2 s = softplus2(
                    __ffma2_rn(f2(uz), xy(z), __ffma2_rn(f2(uy), xy(y), __ffma2_rn(f2(ux), xy(x), xy(b)))));
                const float2 t = softplus2(
                    __ffma2_rn(f2(uz), zw(z), __ffma2_rn(f2(uy), zw(y), __ffma2_rn(f2(ux), zw(x), zw(b)))));
                v[j] = s.x; v[j + 1] = s.y; v[j + 2] = t.x; v[j + 3] = t.y;
            }
            keep(0, tile, c, v);
            split8(v, sc1, h4, l4);
        };
        // 8 columns of a later layer: softplus(acc * f + b)
        auto gate8 = [&](float* v, float f, const float* b) {
#pragma unroll
            for (int j = 0; j < 8; j += 4) {
                const float4 q = ld4(b + j);
                const float2 s = softplus2(__ffma2_rn(make_float2(v[j], v[j + 1]), f2(f), xy(q)));
                const float2 t = softplus2(__ffma2_rn(make_float2(v[j + 2], v[j + 3]), f2(f), zw(q)));
                v[j] = s.x; v[j + 1] = s.y; v[j + 2] = t.x; v[j + 3] = t.y;
            }
        };
        float2 p0, p1, p2;  // this thread's part of k
        auto layer3 = [&](int tile, int c, float* v, float f) {
            gate8(v, f, B.vec(V_B3, c));
#pragma unroll
            for (int j = 0; j < 8; j += 4) {
                const float4 x = ld4(B.vec(V_W4X, c + j)), y = ld4(B.vec(V_W4Y, c + j));
                const float4 q = ld4(B.vec(V_W4Z, c + j));
                const float2 s = make_float2(v[j], v[j + 1]), t = make_float2(v[j + 2], v[j + 3]);
                p0 = __ffma2_rn(t, zw(x), __ffma2_rn(s, xy(x), p0));
                p1 = __ffma2_rn(t, zw(y), __ffma2_rn(s, xy(y), p1));
                p2 = __ffma2_rn(t, zw(q), __ffma2_rn(s, xy(q), p2));
            }
            keep(2, tile, c, v);
        };
        // k and the RK4 update
        auto finish = [&](int item) {
            const int e = eval_of(item), k = e & 3;
            const int64_t row = (int64_t)tile_of(item, e) * TILE + r, s3n = (int64_t)(e >> 2) * 3 * A.n;
            float k0 = p0.x + p0.y, k1 = p1.x + p1.y, k2 = p2.x + p2.y;
            B.template row_sums<SERIAL>(k0, k1, k2, g, r);
            if ((!SERIAL && g > 0) || row >= A.n) return;
            const float kv[3] = {k0 + __ldg(misc + M_B4), k1 + __ldg(misc + M_B4 + 1), k2 + __ldg(misc + M_B4 + 2)};
            const bool late = *B.late != 0;
            const float* x = A.x + s3n;
            float* unext = k < 3 && A.unext ? A.unext + (e >> 2) * A.ustep + k * 3 * A.n : nullptr;
            float* accum = (e | 3) + 1 < A.evals ? A.next + s3n : A.accum;
            const float a = k == 2 ? A.a2 : A.a, wgt = k == 1 || k == 2 ? A.wgt1 : A.wgt;
            const bool init = k == 0 && A.init_acc;
            float un[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const int64_t q = 3 * row + d;
                const float kd = late ? NAN : kv[d];
                if (SERIAL) {
                    un[d] = fmaf(a, kd, sx[d]);
                    sa[d] = fmaf(wgt, kd, k == 0 ? sx[d] : sa[d]);
                    if (k == 3) un[d] = sx[d] = sa[d];
                    if (g == 0) {
                        if (k < 3) unext[q] = un[d];
                        else accum[q] = sa[d];
                    }
                } else {
                    if (unext) unext[q] = fmaf(a, kd, x[q]);
                    accum[q] = fmaf(wgt, kd, init ? x[q] : accum[q]);
                }
            }
            if (SERIAL) {
                ux = un[0];
                uy = un[1];
                uz = un[2];
            }
        };
        // the accumulators of the half that is ready
        auto take = [&](float (&v)[HC]) {
            B.wait_result();
#pragma unroll
            for (int i = 0; i < G8; ++i) tmem_sum4(lane_base + 8 * i, C::NS, v + 8 * i);
        };

        begin1(0);
#pragma unroll
        for (int i = 0; i < G8; ++i) layer1(place(0), c0 + 8 * i, hi[i], lo[i]);
        float f3 = 0.f;
        for (int t = 0; t <= items; ++t) {
            const int tile = place(t);
            constexpr int c1 = (NH - 1) * C::NS;  // the second half's first column
            float f2_, hb;
            {
                float z[HC];
                if (t > 0) take(z);  // layer 3 of the previous item is done: the images are free
                auto last = [&]() {
                    const int prev = place(t - 1);
                    if (NH == 1) p0 = p1 = p2 = f2(0.f);
#pragma unroll
                    for (int i = 0; i < G8; ++i) layer3(prev, c1 + c0 + 8 * i, z + 8 * i, f3);
                    finish(t - 1);
                };
                if (SERIAL && t > 0) {
                    last();
                    if (t == items) break;
                    begin1(t);
#pragma unroll
                    for (int i = 0; i < G8; ++i) layer1(tile, c0 + 8 * i, hi[i], lo[i]);
                }
                f2_ = inv1 * inv2;
                hb = hb1;
                if (t < items) {
#pragma unroll
                    for (int i = 0; i < G8; ++i) B.put8(r, c0 + 8 * i, hi[i], lo[i]);
                    if (NH == 2) {
#pragma unroll 1
                        for (int i = 0; i < G8; ++i) {
                            uint32_t h4[4], l4[4];
                            layer1(tile, c1 + c0 + 8 * i, h4, l4);
                            B.put8(r, c1 + c0 + 8 * i, h4, l4);
                        }
                    }
                    B.publish();
                }
                if (!SERIAL && t > 0) last();
            }
            if (t == items) break;
            // layer 2: activations below sum(W2+) max h1 + max b2 + ln 2
            const float hb2 = fmaf(__ldg(misc + M_N2), hb, __ldg(misc + M_MB2)) + 0.7f;
            hm2 = fmaxf(hm2, hb2);
            float inv;
            const float sc = pow2_scale(hb2, &inv);
            f3 = inv * inv3;
            if (NH == 2) {
                // the first half's images wait in registers for the second half's MMAs
                float v[HC];
                take(v);
                B.release_half();
#pragma unroll
                for (int i = 0; i < G8; ++i) {
                    gate8(v + 8 * i, f2_, B.vec(V_B2, c0 + 8 * i));
                    keep(1, tile, c0 + 8 * i, v + 8 * i);
                    split8(v + 8 * i, sc, hi[i], lo[i]);
                }
            }
            B.wait_result();
            if (NH == 2) {
#pragma unroll
                for (int i = 0; i < G8; ++i) B.put8(r, c0 + 8 * i, hi[i], lo[i]);
            }
#pragma unroll 1
            for (int i = 0; i < G8; ++i) {
                const int c = c1 + c0 + 8 * i;
                float v[8];
                uint32_t h4[4], l4[4];
                tmem_sum4(lane_base + 8 * i, C::NS, v);
                gate8(v, f2_, B.vec(V_B2, c));
                keep(1, tile, c, v);
                split8(v, sc, h4, l4);
                B.put8(r, c, h4, l4);
            }
            B.publish();
            if (!SERIAL && t + 1 < items) {
                // its input is at least `tiles` items old, and between two items
                // every thread has met the others (row_sums) unless there are two
                if (tiles == 2) epi_sync();
                const int then = place(t + 1);
                begin1(t + 1);
#pragma unroll
                for (int i = 0; i < G8; ++i) layer1(then, c0 + 8 * i, hi[i], lo[i]);
            }
            if (NH == 2) {
                float z[HC];
                take(z);
                B.release_half();
                p0 = p1 = p2 = f2(0.f);
#pragma unroll
                for (int i = 0; i < G8; ++i) layer3(tile, c0 + 8 * i, z + 8 * i, f3);
            }
        }
        const uint32_t m1 = __reduce_max_sync(0xffffffffu, __float_as_uint(hm1));
        const uint32_t m2 = __reduce_max_sync(0xffffffffu, __float_as_uint(hm2));
        if (lane == 0) {
            uint32_t* mx = reinterpret_cast<uint32_t*>(A.pack + C::P_MAX);
            atomicMax(mx, m1);
            atomicMax(mx + 1, m2);
            if (w == 0) B.hand_on(A.pack);
        }
    }
    B.finish();
}

// ---- vector-Jacobian product ------------------------------------------------
struct BwdArgs {
    const float *a, *gprev;  // dL/dk = ca*a + cg*gprev (gprev may be NULL)
    float ca, cg;
    const float* u;
    int64_t n;
    unsigned char* pack;
    const float* store;  // H1, H2, H3 of the evaluation at store + l*astride
    int64_t astride;
    float *gz2, *gz3;    // n-padded x W, blocks of 8 columns
    const float* dx_in;  // dx_out = dx_in + dL/du
    float *dx_out, *gu;
    float* partial;      // [blocks][16][W]: dW4 (3), db4, dW1 (3), db1, and their rounding errors
    int first;           // partial: 1 set, 0 add
    int chained;
};

// A step's four products, last evaluation first: product j has the arrays of
// evaluation 3 - j, the inputs u - j*3n (x for the last), the weights ca or ca1 and
// cg, cg1 or cg2, the product before's dx_out and gradient.  (A type of its own: with
// these fields the other kernel spilled 172 bytes a thread instead of 104.)
struct StepArgs : BwdArgs {
    float ca1, cg1, cg2;
    const float* x;
};

// The last layer's gate, two layers back through the tensor cores, and the
// column sums of the small gradients: dW4 from H3 read by column while the
// first MMAs run, dW1 and db1 from the tile of g_z1, laid out as FP32 in the
// (then free) activation images; four lanes keep the sums of one column over
// all of the block's tiles.
//
// Bound (n = 49,688, W = 256): 45,000 clocks a tile of issue, waits for the MMAs
// and shared memory, and 12,000 more behind L2 (256 MB read and written, and H3
// again).  The activations are asked for half a layer ahead and the columns
// summed eight by four rows a warp: 105 -> 95.6 us, width 64 at 2,563 rows 12.6 ->
// 11.0.  A prefetch of them to L2, a tile or a layer ahead, was no faster or
// slower (117 us); dW4 by shared memory instead of L2 134 against 113.
//
// STEP: a step's four products, for one tile a block, whose row keeps its gradient in
// registers (10 steps of 2,563 rows with their flow, W = 64: 758 -> 703 us).  With more
// tiles a block the same launch was slower than four (W = 256, 49,688 rows: 22.1 ms
// against 21.4: 304 bytes of spills a thread against 104).
template <int W, bool STEP>
__global__ void __launch_bounds__(THREADS, 1) k_tc_bwd(std::conditional_t<STEP, StepArgs, BwdArgs> A) {
    using C = Cfg<W>;
    extern __shared__ __align__(1024) unsigned char smem[];
    Block<W> B;
    chain_start();
    if (!A.chained) chain_wait();  // the packed weights may be what is waited for
    B.init(smem, A.pack);
    const int tiles_all = (int)((A.n + TILE - 1) / TILE);
    const int tiles = STEP ? 1 : (tiles_all - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    const int items = STEP ? 4 : tiles;
    const int w = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    if (w >= EPI / 32) {
        regs_down();
        if (w == EPI / 32 && lane == 0) B.produce(A.pack + 3 * C::IMAGE, A.pack + 2 * C::IMAGE, items);
        if (w == EPI / 32 + 1) B.issue(items);
        __syncwarp();
    } else {
        regs_up();
        chain_wait();
        constexpr int HC = C::HC, NH = C::NH, G8 = HC / 8;
        const int g = w >> 2, r = 32 * (w & 3) + lane, c0 = g * HC;
        const uint32_t lane_base = B.tmem + ((uint32_t)(32 * (w & 3)) << 16) + c0;
        const float* misc = reinterpret_cast<const float*>(A.pack + C::P_MISC);
        const float inv2 = __ldg(misc + M_INV2), inv3 = __ldg(misc + M_INV3);
        float* scratch = reinterpret_cast<float*>(smem);
        float* rows = reinterpret_cast<float*>(smem + C::ROWS);  // [3][TILE]
        // Column sums: a lane has a column of an 8-column block and every fourth
        // row, so a warp's access is 128 consecutive bytes of a block.
        constexpr int SB = C::SUM_BLOCKS, PART_ROWS = TILE / C::SUM_PARTS;
        const int blk = w % (W / 8), row0 = w / (W / 8) % C::SUM_PARTS * PART_ROWS, cl = lane & 7, rl = lane >> 3;
        float gm2 = 0.f, gm3 = 0.f;  // bounds of the gradients seen
        auto at8 = [&](int tile, int c) { return (((int64_t)tile * (W / 8) + c / 8) * TILE + r) * 8; };
        // FP32 tile in shared memory, 16-byte chunks swizzled by the row
        auto put_scratch = [&](int c, const float* v) {
            const int s = r & 7;
            *reinterpret_cast<float4*>(scratch + r * W + (((c >> 2) ^ s) << 2)) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(scratch + r * W + ((((c >> 2) + 1) ^ s) << 2)) =
                make_float4(v[4], v[5], v[6], v[7]);
        };
        // v = acc * f * softplus' of 8 columns (h: the activations)
        auto gate8 = [&](float* v, const float* h, float f) {
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                const float2 s = sigmoid_of_h2(make_float2(h[j], h[j + 1]));
                const float2 x = __fmul2_rn(__fmul2_rn(make_float2(v[j], v[j + 1]), f2(f)), s);
                v[j] = x.x;
                v[j + 1] = x.y;
            }
        };

        // The activations are used half by half, H3, H2, H1; x holds the next
        // half: a group of 8 columns is asked for as soon as the last half's
        // group is used up.  (Asked for where they were needed, they were
        // waited for.)
        float x[HC];
        auto ask = [&](int l, int tile, int half, int i) {
            ldg8(A.store + l * A.astride + at8(tile, half * C::NS + c0 + 8 * i), x + 8 * i);
        };
        float ga[3], gp[3];  // the next item's a and gprev
        auto ask_row = [&](int tile) {
            const int64_t row = (int64_t)tile * TILE + r;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                ga[d] = row < A.n ? A.a[3 * row + d] : 0.f;
                gp[d] = row < A.n && A.gprev ? A.gprev[3 * row + d] : 0.f;
            }
        };
        ask_row(blockIdx.x);
#pragma unroll
        for (int i = 0; i < G8; ++i) ask(2, blockIdx.x, 0, i);
        for (int j = 0; j < (STEP ? 4 : 1); ++j) {
            float s4[SB][3] = {}, s1[SB][4] = {}, sg[3] = {0.f, 0.f, 0.f};
            for (int t = 0; t < tiles; ++t) {
                // the tile's place in the arrays of the evaluations, and the next item's
                const int tile = STEP ? (int)blockIdx.x - j * tiles_all : (int)blockIdx.x + t * (int)gridDim.x;
                const int then = STEP ? tile - tiles_all : tile + (int)gridDim.x;
                const bool more = STEP ? j < 3 : t + 1 < tiles;
                const int64_t row = (int64_t)(STEP ? (int)blockIdx.x : tile) * TILE + r;
                float gd[3];
                float ca = A.ca, cg = A.cg;
                if constexpr (STEP) {
                    if (j == 1 || j == 2) ca = A.ca1;
                    if (j > 0) cg = j == 1 ? A.cg1 : A.cg2;
                }
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    gd[d] = ca * ga[d];
                    if ((STEP && j > 0) || A.gprev) gd[d] = fmaf(cg, gp[d], gd[d]);
                }
                if (g == 0) {
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        rows[d * TILE + r] = gd[d];
                        sg[d] += gd[d];
                    }
                }
                // g_z3 = (g W4) * softplus'(z3), below |g|_1 max |W4|; g_z2 below that times |W3^T|_1
                const float gb3 = (fabsf(gd[0]) + fabsf(gd[1]) + fabsf(gd[2])) * __ldg(misc + M_M4);
                const float gb2 = gb3 * __ldg(misc + M_N3);
                gm3 = fmaxf(gm3, gb3);
                gm2 = fmaxf(gm2, gb2);
                float inv_3, inv_2;
                const float sc3 = pow2_scale(gb3, &inv_3), sc2 = pow2_scale(gb2, &inv_2);
#pragma unroll
                for (int h = 0; h < NH; ++h)
#pragma unroll
                    for (int i = 0; i < G8; ++i) {
                        const int c = h * C::NS + c0 + 8 * i;
                        float v[8];
                        uint32_t h4[4], l4[4];
#pragma unroll
                        for (int j = 0; j < 8; j += 4) {
                            const float4 wx = ld4(B.vec(V_W4X, c + j)), wy = ld4(B.vec(V_W4Y, c + j));
                            const float4 wz = ld4(B.vec(V_W4Z, c + j));
                            const float2 p = __ffma2_rn(f2(gd[2]), xy(wz),
                                                        __ffma2_rn(f2(gd[1]), xy(wy), __fmul2_rn(f2(gd[0]), xy(wx))));
                            const float2 q = __ffma2_rn(f2(gd[2]), zw(wz),
                                                        __ffma2_rn(f2(gd[1]), zw(wy), __fmul2_rn(f2(gd[0]), zw(wx))));
                            v[j] = p.x; v[j + 1] = p.y; v[j + 2] = q.x; v[j + 3] = q.y;
                        }
                        gate8(v, x + 8 * i, 1.0f);
                        if (h + 1 < NH) ask(2, tile, h + 1, i);
                        else ask(1, tile, 0, i);
                        stg8(A.gz3 + at8(tile, c), v);
                        split8(v, sc3, h4, l4);
                        B.put8(r, c, h4, l4);
                    }
                B.publish();
                epi_sync();
                {   // dW4 += g^T H3, from L2 (beside the first MMAs)
                    const float* H3 = A.store + 2 * A.astride + ((int64_t)tile * (W / 8) + blk) * TILE * 8 + cl;
#pragma unroll 8
                    for (int k = 0; k < PART_ROWS / 4; ++k) {
                        const int rr = row0 + 4 * k + rl;
                        const float g0 = rows[rr], g1 = rows[TILE + rr], g2 = rows[2 * TILE + rr];
#pragma unroll
                        for (int q = 0; q < SB; ++q) {
                            const float h = H3[(q * 16 * TILE + rr) * 8];
                            s4[q][0] = fmaf(g0, h, s4[q][0]);
                            s4[q][1] = fmaf(g1, h, s4[q][1]);
                            s4[q][2] = fmaf(g2, h, s4[q][2]);
                        }
                    }
                }
                float e3[3] = {0.f, 0.f, 0.f};  // this row's dx (group 0) or u (group 1)
                // two layers back
                float p0 = 0.f, p1 = 0.f, p2 = 0.f;
#pragma unroll
                for (int l = 0; l < 2; ++l) {
                    if (l == 1) {
                        if (!STEP && more) ask_row(then);
                        const float* e = g == 0 ? A.dx_in : A.u;
                        if constexpr (STEP)
                            if (j > 0) e = g == 0 ? A.dx_out : j == 3 ? A.x : A.u - j * 3 * A.n;
                        if (g < 2 && row < A.n) {
#pragma unroll
                            for (int d = 0; d < 3; ++d) e3[d] = e[3 * row + d];
                        }
                    }
                    const float f = l == 0 ? inv_3 * inv3 : inv_2 * inv2;
                    float v[HC];
                    uint32_t ph[G8][4], pl[G8][4];
                    // one 8-column group: l = 0 g_z2 -> global and images, l = 1 g_z1 -> g_u
                    auto finish8 = [&](float* q, int c, uint32_t* h4, uint32_t* l4) {
                        if (l == 0) {
                            const float o[8] = {q[0], q[1], q[2], q[3], q[4], q[5], q[6], q[7]};
                            stg8(A.gz2 + at8(tile, c), o);
                            split8(q, sc2, h4, l4);
                            return;
                        }
#pragma unroll
                        for (int j = 0; j < 8; j += 4) {
                            const float4 x = ld4(B.vec(V_W1X, c + j)), y = ld4(B.vec(V_W1Y, c + j));
                            const float4 z = ld4(B.vec(V_W1Z, c + j));
                            p0 = fmaf(q[j + 3], x.w, fmaf(q[j + 2], x.z, fmaf(q[j + 1], x.y, fmaf(q[j], x.x, p0))));
                            p1 = fmaf(q[j + 3], y.w, fmaf(q[j + 2], y.z, fmaf(q[j + 1], y.y, fmaf(q[j], y.x, p1))));
                            p2 = fmaf(q[j + 3], z.w, fmaf(q[j + 2], z.z, fmaf(q[j + 1], z.y, fmaf(q[j], z.x, p2))));
                        }
                    };
                    if (NH == 2) {
                        B.wait_result();
#pragma unroll
                        for (int i = 0; i < G8; ++i) tmem_sum4(lane_base + 8 * i, C::NS, v + 8 * i);
                        B.release_half();
#pragma unroll
                        for (int i = 0; i < G8; ++i) {
                            gate8(v + 8 * i, x + 8 * i, f);
                            ask(1 - l, tile, 1, i);
                            finish8(v + 8 * i, c0 + 8 * i, ph[i], pl[i]);
                        }
                    }
                    B.wait_result();
                    if (NH == 2) {
#pragma unroll
                        for (int i = 0; i < G8; ++i) {
                            if (l == 0) B.put8(r, c0 + 8 * i, ph[i], pl[i]);
                            else put_scratch(c0 + 8 * i, v + 8 * i);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < G8; ++i) {
                        const int c = (NH - 1) * C::NS + c0 + 8 * i;
                        float q[8];
                        uint32_t h4[4], l4[4];
                        tmem_sum4(lane_base + 8 * i, C::NS, q);
                        gate8(q, x + 8 * i, f);
                        if (l == 0) ask(0, tile, 0, i);
                        else if (more) ask(2, then, 0, i);
                        finish8(q, c, h4, l4);
                        if (l == 0) B.put8(r, c, h4, l4);
                        else put_scratch(c, q);
                    }
                    if (l == 0) B.publish();
                }
                B.template row_sums<STEP>(p0, p1, p2, g, r);
                if (STEP) {
                    const bool late = *B.late != 0;
                    gp[0] = row >= A.n ? 0.f : late ? NAN : p0;
                    gp[1] = row >= A.n ? 0.f : late ? NAN : p1;
                    gp[2] = row >= A.n ? 0.f : late ? NAN : p2;
                }
                if (g == 0 && row < A.n) {
                    if (*B.late) p0 = p1 = p2 = NAN;
                    if (!STEP) {
                        A.gu[3 * row] = p0;
                        A.gu[3 * row + 1] = p1;
                        A.gu[3 * row + 2] = p2;
                    }
                    A.dx_out[3 * row] = e3[0] + p0;
                    A.dx_out[3 * row + 1] = e3[1] + p1;
                    A.dx_out[3 * row + 2] = e3[2] + p2;
                }
                if (g == 1) {
#pragma unroll
                    for (int d = 0; d < 3; ++d) rows[d * TILE + r] = e3[d];
                }
                epi_sync();
                {   // dW1 += g_z1^T u, db1 += g_z1 (every other row of a lane's eight: no two lanes in a bank)
#pragma unroll 4
                    for (int k = 0; k < PART_ROWS / 4; ++k) {
                        const int rr = row0 + 8 * (k >> 1) + (k & 1) + 2 * rl;
                        const float u0 = rows[rr], u1 = rows[TILE + rr], u2 = rows[2 * TILE + rr];
#pragma unroll
                        for (int q = 0; q < SB; ++q) {
                            const int c = 8 * (blk + 16 * q) + cl;
                            const float x1 = scratch[rr * W + ((((c >> 2) ^ (rr & 7)) << 2) | (c & 3))];
                            s1[q][0] = fmaf(u0, x1, s1[q][0]);
                            s1[q][1] = fmaf(u1, x1, s1[q][1]);
                            s1[q][2] = fmaf(u2, x1, s1[q][2]);
                            s1[q][3] += x1;
                        }
                    }
                }
                epi_sync();
            }
            // a column's four lanes (and row ranges) together; db4: the rows of group 0
            float* sums = scratch;  // [SUM_PARTS][8][W]: dW4 (3), -, dW1 (3), db1
            float* xs = reinterpret_cast<float*>(smem + C::ROWS);
#pragma unroll
            for (int q = 0; q < SB; ++q)
#pragma unroll
                for (int d = 0; d < 7; ++d) {
                    float v = d < 3 ? s4[q][d < 3 ? d : 0] : s1[q][d < 3 ? 0 : d - 3];
                    v += __shfl_xor_sync(0xffffffffu, v, 8);
                    v += __shfl_xor_sync(0xffffffffu, v, 16);
                    if (lane < 8) sums[(row0 / PART_ROWS * 8 + d + (d >= 3)) * W + 8 * (blk + 16 * q) + cl] = v;
                }
            if (g == 0) {
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    for (int o = 16; o > 0; o >>= 1) sg[d] += __shfl_xor_sync(0xffffffffu, sg[d], o);
                    if (lane == 0) xs[4 * d + w] = sg[d];
                }
            }
            epi_sync();
            // the sums over all products of a backward pass, with their rounding errors beside them
            for (int e = threadIdx.x; e < 8 * W; e += EPI) {
                const int k = e / W, c = e % W;
                float v = sums[e];
                if (C::SUM_PARTS == 2) v += sums[8 * W + e];
                if (*B.late || isnan(inv2)) v = NAN;
                else if (k == 3) v = c < 3 ? (xs[4 * c] + xs[4 * c + 1]) + (xs[4 * c + 2] + xs[4 * c + 3]) : 0.f;
                float* out = A.partial + (int64_t)blockIdx.x * 16 * W + e;
                const bool first = A.first && j == 0;
                const float h = first ? 0.f : *out, y = first ? v : __fadd_rn(v, out[8 * W]);
                const float t = __fadd_rn(h, y), b = __fsub_rn(t, h);
                *out = t;
                out[8 * W] = __fadd_rn(__fsub_rn(h, __fsub_rn(t, b)), __fsub_rn(y, b));
            }
            if (STEP && j < 3) epi_sync();
        }
        const uint32_t m2 = __reduce_max_sync(0xffffffffu, __float_as_uint(gm2));
        const uint32_t m3 = __reduce_max_sync(0xffffffffu, __float_as_uint(gm3));
        if (lane == 0) {
            uint32_t* mx = reinterpret_cast<uint32_t*>(A.pack + C::P_MAX);
            atomicMax(mx + 2, m2);
            atomicMax(mx + 3, m3);
            if (w == 0) B.hand_on(A.pack);
        }
    }
    B.finish();
}

// ---- weight gradients --------------------------------------------------------
// partial[split][o][i] (+)= sum over the split's rows of G[row][o] * H[row][i]
// for the 128 x 128 block of (o, i) of blockIdx.x; db[split][o] (+)= the column
// sums of G (blocks with i0 = 0).
//
// The contraction runs over rows, so both operands are MN-major: a row's 64
// columns are one 128-byte line, the layout the split values are written in.
// Chunks of 64 rows, two operand stages and two accumulators: while the tensor
// cores work on one chunk the 16 warps split the next one and add the one
// before to FP32 registers, so no truncating chain is longer than 4 steps.
// Bound: the two reads of G and H (DRAM once, L2 once more for the other
// blocks).
template <int W>
struct WCfg {
    static constexpr int NB = W < 128 ? W : 128;   // columns of a block (M is always 128: zero rows for W = 64)
    static constexpr int BLOCKS = (W / NB) * (W / NB);
    static constexpr int ROWS = 64;                // rows of a chunk
    static constexpr int OP = 2 * ROWS * 128;      // bytes of one piece of an operand: two column blocks
    static constexpr int STAGE = 4 * OP;           // G hi, G lo, H hi, H lo
    static constexpr int BARS = 2 * STAGE;
    static constexpr int SMEM = BARS + 64;
    static constexpr int TMEM = 2 * NB;
    static constexpr int DB = W < 128 ? 2 : 1;     // warps that sum the same columns of G
};
constexpr int WTHREADS = EPI + 32;

struct WgradArgs {
    const float *G, *H;  // rows x W, blocks of 8 columns
    int64_t chunks;      // 64-row chunks
    const uint32_t *gmax, *hmax;
    float* misc;
    float *partial, *db;
    int first;
};

template <int W>
__global__ void __launch_bounds__(WTHREADS, 1) k_tc_wgrad(WgradArgs A) {
    using C = WCfg<W>;
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t sm = s32(smem), full = sm + C::BARS, done = full + 16, slot = done + 16, idle = slot + 16;
    volatile int* late = reinterpret_cast<volatile int*>(smem + C::BARS + 40);
    const int w = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    if (w == EPI / 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "n"(C::TMEM)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            bar_init(full + 8 * i, EPI);
            bar_init(done + 8 * i, 1);
        }
        bar_init(idle, 1);
        *late = (sm & 1023u) ? 1 : 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (C::NB < 128)  // the second column block of G stays zero
        for (int i = threadIdx.x; i < 2 * 2 * C::ROWS * 32; i += WTHREADS) {
            const int s = i / (2 * C::ROWS * 32), p = (i / (C::ROWS * 32)) & 1, o = i % (C::ROWS * 32);
            *reinterpret_cast<uint32_t*>(smem + s * C::STAGE + p * C::OP + C::ROWS * 128 + 4 * o) = 0u;
        }
    fence_async();
    fence_before();
    __syncthreads();
    fence_after();
    chain_start();
    chain_wait();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(smem + C::BARS + 32), 0);
    const int o0 = (blockIdx.x / (W / C::NB)) * C::NB, i0 = (blockIdx.x % (W / C::NB)) * C::NB;
    const int64_t per = (A.chunks + gridDim.y - 1) / gridDim.y;
    const int64_t k0 = min(A.chunks, per * (int64_t)blockIdx.y);
    const int nk = (int)(min(A.chunks, k0 + per) - k0);

    if (w == EPI / 32) {
        constexpr uint32_t inst = inst_desc(128, C::NB, true);
        constexpr uint32_t lbo = C::ROWS * 128;
        for (int k = 0; k < nk; ++k) {
            const int s = k & 1;
            bar_wait(full + 8 * s, (k >> 1) & 1, late);
            fence_after();
            const uint32_t d = tmem + s * C::NB;
            const uint64_t gh = smem_desc(sm, lbo) + (uint64_t)(s * (C::STAGE >> 4));
            const uint64_t gl = gh + (C::OP >> 4), hh = gh + (2 * C::OP >> 4), hl = gh + (3 * C::OP >> 4);
#pragma unroll
            for (int q = 0; q < C::ROWS / 16; ++q) {
                mma(d, gh + 128 * q, hl + 128 * q, inst, q > 0);
                mma(d, gl + 128 * q, hh + 128 * q, inst, true);
            }
#pragma unroll
            for (int q = 0; q < C::ROWS / 16; ++q) mma(d, gh + 128 * q, hh + 128 * q, inst, true);
            commit(done + 8 * s);
        }
        if (__any_sync(0xffffffffu, *late)) {  // nobody else has waited for the last MMAs then
            commit(idle);
            bar_wait<true>(idle, 0, late);
        }
        __syncwarp();
    } else {
        constexpr int NC = C::NB / 4;            // accumulator columns of a thread
        constexpr int IT = C::NB / 64;           // items (8 columns x 32 rows) of a warp per operand
        const int c8 = C::NB < 128 ? (w & 7) : w;
        float ginv, hinv;
        const bool was_late = isnan(A.misc[M_INV2]);
        const float gs = pow2_scale(__uint_as_float(*A.gmax), &ginv), hs = pow2_scale(__uint_as_float(*A.hmax), &hinv);
        const uint32_t lane_base = tmem + ((uint32_t)(32 * (w & 3)) << 16) + (w >> 2) * NC;
        float acc[NC];
#pragma unroll
        for (int j = 0; j < NC; ++j) acc[j] = 0.f;
        float cs[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        float g8[IT][8], h8[IT][8];
        // chunk k: rows 64*(k&1).. of tile k>>1
        auto load = [&](int64_t k) {
#pragma unroll
            for (int i = 0; i < IT; ++i) {
                const int half = C::NB < 128 ? w >> 3 : i;
                const int64_t rr = (k & 1) * 64 + 32 * half + lane;
                ldg8(A.G + (((k >> 1) * (W / 8) + o0 / 8 + c8) * TILE + rr) * 8, g8[i]);
                ldg8(A.H + (((k >> 1) * (W / 8) + i0 / 8 + c8) * TILE + rr) * 8, h8[i]);
            }
        };
        auto put = [&](uint32_t at, int half, const float (&v)[8], float sc) {
            const int rr = 32 * half + lane;
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) split2(v[2 * j] * sc, v[2 * j + 1] * sc, hi[j], lo[j]);
            const uint32_t p = at + (c8 >> 3) * (C::ROWS * 128) + rr * 128 + (((c8 & 7) ^ (rr & 7)) << 4);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(p), "r"(hi[0]), "r"(hi[1]), "r"(hi[2]),
                         "r"(hi[3])
                         : "memory");
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(p + C::OP), "r"(lo[0]), "r"(lo[1]),
                         "r"(lo[2]), "r"(lo[3])
                         : "memory");
        };
        auto drain = [&](int s) {
            fence_after();
#pragma unroll
            for (int o = 0; o < NC; o += 8) {
                float p[8];
                tmem_ld8(lane_base + s * C::NB + o, p);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[o + j] += p[j];
            }
            fence_before();
        };
        if (nk > 0) load(k0);
        for (int k = 0; k < nk; ++k) {
            const int s = k & 1;
            if (k >= 2) {  // the MMAs that read this stage are done: their sums, then the stage again
                bar_wait(done + 8 * s, ((k >> 1) - 1) & 1, late);
                drain(s);
            }
#pragma unroll
            for (int i = 0; i < IT; ++i) {
                const int half = C::NB < 128 ? w >> 3 : i;
                put(sm + s * C::STAGE, half, g8[i], gs);
                put(sm + s * C::STAGE + 2 * C::OP, half, h8[i], hs);
#pragma unroll
                for (int j = 0; j < 8; ++j) cs[j] += g8[i][j];
            }
            if (k + 1 < nk) load(k0 + k + 1);
            fence_async();
            bar_arrive(full + 8 * s);
        }
        for (int k = max(0, nk - 2); k < nk; ++k) {
            bar_wait(done + 8 * (k & 1), (k >> 1) & 1, late);
            drain(k & 1);
        }
        // the two inverse scales as two factors of about the same size: neither alone overflows
        const int e = (__float_as_int(ginv) >> 23) + (__float_as_int(hinv) >> 23) - 254, e1 = e >> 1;
        const float s1 = __int_as_float((127 + e1) << 23), s2 = __int_as_float((127 + e - e1) << 23);
        const int o = 32 * (w & 3) + lane;
        const bool bad = *late || was_late;
        if (bad) spoil(A.misc);
        if (C::NB == 128 || o < C::NB) {
            float* out = A.partial + ((int64_t)blockIdx.y * W + o0 + o) * W + i0 + (w >> 2) * NC;
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                const float x = acc[j] * s1 * s2;
                const float v = bad ? NAN : fmaf(x, 2e-8f, x);  // the mean loss of 4-step chains
                out[j] = A.first ? v : out[j] + v;
            }
        }
        if (i0 == 0) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                for (int q = 16; q > 0; q >>= 1) cs[j] += __shfl_xor_sync(0xffffffffu, cs[j], q);
            if (lane == 0) {
                float* out = A.db + ((int64_t)blockIdx.y * C::DB + (C::NB < 128 ? w >> 3 : 0)) * W + o0 + 8 * c8;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float v = bad ? NAN : cs[j];
                    out[j] = A.first ? v : out[j] + v;
                }
            }
        }
    }
    fence_before();
    __syncthreads();
    if (w == EPI / 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(C::TMEM));
}

// ---- gradients from the partial sums, in a fixed order ------------------------
struct ReduceArgs {
    const float *small;          // [rows][16][W]
    int rows;
    const float *w2, *w3, *db2, *db3;  // [splits][W][W], [splits * DB][W]
    int splits, dbrows, W, m;
    float *dW1, *db1, *dW2, *dbb2, *dW3, *dbb3, *dW4, *db4;
};

// The sum of n values at distance `stride`, and of its rounding errors (a plain
// chain of 300 would lose 2e-7).
__device__ __forceinline__ float2 sum_exactly(const float* p, int n, int64_t stride) {
    float s = 0.f, c = 0.f;
#pragma unroll 4
    for (int k = 0; k < n; ++k) {
        const float x = p[k * stride], t = __fadd_rn(s, x), b = __fsub_rn(t, s);
        c += __fadd_rn(__fsub_rn(s, __fsub_rn(t, b)), __fsub_rn(x, b));
        s = t;
    }
    return make_float2(s, c);
}

// 32 gradients a block; each warp sums an eighth of their partial sums, the
// first one the eighths, both with their rounding errors.  (One thread a
// gradient was 71 us at width 64: a chain of 152 loads and additions on 35
// blocks; here 10.3, and 51.8 -> 27.4 at width 256.)
constexpr int RED_PARTS = 8;
__global__ void __launch_bounds__(32 * RED_PARTS) k_tc_reduce(ReduceArgs A) {
    __shared__ float2 sh[RED_PARTS][32];
    chain_wait();
    const int m = A.m, W = A.W, lane = threadIdx.x & 31, part = threadIdx.x >> 5;
    const int64_t mm = (int64_t)m * m;
    int64_t e = (int64_t)blockIdx.x * 32 + lane;
    const float *p = nullptr, *more = nullptr;  // more: the rounding errors kept beside p's sums
    float* out = nullptr;
    int n = 0;
    int64_t stride = W;
    if (e < 2 * mm) {
        const bool third = e >= mm;
        if (third) e -= mm;
        p = (third ? A.w3 : A.w2) + (e / m) * W + e % m;
        out = (third ? A.dW3 : A.dW2) + e;
        n = A.splits;
        stride = (int64_t)W * W;
    } else if ((e -= 2 * mm) < 2 * m) {
        const bool third = e >= m;
        if (third) e -= m;
        p = (third ? A.db3 : A.db2) + e;
        out = (third ? A.dbb3 : A.dbb2) + e;
        n = A.dbrows;
    } else if ((e -= 2 * m) < 7 * m + 3) {  // dW4 (3), dW1 (3), db1 of every unit, then db4
        const int j = (int)(e / m);
        const int k = e >= 7 * m ? 3 : j < 3 ? j : j + 1, c = e >= 7 * m ? (int)e - 7 * m : (int)(e % m);
        p = A.small + (int64_t)k * W + c;
        more = p + 8 * W;
        out = k < 3 ? A.dW4 + k * m + c : k == 3 ? A.db4 + c : k < 7 ? A.dW1 + 3 * c + k - 4 : A.db1 + c;
        n = A.rows;
        stride = 16 * W;
    }
    const int per = (n + RED_PARTS - 1) / RED_PARTS, k0 = min(n, part * per), k1 = min(n, k0 + per);
    float2 s = sum_exactly(p + k0 * stride, k1 - k0, stride);
    if (more) {
        const float2 q = sum_exactly(more + k0 * stride, k1 - k0, stride);
        s.y += q.x + q.y;
    }
    sh[part][lane] = s;
    __syncthreads();
    if (part != 0 || !out) return;
    const float2 t = sum_exactly(&sh[0][lane].x, RED_PARTS, 64);
    const float2 c = sum_exactly(&sh[0][lane].y, RED_PARTS, 64);
    *out = t.x + (t.y + c.x);
}

template <int W>
int set_attrs() {
    MO_CUDA(cudaFuncSetAttribute(k_tc_fwd<W, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<W>::SMEM));
    MO_CUDA(cudaFuncSetAttribute(k_tc_fwd<W, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<W>::SMEM));
    MO_CUDA(cudaFuncSetAttribute(k_tc_fwd<W, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<W>::SMEM));
    MO_CUDA(cudaFuncSetAttribute(k_tc_fwd<W, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<W>::SMEM));
    MO_CUDA(cudaFuncSetAttribute(k_tc_bwd<W, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<W>::SMEM));
    MO_CUDA(cudaFuncSetAttribute(k_tc_bwd<W, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<W>::SMEM));
    MO_CUDA(cudaFuncSetAttribute(k_tc_wgrad<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, WCfg<W>::SMEM));
    return MO_OK;
}

int64_t tiles_of(int64_t n) { return (n + TILE - 1) / TILE; }
int blocks_for(int64_t n) { return (int)std::min<int64_t>(tiles_of(n), device_sm_count()); }
int splits_for(int64_t rows, int W) {
    const int blocks = W == 256 ? 4 : 1;
    return (int)std::max<int64_t>(1, std::min<int64_t>(device_sm_count() / blocks, rows / 64));
}

}  // namespace tc
}  // namespace mo

using namespace mo;
using namespace mo::tc;

// A launch that may start beside the one before it (chained; see chain_wait).
template <class... P, class... Q>
static cudaError_t launch(void (*kernel)(P...), dim3 grid, int threads, int smem, void* stream, bool chained, Q... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = as_stream(stream);
    cfg.attrs = &at;
    cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}
#define TC_LAUNCH(...) MO_CUDA(launch(__VA_ARGS__))

#define TC_WIDTH(W_, ...)                          \
    do {                                           \
        if ((W_) == 64) { constexpr int W = 64; __VA_ARGS__; }        \
        else if ((W_) == 128) { constexpr int W = 128; __VA_ARGS__; } \
        else { constexpr int W = 256; __VA_ARGS__; }                  \
    } while (0)

static int check_width(int W) {
    MO_CHECK_ARG(W == 64 || W == 128 || W == 256, "padded width must be 64, 128 or 256, got %d", W);
    return MO_OK;
}

extern "C" int mo_mlp_tc_width(int m) { return m <= 0 || m > 256 ? -1 : m <= 64 ? 64 : m <= 128 ? 128 : 256; }
extern "C" int64_t mo_mlp_tc_rows(int64_t n) { return n < 0 ? -1 : tiles_of(n) * TILE; }
extern "C" size_t mo_mlp_tc_pack_bytes(int W) {
    return W == 64 ? Cfg<64>::PACK : W == 128 ? Cfg<128>::PACK : W == 256 ? Cfg<256>::PACK : 0;
}
extern "C" int64_t mo_mlp_tc_partial_floats(int64_t n, int W) {
    if (n <= 0 || (W != 64 && W != 128 && W != 256)) return 0;
    return (int64_t)blocks_for(n) * 16 * W;
}
extern "C" int64_t mo_mlp_tc_wgrad_floats(int64_t rows, int W) {
    if (rows <= 0 || (W != 64 && W != 128 && W != 256)) return 0;
    return (int64_t)splits_for(rows, W) * (W * W + (W < 128 ? 2 : 1) * W);
}

extern "C" int mo_mlp_tc_pack(const float* W1, const float* b1, const float* W2, const float* b2, const float* W3,
                              const float* b3, const float* W4, const float* b4, int m, void* pack, void* stream) {
    const int Wp = mo_mlp_tc_width(m);
    MO_CHECK_ARG(Wp > 0, "hidden width %d is not in [1, 256]", m);
    MO_CHECK_ARG(W1 && b1 && W2 && b2 && W3 && b3 && W4 && b4 && pack, "null pointer");
    MO_CHECK_ARG(aligned(pack, 128), "the packed parameters must be 128-byte aligned");
    TC_WIDTH(Wp, {
        int rc = set_attrs<W>();
        if (rc) return rc;
        MO_CUDA(cudaMemsetAsync(reinterpret_cast<unsigned char*>(pack) + Cfg<W>::P_MISC, 0,
                                Cfg<W>::PACK - Cfg<W>::P_MISC, as_stream(stream)));
        k_tc_pack<W><<<dim3(4, 8), 256, 0, as_stream(stream)>>>(Params{W1, b1, W2, b2, W3, b3, W4, b4, m},
                                                                reinterpret_cast<unsigned char*>(pack));
    });
    ::mo::note_launch();
    MO_LAUNCH_CHECK("k_tc_pack");
    return MO_OK;
}

static int issue_fwd(const float* u, const float* x, int64_t n, void* pack, int W_, float a, float w, int init_acc,
                     float* unext, float* acc, float* store, int64_t astride, void* stream, bool chained) {
    int rc = check_width(W_);
    if (rc) return rc;
    MO_CHECK_ARG(n >= 0 && n < ((int64_t)1 << 31), "bad row count %lld", (long long)n);
    if (n == 0) return MO_OK;
    MO_CHECK_ARG(u && x && pack && acc, "null pointer");
    MO_CHECK_ARG(aligned(pack, 128), "the packed parameters must be 128-byte aligned");
    MO_CHECK_ARG(!store || (aligned(store, 32) && astride >= mo_mlp_tc_rows(n) * W_ && astride % 8 == 0),
                 "store must be 32-byte aligned with an array stride of at least the padded rows times the width");
    const FwdArgs A{u,     x,   n,     reinterpret_cast<unsigned char*>(pack), a, 0.f, w, 0.f, init_acc,
                    unext, acc, store, astride, chained, 1, 0, nullptr};
    TC_WIDTH(W_, TC_LAUNCH(store ? k_tc_fwd<W, true, false> : k_tc_fwd<W, false, false>, blocks_for(n), THREADS,
                           Cfg<W>::SMEM, stream, chained, A));
    ::mo::note_launch();
    return MO_OK;
}

extern "C" int mo_mlp_tc_fwd(const float* u, const float* x, int64_t n, void* pack, int W, float a, float w,
                             int init_acc, float* unext, float* acc, float* store, int64_t astride, void* stream) {
    return issue_fwd(u, x, n, pack, W, a, w, init_acc, unext, acc, store, astride, stream, false);
}

static int issue_bwd(const float* a, float ca, const float* gprev, float cg, const float* u, int64_t n, void* pack,
                     int W_, const float* store, int64_t astride, float* gz2, float* gz3, const float* dx_in,
                     float* dx_out, float* gu, float* partial, int first, void* stream, bool chained) {
    int rc = check_width(W_);
    if (rc) return rc;
    MO_CHECK_ARG(n >= 0 && n < ((int64_t)1 << 31), "bad row count %lld", (long long)n);
    if (n == 0) return MO_OK;
    MO_CHECK_ARG(a && u && pack && store && gz2 && gz3 && dx_in && dx_out && gu && partial, "null pointer");
    MO_CHECK_ARG(aligned(pack, 128), "the packed parameters must be 128-byte aligned");
    MO_CHECK_ARG(aligned(store, 32) && aligned(gz2, 32) && aligned(gz3, 32) && astride % 8 == 0 &&
                     astride >= mo_mlp_tc_rows(n) * W_,
                 "activations and gradients must be 32-byte aligned and padded to whole tiles");
    const BwdArgs A{a,   gprev, ca,  cg,    u,      n,  reinterpret_cast<unsigned char*>(pack), store, astride,
                    gz2, gz3,   dx_in, dx_out, gu, partial, first, chained};
    TC_WIDTH(W_, TC_LAUNCH((k_tc_bwd<W, false>), blocks_for(n), THREADS, Cfg<W>::SMEM, stream, chained, A));
    ::mo::note_launch();
    return MO_OK;
}

extern "C" int mo_mlp_tc_bwd(const float* a, float ca, const float* gprev, float cg, const float* u, int64_t n,
                             void* pack, int W, const float* store, int64_t astride, float* gz2, float* gz3,
                             const float* dx_in, float* dx_out, float* gu, float* partial, int first, void* stream) {
    return issue_bwd(a, ca, gprev, cg, u, n, pack, W, store, astride, gz2, gz3, dx_in, dx_out, gu, partial, first,
                     stream, false);
}

// layer 2: G = gz2, H = H1; layer 3: G = gz3, H = H2 (rows: padded rows of all
// evaluations, a multiple of 128)
static int issue_wgrad(const float* G, const float* H, int64_t rows, void* pack, int W_, int layer, float* partial,
                       int first, void* stream, bool chained) {
    int rc = check_width(W_);
    if (rc) return rc;
    MO_CHECK_ARG(rows >= 0 && rows % TILE == 0, "rows must be a multiple of %d", TILE);
    MO_CHECK_ARG(layer == 2 || layer == 3, "layer must be 2 or 3");
    if (rows == 0) return MO_OK;
    MO_CHECK_ARG(G && H && pack && partial, "null pointer");
    MO_CHECK_ARG(aligned(G, 32) && aligned(H, 32), "arrays must be 32-byte aligned");
    const int splits = splits_for(rows, W_);
    TC_WIDTH(W_, {
        uint32_t* mx = reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(pack) + Cfg<W>::P_MAX);
        const WgradArgs A{G, H, rows / 64, mx + layer, mx + layer - 2,
                          reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(pack) + Cfg<W>::P_MISC), partial, partial + (int64_t)splits * W * W, first};
        TC_LAUNCH(k_tc_wgrad<W>, dim3(WCfg<W>::BLOCKS, splits), WTHREADS, WCfg<W>::SMEM, stream, chained, A);
    });
    ::mo::note_launch();
    return MO_OK;
}

extern "C" int mo_mlp_tc_wgrad(const float* G, const float* H, int64_t rows, void* pack, int W, int layer,
                               float* partial, int first, void* stream) {
    return issue_wgrad(G, H, rows, pack, W, layer, partial, first, stream, false);
}

static int issue_reduce(const float* partial, int64_t n, const float* wpart2, const float* wpart3, int64_t rows,
                        int W_, int m, float* dW1, float* db1, float* dW2, float* db2, float* dW3, float* db3,
                        float* dW4, float* db4, void* stream, bool chained) {
    int rc = check_width(W_);
    if (rc) return rc;
    MO_CHECK_ARG(n > 0 && rows > 0 && m > 0 && m <= W_, "bad sizes");
    MO_CHECK_ARG(partial && wpart2 && wpart3 && dW1 && db1 && dW2 && db2 && dW3 && db3 && dW4 && db4, "null pointer");
    const int splits = splits_for(rows, W_);
    const int64_t ww = (int64_t)splits * W_ * W_;
    const ReduceArgs A{partial, blocks_for(n), wpart2, wpart3, wpart2 + ww, wpart3 + ww, splits,
                       splits * (W_ < 128 ? 2 : 1), W_, m, dW1, db1, dW2, db2, dW3, db3, dW4, db4};
    TC_LAUNCH(k_tc_reduce, ceil_div(2 * (int64_t)m * m + 9 * m + 3, 32), 32 * RED_PARTS, 0, stream, chained, A);
    ::mo::note_launch();
    return MO_OK;
}

extern "C" int mo_mlp_tc_reduce(const float* partial, int64_t n, const float* wpart2, const float* wpart3,
                                int64_t rows, int W, int m, float* dW1, float* db1, float* dW2, float* db2,
                                float* dW3, float* db3, float* dW4, float* db4, void* stream) {
    return issue_reduce(partial, n, wpart2, wpart3, rows, W, m, dW1, db1, dW2, db2, dW3, db3, dW4, db4, stream, false);
}

// ---------------------------------------------------------------------------
// The whole RK4 flow and its adjoint, issued in one call each: an evaluation
// at a few thousand vertices is 10 us of the GPU's time, less than a call
// through the bindings takes.
// ---------------------------------------------------------------------------
namespace {
constexpr int64_t FLOW_ALIGN = 32;  // floats
int64_t flow_pad(int64_t floats) { return (floats + FLOW_ALIGN - 1) / FLOW_ALIGN * FLOW_ALIGN; }

// The steps of a flow that one launch takes, or 0: a launch an evaluation.  Where
// some blocks have two tiles and others one, the ones would wait for their k while
// the twos need not.  FLOW_ITEMS keeps a launch below 20 ms (17 us a tile and
// evaluation at W = 256).
constexpr int64_t FLOW_ITEMS = 1024;
int flow_launch_steps(int64_t n, int steps) {
    const int64_t tiles = tiles_of(n), sms = device_sm_count();
    if (tiles > sms && tiles < 2 * sms) return 0;
    return (int)std::max<int64_t>(1, std::min<int64_t>(steps, FLOW_ITEMS / (4 * ((tiles + sms - 1) / sms))));
}

// `steps` RK4 steps of states ckpt [steps][n][3], the last one to out, with the
// stage inputs in u ([3][n][3] every ustep floats); act: a step's four evaluations'
// H1, H2, H3 ([3][4][rows][W]), one step after the other, or NULL.
int flow_launch(float* ckpt, int64_t n, int steps, void* pack, int W_, double h, float* u, int64_t ustep, float* act,
                float* out, void* stream, bool chained) {
    MO_CHECK_ARG(aligned(pack, 128), "the packed parameters must be 128-byte aligned");
    MO_CHECK_ARG(!act || aligned(act, 32), "the activations must be 32-byte aligned");
    const FwdArgs A{ckpt, ckpt, n, reinterpret_cast<unsigned char*>(pack), (float)(h / 2), (float)h, (float)(h / 6),
                    (float)(h / 3), 1, u, out, act, 4 * mo_mlp_tc_rows(n) * W_, chained, 4 * steps, ustep,
                    ckpt + 3 * n};
    const bool serial = tiles_of(n) <= device_sm_count();
    TC_WIDTH(W_, TC_LAUNCH(act ? (serial ? k_tc_fwd<W, true, true> : k_tc_fwd<W, true, false>)
                               : (serial ? k_tc_fwd<W, false, true> : k_tc_fwd<W, false, false>),
                           blocks_for(n), THREADS, Cfg<W>::SMEM, stream, chained, A));
    ::mo::note_launch();
    return MO_OK;
}

// x_next = RK4(x) with the stage inputs in u [3][n][3]; act: the four
// evaluations' H1, H2, H3 ([3][4][rows][W]) or NULL.
int flow_step(const float* x, int64_t n, void* pack, int W, double h, float* u, float* act, float* x_next,
              void* stream, bool chained) {
    if (flow_launch_steps(n, 1))
        return flow_launch(const_cast<float*>(x), n, 1, pack, W, h, u, 0, act, x_next, stream, chained);
    const int64_t size = mo_mlp_tc_rows(n) * W;
    const float a[4] = {(float)(h / 2), (float)(h / 2), (float)h, 0.f};
    const float w[4] = {(float)(h / 6), (float)(h / 3), (float)(h / 3), (float)(h / 6)};
    for (int k = 0; k < 4; ++k) {
        const int rc = issue_fwd(k ? u + (k - 1) * 3 * n : x, x, n, pack, W, a[k], w[k], k == 0,
                                 k < 3 ? u + k * 3 * n : nullptr, x_next, act ? act + k * size : nullptr,
                                 act ? 4 * size : 0, stream, chained || k > 0);
        if (rc) return rc;
    }
    return MO_OK;
}
}  // namespace

extern "C" int64_t mo_ode_act_floats(int64_t n, int W) {
    return n <= 0 || check_width(W) ? 0 : 12 * mo_mlp_tc_rows(n) * W;
}

extern "C" int64_t mo_ode_backward_floats(int64_t n, int W, int stored) {
    if (n <= 0 || check_width(W)) return 0;
    const int64_t rows = mo_mlp_tc_rows(n);
    return flow_pad(8 * rows * W) + flow_pad(mo_mlp_tc_partial_floats(n, W)) +
           2 * flow_pad(mo_mlp_tc_wgrad_floats(4 * rows, W)) + 2 * flow_pad(3 * n) +
           (stored ? 0 : flow_pad(mo_ode_act_floats(n, W)) + flow_pad(9 * n));
}

extern "C" int mo_ode_flow(const float* x0, int64_t n, int steps, void* pack, int W, float* ckpt, float* act, float* u,
                           float* out, void* stream) {
    int rc = check_width(W);
    if (rc) return rc;
    MO_CHECK_ARG(n >= 0 && n < ((int64_t)1 << 31) && steps >= 1, "bad sizes");
    if (n == 0) return MO_OK;
    MO_CHECK_ARG(x0 && pack && ckpt && u && out, "null pointer");
    MO_CUDA(cudaMemcpyAsync(ckpt, x0, sizeof(float) * 3 * n, cudaMemcpyDeviceToDevice, as_stream(stream)));
    const double h = 1.0 / steps;
    if (const int some = flow_launch_steps(n, steps)) {
        for (int k = 0; k < steps && !rc; k += some) {
            const int m = std::min(some, steps - k);
            rc = flow_launch(ckpt + 3 * n * k, n, m, pack, W, h, act ? u + 9 * n * k : u, act ? 9 * n : 0,
                             act ? act + mo_ode_act_floats(n, W) * k : nullptr,
                             k + m < steps ? ckpt + 3 * n * (k + m) : out, stream, k > 0);
        }
        return rc;
    }
    for (int k = 0; k < steps; ++k) {
        rc = flow_step(ckpt + 3 * n * k, n, pack, W, h, act ? u + 9 * n * k : u,
                       act ? act + mo_ode_act_floats(n, W) * k : nullptr, k + 1 < steps ? ckpt + 3 * n * (k + 1) : out,
                       stream, k > 0);
        if (rc) return rc;
    }
    return MO_OK;
}

extern "C" int mo_ode_flow_backward(const float* ckpt, int64_t n, int steps, void* pack, int W, int m, float* act,
                                    float* u, const float* a_out, float* scratch, int64_t scratch_floats, float* dx0,
                                    float* dx1, float* dW1, float* db1, float* dW2, float* db2, float* dW3, float* db3,
                                    float* dW4, float* db4, void* stream) {
    int rc = check_width(W);
    if (rc) return rc;
    MO_CHECK_ARG(n > 0 && n < ((int64_t)1 << 31) && steps >= 1, "bad sizes");
    MO_CHECK_ARG(ckpt && pack && a_out && scratch && dx0 && dx1 && (!act || u), "null pointer");
    MO_CHECK_ARG(aligned(scratch, 128), "scratch must be 128-byte aligned");
    MO_CHECK_ARG(aligned(pack, 128), "the packed parameters must be 128-byte aligned");
    MO_CHECK_ARG(!act || aligned(act, 32), "the activations must be 32-byte aligned");
    const bool stored = act != nullptr;
    if (scratch_floats < mo_ode_backward_floats(n, W, stored)) {
        set_error("flow scratch too small: %lld < %lld floats", (long long)scratch_floats,
                  (long long)mo_ode_backward_floats(n, W, stored));
        return MO_ERR_SCRATCH;
    }
    const int64_t rows = mo_mlp_tc_rows(n), size = rows * W, act_step = mo_ode_act_floats(n, W);
    float* next = scratch;
    auto take = [&](int64_t floats) {
        float* q = next;
        next += flow_pad(floats);
        return q;
    };
    float* gz = take(8 * size);
    float* partial = take(mo_mlp_tc_partial_floats(n, W));
    float* wpart[2] = {take(mo_mlp_tc_wgrad_floats(4 * rows, W)), take(mo_mlp_tc_wgrad_floats(4 * rows, W))};
    float* gu[2] = {take(3 * n), take(3 * n)};
    float* dx[2] = {dx0, dx1};
    if (!stored) {
        act = take(act_step);
        u = take(9 * n);
    }
    const double h = 1.0 / steps;
    const float* a = a_out;
    int evals = 0;
    for (int k = steps - 1; k >= 0; --k) {
        const float* x = ckpt + 3 * n * k;
        float* ak = stored ? act + act_step * k : act;
        float* uk = stored ? u + 9 * n * k : u;
        // the recompute's end state is not needed: it goes where this step's
        // gradient is written next
        if (!stored) {
            rc = flow_step(x, n, pack, W, h, uk, ak, dx[k & 1], stream, k < steps - 1);
            if (rc) return rc;
        }
        // dk4 = a h/6, dk3 = a h/3 + h g4, dk2 = a h/3 + h/2 g3, dk1 = a h/6 + h/2 g2;
        // dL/dx = a + g4 + g3 + g2 + g1
        const float ca[4] = {(float)(h / 6), (float)(h / 3), (float)(h / 3), (float)(h / 6)};
        const float cg[4] = {(float)(h / 2), (float)(h / 2), (float)h, 0.f};
        if (tiles_of(n) <= device_sm_count()) {
            const bool chained = !stored || k < steps - 1;
            const StepArgs A{{a, nullptr, ca[3], cg[3], uk + 6 * n, n, reinterpret_cast<unsigned char*>(pack),
                              ak + 3 * size, 4 * size, gz + 3 * size, gz + 7 * size, a, dx[k & 1], nullptr, partial,
                              k == steps - 1, chained},
                             ca[2], cg[2], cg[1], x};
            TC_WIDTH(W, TC_LAUNCH((k_tc_bwd<W, true>), blocks_for(n), THREADS, Cfg<W>::SMEM, stream, chained, A));
            ::mo::note_launch();
        } else {
            for (int e = 3; e >= 0; --e, ++evals) {
                rc = issue_bwd(a, ca[e], e == 3 ? nullptr : gu[evals & 1], cg[e], e ? uk + (e - 1) * 3 * n : x, n, pack,
                               W, ak + e * size, 4 * size, gz + e * size, gz + (4 + e) * size, e == 3 ? a : dx[k & 1],
                               dx[k & 1], gu[1 - (evals & 1)], partial, evals == 0, stream, !stored || evals > 0);
                if (rc) return rc;
            }
        }
        for (int l = 0; l < 2; ++l) {
            rc = issue_wgrad(gz + 4 * l * size, ak + 4 * l * size, 4 * rows, pack, W, 2 + l, wpart[l], k == steps - 1,
                             stream, true);
            if (rc) return rc;
        }
        a = dx[k & 1];
    }
    return issue_reduce(partial, n, wpart[0], wpart[1], 4 * rows, W, m, dW1, db1, dW2, db2, dW3, db3, dW4, db4, stream,
                        true);
}
