// The loss of a layer and its gradient, each in one pass: the distance-field
// term and the edge term together (src/python/layers/rigid_loss_layer.py:7-27,
// graph_loss_layer.py:9-43).
//
// As separate calls an evaluation wrote d^2 per vertex and three squares per
// half-edge, scaled both, summed both and added the sums: eight launches of
// 2-8 us for 10k vertices, each behind its own call from the host (445 us for
// an evaluation with its gradient, 291 now, nearly all of it the host), and 12
// bytes a half-edge written and read twice.  Here the terms are summed where
// they are made.  Every term is rounded as before; a thread's sum keeps its
// rounding errors, a block's is in double in the order of its threads, so the loss
// is the same in every run.
#include <algorithm>

#include "mo_df_eval.cuh"
#include "mo_edge.cuh"

namespace mo {

constexpr int LAYER_THREADS = 256;

__device__ __forceinline__ double block_sum(double v, double* sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) sh[w] = v;
    __syncthreads();
    v = 0.0;
    if (threadIdx.x == 0)
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) v += sh[k];
    return v;  // thread 0
}

// A sum of floats that are not negative and its rounding errors (Knuth's two-sum):
// as good as double for a fraction of the time of 2 FP64 lanes a clock and SM.
struct Sum {
    float hi = 0.f, lo = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float t = ADD(hi, x), b = SUB(t, hi);
        lo = ADD(lo, ADD(SUB(hi, SUB(t, b)), SUB(x, b)));
        hi = t;
    }
    __device__ __forceinline__ double value() const { return isfinite(hi) ? (double)hi + (double)lo : (double)hi; }
};

// Blocks of a kind at most: past them a thread takes several vertices or half-edges,
// since a block's sum in double costs 5 FP64 instructions a thread.  (With one each and
// all sums in double a loss over 60 M half-edges took 1640 us, as separate calls 890.
// 378 here.)
constexpr int LAYER_BLOCKS = 2048;
static int layer_blocks(int64_t n) { return (int)std::min<int64_t>((n + LAYER_THREADS - 1) / LAYER_THREADS, LAYER_BLOCKS); }

// Blocks [0, vblocks): 0.5 d^2 of the vertices (and with GRAD the
// distance term's gradient, zeroed where 0.5 d^2 >= mask).  The others:
// 0.5 r^2 of the half-edges.  partial[block] = the block's sum.
template <int LAYOUT, bool GRAD>
__global__ void __launch_bounds__(LAYER_THREADS)
    k_layer_forward(const float* __restrict__ V, int64_t nv, const float* __restrict__ grid, int N, float Nf, float Cf,
                    const int32_t* __restrict__ idx, int64_t nh, int kind, const float* __restrict__ off, int vblocks,
                    float mask, double* __restrict__ partial, float* __restrict__ grad) {
    __shared__ double sh[LAYER_THREADS / 32];
    Sum sum;
    if ((int)blockIdx.x < vblocks) {
        for (int64_t i = (int64_t)blockIdx.x * LAYER_THREADS + threadIdx.x; i < nv;
             i += (int64_t)vblocks * LAYER_THREADS) {
            const DFJet j = df_eval<LAYOUT, GRAD>(grid, N, Nf, Cf, V[3 * i], V[3 * i + 1], V[3 * i + 2]);
            const float half = MUL(MUL(j.d, j.d), 0.5f);
            sum.add(half);
            if (GRAD) {
                const float m = half < mask ? 1.0f : 0.0f;
                grad[3 * i] = MUL(df_grad_component(j.d, j.gx), m);
                grad[3 * i + 1] = MUL(df_grad_component(j.d, j.gy), m);
                grad[3 * i + 2] = MUL(df_grad_component(j.d, j.gz), m);
            }
        }
    } else {
        const int64_t step = (int64_t)(gridDim.x - vblocks) * LAYER_THREADS;
#pragma unroll 2
        for (int64_t h = (int64_t)(blockIdx.x - vblocks) * LAYER_THREADS + threadIdx.x; h < nh; h += step) {
            int v0, v1;
            he_ends(idx, kind, h, v0, v1);
            const bool ok = in_range(v0, nv) && in_range(v1, nv);
            for (int c = 0; c < 3; ++c) {
                const float r = ok ? SUB(SUB(V[3 * (int64_t)v1 + c], V[3 * (int64_t)v0 + c]), off[3 * h + c])
                                   : __int_as_float(0x7fc00000);
                sum.add(MUL(MUL(r, r), 0.5f));
            }
        }
    }
    const double total = block_sum(sum.value(), sh);
    if (threadIdx.x == 0) partial[blockIdx.x] = total;
}

// loss = sum of the vertex blocks + r2 * sum of the edge blocks, the two sums
// rounded to float first, as torch's were.
constexpr int LAYER_SUM_THREADS = 512;
__global__ void __launch_bounds__(LAYER_SUM_THREADS) k_layer_sum(const double* __restrict__ partial, int vblocks,
                                                                 int blocks, float r2, float* __restrict__ loss) {
    __shared__ double sh[2][LAYER_SUM_THREADS / 32];
    double d = 0.0, r = 0.0;
    for (int k = threadIdx.x; k < vblocks; k += LAYER_SUM_THREADS) d += partial[k];
    for (int k = vblocks + threadIdx.x; k < blocks; k += LAYER_SUM_THREADS) r += partial[k];
    d = block_sum(d, sh[0]);
    r = block_sum(r, sh[1]);
    if (threadIdx.x == 0) *loss = ADD((float)d, MUL((float)r, r2));
}

// grad[i] = distance term + r2 * edge term, a vertex a thread.  gd: the
// distance term's gradient where the forward pass made it, else it is
// evaluated here.
template <int LAYOUT>
__global__ void __launch_bounds__(LAYER_THREADS)
    k_layer_backward(const float* __restrict__ V, int64_t nv, const float* __restrict__ grid, int N, float Nf, float Cf,
                     const int* __restrict__ row_ptr, const int* __restrict__ key, const int* __restrict__ other,
                     const float* __restrict__ off, const float* __restrict__ gd, float r2, float* __restrict__ grad) {
    const int64_t i = (int64_t)blockIdx.x * LAYER_THREADS + threadIdx.x;
    if (i >= nv) return;
    float d0, d1, d2, gx, gy, gz;
    if (gd) {
        d0 = gd[3 * i]; d1 = gd[3 * i + 1]; d2 = gd[3 * i + 2];
    } else {
        const DFJet j = df_eval<LAYOUT, true>(grid, N, Nf, Cf, V[3 * i], V[3 * i + 1], V[3 * i + 2]);
        d0 = df_grad_component(j.d, j.gx);
        d1 = df_grad_component(j.d, j.gy);
        d2 = df_grad_component(j.d, j.gz);
    }
    edge_gather(V, i, row_ptr, key, other, off, gx, gy, gz);
    grad[3 * i] = ADD(d0, MUL(gx, r2));
    grad[3 * i + 1] = ADD(d1, MUL(gy, r2));
    grad[3 * i + 2] = ADD(d2, MUL(gz, r2));
}

static inline float far_offset(int N) { return (float)((double)(N - 1) - 1e-3); }

static int check_layer(const float* V, int64_t nv, const float* grid, int N, int layout, int64_t nh,
                       const float* off) {
    MO_CHECK_ARG(nv >= 0 && nh >= 0, "negative size");
    MO_CHECK_ARG(N >= 2, "grid resolution must be >= 2 (got %d)", N);
    MO_CHECK_ARG(layout == MO_LAYOUT_LINEAR || layout == MO_LAYOUT_CELL || layout == MO_LAYOUT_BRICK4,
                 "unknown grid layout %d", layout);
    MO_CHECK_ARG(nv == 0 || (V && grid), "null vertex or grid pointer");
    MO_CHECK_ARG(nh == 0 || off, "null rest offsets");
    MO_CHECK_ARG(layout != MO_LAYOUT_CELL || aligned(grid, 16), "cell-layout grid must be 16-byte aligned");
    MO_CHECK_ARG(layout != MO_LAYOUT_BRICK4 || N <= 1280, "brick layout supports N <= 1280");
    return MO_OK;
}

}  // namespace mo

using namespace mo;

extern "C" size_t mo_layer_scratch_bytes(int64_t nv, int64_t nh) {
    if (nv < 0 || nh < 0) return 0;
    return sizeof(double) * ((size_t)layer_blocks(nv) + (size_t)layer_blocks(nh) + 1);
}

extern "C" int mo_layer_forward(const float* V, int64_t nv, const float* grid, int N, int layout, const int32_t* idx,
                                int64_t n_items, int kind, const float* off, float r2, float* df_grad, float mask,
                                void* scratch, size_t scratch_bytes, float* loss, void* stream) {
    MO_CHECK_ARG(kind == MO_EDGES_FACES || kind == MO_EDGES_LIST, "unknown edge kind %d", kind);
    const int64_t nh = mo_edge_count(n_items, kind);
    const int rc = check_layer(V, nv, grid, N, layout, nh, off);
    if (rc) return rc;
    MO_CHECK_ARG(loss && scratch && (nh == 0 || idx), "null pointer");
    MO_CHECK_ARG(aligned(scratch, 8), "scratch must be 8-byte aligned");
    if (scratch_bytes < mo_layer_scratch_bytes(nv, nh)) {
        set_error("layer scratch too small: %zu < %zu", scratch_bytes, mo_layer_scratch_bytes(nv, nh));
        return MO_ERR_SCRATCH;
    }
    cudaStream_t s = as_stream(stream);
    double* partial = reinterpret_cast<double*>(scratch);
    const int vblocks = layer_blocks(nv), blocks = vblocks + layer_blocks(nh);
    const float Nf = (float)N, Cf = far_offset(N);
    if (blocks > 0) {
#define MO_LAYER(LAYOUT, GRAD)                                                                                     \
    k_layer_forward<LAYOUT, GRAD><<<blocks, LAYER_THREADS, 0, s>>>(V, nv, grid, N, Nf, Cf, idx, nh, kind, off,     \
                                                                   vblocks, mask, partial, df_grad)
        if (layout == MO_LAYOUT_CELL) {
            if (df_grad) MO_LAYER(MO_LAYOUT_CELL, true); else MO_LAYER(MO_LAYOUT_CELL, false);
        } else if (layout == MO_LAYOUT_BRICK4) {
            if (df_grad) MO_LAYER(MO_LAYOUT_BRICK4, true); else MO_LAYER(MO_LAYOUT_BRICK4, false);
        } else {
            if (df_grad) MO_LAYER(MO_LAYOUT_LINEAR, true); else MO_LAYER(MO_LAYOUT_LINEAR, false);
        }
#undef MO_LAYER
        ::mo::note_launch();
    }
    k_layer_sum<<<1, LAYER_SUM_THREADS, 0, s>>>(partial, vblocks, blocks, r2, loss); ::mo::note_launch();
    MO_LAUNCH_CHECK("k_layer_forward");
    return MO_OK;
}

extern "C" int mo_layer_backward(const float* V, int64_t nv, const float* grid, int N, int layout, const void* csr,
                                 int64_t nh, const float* off, const float* df_grad, float r2, float* grad_out,
                                 void* stream) {
    const int rc = check_layer(V, nv, grid, N, layout, nh, off);
    if (rc) return rc;
    if (nv == 0) return MO_OK;
    MO_CHECK_ARG(csr && grad_out, "null pointer");
    const CsrView c = csr_view(const_cast<void*>(csr), nv, nh);
    cudaStream_t s = as_stream(stream);
    const float Nf = (float)N, Cf = far_offset(N);
    const int blocks = ceil_div(nv, LAYER_THREADS);
#define MO_LAYER(LAYOUT)                                                                                            \
    k_layer_backward<LAYOUT><<<blocks, LAYER_THREADS, 0, s>>>(V, nv, grid, N, Nf, Cf, c.row_ptr, c.key, c.other,    \
                                                              off, df_grad, r2, grad_out)
    if (layout == MO_LAYOUT_CELL) MO_LAYER(MO_LAYOUT_CELL);
    else if (layout == MO_LAYOUT_BRICK4) MO_LAYER(MO_LAYOUT_BRICK4);
    else MO_LAYER(MO_LAYOUT_LINEAR);
#undef MO_LAYER
    ::mo::note_launch();
    MO_LAUNCH_CHECK("k_layer_backward");
    return MO_OK;
}
