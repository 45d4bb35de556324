// Optimiser-step kernels: the stand-alone Adam update and the fused
// multi-pair step (DF loss + gradient, CSR-ordered edge gradient, mask and
// weights, Adam, loss partials) that advances every active deformation pair
// by one step per launch.
// Reference: the loop body of src/python/rigid_deform.py:35-39 with
// RigidLossFunction (src/python/layers/rigid_loss_layer.py:7-27) or
// GraphLossFunction (src/python/layers/graph_loss_layer.py:9-43) and
// torch.optim.Adam.
#include <algorithm>

#include "mo_lazydf.cuh"
#include "mo_wait.cuh"

namespace mo {

// torch/optim/adam.py _single_tensor_adam for one element:
//   m.lerp_(g, 1-b1); v.mul_(b2).addcmul_(g, g, value=1-b2);
//   denom = v.sqrt()/bc2_sqrt + eps; p.addcdiv_(m, denom, value=-step_size)
__device__ __forceinline__ void adam_elem(float& p, float g, float& m, float& v, float omb1, float b2, float omb2,
                                          float eps, float step_size, float bc2s) {
    m = fmaf(omb1, g - m, m);
    v = ADD(MUL(v, b2), MUL(MUL(omb2, g), g));
    const float denom = ADD(__fdiv_rn(__fsqrt_rn(v), bc2s), eps);
    p = fmaf(-step_size, __fdiv_rn(m, denom), p);
}

__global__ void __launch_bounds__(256) k_adam(float* __restrict__ P, const float* __restrict__ G,
                                              float* __restrict__ M, float* __restrict__ Vs, int64_t n,
                                              float omb1, float b2, float omb2, float eps, float step_size,
                                              float bc2s) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float p = P[i], m = M[i], v = Vs[i];
    adam_elem(p, G[i], m, v, omb1, b2, omb2, eps, step_size, bc2s);
    P[i] = p; M[i] = m; Vs[i] = v;
}

constexpr int STEP_THREADS = 256;  // 8 warps = up to 8 slices of 32 vertices
constexpr int TILE_WARPS = STEP_THREADS / 32;
static_assert(TILE_WARPS == MO_TILE_WARPS, "tile warps");
constexpr int REC_UNROLL = 3;      // record rows whose neighbours are gathered together

template <int LAYOUT>
__device__ __forceinline__ DFJet df_eval_layout(const float* grid, int N, float Nf, float Cf, float x, float y,
                                                float z) {
    return df_eval<LAYOUT, true>(grid, N, Nf, Cf, x, y, z);
}

// Every warp owns one 32-vertex slice of a tile and never waits for the
// other warps of its block.  ON_DEMAND: the pairs' grids are filled on
// demand, and a vertex moving into a cell not yet filled queues it (a
// separate instantiation: the queueing code slows the plain kernel down even
// when it is skipped).  WEIGHTED: every record carries a weight
// (MoPair.sell_w, NULL: 1): the gradient takes r * w^2 and the energy
// (r * w)^2 (CadEdgeLoss), another separate instantiation.
template <bool ON_DEMAND, bool WEIGHTED = false>
__global__ void __launch_bounds__(STEP_THREADS, 4) k_fused_step(const MoPair* __restrict__ pairs,
                                                             const MoTile* __restrict__ tiles,
                                                             const int* __restrict__ ntiles_p, int max_tiles,
                                                             int k, float* __restrict__ tile_loss) {
    const int ntiles = min(*ntiles_p, max_tiles);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const MoTile T = tiles[tile];
        const MoPair& P = pairs[T.pair];
        float* out = tile_loss + ((int64_t)k * max_tiles + tile) * TILE_WARPS + w;
        const int t = P.t0 + k + 1;
        if (t > P.t_end || w >= T.nslices) {  // warp-uniform
            if (lane == 0) *out = 0.f;
            continue;
        }
        const int slice = T.slice0 + w;
        const int nv = P.nv;
        const int i = slice * 32 + lane;
        const bool valid = i < nv;
        const float4* __restrict__ Vin = reinterpret_cast<const float4*>((t & 1) ? P.pos0 : P.pos1);
        float4* __restrict__ Vout = reinterpret_cast<float4*>((t & 1) ? P.pos1 : P.pos0);
        const float4* __restrict__ R = reinterpret_cast<const float4*>(P.rest);
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 p = valid ? Vin[i] : zero;
        const float4 r0 = valid ? __ldg(R + i) : zero;
        float* __restrict__ Mm = P.adam_m + 3 * (int64_t)i;
        float* __restrict__ Vv = P.adam_v + 3 * (int64_t)i;
        if (valid) {  // the moments are read after the edge loop
            asm volatile("prefetch.global.L1 [%0];" :: "l"(Mm));
            asm volatile("prefetch.global.L1 [%0];" :: "l"(Vv));
        }
        // The first record rows are requested before the distance-field cell
        // so that both gathers are in flight together.
        const int rb = P.slice_ptr[slice];
        const int rows = (P.slice_ptr[slice + 1] - rb) >> 5;
        const int* __restrict__ rec = P.sell + rb + lane;
        int c[REC_UNROLL];
#pragma unroll
        for (int u = 0; u < REC_UNROLL; ++u) c[u] = (u < rows) ? __ldg(rec + u * 32) : -1;
        const float* __restrict__ recw = WEIGHTED && P.sell_w ? P.sell_w + rb + lane : nullptr;
        const int N = P.N;
        const float Nf = (float)N, Cf = (float)((double)(N - 1) - 1e-3);
        const DFJet j = (P.layout == MO_LAYOUT_CELL)
                            ? df_eval_layout<MO_LAYOUT_CELL>(P.grid, N, Nf, Cf, p.x, p.y, p.z)
                            : (P.layout == MO_LAYOUT_BRICK4)
                                  ? df_eval_layout<MO_LAYOUT_BRICK4>(P.grid, N, Nf, Cf, p.x, p.y, p.z)
                                  : df_eval_layout<MO_LAYOUT_LINEAR>(P.grid, N, Nf, Cf, p.x, p.y, p.z);
        const float dsq = MUL(j.d, j.d);
        float gdx = df_grad_component(j.d, j.gx);
        float gdy = df_grad_component(j.d, j.gy);
        float gdz = df_grad_component(j.d, j.gz);
        if (P.use_mask) {
            const float mk = (MUL(dsq, 0.5f) < P.mask_thresh) ? 1.0f : 0.0f;
            gdx = MUL(gdx, mk); gdy = MUL(gdy, mk); gdz = MUL(gdz, mk);
        }
        // Edge residuals over this vertex's sliced-ELL column, in the order
        // of the reference's serial scatter.  Rest offset = rest[v1] - rest[v0].
        // The next rows' records are requested while this row's neighbours
        // are gathered.
        float grx = 0.f, gry = 0.f, grz = 0.f, esq = 0.f;
        for (int row = 0; row < rows; row += REC_UNROLL) {
            float4 q[REC_UNROLL], sr[REC_UNROLL];
#pragma unroll
            for (int u = 0; u < REC_UNROLL; ++u) {
                if (c[u] != -1) {
                    const int o = c[u] & 0x7fffffff;
                    q[u] = Vin[o];
                    sr[u] = __ldg(R + o);
                } else {
                    q[u] = zero;
                    sr[u] = zero;
                }
            }
            int cn[REC_UNROLL];
#pragma unroll
            for (int u = 0; u < REC_UNROLL; ++u)
                cn[u] = (row + REC_UNROLL + u < rows) ? __ldg(rec + (row + REC_UNROLL + u) * 32) : -1;
            // As v0 of a half-edge the vertex takes g -= r with r = (v1 - v0) - off;
            // as v1 it takes g += (v0 - v1) - (-off), which is the same
            // rounding of the same r with its sign flipped, so both roles
            // subtract r = (q - p) - (rest[q] - rest[p]); only v0 adds the
            // edge's energy.  Padding (-1) follows the last real record.
#pragma unroll
            for (int u = 0; u < REC_UNROLL; ++u) {
                const float rx = SUB(SUB(q[u].x, p.x), SUB(sr[u].x, r0.x));
                const float ry = SUB(SUB(q[u].y, p.y), SUB(sr[u].y, r0.y));
                const float rz = SUB(SUB(q[u].z, p.z), SUB(sr[u].z, r0.z));
                if (WEIGHTED) {
                    // (v1 - v0 - off) * (w * w) as cad_layer.cc:195-202
                    // rounds it; the v1 role's r is the v0 role's negated
                    const float we_ = (recw && c[u] != -1) ? __ldg(recw + (row + u) * 32) : 1.0f;
                    const float l2 = MUL(we_, we_);
                    if (c[u] != -1) {
                        grx = SUB(grx, MUL(rx, l2)); gry = SUB(gry, MUL(ry, l2)); grz = SUB(grz, MUL(rz, l2));
                    }
                    if (c[u] >= 0) {
                        const float ex = MUL(rx, we_), ey = MUL(ry, we_), ez = MUL(rz, we_);
                        esq += ex * ex + ey * ey + ez * ez;
                    }
                } else {
                    if (c[u] != -1) {
                        grx = SUB(grx, rx); gry = SUB(gry, ry); grz = SUB(grz, rz);
                    }
                    if (c[u] >= 0) esq += rx * rx + ry * ry + rz * rz;
                }
            }
            if (c[REC_UNROLL - 1] == -1) break;
#pragma unroll
            for (int u = 0; u < REC_UNROLL; ++u) c[u] = cn[u];
        }
        // grad_h * (gD + gR * w)  (graph_loss_layer.py:42, rigid_loss_layer.py:27)
        const float we = P.w_edge, gh = P.grad_scale;
        const float gx = MUL(gh, ADD(gdx, MUL(grx, we)));
        const float gy = MUL(gh, ADD(gdy, MUL(gry, we)));
        const float gz = MUL(gh, ADD(gdz, MUL(grz, we)));
        float part = 0.f;
        if (valid) {
            if (P.grad_dbg) {
                P.grad_dbg[3 * (int64_t)i] = gx;
                P.grad_dbg[3 * (int64_t)i + 1] = gy;
                P.grad_dbg[3 * (int64_t)i + 2] = gz;
            }
            const float2 ab = __ldg(reinterpret_cast<const float2*>(P.adam_tab) + (t - 1));
            float m0 = Mm[0], m1 = Mm[1], m2 = Mm[2];
            float v0 = Vv[0], v1 = Vv[1], v2 = Vv[2];
            float px = p.x, py = p.y, pz = p.z;
            adam_elem(px, gx, m0, v0, P.one_minus_b1, P.b2, P.one_minus_b2, P.eps, ab.x, ab.y);
            adam_elem(py, gy, m1, v1, P.one_minus_b1, P.b2, P.one_minus_b2, P.eps, ab.x, ab.y);
            adam_elem(pz, gz, m2, v2, P.one_minus_b1, P.b2, P.one_minus_b2, P.eps, ab.x, ab.y);
            Mm[0] = m0; Mm[1] = m1; Mm[2] = m2;
            Vv[0] = v0; Vv[1] = v1; Vv[2] = v2;
            Vout[i] = make_float4(px, py, pz, 0.f);
            if (ON_DEMAND && P.df_cells != nullptr && t < P.t_end) {  // the next step's cell
                int cn = lazy_cell_of(N, px, py, pz);
                if (cn == lazy_cell_of(N, p.x, p.y, p.z)) cn = -1;  // read by this step: written
                lazy_queue_cell(P, T.pair, cn, P.df_queue, P.df_pqueue, P.df_queue_count + 2 * k,
                                P.df_queue_cap);
            }
            part = 0.5f * dsq + we * (0.5f * esq);
        }
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        if (lane == 0) *out = part;
    }
}

// ---------------------------------------------------------------------------
// Many steps of one pair in one cooperative launch, for pairs whose every vertex
// can stay on the chip.  A launch per step is a chain of dependent loads (tile,
// pair, position, record, neighbour) behind a launch, and from 80k vertices on
// 370 bytes a vertex from L2.  Here a vertex's position, moments, records and
// rest offsets stay in registers and shared memory for all steps; a step is one
// gather of the neighbours' positions (L2), the arithmetic, one store and a grid
// barrier, beside which the next step's distance lookup and the loss partials
// run.  Bound: the latency of that gather and barrier.  Every operation on a
// value is k_fused_step's, in its order.
// ---------------------------------------------------------------------------
constexpr int RUN_REC = 12;  // records a thread keeps (a closed mesh's six neighbours twice); further ones are re-read
constexpr int RUN_CHUNK = 4096;  // steps of a launch

// The block's writes come before the release, by its barrier, and the release
// publishes them all; run_wait's acquire, before its block's barrier, is as good
// for every thread behind it.  (A full fence beside each cost 0.5 us a step.)
__device__ __forceinline__ void run_arrive(unsigned* bar) {
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
}

// Waits until every block has arrived `target` times in total; after two seconds
// of polling (or another block's) it gives up: false.
__device__ __forceinline__ bool run_wait(unsigned* bar, unsigned target) {
    __shared__ int ok;
    if (threadIdx.x == 0) {
        ok = 1;
        unsigned v, stop;
        WaitLimit limit(0);
        for (int n = 0;; ++n) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if ((int)(v - target) >= 0) break;
            if ((n & 1023) == 1023) {
                const uint32_t now = wait_clock();
                if (n == 1023) limit = WaitLimit(now);  // a clock reading a millisecond, none for a short wait
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(stop) : "l"(bar + 1) : "memory");
                if (stop || limit.over(now)) {
                    atomicExch(bar + 1, 1u);
                    ok = 0;
                    break;
                }
            }
        }
    }
    __syncthreads();
    return ok != 0;
}

// K vertices a thread, blocks of up to T threads; LOSS: with the steps' loss
// partials (else the energy is not summed).  What a thread keeps is 21
// registers a vertex and, in shared memory, 144 bytes of rest offsets:
//   T = 256, K = 1: two blocks an SM, all twelve neighbours gathered together;
//   T = 1024, K = 1: one block, 64 registers, four neighbours at a time;
//   T = 768, K = 2: one block, 80 registers, its offsets ~all of the shared
//     memory.  (Three vertices a thread of 512 were slower: 10.3 us a step at
//     200k vertices against 8.7, each vertex's gathers waiting for the one's before.)
// Measured, us a step (a launch per step, here): 10k 4.7, 2.65; 77k 5.6, 3.5;
// 150k 8.3, 5.4; 200k 10.4, 7.9; 230k 11.8, 8.5.
constexpr int RUN_WARPS1 = 32, RUN_WARPS2 = 24;
template <bool WEIGHTED, bool LOSS, int K, int T>
__global__ void __launch_bounds__(T, T == STEP_THREADS ? 2 : 1)
    k_fused_run(const __grid_constant__ MoPair P, int nsteps, float* __restrict__ tile_loss, int64_t loss_stride,
                unsigned* bar) {
    extern __shared__ float offs[];  // [K][RUN_REC][3][threads] rest offsets of the kept records
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nt = blockDim.x, warps = nt >> 5;
    const int slice0 = blockIdx.x * warps * K + w;  // and every warps-th after it
    const float4* __restrict__ R = reinterpret_cast<const float4*>(P.rest);
    float4* const pos0 = reinterpret_cast<float4*>(P.pos0);
    float4* const pos1 = reinterpret_cast<float4*>(P.pos1);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const int N = P.N;
    const float Nf = (float)N, Cf = (float)((double)(N - 1) - 1e-3);
    const float we = P.w_edge, gh = P.grad_scale;
    float3 p[K] = {}, m[K], v[K];
    int c[K][RUN_REC];
    bool valid[K];
    float dsq[K];
    float3 gd[K];
    auto rows_of = [&](int slice) { return (P.slice_ptr[slice + 1] - P.slice_ptr[slice]) >> 5; };
    auto lookup = [&](int j) {
        const float x = p[j].x, y = p[j].y, z = p[j].z;
        const DFJet d = (P.layout == MO_LAYOUT_CELL) ? df_eval_layout<MO_LAYOUT_CELL>(P.grid, N, Nf, Cf, x, y, z)
                        : (P.layout == MO_LAYOUT_BRICK4)
                            ? df_eval_layout<MO_LAYOUT_BRICK4>(P.grid, N, Nf, Cf, x, y, z)
                            : df_eval_layout<MO_LAYOUT_LINEAR>(P.grid, N, Nf, Cf, x, y, z);
        dsq[j] = MUL(d.d, d.d);
        gd[j] = make_float3(df_grad_component(d.d, d.gx), df_grad_component(d.d, d.gy), df_grad_component(d.d, d.gz));
        if (P.use_mask) {
            const float mk = (MUL(dsq[j], 0.5f) < P.mask_thresh) ? 1.0f : 0.0f;
            gd[j].x = MUL(gd[j].x, mk); gd[j].y = MUL(gd[j].y, mk); gd[j].z = MUL(gd[j].z, mk);
        }
    };
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const int slice = slice0 + j * warps;  // warp-uniform
        const int i = slice * 32 + lane;
        valid[j] = slice < P.nslices && i < P.nv;
        p[j] = m[j] = v[j] = make_float3(0.f, 0.f, 0.f);
        float4 r0 = zero;
        if (valid[j]) {
            const float4 q = ((P.t0 & 1) ? pos1 : pos0)[i];
            p[j] = make_float3(q.x, q.y, q.z);
            r0 = __ldg(R + i);
            const float* Mm = P.adam_m + 3 * (int64_t)i;
            const float* Vv = P.adam_v + 3 * (int64_t)i;
            m[j] = make_float3(Mm[0], Mm[1], Mm[2]);
            v[j] = make_float3(Vv[0], Vv[1], Vv[2]);
        }
        const int rows = slice < P.nslices ? rows_of(slice) : 0;
        const int* __restrict__ rec = P.sell + (rows ? P.slice_ptr[slice] : 0) + lane;
        float* o = offs + j * 3 * RUN_REC * nt + threadIdx.x;
#pragma unroll
        for (int u = 0; u < RUN_REC; ++u) {
            c[j][u] = u < rows ? __ldg(rec + u * 32) : -1;
            if (c[j][u] != -1) {
                const float4 s = __ldg(R + (c[j][u] & 0x7fffffff));
                o[(3 * u) * nt] = SUB(s.x, r0.x);
                o[(3 * u + 1) * nt] = SUB(s.y, r0.y);
                o[(3 * u + 2) * nt] = SUB(s.z, r0.z);
            }
        }
        lookup(j);
    }
    float2 ab = __ldg(reinterpret_cast<const float2*>(P.adam_tab) + P.t0);
    for (int k = 0; k < nsteps; ++k) {
        const int t = P.t0 + k + 1;
        const float4* Vin = (t & 1) ? pos0 : pos1;
        float4* Vout = (t & 1) ? pos1 : pos0;
        float part[K];
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const int slice = slice0 + j * warps;
            const int i = slice * 32 + lane;
            const float* o = offs + j * 3 * RUN_REC * nt + threadIdx.x;
            const float* __restrict__ recw =
                WEIGHTED && P.sell_w && slice < P.nslices ? P.sell_w + P.slice_ptr[slice] + lane : nullptr;
            float grx = 0.f, gry = 0.f, grz = 0.f, esq = 0.f;
            auto edge = [&](int cu, float4 qu, float ox, float oy, float oz, int row) {
                const float rx = SUB(SUB(qu.x, p[j].x), ox);
                const float ry = SUB(SUB(qu.y, p[j].y), oy);
                const float rz = SUB(SUB(qu.z, p[j].z), oz);
                if (WEIGHTED) {
                    const float we_ = recw ? __ldg(recw + row * 32) : 1.0f;
                    const float l2 = MUL(we_, we_);
                    grx = SUB(grx, MUL(rx, l2)); gry = SUB(gry, MUL(ry, l2)); grz = SUB(grz, MUL(rz, l2));
                    if (LOSS && cu >= 0) {
                        const float ex = MUL(rx, we_), ey = MUL(ry, we_), ez = MUL(rz, we_);
                        esq += ex * ex + ey * ey + ez * ez;
                    }
                } else {
                    grx = SUB(grx, rx); gry = SUB(gry, ry); grz = SUB(grz, rz);
                    if (LOSS && cu >= 0) esq += rx * rx + ry * ry + rz * rz;
                }
            };
            constexpr int B = T == STEP_THREADS ? RUN_REC : 4;  // gathered together
#pragma unroll
            for (int u0 = 0; u0 < RUN_REC; u0 += B) {
                float4 q[B];
#pragma unroll
                for (int u = 0; u < B; ++u) q[u] = c[j][u0 + u] != -1 ? Vin[c[j][u0 + u] & 0x7fffffff] : zero;
#pragma unroll
                for (int u = 0; u < B; ++u)
                    if (c[j][u0 + u] != -1)
                        edge(c[j][u0 + u], q[u], o[(3 * (u0 + u)) * nt], o[(3 * (u0 + u) + 1) * nt],
                             o[(3 * (u0 + u) + 2) * nt], u0 + u);
            }
            if (c[j][RUN_REC - 1] != -1) {  // the records that were not kept
                const int rows = rows_of(slice);
                const int* __restrict__ rec = P.sell + P.slice_ptr[slice] + lane;
                const float4 r0 = __ldg(R + i);
                if (T == STEP_THREADS) {
                    // a vertex of a CAD mesh can have hundreds: four at a time, their
                    // numbers a round ahead (5,912 vertices with up to 60: 18.3 us a step
                    // one after the other, 6.3 so, 10.7 with a launch per step)
                    constexpr int MORE = 4;
                    int cu[MORE];
#pragma unroll
                    for (int u = 0; u < MORE; ++u) cu[u] = RUN_REC + u < rows ? __ldg(rec + (RUN_REC + u) * 32) : -1;
                    for (int row = RUN_REC; row < rows; row += MORE) {
                        float4 q[MORE], s[MORE];
#pragma unroll
                        for (int u = 0; u < MORE; ++u) {
                            const int n = cu[u] != -1 ? cu[u] & 0x7fffffff : i;
                            q[u] = Vin[n];
                            s[u] = __ldg(R + n);
                        }
                        int cn[MORE];
#pragma unroll
                        for (int u = 0; u < MORE; ++u)
                            cn[u] = row + MORE + u < rows ? __ldg(rec + (row + MORE + u) * 32) : -1;
#pragma unroll
                        for (int u = 0; u < MORE; ++u)
                            if (cu[u] != -1)
                                edge(cu[u], q[u], SUB(s[u].x, r0.x), SUB(s[u].y, r0.y), SUB(s[u].z, r0.z), row + u);
                        if (cu[MORE - 1] == -1) break;  // padding follows the last record
#pragma unroll
                        for (int u = 0; u < MORE; ++u) cu[u] = cn[u];
                    }
                } else {  // no registers for that: see mo_fused_run_pays
                    for (int row = RUN_REC; row < rows; ++row) {
                        const int cu = __ldg(rec + row * 32);
                        if (cu == -1) break;  // padding follows the last record
                        const int n = cu & 0x7fffffff;
                        const float4 s = __ldg(R + n);
                        edge(cu, Vin[n], SUB(s.x, r0.x), SUB(s.y, r0.y), SUB(s.z, r0.z), row);
                    }
                }
            }
            const float gx = MUL(gh, ADD(gd[j].x, MUL(grx, we)));
            const float gy = MUL(gh, ADD(gd[j].y, MUL(gry, we)));
            const float gz = MUL(gh, ADD(gd[j].z, MUL(grz, we)));
            part[j] = 0.f;
            if (valid[j]) {
                if (LOSS) part[j] = 0.5f * dsq[j] + we * (0.5f * esq);
                if (P.grad_dbg) {
                    P.grad_dbg[3 * (int64_t)i] = gx;
                    P.grad_dbg[3 * (int64_t)i + 1] = gy;
                    P.grad_dbg[3 * (int64_t)i + 2] = gz;
                }
                adam_elem(p[j].x, gx, m[j].x, v[j].x, P.one_minus_b1, P.b2, P.one_minus_b2, P.eps, ab.x, ab.y);
                adam_elem(p[j].y, gy, m[j].y, v[j].y, P.one_minus_b1, P.b2, P.one_minus_b2, P.eps, ab.x, ab.y);
                adam_elem(p[j].z, gz, m[j].z, v[j].z, P.one_minus_b1, P.b2, P.one_minus_b2, P.eps, ab.x, ab.y);
                Vout[i] = make_float4(p[j].x, p[j].y, p[j].z, 0.f);
            }
        }
        const bool more = k + 1 < nsteps;
        if (more) run_arrive(bar);
        if (LOSS) {
#pragma unroll
            for (int j = 0; j < K; ++j) {
                const int slice = slice0 + j * warps;
                if (slice >= P.ntiles * TILE_WARPS) continue;
                float s = part[j];
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (lane == 0) tile_loss[(int64_t)k * loss_stride + slice] = s;
            }
        }
        if (!more) break;
        ab = __ldg(reinterpret_cast<const float2*>(P.adam_tab) + t);
#pragma unroll
        for (int j = 0; j < K; ++j) lookup(j);
        if (!run_wait(bar, (unsigned)(k + 1) * gridDim.x)) {  // never in a working launch: no result
#pragma unroll
            for (int j = 0; j < K; ++j) {
                const int i = (slice0 + j * warps) * 32 + lane;
                if (valid[j]) pos0[i] = pos1[i] = make_float4(NAN, NAN, NAN, 0.f);
            }
            return;
        }
    }
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const int i = (slice0 + j * warps) * 32 + lane;
        if (!valid[j]) continue;
        float* Mm = P.adam_m + 3 * (int64_t)i;
        float* Vv = P.adam_v + 3 * (int64_t)i;
        Mm[0] = m[j].x; Mm[1] = m[j].y; Mm[2] = m[j].z;
        Vv[0] = v[j].x; Vv[1] = v[j].y; Vv[2] = v[j].z;
    }
}

// Vertices a thread, warps of a block and blocks of a run over nslices slices
// (blocks 0: they do not fit the chip at once): an SM's share of them in two
// blocks of up to 8, in one of up to 32, or in one of up to 24 warps twice.
static void run_shape(int nslices, int* per_thread, int* warps, int* blocks) {
    const int sms = device_sm_count();
    const int share = (nslices + sms - 1) / sms;
    int max_blocks = sms;
    if (share <= 2 * TILE_WARPS) {
        *per_thread = 1;
        *warps = std::max(1, std::min(TILE_WARPS, share));
        max_blocks = 2 * sms;
    } else if (share <= RUN_WARPS1) {
        *per_thread = 1;
        *warps = share;
    } else {
        *per_thread = 2;
        *warps = std::min(RUN_WARPS2, (share + 1) / 2);
    }
    const int per_block = *warps * *per_thread;
    *blocks = (nslices + per_block - 1) / per_block;
    if (*blocks > max_blocks) *blocks = 0;
}

template <bool WEIGHTED, bool LOSS>
static const void* run_kernel_of(int per_thread, int warps) {
    if (per_thread == 2) return (const void*)k_fused_run<WEIGHTED, LOSS, 2, 32 * RUN_WARPS2>;
    if (warps > TILE_WARPS) return (const void*)k_fused_run<WEIGHTED, LOSS, 1, 32 * RUN_WARPS1>;
    return (const void*)k_fused_run<WEIGHTED, LOSS, 1, STEP_THREADS>;
}

static const void* run_kernel(bool weighted, bool loss, int per_thread, int warps) {
    if (weighted) return loss ? run_kernel_of<true, true>(per_thread, warps) : run_kernel_of<true, false>(per_thread, warps);
    return loss ? run_kernel_of<false, true>(per_thread, warps) : run_kernel_of<false, false>(per_thread, warps);
}

// One warp per (pair, launch): lane l sums the pair's tile partials l, l+32,
// ... in double, then a fixed shuffle tree adds the 32 lane sums.  The order
// is fixed, so the result does not depend on scheduling.
__global__ void __launch_bounds__(128) k_pair_loss(const MoPair* __restrict__ pairs, int npairs, int max_tiles,
                                                   int nlaunch, const float* __restrict__ tile_loss,
                                                   double* __restrict__ out) {
    const int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (q >= (int64_t)npairs * nlaunch) return;  // warp-uniform
    const int p = (int)(q % npairs), k = (int)(q / npairs);
    const MoPair& P = pairs[p];
    const float* base = tile_loss + (int64_t)k * max_tiles * TILE_WARPS;
    const int64_t t0 = (int64_t)P.tile0 * TILE_WARPS, t1 = (int64_t)(P.tile0 + P.ntiles) * TILE_WARPS;
    double s = 0.0;
    for (int64_t t = t0 + lane; t < t1; t += 32) s += (double)base[t];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) out[(int64_t)k * npairs + p] = s;
}

__global__ void k_pack(const float* __restrict__ V, int64_t n, float4* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = make_float4(V[3 * i], V[3 * i + 1], V[3 * i + 2], 0.f);
}

__global__ void k_unpack(const float4* __restrict__ P, int64_t n, float* __restrict__ V) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const float4 p = P[i];
        V[3 * i] = p.x; V[3 * i + 1] = p.y; V[3 * i + 2] = p.z;
    }
}

static int g_step_ctas = 0;

static int step_ctas() {
    if (g_step_ctas == 0) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fused_step<false>, STEP_THREADS, 0) !=
                cudaSuccess ||
            per_sm <= 0)
            per_sm = 4;
        g_step_ctas = per_sm * device_sm_count();
    }
    return g_step_ctas;
}

}  // namespace mo

using namespace mo;

extern "C" int mo_adam_step(float* P, const float* G, float* M, float* Vsq, int64_t n, float one_minus_b1, float b2,
                            float one_minus_b2, float eps, float step_size, float bc2_sqrt, void* stream) {
    MO_CHECK_ARG(n >= 0, "negative size");
    if (n == 0) return MO_OK;
    MO_CHECK_ARG(P && G && M && Vsq, "null pointer");
    k_adam<<<ceil_div(n, 256), 256, 0, as_stream(stream)>>>(P, G, M, Vsq, n, one_minus_b1, b2, one_minus_b2, eps,
                                                           step_size, bc2_sqrt); ::mo::note_launch();
    MO_LAUNCH_CHECK("k_adam");
    return MO_OK;
}

static int launch_fused_step(int variant, const MoPair* pairs, const MoTile* tiles, const int32_t* ntiles,
                             int max_tiles, int launch_index, float* tile_loss, int grid_ctas, void* stream) {
    MO_CHECK_ARG(pairs && tiles && ntiles && tile_loss, "null pointer");
    MO_CHECK_ARG(max_tiles >= 0 && launch_index >= 0, "negative size");
    if (max_tiles == 0) return MO_OK;
    int ctas = grid_ctas > 0 ? grid_ctas : step_ctas();
    if (ctas > max_tiles) ctas = max_tiles;
    if (variant == 1)
        k_fused_step<true><<<ctas, STEP_THREADS, 0, as_stream(stream)>>>(pairs, tiles, ntiles, max_tiles,
                                                                         launch_index, tile_loss);
    else if (variant == 2)
        k_fused_step<false, true><<<ctas, STEP_THREADS, 0, as_stream(stream)>>>(pairs, tiles, ntiles, max_tiles,
                                                                                launch_index, tile_loss);
    else
        k_fused_step<false><<<ctas, STEP_THREADS, 0, as_stream(stream)>>>(pairs, tiles, ntiles, max_tiles,
                                                                          launch_index, tile_loss);
    ::mo::note_launch();
    MO_LAUNCH_CHECK("k_fused_step");
    return MO_OK;
}

extern "C" int mo_fused_step(const MoPair* pairs, const MoTile* tiles, const int32_t* ntiles, int max_tiles,
                             int launch_index, float* tile_loss, int grid_ctas, void* stream) {
    return launch_fused_step(0, pairs, tiles, ntiles, max_tiles, launch_index, tile_loss, grid_ctas, stream);
}

extern "C" int mo_fused_step_weighted(const MoPair* pairs, const MoTile* tiles, const int32_t* ntiles, int max_tiles,
                                      int launch_index, float* tile_loss, int grid_ctas, void* stream) {
    return launch_fused_step(2, pairs, tiles, ntiles, max_tiles, launch_index, tile_loss, grid_ctas, stream);
}

extern "C" int mo_fused_step_on_demand(const MoPair* pairs, const MoTile* tiles, const int32_t* ntiles,
                                       int max_tiles, int launch_index, float* tile_loss, int grid_ctas,
                                       void* stream) {
    return launch_fused_step(1, pairs, tiles, ntiles, max_tiles, launch_index, tile_loss, grid_ctas, stream);
}

extern "C" int mo_fused_run_fits(int64_t nv) {
    if (nv <= 0 || nv > ((int64_t)1 << 30)) return 0;
    int per_thread, warps, blocks;
    run_shape((int)((nv + 31) / 32), &per_thread, &warps, &blocks);
    return blocks > 0 ? 1 : 0;
}

// With more than 512 vertices an SM the records past the kept ones are read one
// after the other, 0.26 us a step for each of the longest row: with nine of them
// a launch per step is as fast (93k vertices with up to 60 records: 10.8 us against
// 17.0; without long rows 6.7 against 4.5).
extern "C" int mo_fused_run_pays(int64_t nv, int max_rows) {
    if (nv <= 0 || nv > ((int64_t)1 << 30)) return 0;
    int per_thread, warps, blocks;
    run_shape((int)((nv + 31) / 32), &per_thread, &warps, &blocks);
    return blocks > 0 && (warps <= TILE_WARPS || max_rows <= RUN_REC + 8) ? 1 : 0;
}

extern "C" int mo_fused_run(const MoPair* pair, int weighted, int nsteps, float* tile_loss, int64_t loss_stride,
                            uint32_t* sync, void* stream) {
    MO_CHECK_ARG(pair && sync, "null pointer");
    MO_CHECK_ARG(nsteps >= 0, "negative step count");
    const MoPair& q = *pair;
    MO_CHECK_ARG(q.nv > 0 && q.nslices == (q.nv + 31) / 32 && q.N >= 2, "bad pair sizes");
    MO_CHECK_ARG(q.grid && q.slice_ptr && q.sell && q.rest && q.pos0 && q.pos1 && q.adam_m && q.adam_v && q.adam_tab,
                 "null pointer in the pair");
    MO_CHECK_ARG(!tile_loss || (q.ntiles >= (q.nslices + TILE_WARPS - 1) / TILE_WARPS &&
                                loss_stride >= (int64_t)q.ntiles * TILE_WARPS),
                 "loss partials need whole tiles of %d slices", TILE_WARPS);
    MO_CHECK_ARG(q.t0 >= 0 && nsteps <= q.t_end - q.t0, "more steps than the pair has left");
    int per_thread, warps, blocks;
    run_shape(q.nslices, &per_thread, &warps, &blocks);
    MO_CHECK_ARG(blocks > 0, "%d vertices do not fit one launch (mo_fused_run_fits)", q.nv);
    if (tile_loss) {  // the slices past the last one of its tile
        const int pad = q.ntiles * TILE_WARPS - q.nslices;
        if (pad > 0 && nsteps > 0)
            MO_CUDA(cudaMemset2DAsync(tile_loss + q.nslices, sizeof(float) * loss_stride, 0, sizeof(float) * pad, nsteps,
                                      as_stream(stream)));
    }
    auto smem_of = [](int slices) { return RUN_REC * 3 * (int)sizeof(float) * 32 * slices; };
    const int smem = smem_of(warps * per_thread);
    const void* kernel = run_kernel(weighted != 0, tile_loss != nullptr, per_thread, warps);
    // a limit belongs to the kernel and not to a call: every thread sets the kernel's largest
    if (per_thread == 2 || warps > TILE_WARPS)
        MO_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     smem_of(per_thread == 2 ? 2 * RUN_WARPS2 : RUN_WARPS1)));
    for (int done = 0; done < nsteps;) {
        int n = std::min(RUN_CHUNK, nsteps - done);
        MoPair p = q;
        p.t0 += done;
        float* loss = tile_loss ? tile_loss + (int64_t)done * loss_stride : nullptr;
        unsigned* bar = sync;
        MO_CUDA(cudaMemsetAsync(sync, 0, 8, as_stream(stream)));
        void* args[] = {&p, &n, &loss, &loss_stride, &bar};
        const cudaError_t e =
            cudaLaunchCooperativeKernel(kernel, dim3(blocks), dim3(32 * warps), args, smem, as_stream(stream));
        if (e == cudaErrorCooperativeLaunchTooLarge && done == 0) {
            cudaGetLastError();
            set_error("%d blocks do not fit this context's SMs at once", blocks);
            return MO_ERR_TOO_LARGE;
        }
        MO_CUDA(e);
        ::mo::note_launch();
        done += n;
    }
    return MO_OK;
}

extern "C" int mo_pair_loss(const MoPair* pairs, int npairs, int max_tiles, int nlaunch, const float* tile_loss,
                            double* pair_loss, void* stream) {
    MO_CHECK_ARG(npairs >= 0 && nlaunch >= 0 && max_tiles >= 0, "negative size");
    const int64_t n = (int64_t)npairs * nlaunch;
    if (n == 0) return MO_OK;
    MO_CHECK_ARG(pairs && tile_loss && pair_loss, "null pointer");
    k_pair_loss<<<ceil_div(n, 4), 128, 0, as_stream(stream)>>>(pairs, npairs, max_tiles, nlaunch, tile_loss,
                                                              pair_loss); ::mo::note_launch();
    MO_LAUNCH_CHECK("k_pair_loss");
    return MO_OK;
}

extern "C" int mo_pack_pos(const float* V, int64_t n, float* pos4, void* stream) {
    MO_CHECK_ARG(n >= 0, "negative size");
    if (n == 0) return MO_OK;
    MO_CHECK_ARG(V && pos4 && aligned(pos4, 16), "null or misaligned pointer");
    k_pack<<<ceil_div(n, 256), 256, 0, as_stream(stream)>>>(V, n, reinterpret_cast<float4*>(pos4)); ::mo::note_launch();
    MO_LAUNCH_CHECK("k_pack");
    return MO_OK;
}

extern "C" int mo_unpack_pos(const float* pos4, int64_t n, float* V, void* stream) {
    MO_CHECK_ARG(n >= 0, "negative size");
    if (n == 0) return MO_OK;
    MO_CHECK_ARG(V && pos4 && aligned(pos4, 16), "null or misaligned pointer");
    k_unpack<<<ceil_div(n, 256), 256, 0, as_stream(stream)>>>(reinterpret_cast<const float4*>(pos4), n, V); ::mo::note_launch();
    MO_LAUNCH_CHECK("k_unpack");
    return MO_OK;
}

extern "C" int mo_abi_sizes(size_t* pair_bytes, size_t* tile_bytes) {
    MO_CHECK_ARG(pair_bytes && tile_bytes, "null pointer");
    *pair_bytes = sizeof(MoPair);
    *tile_bytes = sizeof(MoTile);
    return MO_OK;
}
