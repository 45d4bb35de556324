// Nearest source vertex of every target vertex, and the reverse
// (target -> source) loss of src/python/layers/reverse_loss_layer.py:14-25:
//   ii = cKDTree(src).query(tar, k=1);  loss = 0.5 * sum |src[ii] - tar|^2.
//
// The query builds an LBVH over the source points (Morton codes in the points'
// bounding cube, stable radix sort, Karras tree, node boxes: the stages of the
// distance-field build) and walks it once per target point, one thread per
// query, queries taken in Morton order so a warp's queries are neighbours.
// Distances are squared Euclidean in double, summed x, y, z like cKDTree's
// (src/scipy cKDTree evaluates them in float64 from the float32 input), boxes
// culled by float lower bounds; among exactly equal distances the lowest source
// index wins.
#include <cfloat>

#include "mo_bbox.cuh"
#include "mo_common.cuh"
#include "mo_lbvh.cuh"

namespace mo {
namespace {

constexpr int NN_STACK = 64;
constexpr int CHUNK = 256;

// Points and queries are sorted in one go, the queries' codes above the points'.
bool sort_together(int64_t np, int64_t nq) { return np + nq < ((int64_t)1 << 30); }
constexpr uint32_t QUERY = 1u << 30;

struct NnScratch {
    int* bbox;        // 6 ordered ints
    float4* cube;     // lo.xyz, 1/extent
    int* status;
    uint32_t* codes_a;  // points, then queries
    uint32_t* codes_b;
    int* ids_a;
    int* ids_b;
    float4* nodes;
    float4* boxes;
    int* parent;
    int* flags;
    int2* range;
    float4* chunks;   // boxes of CHUNK leaves
    int* hist;
    size_t bytes;
};

size_t a256(size_t x) { return (x + 255) & ~(size_t)255; }

NnScratch plan(char* base, int64_t np, int64_t nq) {
    NnScratch s;
    size_t o = 0;
    auto take = [&](size_t bytes) {
        char* p = base ? base + o : nullptr;
        o += a256(bytes);
        return p;
    };
    s.bbox = reinterpret_cast<int*>(take(32));
    s.cube = reinterpret_cast<float4*>(take(16));
    s.status = reinterpret_cast<int*>(take(16));
    const size_t all = (size_t)np + (size_t)nq;
    s.codes_a = reinterpret_cast<uint32_t*>(take(4 * all));
    s.codes_b = reinterpret_cast<uint32_t*>(take(4 * all));
    s.ids_a = reinterpret_cast<int*>(take(4 * all));
    s.ids_b = reinterpret_cast<int*>(take(4 * all));
    s.nodes = reinterpret_cast<float4*>(take(64 * (size_t)(np > 1 ? np - 1 : 1)));
    s.boxes = reinterpret_cast<float4*>(take(32 * (size_t)np));
    s.parent = reinterpret_cast<int*>(take(8 * (size_t)np));
    s.flags = reinterpret_cast<int*>(take(4 * (size_t)np));
    s.range = reinterpret_cast<int2*>(take(8 * (size_t)np));
    s.chunks = reinterpret_cast<float4*>(take(32 * (size_t)((np + CHUNK - 1) / CHUNK)));
    const size_t most = sort_together(np, nq) ? all : (size_t)(np > nq ? np : nq);
    s.hist = reinterpret_cast<int*>(take(4 * radix_hist_ints((int)most)));
    s.bytes = o;
    return s;
}

__global__ void k_pt_bbox_init(int* bb) {
    if (threadIdx.x < 3) bb[threadIdx.x] = INT_MAX;
    else if (threadIdx.x < 6) bb[threadIdx.x] = INT_MIN;
}

// Exact per-axis extremes of the finite coordinates (ordered-int encoding).
__global__ void __launch_bounds__(256) k_pt_bbox(const float* __restrict__ P, int64_t n, int* __restrict__ bb) {
    int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {INT_MIN, INT_MIN, INT_MIN};
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        for (int c = 0; c < 3; ++c) {
            const float f = P[3 * i + c];
            if (!isfinite(f)) continue;
            const int k = float_to_ordered(f);
            lo[c] = min(lo[c], k);
            hi[c] = max(hi[c], k);
        }
    }
    for (int c = 0; c < 3; ++c) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[c] = min(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
            hi[c] = max(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
        }
    }
    if ((threadIdx.x & 31) == 0) {
        for (int c = 0; c < 3; ++c) {
            atomicMin(&bb[c], lo[c]);
            atomicMax(&bb[3 + c], hi[c]);
        }
    }
}

// The cube the Morton codes quantise: lower corner and 1/longest extent.
__device__ void pt_cube(const int* bb, float4* __restrict__ cube) {
    float lo[3], ext = 0.f;
    for (int c = 0; c < 3; ++c) {
        lo[c] = bb[c] == INT_MAX ? 0.f : ordered_to_float(bb[c]);
        const float h = bb[3 + c] == INT_MIN ? 0.f : ordered_to_float(bb[3 + c]);
        ext = fmaxf(ext, h - lo[c]);
    }
    *cube = make_float4(lo[0], lo[1], lo[2], ext > 0.f && isfinite(ext) ? 1.0f / ext : 0.f);
}

__global__ void k_pt_cube(const int* __restrict__ bb, float4* __restrict__ cube) { pt_cube(bb, cube); }

__global__ void __cluster_dims__(BBOX_BLOCKS, 1, 1) __launch_bounds__(BBOX_THREADS)
    k_pt_cube_cluster(const float* __restrict__ P, int64_t n, float4* __restrict__ cube) {
    __shared__ int box[6];
    if (bbox_cluster<true>(P, n, box)) pt_cube(box, cube);
}

__device__ __forceinline__ uint32_t pt_code(const float* __restrict__ p, float4 cube) {
    return morton30((p[0] - cube.x) * cube.w, (p[1] - cube.y) * cube.w, (p[2] - cube.z) * cube.w);
}

// Codes of the points, and behind them of the queries.
__global__ void k_pt_morton(const float* __restrict__ P, int64_t np, const float* __restrict__ Q, int64_t nq,
                            const float4* __restrict__ cube, uint32_t* __restrict__ codes, int* __restrict__ ids) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= np + nq) return;
    const bool query = i >= np;
    const int64_t j = query ? i - np : i;
    codes[i] = pt_code(query ? Q + 3 * j : P + 3 * j, *cube) | (query ? QUERY : 0u);
    ids[i] = (int)j;
}

struct Box {
    float3 lo, hi;
    __device__ void none() { lo = make_float3(NAN, NAN, NAN); hi = lo; }
    __device__ __forceinline__ void add(float3 l, float3 h) {
        lo = make_float3(fminf(lo.x, l.x), fminf(lo.y, l.y), fminf(lo.z, l.z));
        hi = make_float3(fmaxf(hi.x, h.x), fmaxf(hi.y, h.y), fmaxf(hi.z, h.z));
    }
    __device__ __forceinline__ void add(const float4* __restrict__ b) {  // (lo, hi) pair
        const float4 l = __ldg(b), h = __ldg(b + 1);
        add(make_float3(l.x, l.y, l.z), make_float3(h.x, h.y, h.z));
    }
    __device__ __forceinline__ void warp() {
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned F = 0xffffffffu;
            const float3 l = make_float3(__shfl_xor_sync(F, lo.x, o), __shfl_xor_sync(F, lo.y, o), __shfl_xor_sync(F, lo.z, o));
            const float3 h = make_float3(__shfl_xor_sync(F, hi.x, o), __shfl_xor_sync(F, hi.y, o), __shfl_xor_sync(F, hi.z, o));
            add(l, h);
        }
    }
};

// Leaf k's box is its point (a NaN coordinate stays out of its ancestors'
// boxes; such a point is never nearest).  Also the boxes of CHUNK leaves.
__global__ void __launch_bounds__(CHUNK) k_pt_leaves(const float* __restrict__ P, const int* __restrict__ order, int n,
                                                     float4* __restrict__ boxes, float4* __restrict__ chunks) {
    __shared__ Box sh[CHUNK / 32];
    const int k = blockIdx.x * CHUNK + threadIdx.x;
    Box b;
    b.none();
    if (k < n) {
        const float* p = P + 3 * (int64_t)order[k];
        b.lo = b.hi = make_float3(p[0], p[1], p[2]);
        boxes[2 * (int64_t)k] = make_float4(p[0], p[1], p[2], 0.f);
        boxes[2 * (int64_t)k + 1] = make_float4(p[0], p[1], p[2], 0.f);
    }
    b.warp();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < CHUNK / 32; ++w) b.add(sh[w].lo, sh[w].hi);
    chunks[2 * (int64_t)blockIdx.x] = make_float4(b.lo.x, b.lo.y, b.lo.z, 0.f);
    chunks[2 * (int64_t)blockIdx.x + 1] = make_float4(b.hi.x, b.hi.y, b.hi.z, 0.f);
}

__device__ __forceinline__ void write_box(float4* nodes, int slot, const Box& b) {  // slot: 2 * node + side
    float* r = reinterpret_cast<float*>(nodes + 4 * (int64_t)(slot >> 1) + 2 * (slot & 1));
    r[0] = b.lo.x; r[1] = b.lo.y; r[2] = b.lo.z;
    r[4] = b.hi.x; r[5] = b.hi.y; r[6] = b.hi.z;
}

// Every node's box, into its parent's record, from its leaves: a thread for up
// to NB_SMALL of them, a warp for up to NB_WIDE, else the whole block, which
// takes the chunks inside the node whole.  All nodes at once: climbing the tree
// (k_refit) is a chain of its depth in atomics and fences, 43 us for 50k
// points against 13.0 here.
constexpr int NB_THREADS = 256, NB_SMALL = 16, NB_WIDE = 1024;
__global__ void __launch_bounds__(NB_THREADS) k_pt_boxes(const float4* __restrict__ boxes,
                                                         const float4* __restrict__ chunks, int n,
                                                         const int2* __restrict__ range,
                                                         const int* __restrict__ parent, float4* __restrict__ nodes) {
    __shared__ int n_wide, wide[NB_THREADS];
    __shared__ Box sh[NB_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i = blockIdx.x * NB_THREADS + threadIdx.x;
    if (threadIdx.x == 0) n_wide = 0;
    __syncthreads();
    Box b;
    b.none();
    if (i < n) {  // leaf i
        b.add(boxes + 2 * (int64_t)i);
        write_box(nodes, parent[n - 1 + i], b);
    }
    int2 r = make_int2(0, -1);
    if (i > 0 && i < n - 1) r = range[i];  // the root's box is nobody's
    const int size = r.y - r.x + 1;
    if (size > 0 && size <= NB_SMALL) {
        b.none();
#pragma unroll 4
        for (int k = r.x; k <= r.y; ++k) b.add(boxes + 2 * (int64_t)k);
        write_box(nodes, parent[i], b);
    } else if (size > NB_WIDE) {
        wide[atomicAdd(&n_wide, 1)] = i;
    }
    unsigned m = __ballot_sync(0xffffffffu, size > NB_SMALL && size <= NB_WIDE);
    while (m) {
        const int l = __ffs(m) - 1;
        m &= m - 1;
        const int first = __shfl_sync(0xffffffffu, r.x, l), last = __shfl_sync(0xffffffffu, r.y, l);
        b.none();
        for (int k = first + lane; k <= last; k += 32) b.add(boxes + 2 * (int64_t)k);
        b.warp();
        if (lane == l) write_box(nodes, parent[i], b);
    }
    __syncthreads();
    const int cnt = n_wide;
    for (int q = 0; q < cnt; ++q) {
        const int node = wide[q];
        r = range[node];
        // leaves [r.x, c0 * CHUNK), chunks [c0, c1), leaves [c1 * CHUNK, r.y]
        const int c0 = (r.x + CHUNK - 1) / CHUNK, c1 = (r.y + 1) / CHUNK;
        b.none();
        for (int k = r.x + threadIdx.x; k < c0 * CHUNK; k += NB_THREADS) b.add(boxes + 2 * (int64_t)k);
        for (int k = c0 + threadIdx.x; k < c1; k += NB_THREADS) b.add(chunks + 2 * (int64_t)k);
        for (int k = c1 * CHUNK + threadIdx.x; k <= r.y; k += NB_THREADS) b.add(boxes + 2 * (int64_t)k);
        b.warp();
        if (lane == 0) sh[w] = b;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int k = 1; k < NB_THREADS / 32; ++k) b.add(sh[k].lo, sh[k].hi);
            write_box(nodes, parent[node], b);
        }
        __syncthreads();
    }
}
static_assert(NB_WIDE >= 2 * CHUNK, "a wide node holds a chunk");

// Squared distance of two points, summed x, y, z in double with every product
// and sum rounded on its own (no fused multiply-add): cKDTree's evaluation.
__device__ __forceinline__ double sum_sq(double dx, double dy, double dz) {
    return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

__device__ __forceinline__ double pt_d2(double qx, double qy, double qz, float px, float py, float pz) {
    return sum_sq(__dsub_rn((double)px, qx), __dsub_rn((double)py, qy), __dsub_rn((double)pz, qz));
}

// A float lower bound of the squared distance from q to a box, per axis
// max(lo - q, q - hi, 0): every operation rounded down (an overflow stays at
// FLT_MAX, a NaN corner counts as 0, as fmaxf drops it).
__device__ __forceinline__ float box_lb(float qx, float qy, float qz, float4 lo, float4 hi) {
    const float dx = fmaxf(fmaxf(__fsub_rd(lo.x, qx), __fsub_rd(qx, hi.x)), 0.f);
    const float dy = fmaxf(fmaxf(__fsub_rd(lo.y, qy), __fsub_rd(qy, hi.y)), 0.f);
    const float dz = fmaxf(fmaxf(__fsub_rd(lo.z, qz), __fsub_rd(qz, hi.z)), 0.f);
    return __fadd_rd(__fadd_rd(__fmul_rd(dx, dx), __fmul_rd(dy, dy)), __fmul_rd(dz, dz));
}

// The same of the nearest point of a box: never above that of a point in it.
__device__ __forceinline__ double box_d2(double qx, double qy, double qz, float4 lo, float4 hi) {
    const double dx = fmax(fmax(__dsub_rn((double)lo.x, qx), __dsub_rn(qx, (double)hi.x)), 0.0);
    const double dy = fmax(fmax(__dsub_rn((double)lo.y, qy), __dsub_rn(qy, (double)hi.y)), 0.0);
    const double dz = fmax(fmax(__dsub_rn((double)lo.z, qz), __dsub_rn(qz, (double)hi.z)), 0.0);
    return sum_sq(dx, dy, dz);
}

__device__ __forceinline__ void take(double d, int id, double& best, int& best_id) {
    if (d < best || (d == best && id < best_id)) {
        best = d;
        best_id = id;
    }
}

// A query's nearest point so far.  Distances are compared in float as long as
// that decides: box_lb of a point is at most its double distance, and NN_UP times
// it (plus NN_TINY, for what underflows) at least.  The points that may still be
// nearest wait in a short list; only they are measured in double (2 lanes a
// clock and SM), when the list is full and at the end: about one per query.
// A list that fills up again and again means points that floats cannot tell apart
// (a dense line, seen from beside it): from the NN_FILLS-th time on the query
// measures what passes in float, and boxes that may be no nearer than the best,
// in double at once.  300k queries beside 300k points of a line: 8.9 ms with every
// box in double, 25.9 with the list alone, 10.5 here (10.1, 10.9 and 11.2 with 1, 3
// and 4 fills, but a cluster of a million points seen from afar 0.61 to 0.78 ms with 1
// and 0.47 with more, and with the list alone).
constexpr int NN_LIST = 4, NN_FILLS = 2;
constexpr float NN_UP = 1.0f + 1e-6f, NN_TINY = 1e-37f;

struct Nearest {
    float lo = INFINITY;   // least lower bound in the list
    float lim = INFINITY;  // upper bound of the nearest distance: what lies beyond is not opened
    int n = 0;
    int fills = 0;         // how often the list was full
    bool exact = false;    // too often: `best` is the nearest of all points so far
    int leaf[NN_LIST];     // sorted points

    // The exact nearest of the list (and of `best`, `best_id` before it).
    __device__ void resolve(const float4* __restrict__ boxes, const int* __restrict__ order, double qx, double qy,
                            double qz, double& best, int& best_id) {
        for (int k = 0; k < n; ++k) {
            const float4 p = __ldg(boxes + 2 * (int64_t)leaf[k]);
            take(pt_d2(qx, qy, qz, p.x, p.y, p.z), order[leaf[k]], best, best_id);
        }
        n = 0;
    }
    __device__ void measure(int k, const float4* __restrict__ boxes, const int* __restrict__ order, double qx,
                            double qy, double qz, double& best, int& best_id) {
        const float4 p = __ldg(boxes + 2 * (int64_t)k);
        take(pt_d2(qx, qy, qz, p.x, p.y, p.z), order[k], best, best_id);
        lim = fminf(lim, __double2float_ru(best));
    }
    // A point whose lower bound d is not above lim.
    __device__ __forceinline__ void add(int k, float d, const float4* __restrict__ boxes,
                                        const int* __restrict__ order, double qx, double qy, double qz, double& best,
                                        int& best_id) {
        if (exact) {
            measure(k, boxes, order, qx, qy, qz, best, best_id);
            return;
        }
        const float up = fmaf(d, NN_UP, NN_TINY);
        if (up < lo) {  // nearer than everything before it
            n = 0;
            best = DBL_MAX;
            best_id = -1;
            lo = d;
        }
        lo = fminf(lo, d);
        lim = fminf(lim, up);
        if (n == NN_LIST) {
            resolve(boxes, order, qx, qy, qz, best, best_id);
            lim = fminf(lim, __double2float_ru(best));
            exact = ++fills == NN_FILLS;
            if (exact) {
                measure(k, boxes, order, qx, qy, qz, best, best_id);
                return;
            }
        }
        leaf[0] = n == 0 ? k : leaf[0];
        leaf[1] = n == 1 ? k : leaf[1];
        leaf[2] = n == 2 ? k : leaf[2];
        leaf[3] = n == 3 ? k : leaf[3];
        ++n;
    }
};
static_assert(NN_LIST == 4, "add writes four entries");

// One query a thread, queries in Morton order.  Measured: 50k queries over 50k
// points 788 us with every box in double, 150 with every passing point in
// double, 65.5 with the list.  A walk of the whole warp together, opening what
// any of its queries needs, was slower at every size from 1k to 200k points and
// queries (50k: by 120 us): neighbours in Morton order share little below
// the upper levels.
__global__ void __launch_bounds__(128) k_nn(const float4* __restrict__ nodes, const float4* __restrict__ boxes,
                                            const int* __restrict__ order, const float* __restrict__ P, int np,
                                            const float* __restrict__ Q, const int* __restrict__ qorder, int nq,
                                            int32_t* __restrict__ idx_out, double* __restrict__ d2_out,
                                            int* __restrict__ status) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nq) return;
    const int q = qorder[t];
    const float fx = Q[3 * (int64_t)q], fy = Q[3 * (int64_t)q + 1], fz = Q[3 * (int64_t)q + 2];
    const double qx = fx, qy = fy, qz = fz;
    double best = DBL_MAX;  // a point at DBL_MAX or NaN distance is never taken
    int best_id = -1;
    if (!isfinite(fx) || !isfinite(fy) || !isfinite(fz)) {
        atomicOr(status, 16);
        idx_out[q] = 0;
        if (d2_out) d2_out[q] = DBL_MAX;
        return;
    }
    if (np == 1) {
        take(pt_d2(qx, qy, qz, P[0], P[1], P[2]), 0, best, best_id);
    } else {
        Nearest near;
        // a leaf's box is its point; one that is not finite is never nearest
        auto leaf = [&](int k, float4 at, float d) {
            if (d <= near.lim && isfinite(at.x) && isfinite(at.y) && isfinite(at.z))
                near.add(k, d, boxes, order, qx, qy, qz, best, best_id);
        };
        int stack[NN_STACK];
        int sp = 0, node = 0;
        const int64_t max_iter = 2 * (int64_t)np + 64;  // each node is entered at most once
        for (int64_t iter = 0;; ++iter) {
            if (iter > max_iter) {
                atomicOr(status, 4);
                break;
            }
            const float4* nd = nodes + 4 * (int64_t)node;
            const float4 a = __ldg(nd), b = __ldg(nd + 1), c = __ldg(nd + 2), d = __ldg(nd + 3);
            const int L = __float_as_int(a.w), R = __float_as_int(b.w);
            const float dl = box_lb(fx, fy, fz, a, b), dr = box_lb(fx, fy, fz, c, d);
            // boxes at exactly the best distance are opened too: a lower index
            // may tie
            if (L < 0) leaf(~L, a, dl);
            if (R < 0) leaf(~R, c, dr);
            bool wl = L >= 0 && dl <= near.lim, wr = R >= 0 && dr <= near.lim;
            if (near.exact) {  // what floats cannot tell from the best
                if (wl && fmaf(dl, NN_UP, NN_TINY) >= near.lim) wl = box_d2(qx, qy, qz, a, b) <= best;
                if (wr && fmaf(dr, NN_UP, NN_TINY) >= near.lim) wr = box_d2(qx, qy, qz, c, d) <= best;
            }
            if (wl && wr) {
                if (sp >= NN_STACK) {  // cannot happen for trees of depth <= 64
                    atomicOr(status, 2);
                    break;
                }
                const bool lfirst = dl <= dr;
                stack[sp++] = lfirst ? R : L;
                node = lfirst ? L : R;
            } else if (wl) {
                node = L;
            } else if (wr) {
                node = R;
            } else {
                if (sp == 0) break;
                node = stack[--sp];
            }
        }
        near.resolve(boxes, order, qx, qy, qz, best, best_id);
    }
    if (best_id < 0) atomicOr(status, 8);  // every source coordinate non-finite
    idx_out[q] = best_id < 0 ? 0 : best_id;
    if (d2_out) d2_out[q] = best;
}

// ---- reverse loss ----------------------------------------------------------
constexpr int RL_THREADS = 256;

// Block b sums 0.5*|src[idx[t]] - tar[t]|^2 (float differences and squares
// as the reference's tensors compute them, accumulated in double) over its
// chunk in a fixed tree order.
__global__ void __launch_bounds__(RL_THREADS) k_rev_partial(const float* __restrict__ src, int64_t ns,
                                                           const float* __restrict__ tar,
                                                           const int32_t* __restrict__ idx, int64_t nt,
                                                           double* __restrict__ partial, int* __restrict__ status) {
    __shared__ double sh[RL_THREADS];
    double acc = 0.0;
    for (int64_t t = (int64_t)blockIdx.x * RL_THREADS + threadIdx.x; t < nt; t += (int64_t)gridDim.x * RL_THREADS) {
        const int64_t i = idx[t];
        if (i < 0 || i >= ns) {  // skipped and reported
            atomicOr(status, 1);
            continue;
        }
        for (int c = 0; c < 3; ++c) {
            const float l = SUB(src[3 * i + c], tar[3 * t + c]);
            acc += (double)MUL(l, l);
        }
    }
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int o = RL_THREADS / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

__global__ void __launch_bounds__(RL_THREADS) k_rev_total(const double* __restrict__ partial, int n,
                                                         double* __restrict__ loss) {
    __shared__ double sh[RL_THREADS];
    double acc = 0.0;
    for (int i = threadIdx.x; i < n; i += RL_THREADS) acc += partial[i];
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int o = RL_THREADS / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *loss = 0.5 * sh[0];
}

// Segment bounds of the targets grouped by their nearest source vertex.
__global__ void k_rev_segments(const uint32_t* __restrict__ keys, int nt, int64_t ns, int* __restrict__ seg_begin,
                               int* __restrict__ seg_end, int* __restrict__ status) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nt) return;
    const uint32_t key = keys[k];
    if ((int64_t)key >= ns) {  // out-of-range (or negative) index: skipped and reported
        atomicOr(status, 1);
        return;
    }
    if (k == 0 || keys[k - 1] != key) seg_begin[key] = k;
    if (k == nt - 1 || keys[k + 1] != key) seg_end[key] = k + 1;
}

// grad_src[i] = sum over the targets t matched to i, in increasing t, of
// (g*l + g*l) with l = src[i] - tar[t] and g = 0.5 * grad_out: torch's
// backward of 0.5*(l*l).sum() through src_V[ii], whose index_put_
// accumulation adds the matched rows in order, from zero.
__global__ void k_rev_grad(const float* __restrict__ src, const float* __restrict__ tar,
                           const int* __restrict__ sorted_t, const int* __restrict__ seg_begin,
                           const int* __restrict__ seg_end, int64_t ns, const float* __restrict__ grad_out,
                           float* __restrict__ grad_src) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ns) return;
    const float g = MUL(0.5f, *grad_out);
    float a0 = 0.f, a1 = 0.f, a2 = 0.f;
    const int b = seg_begin[i], e = seg_end[i];
    for (int k = b; k < e; ++k) {
        const int64_t t = sorted_t[k];
        const float l0 = SUB(src[3 * i], tar[3 * t]), l1 = SUB(src[3 * i + 1], tar[3 * t + 1]);
        const float l2 = SUB(src[3 * i + 2], tar[3 * t + 2]);
        const float g0 = MUL(g, l0), g1 = MUL(g, l1), g2 = MUL(g, l2);
        a0 = ADD(a0, ADD(g0, g0));
        a1 = ADD(a1, ADD(g1, g1));
        a2 = ADD(a2, ADD(g2, g2));
    }
    grad_src[3 * i] = a0;
    grad_src[3 * i + 1] = a1;
    grad_src[3 * i + 2] = a2;
}

struct RevScratch {
    int* status;
    double* partial;
    uint32_t* keys_a;
    uint32_t* keys_b;
    int* vals_a;
    int* vals_b;
    int* hist;
    int* seg_begin;
    int* seg_end;
    size_t bytes;
};

constexpr int RL_BLOCKS = 1024;

RevScratch plan_rev(char* base, int64_t ns, int64_t nt) {
    RevScratch s;
    size_t o = 0;
    auto take = [&](size_t bytes) {
        char* p = base ? base + o : nullptr;
        o += a256(bytes);
        return p;
    };
    s.status = reinterpret_cast<int*>(take(16));
    s.partial = reinterpret_cast<double*>(take(8 * RL_BLOCKS));
    s.keys_a = reinterpret_cast<uint32_t*>(take(4 * (size_t)nt));
    s.keys_b = reinterpret_cast<uint32_t*>(take(4 * (size_t)nt));
    s.vals_a = reinterpret_cast<int*>(take(4 * (size_t)nt));
    s.vals_b = reinterpret_cast<int*>(take(4 * (size_t)nt));
    s.hist = reinterpret_cast<int*>(take(4 * radix_hist_ints((int)nt)));
    s.seg_begin = reinterpret_cast<int*>(take(4 * (size_t)ns));
    s.seg_end = reinterpret_cast<int*>(take(4 * (size_t)ns));
    s.bytes = o;
    return s;
}

__global__ void k_rev_keys(const int32_t* __restrict__ idx, int64_t nt, uint32_t* __restrict__ keys,
                           int* __restrict__ vals) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nt) return;
    keys[t] = (uint32_t)idx[t];
    vals[t] = (int)t;
}

int bits_for(int64_t n) {
    int b = 1;
    while (b < 32 && ((int64_t)1 << b) < n) ++b;
    return b;
}

// status_out given: OR the index error into it; else synchronise and report.
int finish_status(RevScratch& S, int32_t* status_out, cudaStream_t s) {
    if (status_out) return MO_OK;
    int status = 0;
    cudaError_t e = cudaMemcpyAsync(&status, S.status, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_status(e, "reverse loss status");
    if (status & 1) {
        set_error("nearest-point index out of range");
        return MO_ERR_DEVICE;
    }
    return MO_OK;
}

}  // namespace
}  // namespace mo

using namespace mo;

extern "C" size_t mo_nn_scratch_bytes(int64_t np, int64_t nq) {
    if (np < 0 || nq < 0) return 0;
    return plan(nullptr, np, nq).bytes;
}

extern "C" int mo_nn_query(const float* P, int64_t np, const float* Q, int64_t nq, int32_t* idx_out,
                           double* d2_out, void* scratch, size_t scratch_bytes, void* stream) {
    MO_CHECK_ARG(np > 0 && nq >= 0, "need at least one source point (np=%lld)", (long long)np);
    MO_CHECK_ARG(np < ((int64_t)1 << 30) && nq < ((int64_t)1 << 31), "too many points");
    if (nq == 0) return MO_OK;
    MO_CHECK_ARG(P && Q && idx_out, "null pointer");
    cudaStream_t s = as_stream(stream);
    const size_t need = plan(nullptr, np, nq).bytes;
    void* owned = nullptr;
    if (!scratch) {
        MO_CUDA(cudaMallocAsync(&owned, need, s));
        scratch = owned;
    } else if (scratch_bytes < need) {
        set_error("NN query scratch too small: %zu < %zu", scratch_bytes, need);
        return MO_ERR_SCRATCH;
    }
    NnScratch S = plan(reinterpret_cast<char*>(scratch), np, nq);
    int rc = MO_OK;
    do {
        cudaError_t e = cudaMemsetAsync(S.status, 0, 16, s);
        if (e != cudaSuccess) { rc = cuda_status(e, "memset"); break; }
        if (np <= BBOX_CLUSTER_MAX) {
            k_pt_cube_cluster<<<BBOX_BLOCKS, BBOX_THREADS, 0, s>>>(P, np, S.cube); ::mo::note_launch();
        } else {
            k_pt_bbox_init<<<1, 32, 0, s>>>(S.bbox); ::mo::note_launch();
            k_pt_bbox<<<std::min(ceil_div(np, 256), 4 * device_sm_count()), 256, 0, s>>>(P, np, S.bbox);
            ::mo::note_launch();
            k_pt_cube<<<1, 1, 0, s>>>(S.bbox, S.cube); ::mo::note_launch();
        }
        // the queries in Morton order of the same cube
        k_pt_morton<<<ceil_div(np + nq, 256), 256, 0, s>>>(P, np, Q, nq, S.cube, S.codes_a, S.ids_a);
        ::mo::note_launch();
        if (sort_together(np, nq)) {
            e = radix_sort_pairs(S.codes_a, S.ids_a, S.codes_b, S.ids_b, (int)(np + nq), 31, S.hist, s);
        } else {
            e = radix_sort_pairs(S.codes_a, S.ids_a, S.codes_b, S.ids_b, (int)np, 30, S.hist, s);
            if (e == cudaSuccess)
                e = radix_sort_pairs(S.codes_a + np, S.ids_a + np, S.codes_b + np, S.ids_b + np, (int)nq, 30, S.hist, s);
        }
        if (e != cudaSuccess) { rc = cuda_status(e, "radix_sort_pairs"); break; }
        if (np > 1) {
            k_pt_leaves<<<ceil_div(np, CHUNK), CHUNK, 0, s>>>(P, S.ids_a, (int)np, S.boxes, S.chunks);
            ::mo::note_launch();
            k_karras<<<ceil_div(np - 1, 256), 256, 0, s>>>(S.codes_a, (int)np, S.nodes, S.parent, S.flags, S.range);
            ::mo::note_launch();
            k_pt_boxes<<<ceil_div(np, NB_THREADS), NB_THREADS, 0, s>>>(S.boxes, S.chunks, (int)np, S.range, S.parent,
                                                                       S.nodes);
            ::mo::note_launch();
        }
        k_nn<<<ceil_div(nq, 128), 128, 0, s>>>(S.nodes, S.boxes, S.ids_a, P, (int)np, Q, S.ids_a + np, (int)nq, idx_out,
                                               d2_out, S.status);
        ::mo::note_launch();
        e = cudaGetLastError();
        if (e != cudaSuccess) { rc = cuda_status(e, "nn kernels"); break; }
        int status = 0;
        e = cudaMemcpyAsync(&status, S.status, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) { rc = cuda_status(e, "nn status"); break; }
        if (status & 16) { set_error("a query point has non-finite coordinates"); rc = MO_ERR_DEVICE; }
        else if (status & 8) { set_error("no source point has finite coordinates"); rc = MO_ERR_DEVICE; }
        else if (status & 6) { set_error("point LBVH is malformed (status %d)", status); rc = MO_ERR_DEVICE; }
    } while (0);
    if (owned) cudaFreeAsync(owned, s);
    return rc;
}

extern "C" size_t mo_reverse_loss_scratch_bytes(int64_t ns, int64_t nt) {
    if (ns < 0 || nt < 0) return 0;
    return plan_rev(nullptr, ns, nt).bytes;
}

extern "C" int mo_reverse_loss_forward(const float* src, int64_t ns, const float* tar, int64_t nt,
                                       const int32_t* idx, double* loss_out, void* scratch, size_t scratch_bytes,
                                       int32_t* status_out, void* stream) {
    MO_CHECK_ARG(ns > 0 && nt >= 0 && nt < ((int64_t)1 << 31), "bad sizes");
    MO_CHECK_ARG(src && loss_out && (nt == 0 || (tar && idx)), "null pointer");
    MO_CHECK_ARG(scratch && scratch_bytes >= plan_rev(nullptr, ns, nt).bytes, "reverse loss scratch too small");
    cudaStream_t s = as_stream(stream);
    RevScratch S = plan_rev(reinterpret_cast<char*>(scratch), ns, nt);
    int* st = status_out ? reinterpret_cast<int*>(status_out) : S.status;
    if (!status_out) MO_CUDA(cudaMemsetAsync(S.status, 0, 16, s));
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(RL_BLOCKS, (nt + RL_THREADS - 1) / RL_THREADS));
    k_rev_partial<<<blocks, RL_THREADS, 0, s>>>(src, ns, tar, idx, nt, S.partial, st); ::mo::note_launch();
    k_rev_total<<<1, RL_THREADS, 0, s>>>(S.partial, blocks, loss_out); ::mo::note_launch();
    MO_LAUNCH_CHECK("reverse loss forward");
    return finish_status(S, status_out, s);
}

extern "C" int mo_reverse_loss_backward(const float* src, int64_t ns, const float* tar, int64_t nt,
                                        const int32_t* idx, const float* grad_out, float* grad_src, void* scratch,
                                        size_t scratch_bytes, int32_t* status_out, void* stream) {
    MO_CHECK_ARG(ns > 0 && nt >= 0 && nt < ((int64_t)1 << 31) && ns < ((int64_t)1 << 31), "bad sizes");
    MO_CHECK_ARG(src && grad_out && grad_src && (nt == 0 || (tar && idx)), "null pointer");
    MO_CHECK_ARG(scratch && scratch_bytes >= plan_rev(nullptr, ns, nt).bytes, "reverse loss scratch too small");
    cudaStream_t s = as_stream(stream);
    RevScratch S = plan_rev(reinterpret_cast<char*>(scratch), ns, nt);
    int* st = status_out ? reinterpret_cast<int*>(status_out) : S.status;
    if (!status_out) MO_CUDA(cudaMemsetAsync(S.status, 0, 16, s));
    MO_CUDA(cudaMemsetAsync(S.seg_begin, 0, 4 * (size_t)ns, s));
    MO_CUDA(cudaMemsetAsync(S.seg_end, 0, 4 * (size_t)ns, s));
    if (nt > 0) {
        k_rev_keys<<<ceil_div(nt, 256), 256, 0, s>>>(idx, nt, S.keys_a, S.vals_a); ::mo::note_launch();
        MO_CUDA(radix_sort_pairs(S.keys_a, S.vals_a, S.keys_b, S.vals_b, (int)nt, bits_for(ns), S.hist, s));
        k_rev_segments<<<ceil_div(nt, 256), 256, 0, s>>>(S.keys_a, (int)nt, ns, S.seg_begin, S.seg_end, st);
        ::mo::note_launch();
    }
    k_rev_grad<<<ceil_div(ns, 256), 256, 0, s>>>(src, tar, S.vals_a, S.seg_begin, S.seg_end, ns, grad_out, grad_src);
    ::mo::note_launch();
    MO_LAUNCH_CHECK("reverse loss backward");
    return finish_status(S, status_out, s);
}
