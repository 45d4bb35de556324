// SolveLinear (src/interface/linear_layer.cc:5-79): the sparse linear
// propagation after a graph or flow deformation.
//
// LinearEstimation (src/lib/linear.cc:10-112), in double:
//   minimise  sum_g (w_g * sum_{j in cell g} x_j - w_g * G_g)^2      w_g = 1/|cell g|
//           + 1e-6 * sum_i |x_i - G_{ref(i)}|^2
//           + sum_edges reg_e |(x_a - x_b) - (V_a - V_b)|^2          reg_e = (0.02 r / (|V_a - V_b| + 1e-8))^2
// over the three coordinates, edges = the faces' half-edges then E; cell g
// holds the vertices i with ref(i) = g.
// LinearEstimationWithRot (linear.cc:114-230): per vertex the rotation
// R_i = U V^T of the SVD of sum_{j in N(i)} (G_j - G_i)(V_j - V_i)^T and the
// scale s_i = sum |G_j - G_i| / (sum |V_j - V_i| + 1e-8), then
//   minimise  sum_i |x_i - G_i|^2 + sum over face half-edges (a, b), both
//   directions, reg_ab |(x_b - x_a) - s_a R_a (V_b - V_a)|^2,   reg_ab = 0.02 r / |V_b - V_a|.
//
// The reference assembles A and factorises it with SimplicialLDLT.  Here the
// normal equations A x = B are solved matrix-free with Jacobi-preconditioned
// conjugate gradients in double: A x is gathered per vertex over its unique
// neighbours (and, for the cell term, a cell -> vertex CSR), every dot product is
// a fixed-order reduction, and all iterations run in one cooperative launch
// (k_lin_cg).
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <vector>

#include "mo_common.cuh"
#include "mo_wait.cuh"

namespace mo {
namespace {

constexpr int CG_ROWS = 341;      // vertices a block of the solver handles at a time, a thread per coordinate
constexpr int CG_THREADS = 1024;  // one block per SM
constexpr int CG_MIN_ROWS = 16;   // vertices a block should have before another block is used
constexpr int CG_CHECK = 32;      // iterations between convergence checks
constexpr int CG_MAX_BLOCKS = 512;
constexpr int CG_ROW_BYTES = 160 * 1024;  // shared memory for a block's rows of the matrix
constexpr int CG_FEW = 8;         // members of a cell that one lane sums
constexpr int CG_MERGE = 128;     // half-edges of a vertex whose neighbours are merged

size_t a256(size_t x) { return (x + 255) & ~(size_t)255; }

struct LinScratch {
    int32_t* edges;    // [nh, 2]
    void* csr;         // vertex -> half-edge CSR (mo_edge_csr_build layout)
    size_t csr_bytes;
    double* w;         // per half-edge weight
    double* G;         // [ng, 3] graph positions (LE) or [nv, 3] targets (rot)
    double* V0;        // [nv, 3] input positions
    double* diag;      // [nv]
    double* cellw;     // [ng] 1/|cell|
    int32_t* cell_ptr; // [ng + 1]
    int32_t* cell_mem; // [nv] vertices by cell, increasing
    double* cellsum;   // [ng, 3]
    double* rot;       // [nv, 9] s_i * R_i (row-major)
    int4* nbr;         // [2 nh] unique neighbours: (vertex, -, weight as a double)
    int32_t* nnbr;     // [nv] their number
    double* x;         // [nv, 3]
    double* r;         // [nv, 3]
    double* dinv;      // [nv, 3]
    double* z;         // [nv, 4]
    double* p;         // [2, nv, 4]
    double* partial;   // [3][CG_MAX_BLOCKS, 3]
    double* result;    // iterations, relative residual
    unsigned* bar;     // grid barrier count, then its abort flag
    int* status;
    uint32_t* keys_a;  // cell sort
    uint32_t* keys_b;
    int* vals_a;
    int* vals_b;
    int* hist;
    size_t bytes;
};

LinScratch plan(char* base, int64_t nv, int64_t nf, int64_t ne, int64_t ng, int with_rot) {
    LinScratch s;
    size_t o = 0;
    auto take = [&](size_t bytes) {
        char* p = base ? base + o : nullptr;
        o += a256(bytes ? bytes : 1);
        return p;
    };
    const int64_t nh = 3 * nf + (with_rot ? 0 : ne);
    s.edges = reinterpret_cast<int32_t*>(take(8 * (size_t)nh));
    s.csr_bytes = mo_edge_csr_bytes(nv, nh, MO_EDGES_LIST);
    s.csr = take(s.csr_bytes);
    s.w = reinterpret_cast<double*>(take(8 * (size_t)nh));
    s.G = reinterpret_cast<double*>(take(24 * (size_t)(with_rot ? nv : ng)));
    s.V0 = reinterpret_cast<double*>(take(24 * (size_t)nv));
    s.diag = reinterpret_cast<double*>(take(8 * (size_t)nv));
    s.cellw = reinterpret_cast<double*>(take(8 * (size_t)ng));
    s.cell_ptr = reinterpret_cast<int32_t*>(take(4 * (size_t)(ng + 1)));
    s.cell_mem = reinterpret_cast<int32_t*>(take(4 * (size_t)nv));
    s.cellsum = reinterpret_cast<double*>(take(24 * (size_t)ng));
    s.rot = reinterpret_cast<double*>(take(with_rot ? 72 * (size_t)nv : 0));
    s.nbr = reinterpret_cast<int4*>(take(32 * (size_t)nh));
    s.nnbr = reinterpret_cast<int32_t*>(take(4 * (size_t)nv));
    s.x = reinterpret_cast<double*>(take(24 * (size_t)nv));
    s.r = reinterpret_cast<double*>(take(24 * (size_t)nv));
    s.dinv = reinterpret_cast<double*>(take(24 * (size_t)nv));
    s.z = reinterpret_cast<double*>(take(32 * (size_t)nv));
    s.p = reinterpret_cast<double*>(take(64 * (size_t)nv));
    s.partial = reinterpret_cast<double*>(take(8 * 9 * (size_t)CG_MAX_BLOCKS));
    s.result = reinterpret_cast<double*>(take(16));
    s.bar = reinterpret_cast<unsigned*>(take(16));
    s.status = reinterpret_cast<int*>(take(16));
    s.keys_a = reinterpret_cast<uint32_t*>(take(4 * (size_t)nv));
    s.keys_b = reinterpret_cast<uint32_t*>(take(4 * (size_t)nv));
    s.vals_a = reinterpret_cast<int*>(take(4 * (size_t)nv));
    s.vals_b = reinterpret_cast<int*>(take(4 * (size_t)nv));
    s.hist = reinterpret_cast<int*>(take(4 * radix_hist_ints((int)nv)));
    s.bytes = o;
    return s;
}

// ---- set-up ----------------------------------------------------------------
__global__ void k_lin_edges(const int32_t* __restrict__ F, int64_t nf, const int32_t* __restrict__ E, int64_t ne,
                            int32_t* __restrict__ out) {
    const int64_t h = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (h < 3 * nf) {
        const int64_t f = h / 3;
        const int j = (int)(h - 3 * f);
        out[2 * h] = F[3 * f + j];
        out[2 * h + 1] = F[3 * f + (j == 2 ? 0 : j + 1)];
    } else if (h < 3 * nf + ne) {
        const int64_t k = h - 3 * nf;
        out[2 * h] = E[2 * k];
        out[2 * h + 1] = E[2 * k + 1];
    }
}

__global__ void k_lin_to_double(const float* __restrict__ a, int64_t n, double* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (double)a[i];
}

__device__ __forceinline__ double norm3(double x, double y, double z) { return sqrt(x * x + y * y + z * z); }

// Half-edge weights from the input positions (edges validated by the CSR).
__global__ void k_lin_weights(const int32_t* __restrict__ edges, int64_t nh, const double* __restrict__ V,
                              double rigidity, int with_rot, double* __restrict__ w) {
    const int64_t h = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= nh) return;
    const int64_t a = edges[2 * h], b = edges[2 * h + 1];
    const double n = norm3(V[3 * a] - V[3 * b], V[3 * a + 1] - V[3 * b + 1], V[3 * a + 2] - V[3 * b + 2]);
    if (with_rot) {
        // linear.cc:206: regulation * 2e-2 / |off| * rigidity, both directions
        w[h] = 2.0 * (1.0 * 2e-2 / n * rigidity);
    } else {
        // linear.cc:62-63: (regular * 2e-2 / (|V0 - V1| + 1e-8))^2
        const double reg = rigidity * 2e-2 / (n + 1e-8);
        w[h] = reg * reg;
    }
}

__global__ void k_lin_cell_keys(const int32_t* __restrict__ ref, int64_t nv, int64_t ng, uint32_t* __restrict__ keys,
                                int* __restrict__ vals, int* __restrict__ status) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nv) return;
    const int g = ref[i];
    if (g < 0 || (int64_t)g >= ng) atomicOr(status, 1);
    keys[i] = (g < 0 || (int64_t)g >= ng) ? 0u : (uint32_t)g;
    vals[i] = (int)i;
}

__global__ void k_lin_cell_ptr(const uint32_t* __restrict__ keys, int64_t nv, int32_t* __restrict__ cell_ptr) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nv) return;
    const uint32_t key = keys[k];
    const uint32_t prev = k == 0 ? 0u : keys[k - 1];
    // cell_ptr[g] = first position of cell g; empty cells take the next start
    for (uint32_t g = (k == 0 ? 0u : prev + 1); g <= key; ++g) cell_ptr[g] = (int32_t)k;
}

__global__ void k_lin_cell_tail(const uint32_t* __restrict__ keys, int64_t nv, int64_t ng,
                                int32_t* __restrict__ cell_ptr) {
    const uint32_t last = nv > 0 ? keys[nv - 1] : 0u;
    for (int64_t g = (nv > 0 ? (int64_t)last + 1 : 0); g <= ng; ++g) cell_ptr[g] = (int32_t)nv;
}

__global__ void k_lin_cellw(const int32_t* __restrict__ cell_ptr, int64_t ng, double* __restrict__ cellw) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ng) return;
    const int c = cell_ptr[g + 1] - cell_ptr[g];
    cellw[g] = c > 0 ? 1.0 / (double)c : 0.0;
}

// Jacobi diagonal and right-hand side (LinearEstimation).
__global__ void k_lin_rhs(int64_t nv, const int* __restrict__ row_ptr, const int* __restrict__ other,
                          const int* __restrict__ key, const double* __restrict__ w, const double* __restrict__ V,
                          const int32_t* __restrict__ ref, const double* __restrict__ G,
                          const double* __restrict__ cellw, double* __restrict__ diag, double* __restrict__ B) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nv) return;
    const int64_t g = ref[i];
    const double wg = cellw[g];
    double d = 1e-6 + wg * wg;
    double b[3];
    for (int c = 0; c < 3; ++c) b[c] = wg * G[3 * g + c] + 1e-6 * G[3 * g + c];
    for (int k = row_ptr[i]; k < row_ptr[i + 1]; ++k) {
        const int64_t o = other[k];
        if (o == i) continue;  // a self-loop's four entries cancel
        const double we = w[key[k] >> 1];
        d += we;
        for (int c = 0; c < 3; ++c) b[c] += we * (V[3 * i + c] - V[3 * o + c]);
    }
    diag[i] = d;
    for (int c = 0; c < 3; ++c) B[3 * i + c] = b[c];
}

// ---- with rotations --------------------------------------------------------
// Symmetric 3x3 eigen-decomposition by cyclic Jacobi rotations (bounded
// sweeps): a = Q diag(e) Q^T, Q columns the eigenvectors.
__device__ void jacobi3(double a[3][3], double Q[3][3], double e[3]) {
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) Q[r][c] = r == c ? 1.0 : 0.0;
    for (int sweep = 0; sweep < 32; ++sweep) {
        const double off = fabs(a[0][1]) + fabs(a[0][2]) + fabs(a[1][2]);
        const double scale = fabs(a[0][0]) + fabs(a[1][1]) + fabs(a[2][2]);
        if (off <= 1e-300 || off <= 1e-18 * scale) break;
        for (int p = 0; p < 2; ++p) {
            for (int q = p + 1; q < 3; ++q) {
                if (a[p][q] == 0.0) continue;
                const double theta = (a[q][q] - a[p][p]) / (2.0 * a[p][q]);
                const double t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
                const double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
                for (int k = 0; k < 3; ++k) {  // a <- J^T a J
                    const double akp = a[k][p], akq = a[k][q];
                    a[k][p] = c * akp - s * akq;
                    a[k][q] = s * akp + c * akq;
                }
                for (int k = 0; k < 3; ++k) {
                    const double apk = a[p][k], aqk = a[q][k];
                    a[p][k] = c * apk - s * aqk;
                    a[q][k] = s * apk + c * aqk;
                }
                for (int k = 0; k < 3; ++k) {
                    const double qkp = Q[k][p], qkq = Q[k][q];
                    Q[k][p] = c * qkp - s * qkq;
                    Q[k][q] = s * qkp + c * qkq;
                }
            }
        }
    }
    for (int k = 0; k < 3; ++k) e[k] = a[k][k];
}

__device__ __forceinline__ void cross3(const double a[3], const double b[3], double c[3]) {
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
}

__device__ __forceinline__ bool unit3(double v[3]) {
    const double n = norm3(v[0], v[1], v[2]);
    if (!(n > 0.0)) return false;
    v[0] /= n; v[1] /= n; v[2] /= n;
    return true;
}

// R = U V^T for M = U S V^T: the orthogonal polar factor of M (unique when M
// is nonsingular).  From M^T M = Q diag(l) Q^T: v_k = q_k, u_k = M v_k /
// sqrt(l_k) for the two largest; when the smallest singular value vanishes
// (neighbours in one plane: every vertex of a surface patch) the third pair
// is completed as u1 x u2, v1 x v2 -- the reference's own choice there is an
// arbitrary sign, and the completed column multiplies only the normal part
// of an edge, which is zero for those neighbourhoods.
__device__ void polar3(const double M[3][3], double R[3][3]) {
    double a[3][3], Q[3][3], e[3];
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) a[r][c] = M[0][r] * M[0][c] + M[1][r] * M[1][c] + M[2][r] * M[2][c];
    jacobi3(a, Q, e);
    int ord[3] = {0, 1, 2};  // descending eigenvalues
    for (int i = 0; i < 3; ++i)
        for (int j = i + 1; j < 3; ++j)
            if (e[ord[j]] > e[ord[i]]) { const int t = ord[i]; ord[i] = ord[j]; ord[j] = t; }
    double u[3][3], v[3][3];
    const double smax = sqrt(fmax(e[ord[0]], 0.0));
    int rank = 0;
    for (int k = 0; k < 3; ++k) {
        for (int c = 0; c < 3; ++c) v[k][c] = Q[c][ord[k]];
        const double sk = sqrt(fmax(e[ord[k]], 0.0));
        if (sk > 1e-12 * smax && sk > 0.0) {
            for (int r = 0; r < 3; ++r) u[k][r] = (M[r][0] * v[k][0] + M[r][1] * v[k][1] + M[r][2] * v[k][2]) / sk;
            ++rank;
        }
    }
    if (rank == 0) {
        for (int r = 0; r < 3; ++r)
            for (int c = 0; c < 3; ++c) R[r][c] = r == c ? 1.0 : 0.0;
        return;
    }
    if (rank == 1) {  // complete u2 orthogonal to u1 along v2's direction
        double t[3] = {v[1][0], v[1][1], v[1][2]};
        const double d = t[0] * u[0][0] + t[1] * u[0][1] + t[2] * u[0][2];
        for (int c = 0; c < 3; ++c) t[c] -= d * u[0][c];
        if (!unit3(t)) {  // v2 parallel to u1: any perpendicular
            double ax[3] = {fabs(u[0][0]) < 0.9 ? 1.0 : 0.0, fabs(u[0][0]) < 0.9 ? 0.0 : 1.0, 0.0};
            cross3(u[0], ax, t);
            unit3(t);
        }
        for (int c = 0; c < 3; ++c) u[1][c] = t[c];
        rank = 2;
    }
    if (rank == 2) {
        cross3(u[0], u[1], u[2]);
        cross3(v[0], v[1], v[2]);
    }
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) R[r][c] = u[0][r] * v[0][c] + u[1][r] * v[1][c] + u[2][r] * v[2][c];
}

// s_i * R_i from the unique neighbours of i (linear.cc:131-163).
__global__ void k_lin_rotations(int64_t nv, const int* __restrict__ row_ptr, const int* __restrict__ other,
                                const double* __restrict__ V, const double* __restrict__ T, double* __restrict__ rot) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nv) return;
    double M[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    double lo = 0.0, lc = 0.0;
    const int b = row_ptr[i], e = row_ptr[i + 1];
    for (int k = b; k < e; ++k) {
        const int o = other[k];
        bool seen = false;  // links[] is a set: each neighbour once
        for (int j = b; j < k && !seen; ++j) seen = other[j] == o;
        if (seen) continue;
        const double d1[3] = {V[3 * o] - V[3 * i], V[3 * o + 1] - V[3 * i + 1], V[3 * o + 2] - V[3 * i + 2]};
        const double d2[3] = {T[3 * o] - T[3 * i], T[3 * o + 1] - T[3 * i + 1], T[3 * o + 2] - T[3 * i + 2]};
        lo += norm3(d1[0], d1[1], d1[2]);
        lc += norm3(d2[0], d2[1], d2[2]);
        for (int r = 0; r < 3; ++r)
            for (int c = 0; c < 3; ++c) M[r][c] += d2[r] * d1[c];
    }
    const double s = lc / (lo + 1e-8);
    double R[3][3];
    polar3(M, R);
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) rot[9 * i + 3 * r + c] = s * R[r][c];
}

// Diagonal and right-hand side with rotations (linear.cc:190-216).
__global__ void k_lin_rhs_rot(int64_t nv, const int* __restrict__ row_ptr, const int* __restrict__ other,
                              const int* __restrict__ key, const double* __restrict__ w,
                              const double* __restrict__ V, const double* __restrict__ T,
                              const double* __restrict__ rot, double* __restrict__ diag, double* __restrict__ B) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nv) return;
    double d = 1.0;
    double b[3] = {T[3 * i], T[3 * i + 1], T[3 * i + 2]};
    for (int k = row_ptr[i]; k < row_ptr[i + 1]; ++k) {
        const int64_t o = other[k];
        if (o == i) continue;
        const double we = w[key[k] >> 1];  // both directions: 2 * reg
        const double reg = 0.5 * we;
        d += we;
        // + reg * s_o R_o (V_i - V_o)  - reg * s_i R_i (V_o - V_i)
        const double e[3] = {V[3 * i] - V[3 * o], V[3 * i + 1] - V[3 * o + 1], V[3 * i + 2] - V[3 * o + 2]};
        for (int r = 0; r < 3; ++r) {
            const double* Ro = rot + 9 * o + 3 * r;
            const double* Ri = rot + 9 * i + 3 * r;
            b[r] += reg * (Ro[0] * e[0] + Ro[1] * e[1] + Ro[2] * e[2]) + reg * (Ri[0] * e[0] + Ri[1] * e[1] + Ri[2] * e[2]);
        }
    }
    diag[i] = d;
    for (int c = 0; c < 3; ++c) B[3 * i + c] = b[c];
}

// ---- CG --------------------------------------------------------------------
// A vertex's unique neighbours with their summed weights, in the order of
// their first half-edge: a closed mesh names every neighbour twice, and the
// product with A is bound by the FP64 pipe (2 lanes a clock and SM).  One thread
// looks at every pair of a vertex's half-edges, so past CG_MERGE of them they stay
// as they are.  Measured, ms a solve with one hub (merged, not): 200 half-edges
// 3.6, 3.15; 400 10.0, 8.2; 1600 121, 74; 3200 452, 257 (of which the vertex ->
// half-edge list 147).
__global__ void k_lin_merge(int64_t nv, const int* __restrict__ row_ptr, const int* __restrict__ other,
                            const int* __restrict__ key, const double* __restrict__ w, int4* __restrict__ nbr,
                            int32_t* __restrict__ nnbr) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nv) return;
    const int b = row_ptr[i], e = row_ptr[i + 1];
    const bool merge = e - b <= CG_MERGE;
    int n = 0;
    for (int k = b; k < e; ++k) {
        const int o = other[k];
        if (o == i) continue;  // a self-loop's entries cancel
        double s = w[key[k] >> 1];
        if (merge) {
            bool seen = false;
            for (int j = b; j < k && !seen; ++j) seen = other[j] == o;
            if (seen) continue;
            for (int j = k + 1; j < e; ++j)
                if (other[j] == o) s += w[key[j] >> 1];
        }
        nbr[b + n] = make_int4(o, 0, __double2loint(s), __double2hiint(s));
        ++n;
    }
    nnbr[i] = n;
}

struct CgArgs {
    int64_t nv, ng;
    const int* row_ptr;
    const int4* nbr;
    const int32_t *nnbr, *ref;  // ref NULL: no cell term
    const double* cellw;
    const int32_t *cell_ptr, *cell_mem;
    double c0;
    const double *V0, *diag;
    double *x, *r, *dinv, *z, *p, *cellsum, *partial, *result;
    unsigned* bar;
    double tol;
    int max_iter;
};

// All blocks of the (cooperative) grid; `target` grows by gridDim.x per call.
// The release publishes the writes that the block's barrier put before it, the
// acquire holds for the threads behind the second one.  (With a full fence beside
// each an iteration took 23.6 us instead of 21.6.)
// A wait of more than two seconds of polling, or another block's, ends the solve: false.
__device__ __forceinline__ bool grid_sync(unsigned* bar, unsigned target) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
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

// Per coordinate: the block's sum of v (thread t holds coordinate t % 3), in a
// fixed order, into out[0..2] of shared memory.  FP64 instructions are the scarce
// resource (a warp's takes 64 clocks of its scheduler), so three warps add what
// all threads put into shared memory instead of every warp shuffling.
__device__ __forceinline__ void block_sum3(double v, double* sh, double* out) {
    sh[threadIdx.x] = v;
    __syncthreads();
    const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (c < 3) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < (CG_ROWS + 31) / 32; ++k) {
            const int row = lane + 32 * k;
            if (row < CG_ROWS) s += sh[3 * row + c];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) out[c] = s;
    }
    __syncthreads();
}

// The block's sums of v per coordinate (as block_sum3's) into its place of part.
__device__ __forceinline__ void store_partial(double v, double* sh, double* part) {
    sh[threadIdx.x] = v;
    __syncthreads();
    const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (c >= 3) return;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int k = 0; k < (CG_ROWS + 31) / 32; ++k) {
        const int row = lane + 32 * k;
        if (row < CG_ROWS) s[k & 3] += sh[3 * row + c];
    }
    double t = (s[0] + s[1]) + (s[2] + s[3]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) part[3 * blockIdx.x + c] = t;
}

// The totals of the blocks' partial sums (every block adds them in the same
// order): then(c, total) in one thread per coordinate, before all go on.
template <class Then>
__device__ __forceinline__ void grid_sum3(const double* part, Then then) {
    constexpr int BATCH = 5;  // 160 blocks
    const int c = threadIdx.x >> 5, lane = threadIdx.x & 31, n = (int)gridDim.x;
    if (c < 3) {
        double s = 0.0;
        for (int b0 = lane; b0 < n; b0 += 32 * BATCH) {
            double v[BATCH];
#pragma unroll
            for (int j = 0; j < BATCH; ++j) v[j] = b0 + 32 * j < n ? __ldcg(part + 3 * (b0 + 32 * j) + c) : 0.0;
            s += ((v[0] + v[1]) + (v[2] + v[3])) + v[4];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) then(c, s);
    }
    __syncthreads();
}

// Every iteration of the conjugate gradients in one cooperative launch.  (Before:
// a graph of seven kernels, 98 us an iteration at 41k vertices and 802 cells, of
// which the launches and the cells, each summed by one thread, were most.)
// Three grid barriers an iteration:
//   A p and p.Ap | alpha; x, r, z = r / diag and r.z | beta; p = z + beta p and
//   its cell sums
// (Sums that are their own barrier, every block polling every block's slot, were
// slower: 24 us an iteration at 15k vertices; the polling fills L2.)
// p is double-buffered, so the cell sums can be taken of z + beta p while the
// vertices write it.  A block owns a contiguous range of vertices, a thread one
// coordinate of a vertex; with at most CG_ROWS vertices (ONE) x, r, z and p stay in
// registers, and the block's rows of the matrix in shared memory where they fit.
// Bound: latency (a trip to L2 for the neighbours, one for the cells, three
// barriers of ~2,500 clocks and two sums of ~5,000 in between), and from ~30k
// vertices the FP64 pipe (2 lanes a clock and SM) in A p, two operations a
// neighbour and coordinate.
// Measured, us an iteration: 4k vertices 17.2, 15k 15.8, 41k 18.8 (20.5, 16.8, 20.2
// with the rows read from L2, two more loads a vertex and chains of eleven
// additions).  Eight lanes a cell instead of a warp: 41k 25; fewer than 16 vertices
// a block were not tried, 64 took 5% longer at 2k to 8k.
//
// MANY (four turns of a warp a sum and more; a cell a vertex at 15k, 100k and 300k
// vertices, where the kernels before took 40, 60 and 123 us an iteration): 39, 158 and
// 447 us with a warp a sum, 20, 32 and 71 so; cells of 16 at 300k 80 and 82.
template <bool ONE, bool MANY>
__global__ void __launch_bounds__(CG_THREADS) k_lin_cg(CgArgs A) {
    extern __shared__ int4 rows[];  // ONE: this block's rows, if they fit
    __shared__ double sh[CG_THREADS], sh2[CG_THREADS];
    __shared__ int longest;
    __shared__ double sum[3], rz[3], bb[3], coef[3];
    __shared__ double rel_sh;
    const int64_t per = (A.nv + gridDim.x - 1) / gridDim.x;
    const int c = threadIdx.x % 3, tid = threadIdx.x;
    const int64_t i0 = per * blockIdx.x + tid / 3;
    const int64_t i1 = tid < 3 * CG_ROWS ? min(A.nv, per * (blockIdx.x + 1)) : 0;
    double* PA = A.partial;
    double* PU = PA + 3 * CG_MAX_BLOCKS;
    double* PR = PU + 3 * CG_MAX_BLOCKS;
    unsigned target = 0;
    double x = 0, r = 0, di = 0, z = 0, pv = 0;  // ONE: this thread's vertex

    // a vertex's neighbours and cell
    struct Row {
        const int4* q;
        const double* sum;
        double w2;
        int n;
    };
    auto row_of = [&](int64_t i) {
        Row w{A.nbr + A.row_ptr[i], nullptr, 0.0, A.nnbr[i]};
        if (A.ref) {
            const int64_t g = A.ref[i];
            w.sum = A.cellsum + 3 * g + c;
            w.w2 = A.cellw[g] * A.cellw[g];
        }
        return w;
    };
    Row mine{};      // ONE
    int stride = 1;  // of its entries
    if (ONE) {
        if (i0 < i1) mine = row_of(i0);
        // entry k of the block's v-th vertex at rows[k * per + v]: no two of a warp's in a bank
        if (tid == 0) longest = 0;
        __syncthreads();
        if (i0 < i1) atomicMax(&longest, mine.n);
        __syncthreads();
        if (longest * per <= CG_ROW_BYTES / (int64_t)sizeof(int4)) {
            for (int k = c; k < mine.n; k += 3) rows[k * per + tid / 3] = mine.q[k];
            mine.q = rows + tid / 3;
            stride = (int)per;
        }
        __syncthreads();
    }
    // coordinate c of A v for vertex i; v in rows of 4
    auto apply = [&](const double* v, int64_t i, double vi) {
        const Row w = ONE ? mine : row_of(i);
        const double cs = w.sum ? __ldcg(w.sum) : 0.0;
        double y = A.c0 * vi;
        const int4* q = w.q;
        const int n = w.n;
#pragma unroll 6
        for (int k = 0; k < n; ++k) {
            const int4 e = ONE ? q[k * stride] : __ldg(q + k);
            y += __hiloint2double(e.w, e.z) * (vi - __ldcg(v + 4 * (int64_t)e.x + c));
        }
        y += w.w2 * cs;
        return y;
    };
    // cellsum = sums of value(member, coordinate) over the cells: a warp per
    // coordinate of a cell, its loads in flight together, or a block where cells
    // are large.  MANY: more sums than the grid's warps take in a few turns; a warp
    // takes up to 32 at once, and a lane each of those with few members
    auto cells = [&](auto value) {
        if (A.nv >= A.ng * 1024) {
            for (int64_t g = blockIdx.x; g < A.ng; g += gridDim.x) {
                double s = 0.0;
                const int e = A.cell_ptr[g + 1];
                if (tid < 3 * CG_ROWS)
                    for (int k = A.cell_ptr[g] + tid / 3; k < e; k += CG_ROWS) s += value(A.cell_mem[k], c);
                block_sum3(s, sh, sum);
                if (tid < 3) A.cellsum[3 * g + tid] = sum[tid];
                __syncthreads();
            }
            return;
        }
        const int lane = tid & 31;
        if (MANY) {
            const int64_t sums = 3 * A.ng, warps = (int64_t)gridDim.x * (CG_THREADS / 32);
            const int at_once = (int)min((int64_t)32, (sums + warps - 1) / warps);
            for (int64_t q0 = (blockIdx.x + gridDim.x * (int64_t)(tid >> 5)) * at_once; q0 < sums;
                 q0 += warps * at_once) {
                const int64_t q = q0 + lane, g = q / 3;
                const int k0 = (int)(q - 3 * g);
                int b = 0, n = -1;
                if (lane < at_once && q < sums) {
                    b = A.cell_ptr[g];
                    n = A.cell_ptr[g + 1] - b;
                    if (n <= CG_FEW) {
                        double s = 0.0;
                        for (int k = b; k < b + n; ++k) s += value(A.cell_mem[k], k0);
                        A.cellsum[q] = s;
                    }
                }
                unsigned m = __ballot_sync(0xffffffffu, n > CG_FEW);
                while (m) {
                    const int l = __ffs(m) - 1;
                    m &= m - 1;
                    const int b0 = __shfl_sync(0xffffffffu, b, l), e = b0 + __shfl_sync(0xffffffffu, n, l);
                    const int kl = __shfl_sync(0xffffffffu, k0, l);
                    double s = 0.0;
#pragma unroll 4
                    for (int k = b0 + lane; k < e; k += 32) s += value(A.cell_mem[k], kl);
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                    if (lane == l) A.cellsum[q] = s;
                }
            }
            return;
        }
        for (int64_t q = blockIdx.x + gridDim.x * (int64_t)(tid >> 5); q < 3 * A.ng; q += gridDim.x * (CG_THREADS / 32)) {
            const int64_t g = q / 3;
            const int k0 = (int)(q - 3 * g), e = A.cell_ptr[g + 1];
            double s = 0.0;
#pragma unroll 4
            for (int k = A.cell_ptr[g] + lane; k < e; k += 32) s += value(A.cell_mem[k], k0);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) A.cellsum[q] = s;
        }
    };
    // r = B - A x0 (B in r), z = r / diag, p = z
    double* p = A.p;
    double* pn = A.p + 4 * A.nv;
    if (A.ref) cells([&](int64_t j, int k) { return A.V0[3 * j + k]; });
    for (int64_t i = i0; i < i1; i += CG_ROWS) pn[4 * i + c] = A.V0[3 * i + c];  // x0 in rows of 4
    if (!grid_sync(A.bar, target += gridDim.x)) return;
    double sz = 0.0, sb = 0.0;
    for (int64_t i = i0; i < i1; i += CG_ROWS) {
        const double x0 = A.V0[3 * i + c], b = A.r[3 * i + c], rc = b - apply(pn, i, x0);
        const double d = 1.0 / A.diag[i], zc = rc * d;
        if (ONE) {
            x = x0;
            r = rc;
            di = d;
            pv = zc;
        } else {
            A.x[3 * i + c] = x0;
            A.r[3 * i + c] = rc;
            A.dinv[3 * i + c] = d;
        }
        A.z[4 * i + c] = zc;
        p[4 * i + c] = zc;
        sz += rc * zc;
        sb += b * b;
    }
    store_partial(sz, sh, PU);
    store_partial(sb, sh2, PR);
    if (!grid_sync(A.bar, target += gridDim.x)) return;
    grid_sum3(PU, [&](int k, double v) { rz[k] = v; });
    grid_sum3(PR, [&](int k, double v) { bb[k] = v; });
    if (A.ref) cells([&](int64_t j, int k) { return __ldcg(A.z + 4 * j + k); });
    if (!grid_sync(A.bar, target += gridDim.x)) return;

    int it = 0;
    double rel = INFINITY;
    while (it < A.max_iter) {
        const bool check = (it + 1) % CG_CHECK == 0 || it + 1 == A.max_iter;
        double y = 0, acc = 0.0;
        for (int64_t i = i0; i < i1; i += CG_ROWS) {
            const double pi = ONE ? pv : p[4 * i + c];
            y = apply(p, i, pi);
            acc += pi * y;
            if (!ONE) pn[4 * i + c] = y;  // A p waits where the next p will be
        }
        store_partial(acc, sh, PA);
        if (!grid_sync(A.bar, target += gridDim.x)) return;
        grid_sum3(PA, [&](int k, double v) { coef[k] = v > 0.0 ? rz[k] / v : 0.0; });
        const double alpha = coef[c];
        double s = 0.0, rr = 0.0;
        for (int64_t i = i0; i < i1; i += CG_ROWS) {
            double rc;
            if (ONE) {
                x += alpha * pv;
                r -= alpha * y;
                rc = r;
                z = rc * di;
            } else {
                A.x[3 * i + c] += alpha * p[4 * i + c];
                rc = A.r[3 * i + c] -= alpha * pn[4 * i + c];
                z = rc * A.dinv[3 * i + c];
            }
            A.z[4 * i + c] = z;
            s += rc * z;
            if (check) rr += rc * rc;
        }
        store_partial(s, sh, PU);
        if (check) store_partial(rr, sh2, PR);
        if (!grid_sync(A.bar, target += gridDim.x)) return;
        grid_sum3(PU, [&](int k, double v) {
            coef[k] = rz[k] > 0.0 ? v / rz[k] : 0.0;
            rz[k] = v;
        });
        ++it;
        if (check) {
            grid_sum3(PR, [&](int k, double v) { sum[k] = v; });
            if (tid == 0) {
                double m = 0.0;
                for (int k = 0; k < 3; ++k) {
                    const double v = bb[k] > 0.0 ? sqrt(sum[k] / bb[k]) : sqrt(sum[k]);
                    if (m < v) m = v;
                }
                rel_sh = m;
            }
            __syncthreads();
            rel = rel_sh;
            if (!(rel > A.tol)) break;
        }
        const double beta = coef[c];
        for (int64_t i = i0; i < i1; i += CG_ROWS) {
            if (ONE) pn[4 * i + c] = pv = fma(beta, pv, z);
            else pn[4 * i + c] = fma(beta, p[4 * i + c], A.z[4 * i + c]);
        }
        if (A.ref) {
            const double b0 = coef[0], b1 = coef[1], b2 = coef[2];
            cells([&](int64_t j, int k) {
                return fma(k == 0 ? b0 : k == 1 ? b1 : b2, __ldcg(p + 4 * j + k), __ldcg(A.z + 4 * j + k));
            });
        }
        double* t = p;
        p = pn;
        pn = t;
        if (!grid_sync(A.bar, target += gridDim.x)) return;
    }
    if (ONE)
        for (int64_t i = i0; i < i1; i += CG_ROWS) A.x[3 * i + c] = x;
    if (blockIdx.x == 0 && tid == 0) {
        A.result[0] = (double)it;
        A.result[1] = rel;
    }
}

__global__ void k_lin_to_float(const double* __restrict__ x, int64_t n, float* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (float)x[i];
}

}  // namespace
}  // namespace mo

using namespace mo;

namespace {
int solve_on(float* V, int64_t nv, const int32_t* F, int64_t nf, const int32_t* E, int64_t ne, const int32_t* ref,
             const float* G, int64_t ng, double rigidity, int with_rot, double tol, int max_iter, void* scratch,
             size_t scratch_bytes, int* iters_out, double* rel_residual_out, cudaStream_t s);
}  // namespace

extern "C" size_t mo_solve_linear_scratch_bytes(int64_t nv, int64_t nf, int64_t ne, int64_t ng, int with_rot) {
    if (nv < 0 || nf < 0 || ne < 0 || ng < 0) return 0;
    return plan(nullptr, nv, nf, ne, ng, with_rot ? 1 : 0).bytes;
}

extern "C" int mo_solve_linear(float* V, int64_t nv, const int32_t* F, int64_t nf, const int32_t* E, int64_t ne,
                               const int32_t* ref, const float* G, int64_t ng, double rigidity, int with_rot,
                               double tol, int max_iter, void* scratch, size_t scratch_bytes, int* iters_out,
                               double* rel_residual_out, void* stream) {
    with_rot = with_rot ? 1 : 0;
    MO_CHECK_ARG(nv > 0 && nf >= 0 && ne >= 0 && ng >= 0, "bad sizes");
    MO_CHECK_ARG(nv < ((int64_t)1 << 30) && 3 * nf + ne < ((int64_t)1 << 30), "system too large");
    MO_CHECK_ARG(V && G && (nf == 0 || F), "null pointer");
    MO_CHECK_ARG(with_rot || ((ne == 0 || E) && ref && ng > 0), "LinearEstimation needs references and a graph");
    MO_CHECK_ARG(!with_rot || ng == nv, "with_rot needs one target position per vertex (ng == nv)");
    MO_CHECK_ARG(tol > 0.0 && max_iter > 0, "bad tolerance or iteration limit");
    MO_CHECK_ARG(std::isfinite(rigidity), "bad rigidity");
    // The solve runs on a stream of its own that first waits for the caller's
    // work.
    cudaStream_t caller = as_stream(stream);
    cudaStream_t s = nullptr;
    cudaEvent_t ready = nullptr;
    MO_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    cudaError_t e0 = cudaEventCreateWithFlags(&ready, cudaEventDisableTiming);
    if (e0 == cudaSuccess) e0 = cudaEventRecord(ready, caller);
    if (e0 == cudaSuccess) e0 = cudaStreamWaitEvent(s, ready, 0);
    if (ready) cudaEventDestroy(ready);
    if (e0 != cudaSuccess) {
        cudaStreamDestroy(s);
        return cuda_status(e0, "solver stream");
    }
    int rc0 = solve_on(V, nv, F, nf, E, ne, ref, G, ng, rigidity, with_rot, tol, max_iter, scratch, scratch_bytes,
                       iters_out, rel_residual_out, s);
    cudaStreamSynchronize(s);
    cudaStreamDestroy(s);
    return rc0;
}

namespace {
int solve_on(float* V, int64_t nv, const int32_t* F, int64_t nf, const int32_t* E, int64_t ne, const int32_t* ref,
             const float* G, int64_t ng, double rigidity, int with_rot, double tol, int max_iter, void* scratch,
             size_t scratch_bytes, int* iters_out, double* rel_residual_out, cudaStream_t s) {
    const LinScratch need = plan(nullptr, nv, nf, ne, ng, with_rot);
    void* owned = nullptr;
    if (!scratch) {
        MO_CUDA(cudaMallocAsync(&owned, need.bytes, s));
        scratch = owned;
    } else if (scratch_bytes < need.bytes) {
        set_error("SolveLinear scratch too small: %zu < %zu", scratch_bytes, need.bytes);
        return MO_ERR_SCRATCH;
    }
    LinScratch S = plan(reinterpret_cast<char*>(scratch), nv, nf, ne, ng, with_rot);
    const int64_t nh = 3 * nf + (with_rot ? 0 : ne);
    int rc = MO_OK;
    auto fail = [&](cudaError_t e, const char* where) { rc = cuda_status(e, where); };
    do {
        cudaError_t e = cudaMemsetAsync(S.status, 0, 16, s);
        if (e == cudaSuccess) e = cudaMemsetAsync(S.bar, 0, 16, s);
        if (e != cudaSuccess) { fail(e, "memset"); break; }
        if (nh > 0) {
            k_lin_edges<<<ceil_div(nh, 256), 256, 0, s>>>(F, nf, with_rot ? nullptr : E, with_rot ? 0 : ne, S.edges);
            ::mo::note_launch();
        }
        rc = mo_edge_csr_build(S.edges, nh, MO_EDGES_LIST, nv, S.csr, S.csr_bytes, S.status, s);
        if (rc) break;
        const int* row_ptr = reinterpret_cast<const int*>(S.csr);
        const int* key = row_ptr + (nv + 1);
        const int* other = key + 2 * nh;
        // the status must be clean before any kernel indexes by the edges
        int status = 0;
        e = cudaMemcpyAsync(&status, S.status, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) { fail(e, "status"); break; }
        if (status) { set_error("edge or face index out of range [0, %lld)", (long long)nv); rc = MO_ERR_DEVICE; break; }
        k_lin_to_double<<<ceil_div(3 * nv, 256), 256, 0, s>>>(V, 3 * nv, S.V0); ::mo::note_launch();
        k_lin_to_double<<<ceil_div(3 * (with_rot ? nv : ng), 256), 256, 0, s>>>(G, 3 * (with_rot ? nv : ng), S.G);
        ::mo::note_launch();
        if (nh > 0) {
            k_lin_weights<<<ceil_div(nh, 256), 256, 0, s>>>(S.edges, nh, S.V0, rigidity, with_rot, S.w);
            ::mo::note_launch();
        }
        double c0;
        if (!with_rot) {
            k_lin_cell_keys<<<ceil_div(nv, 256), 256, 0, s>>>(ref, nv, ng, S.keys_a, S.vals_a, S.status);
            ::mo::note_launch();
            int bits = 1;
            while (bits < 32 && ((int64_t)1 << bits) < ng) ++bits;
            e = radix_sort_pairs(S.keys_a, S.vals_a, S.keys_b, S.vals_b, (int)nv, bits, S.hist, s);
            if (e != cudaSuccess) { fail(e, "radix_sort_pairs"); break; }
            e = cudaMemcpyAsync(&status, S.status, sizeof(int), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) { fail(e, "status"); break; }
            if (status) { set_error("reference index out of range [0, %lld)", (long long)ng); rc = MO_ERR_DEVICE; break; }
            k_lin_cell_ptr<<<ceil_div(nv, 256), 256, 0, s>>>(S.keys_a, nv, S.cell_ptr); ::mo::note_launch();
            k_lin_cell_tail<<<1, 1, 0, s>>>(S.keys_a, nv, ng, S.cell_ptr); ::mo::note_launch();
            e = cudaMemcpyAsync(S.cell_mem, S.vals_a, 4 * (size_t)nv, cudaMemcpyDeviceToDevice, s);
            if (e != cudaSuccess) { fail(e, "copy"); break; }
            k_lin_cellw<<<ceil_div(ng, 256), 256, 0, s>>>(S.cell_ptr, ng, S.cellw); ::mo::note_launch();
            k_lin_rhs<<<ceil_div(nv, 256), 256, 0, s>>>(nv, row_ptr, other, key, S.w, S.V0, ref, S.G, S.cellw,
                                                        S.diag, S.r);
            ::mo::note_launch();
            c0 = 1e-6;
        } else {
            k_lin_rotations<<<ceil_div(nv, 128), 128, 0, s>>>(nv, row_ptr, other, S.V0, S.G, S.rot); ::mo::note_launch();
            k_lin_rhs_rot<<<ceil_div(nv, 256), 256, 0, s>>>(nv, row_ptr, other, key, S.w, S.V0, S.G, S.rot, S.diag,
                                                            S.r);
            ::mo::note_launch();
            c0 = 1.0;
        }
        const int32_t* cref = with_rot ? nullptr : ref;
        k_lin_merge<<<ceil_div(nv, 128), 128, 0, s>>>(nv, row_ptr, other, key, S.w, S.nbr, S.nnbr); ::mo::note_launch();
        // one block per SM, fewer where blocks would have too few vertices for the barriers to pay
        int blocks = (int)std::max<int64_t>(
            1, std::min<int64_t>(std::min(device_sm_count(), CG_MAX_BLOCKS), (nv + CG_MIN_ROWS - 1) / CG_MIN_ROWS));
        CgArgs args{nv, ng, row_ptr, S.nbr, S.nnbr, cref, S.cellw, S.cell_ptr, S.cell_mem, c0, S.V0, S.diag,
                    S.x, S.r, S.dinv, S.z, S.p, S.cellsum, S.partial, S.result, S.bar, tol, max_iter};
        void* argv[] = {&args};
        // half of them as long as the process has only a part of the SMs (a partition of
        // the device): one block always fits
        for (;; blocks /= 2) {
            const bool one = (nv + blocks - 1) / blocks <= CG_ROWS;
            const bool many = cref && nv < ng * 1024 && 3 * ng > (int64_t)4 * blocks * (CG_THREADS / 32);
            const void* kernel = many ? (one ? (const void*)k_lin_cg<true, true> : (const void*)k_lin_cg<false, true>)
                                      : (one ? (const void*)k_lin_cg<true, false> : (const void*)k_lin_cg<false, false>);
            const int smem = one ? CG_ROW_BYTES : 0;
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (e == cudaSuccess)
                e = cudaLaunchCooperativeKernel(kernel, dim3(blocks), dim3(CG_THREADS), argv, smem, s);
            if (e != cudaErrorCooperativeLaunchTooLarge || blocks == 1) break;
            cudaGetLastError();
        }
        ::mo::note_launch();
        if (e != cudaSuccess) { fail(e, "k_lin_cg"); break; }
        double result[2];
        unsigned aborted[2];
        e = cudaMemcpyAsync(result, S.result, sizeof(result), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(aborted, S.bar, sizeof(aborted), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) { fail(e, "conjugate gradients"); break; }
        if (aborted[1]) {
            set_error("conjugate gradients: a grid barrier ran out of time");
            rc = MO_ERR_DEVICE;
            break;
        }
        const int it = (int)result[0];
        const double rel = result[1];
        if (rc) break;
        if (iters_out) *iters_out = it;
        if (rel_residual_out) *rel_residual_out = rel;
        k_lin_to_float<<<ceil_div(3 * nv, 256), 256, 0, s>>>(S.x, 3 * nv, V); ::mo::note_launch();
        e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) { fail(e, "solve"); break; }
        if (!(rel <= tol)) {
            set_error("conjugate gradients did not reach %g in %d iterations (relative residual %g)", tol, it, rel);
            rc = MO_ERR_DEVICE;
        }
    } while (0);
    if (owned) cudaFreeAsync(owned, s);
    return rc;
}
}  // namespace
