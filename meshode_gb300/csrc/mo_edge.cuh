// Half-edges and the vertex->half-edge CSR, shared by the edge losses
// (mo_edge.cu) and the fused layer losses (mo_layer.cu).
//
// CSR buffer layout (int32 words):
//   row_ptr[nv+1] | key[2H] | other[2H] | cursor[nv] | status[1] | pad
// key = 2*h + role, role 0 when the vertex is the half-edge's v0 (the
// reference's `g[v0] -= r`), 1 when it is v1 (`g[v1] += r`).  Rows are sorted
// by key, i.e. in the order the reference's serial loop touches the vertex.
#pragma once

#include "mo_common.cuh"

namespace mo {

struct CsrView {
    int* row_ptr;
    int* key;
    int* other;
    int* cursor;
    int* status;
};

static inline CsrView csr_view(void* base, int64_t nv, int64_t nh) {
    CsrView v;
    int* p = reinterpret_cast<int*>(base);
    v.row_ptr = p;
    v.key = p + (nv + 1);
    v.other = v.key + 2 * nh;
    v.cursor = v.other + 2 * nh;
    v.status = v.cursor + nv;
    return v;
}

__device__ __forceinline__ void he_ends(const int32_t* __restrict__ idx, int kind, int64_t h, int& v0, int& v1) {
    if (kind == MO_EDGES_FACES) {
        const int64_t f = h / 3;
        const int j = (int)(h - 3 * f);
        v0 = idx[3 * f + j];
        v1 = idx[3 * f + (j == 2 ? 0 : j + 1)];
    } else {
        v0 = idx[2 * h];
        v1 = idx[2 * h + 1];
    }
}

__device__ __forceinline__ bool in_range(int v, int64_t nv) { return v >= 0 && (int64_t)v < nv; }

// The gradient of the edge term at vertex i: its half-edges' residuals in the
// order of the reference's serial scatter (rigid_layer.cc:119-129).
__device__ __forceinline__ void edge_gather(const float* __restrict__ V, int64_t i, const int* __restrict__ row_ptr,
                                            const int* __restrict__ key, const int* __restrict__ other,
                                            const float* __restrict__ off, float& gx, float& gy, float& gz) {
    const float px = V[3 * i], py = V[3 * i + 1], pz = V[3 * i + 2];
    gx = 0.0f; gy = 0.0f; gz = 0.0f;
    const int b = row_ptr[i], e = row_ptr[i + 1];
    for (int k = b; k < e; ++k) {
        const int kk = key[k];
        const int64_t h = kk >> 1;
        const int64_t o = other[k];
        const float qx = V[3 * o], qy = V[3 * o + 1], qz = V[3 * o + 2];
        const float ox = off[3 * h], oy = off[3 * h + 1], oz = off[3 * h + 2];
        if ((kk & 1) == 0) {  // this vertex is v0: g[v0] -= (v1 - v0 - off)
            gx = SUB(gx, SUB(SUB(qx, px), ox));
            gy = SUB(gy, SUB(SUB(qy, py), oy));
            gz = SUB(gz, SUB(SUB(qz, pz), oz));
        } else {              // this vertex is v1: g[v1] += (v1 - v0 - off)
            gx = ADD(gx, SUB(SUB(px, qx), ox));
            gy = ADD(gy, SUB(SUB(py, qy), oy));
            gz = ADD(gz, SUB(SUB(pz, qz), oz));
        }
    }
}

}  // namespace mo
