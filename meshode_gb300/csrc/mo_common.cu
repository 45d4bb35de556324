// Error state, device queries and two set-up primitives shared by the
// builders: a single-CTA exclusive scan and a stable LSD radix sort.
#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstring>

#include "mo_common.cuh"

namespace mo {

static thread_local char g_err[512] = "";
static std::atomic<unsigned long long> g_launches{0};

void note_launch(int n) { g_launches.fetch_add((unsigned long long)n, std::memory_order_relaxed); }

void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}

int cuda_status(cudaError_t e, const char* where) {
    set_error("CUDA error %d (%s) in %s", (int)e, cudaGetErrorString(e), where);
    return MO_ERR_CUDA;
}

int device_sm_count() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 1;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 1;
    return sms > 0 ? sms : 1;
}

// ---------------------------------------------------------------------------
// Single-CTA exclusive scan, in tiles of 1024 x 8 ints: coalesced loads into
// shared memory, each thread scans 8 consecutive ints, a block scan of the
// thread sums, coalesced stores; a running carry joins the tiles.
// ---------------------------------------------------------------------------
constexpr int SCAN_THREADS = 1024, SCAN_PER = 8, SCAN_TILE = SCAN_THREADS * SCAN_PER;

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_1cta(int* a, int n, int* total) {
    __shared__ int tile[SCAN_TILE + SCAN_TILE / 32];  // one pad int per 32 breaks bank conflicts
    __shared__ int warp_sums[32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    auto at = [](int i) { return i + (i >> 5); };
    int carry = 0;
    for (int base = 0; base < n; base += SCAN_TILE) {
#pragma unroll
        for (int k = 0; k < SCAN_PER; ++k) {
            const int i = k * SCAN_THREADS + tid;
            tile[at(i)] = base + i < n ? a[base + i] : 0;
        }
        __syncthreads();
        int v[SCAN_PER];
        int s = 0;
#pragma unroll
        for (int k = 0; k < SCAN_PER; ++k) {
            v[k] = s;
            s += tile[at(tid * SCAN_PER + k)];
        }
        int x = s;  // inclusive scan of the thread sums
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sums[w] = x;
        __syncthreads();
        if (w == 0) {
            int ws = warp_sums[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, ws, o);
                if (lane >= o) ws += y;
            }
            warp_sums[lane] = ws;
        }
        __syncthreads();
        const int pre = carry + x - s + (w > 0 ? warp_sums[w - 1] : 0);
#pragma unroll
        for (int k = 0; k < SCAN_PER; ++k) tile[at(tid * SCAN_PER + k)] = pre + v[k];
        const int tile_total = warp_sums[31];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < SCAN_PER; ++k) {
            const int i = k * SCAN_THREADS + tid;
            if (base + i < n) a[base + i] = tile[at(i)];
        }
        carry += tile_total;
        __syncthreads();  // tile and warp_sums are rewritten next round
    }
    if (total && tid == 0) *total = carry;
}

cudaError_t exclusive_scan_i32(int* data, int n, int* total, cudaStream_t s) {
    if (n <= 0) {
        if (total) return cudaMemsetAsync(total, 0, sizeof(int), s);
        return cudaSuccess;
    }
    k_scan_1cta<<<1, 1024, 0, s>>>(data, n, total); ::mo::note_launch();
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort, 8-bit digits, one kernel per digit by decoupled look-back
// (Merrill and Garland 2016; for sorting Adinets and Merrill 2022).  One pass over the
// keys counts every digit of every pass; then each pass is a single kernel:
// a tile ranks its keys (per-warp ranks from __match_any_sync, warps in order),
// publishes its digit counts and adds up its predecessors' by looking back over
// their published words, 16 at a time, until one holds an inclusive prefix.
// Tiles take their number from a counter, so every predecessor is running.  A tile
// that has waited for one for too long all the same counts the keys before its own
// by itself, which needs nobody: the order is complete whatever the waits did.
// (Before: histogram, single-CTA scan and scatter per digit, 12 launches for
// 30-bit codes: 75 us at 20k to 50k keys, 130 us at 355k.)
//
// hist: counts [4][256] | tickets [4] | words [passes][tiles][256], zeroed per sort;
// a word is state << BITS | count, state 1: the tile's count, 2: inclusive prefix.
// 30 bits hold the count of a digit up to 2^30 - 1 keys; from 2^30 on the words
// have 64 bits, twice the bytes to clear and to look back over.
// ---------------------------------------------------------------------------
constexpr int RS_WARPS = 8, RS_PASSES = 4, RS_HEAD = RS_PASSES * 256 + 64;
// keys per thread: small sorts take small tiles, so that more SMs share them
// (the rank loop is serial in a tile's rounds)
constexpr int RS_SMALL = 1 << 17;
static int rs_rounds(int n) { return n <= RS_SMALL ? 2 : 8; }
static int rs_tiles(int n) { return ceil_div(n > 0 ? n : 1, RS_WARPS * 32 * rs_rounds(n)); }

constexpr int RS_WIDE = 1 << 30;
static size_t rs_word_ints(int n) { return 256 * (size_t)rs_tiles(n) * (n >= RS_WIDE ? 2 : 1); }  // of a pass

size_t radix_hist_ints(int n) { return (size_t)RS_HEAD + RS_PASSES * rs_word_ints(n); }

__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed(uint64_t* p, uint64_t v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint64_t ld_relaxed(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__global__ void __launch_bounds__(256) k_rs_count(const uint32_t* __restrict__ keys, int n, int passes,
                                                  int* __restrict__ hist) {
    __shared__ int h[RS_PASSES][256];
    for (int p = 0; p < RS_PASSES; ++p) h[p][threadIdx.x] = 0;
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
        const uint32_t k = keys[i];
        for (int p = 0; p < passes; ++p) atomicAdd(&h[p][(k >> (8 * p)) & 255u], 1);
    }
    __syncthreads();
    for (int p = 0; p < passes; ++p)
        if (h[p][threadIdx.x]) atomicAdd(hist + 256 * p + threadIdx.x, h[p][threadIdx.x]);
}

template <int ROUNDS, class Word>
__global__ void __launch_bounds__(256) k_rs_pass(const uint32_t* __restrict__ kin, const int* __restrict__ vin,
                                                 uint32_t* __restrict__ kout, int* __restrict__ vout, int n, int pass,
                                                 int* __restrict__ hist, Word* __restrict__ words,
                                                 unsigned long long max_wait) {
    constexpr int BITS = 8 * sizeof(Word) - 2;
    constexpr Word COUNT = ((Word)1 << BITS) - 1;
    __shared__ int wh[RS_WARPS][256];
    __shared__ int warp_sum[8];
    __shared__ int tile_sh;
    __shared__ int before[256];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, shift = 8 * pass;
    if (threadIdx.x == 0) tile_sh = atomicAdd(hist + RS_PASSES * 256 + pass, 1);
    for (int d = threadIdx.x; d < RS_WARPS * 256; d += 256) (&wh[0][0])[d] = 0;
    __syncthreads();
    const int tile = tile_sh;
    const int64_t wbeg = ((int64_t)tile * RS_WARPS + w) * ROUNDS * 32;
    const unsigned lt = (1u << lane) - 1u;
    uint32_t key[ROUNDS];
    int val[ROUNDS], digit[ROUNDS], rank[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const int64_t i = wbeg + r * 32 + lane;
        key[r] = i < n ? kin[i] : 0u;
        val[r] = i < n ? vin[i] : 0;
    }
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const bool valid = wbeg + r * 32 + lane < n;
        digit[r] = valid ? (int)((key[r] >> shift) & 255u) : 256 + lane;
        const unsigned peers = __match_any_sync(0xffffffffu, digit[r]);
        int pre = 0;
        if (valid) pre = wh[w][digit[r]];
        __syncwarp();
        if (valid && lane == __ffs(peers) - 1) wh[w][digit[r]] = pre + __popc(peers);
        __syncwarp();
        rank[r] = pre + __popc(peers & lt);
    }
    __syncthreads();
    // thread d owns digit d: the tile's count, the keys of smaller digits (an
    // exclusive scan of the counts over all keys), the predecessors' keys of digit d
    const int d = threadIdx.x;
    int mine = 0;
#pragma unroll
    for (int ww = 0; ww < RS_WARPS; ++ww) mine += wh[ww][d];
    Word* my = words + (int64_t)tile * 256 + d;
    st_relaxed(my, (Word)(tile == 0 ? 2 : 1) << BITS | (Word)mine);
    const int total = hist[256 * pass + d];
    int x = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[w] = x;
    __syncthreads();
    int base = x - total;
    for (int k = 0; k < w; ++k) base += warp_sum[k];
    int prefix = 0;
    bool lost = false;
    if (tile > 0) {
        constexpr int BATCH = 16;
        unsigned long long t0 = 0, now;
        for (int t = tile - 1; t >= 0;) {
            Word v[BATCH];
#pragma unroll
            for (int k = 0; k < BATCH; ++k) v[k] = t - k >= 0 ? ld_relaxed(words + (int64_t)(t - k) * 256 + d) : 0;
            bool end = false, stalled = false;
#pragma unroll
            for (int k = 0; k < BATCH; ++k) {
                if (end || stalled || t < 0) continue;
                const int st = (int)(v[k] >> BITS);
                if (st == 0) {
                    stalled = true;
                    continue;
                }
                prefix += (int)(v[k] & COUNT);
                --t;
                end = st == 2;
            }
            if (end) break;
            if (stalled) {  // a predecessor has not published yet
                asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
                if (t0 == 0) t0 = now;
                lost = now - t0 >= max_wait;
                if (lost) break;
            }
        }
        if (!lost) st_relaxed(my, (Word)2 << BITS | (Word)(prefix + mine));
    }
    if (__syncthreads_or(lost)) {
        before[d] = 0;
        __syncthreads();
        const int64_t first = (int64_t)tile * RS_WARPS * ROUNDS * 32;
        for (int64_t i = d; i < first; i += 256) atomicAdd(&before[(kin[i] >> shift) & 255u], 1);
        __syncthreads();
        if (lost) {
            prefix = before[d];
            st_relaxed(my, (Word)2 << BITS | (Word)(prefix + mine));
        }
    }
    int run = base + prefix;
#pragma unroll
    for (int ww = 0; ww < RS_WARPS; ++ww) {
        const int c = wh[ww][d];
        wh[ww][d] = run;
        run += c;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        if (wbeg + r * 32 + lane < n) {
            const int pos = wh[w][digit[r]] + rank[r];
            if ((unsigned)pos < (unsigned)n) {  // always, unless somebody else writes to the scratch
                kout[pos] = key[r];
                vout[pos] = val[r];
            }
        }
    }
}

cudaError_t radix_sort_pairs(uint32_t* keys_a, int* vals_a, uint32_t* keys_b, int* vals_b, int n,
                             int bits, int* hist, cudaStream_t s, uint64_t max_wait_ns) {
    if (n <= 1) return cudaSuccess;
    const int tiles = rs_tiles(n), passes = (bits + 7) / 8;
    cudaError_t e = cudaMemsetAsync(hist, 0, sizeof(int) * ((size_t)RS_HEAD + passes * rs_word_ints(n)), s);
    if (e != cudaSuccess) return e;
    k_rs_count<<<std::min(ceil_div(n, 1024), 2 * device_sm_count()), 256, 0, s>>>(keys_a, n, passes, hist);
    ::mo::note_launch();
    uint32_t *ki = keys_a, *ko = keys_b;
    int *vi = vals_a, *vo = vals_b;
    for (int p = 0; p < passes; ++p) {
        uint32_t* words = reinterpret_cast<uint32_t*>(hist) + RS_HEAD + p * rs_word_ints(n);
        if (rs_rounds(n) == 2)
            k_rs_pass<2><<<tiles, 256, 0, s>>>(ki, vi, ko, vo, n, p, hist, words, max_wait_ns);
        else if (n < RS_WIDE)
            k_rs_pass<8><<<tiles, 256, 0, s>>>(ki, vi, ko, vo, n, p, hist, words, max_wait_ns);
        else
            k_rs_pass<8><<<tiles, 256, 0, s>>>(ki, vi, ko, vo, n, p, hist, reinterpret_cast<uint64_t*>(words),
                                                 max_wait_ns);
        ::mo::note_launch();
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        uint32_t* tk = ki; ki = ko; ko = tk;
        int* tv = vi; vi = vo; vo = tv;
    }
    if (ki != keys_a) {  // odd number of passes: result is in *_b
        e = cudaMemcpyAsync(keys_a, ki, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) return e;
        e = cudaMemcpyAsync(vals_a, vi, sizeof(int) * n, cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace mo

extern "C" size_t mo_sort_pairs_scratch_bytes(int64_t n) {
    if (n < 0 || n > INT_MAX) return 0;
    return sizeof(int) * mo::radix_hist_ints((int)n) + 8 * (size_t)n;
}

extern "C" int mo_sort_pairs(uint32_t* keys, int32_t* vals, int64_t n, int bits, void* scratch, size_t scratch_bytes,
                             uint64_t max_wait_ns, void* stream) {
    MO_CHECK_ARG(n >= 0 && n <= INT_MAX, "bad number of keys");
    MO_CHECK_ARG(bits >= 1 && bits <= 32, "keys have 1 to 32 bits, got %d", bits);
    if (n <= 1) return MO_OK;
    MO_CHECK_ARG(keys && vals && scratch && mo::aligned(scratch, 8), "null or misaligned pointer");
    if (scratch_bytes < mo_sort_pairs_scratch_bytes(n)) {
        mo::set_error("sort scratch too small: %zu < %zu", scratch_bytes, mo_sort_pairs_scratch_bytes(n));
        return MO_ERR_SCRATCH;
    }
    int* hist = reinterpret_cast<int*>(scratch);
    uint32_t* keys_b = reinterpret_cast<uint32_t*>(hist + mo::radix_hist_ints((int)n));
    MO_CUDA(mo::radix_sort_pairs(keys, vals, keys_b, reinterpret_cast<int*>(keys_b + n), (int)n, bits, hist,
                                 mo::as_stream(stream), max_wait_ns));
    return MO_OK;
}

extern "C" const char* mo_last_error(void) { return mo::g_err; }
extern "C" int mo_version(void) { return 100; }
extern "C" unsigned long long mo_launch_count(void) { return mo::g_launches.load(std::memory_order_relaxed); }
