// COO -> canonical CSR on the device: the canonicalisation the reference's
// Matrix Market loader does on the host (rv-sparse
// tools/src/mtx_to_csr_formatter.c:219-330 and canonicalise_rows :74-151):
// symmetric storage expanded by appending the mirror of every off-diagonal
// entry after all stored ones (:221-244); entries bucketed by row in COO
// order (:246-300); each row sorted by column and repeated (row, column)
// entries summed (:112-131).
//
// Here: one stable LSD radix sort of the packed keys (row << cb | column) with
// the values as payload, so entries with equal keys stay in COO order; then
// each run of equal keys is summed left to right, starting from its first
// value like the reference (acc = first; acc += next ...), and the row pointer
// is written where a run starts a new row. Every pass is a device kernel; the
// only host work is the launch sequence and one read of the output size.
//
// A pass reads and writes every entry once: the digit counts of all passes
// come from one sweep over the list beforehand, and a tile learns where its
// digits go from the tiles before it while the pass runs (k_coo_pass), so no
// pass counts first. Measured (16.8 M entries of 40-bit keys, 5 passes, whole
// call): 2.72 ms with a histogram, a scan and an uncoalesced scatter per pass
// and 16-byte entries, 1.22 ms now; 177 us a pass against 62 us of HBM time for
// its 24 bytes an entry. A tile takes 34,000 cycles, of which the wait for the
// tiles before it 8,000 (without it a pass takes 122 us, without the output
// writes 165). Tried and dropped: tiles of 512 threads with 8 entries each (193
// us with two CTAs an SM, 215 with three), 4 or 16 earlier tiles read at once
// (no difference).

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <utility>

#include "rv_sparse_types.h"
#include "rvsp_cuda.h"
#include "rvsp_internal.h"

using namespace rvsp;

namespace {

constexpr int CS_TPB = 256;
constexpr int CS_ITEMS = 16;
constexpr int CS_TILE = CS_TPB * CS_ITEMS;  // entries per tile
constexpr int CS_WARPS = CS_TPB / 32;
constexpr int RUN_ITEMS = 8;
constexpr int RUN_TILE = CS_TPB * RUN_ITEMS;  // sorted entries per tile of the run kernels
constexpr int CS_PASSES = 8;   // 62-bit keys at most
constexpr int CS_COPIES = 4;   // shared copies of the digit counters (fewer collisions)
constexpr unsigned CS_FULL = 0xffffffffu;
constexpr int COO_BAD = 1;     // error word: an index out of range
constexpr int COO_STUCK = 2;   // a wait on an earlier tile ran out

__device__ __forceinline__ int c_lane() { return threadIdx.x & 31; }

// Digits of the keys: `passes` of db bits.
struct Digits {
    int passes, db;
    __device__ __forceinline__ int of(uint64_t key, int p) const {
        return (int)(key >> (p * db)) & ((1 << db) - 1);
    }
};

// Where a pass reads its keys: the COO list itself or an array of keys.
struct CooKeys {
    const int32_t* r;
    const int32_t* c;
    int32_t rows, cols;
    int cb;
    int32_t* bad;
    __device__ __forceinline__ uint64_t at(int64_t i) const {
        const int32_t ri = r[i], ci = c[i];
        if ((unsigned)ri >= (unsigned)rows || (unsigned)ci >= (unsigned)cols) {
            atomicOr(bad, COO_BAD);
            return 0;
        }
        return ((uint64_t)ri << cb) | (uint64_t)ci;
    }
};

template <class K>
struct ArrayKeys {
    const K* k;
    __device__ __forceinline__ uint64_t at(int64_t i) const { return k[i]; }
};

// Keys and values of a list: used for symmetric lists, whose mirrored entries
// go after the stored ones, in the stored order (mpos = exclusive scan of
// off-diagonal flags), and for keys of no bits, which no pass reads.
template <class K>
__global__ void k_coo_keys(int64_t n, CooKeys src, const float* __restrict__ v, int symmetric,
                           const int64_t* __restrict__ mpos, K* __restrict__ keys,
                           float* __restrict__ vals) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t key = src.at(i);
    keys[i] = (K)key;
    if (v) vals[i] = v[i];
    const int32_t ri = src.r[i], ci = src.c[i];
    if (symmetric && ri != ci) {
        const int64_t j = n + mpos[i];
        // (rows == cols: an index in range is in range mirrored)
        const bool ok = (unsigned)ri < (unsigned)src.rows && (unsigned)ci < (unsigned)src.cols;
        keys[j] = ok ? (K)(((uint64_t)ci << src.cb) | (uint64_t)ri) : (K)0;
        if (v) vals[j] = v[i];
    }
}

__global__ void k_offdiag(int64_t n, const int32_t* __restrict__ r, const int32_t* __restrict__ c,
                          int32_t* __restrict__ flag) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) flag[i] = r[i] != c[i];
}

// Digit counts of every pass in one sweep: counts[p * 256 + digit].
template <class Src>
__global__ void __launch_bounds__(CS_TPB)
    k_coo_digits(int64_t n, Src src, Digits dg, unsigned long long* __restrict__ counts) {
    __shared__ uint32_t h[CS_COPIES][CS_PASSES * 256];
    for (int x = threadIdx.x; x < CS_COPIES * CS_PASSES * 256; x += CS_TPB) (&h[0][0])[x] = 0u;
    __syncthreads();
    uint32_t* mine = h[threadIdx.x & (CS_COPIES - 1)];
    const int64_t step = (int64_t)gridDim.x * CS_TPB;
    for (int64_t i = (int64_t)blockIdx.x * CS_TPB + threadIdx.x; i < n; i += step) {
        const uint64_t key = src.at(i);
        for (int p = 0; p < dg.passes; ++p) atomicAdd(&mine[p * 256 + dg.of(key, p)], 1u);
    }
    __syncthreads();
    for (int x = threadIdx.x; x < dg.passes * 256; x += CS_TPB) {
        uint32_t s = 0;
        for (int k = 0; k < CS_COPIES; ++k) s += h[k][x];
        if (s) atomicAdd(&counts[x], (unsigned long long)s);
    }
}

// Exclusive scan of 256 values, one a thread.
__device__ __forceinline__ uint32_t scan256(uint32_t x, uint32_t* s_warp) {
    const int lane = c_lane(), warp = threadIdx.x >> 5;
    uint32_t incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(CS_FULL, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t before = 0;
    for (int w = 0; w < warp; ++w) before += s_warp[w];
    __syncthreads();
    return before + incl - x;
}

// Where every digit of every pass starts: one CTA a pass.
__global__ void __launch_bounds__(256)
    k_coo_starts(const unsigned long long* __restrict__ counts, uint32_t* __restrict__ starts) {
    __shared__ uint32_t s_warp[8];
    const int x = blockIdx.x * 256 + threadIdx.x;
    starts[x] = scan256((uint32_t)counts[x], s_warp);
}

__device__ __forceinline__ unsigned long long load_word(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void store_word(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" : : "l"(p), "l"(v));
}

// Lanes whose digit equals the caller's (ok lanes only), a ballot a bit
// (match_any instead: 195 us a pass against 177).
__device__ __forceinline__ unsigned same_digit(int d, bool ok) {
    unsigned peers = __ballot_sync(CS_FULL, ok);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = d >> b & 1;
        const unsigned bal = __ballot_sync(CS_FULL, bit);
        peers &= bit ? bal : ~bal;
    }
    return peers;
}

// Polls of one wait before it gives up (a second or more; a tile waits only
// for tiles that started before it, so an ordinary wait is microseconds).
constexpr int CS_POLLS = 1 << 20;
constexpr int CS_BACK = 16;  // earlier tiles read at once

// One stable pass by digit p. Tiles are numbered in the order they start, so
// every tile a tile waits for is running or done. Per tile: ranks of its
// entries within their digits (warp by warp, step by step: ballots give
// the lanes of one digit, counters of half a warp's entries those before), entries to
// shared memory in digit order, then written out run by run. Where each
// digit's run goes: the tile publishes its digit counts as soon as it has them
// (tag 2p + 1), thread d adds up digit d's counts of the tiles before it back
// to one that has published its running total (tag 2p + 2), and publishes its
// own. A word holds tag and count, so reading it needs no fence; words of
// earlier passes carry smaller tags and read as not yet there.
template <class K, class Src, bool VAL>
__global__ void __launch_bounds__(CS_TPB, 3)
    k_coo_pass(int64_t n, Src src, const float* __restrict__ vals, Digits dg, int p,
               const uint32_t* __restrict__ starts, unsigned long long* __restrict__ status,
               int32_t* __restrict__ ticket, K* __restrict__ keys_out,
               float* __restrict__ vals_out, int32_t* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char smem[];
    K* s_key = reinterpret_cast<K*>(smem);
    float* s_val = reinterpret_cast<float*>(s_key + CS_TILE);
    uint16_t* s_cnt = reinterpret_cast<uint16_t*>(s_val + (VAL ? CS_TILE : 0));  // [half of a warp][256]
    __shared__ uint32_t s_first[256];  // digit d's first entry in the tile
    __shared__ int64_t s_to[256];      // its place in the output less s_first
    __shared__ uint32_t s_warp[8];
    __shared__ int s_tile, s_dead;
    const int t = threadIdx.x, lane = c_lane(), warp = t >> 5;
    if (t == 0) {
        s_tile = atomicAdd(ticket, 1);
        s_dead = 0;
    }
    for (int x = t; x < CS_WARPS * 256; x += CS_TPB) reinterpret_cast<uint32_t*>(s_cnt)[x] = 0u;
    __syncthreads();
    const int tile = s_tile;
    const int64_t base = (int64_t)tile * CS_TILE + warp * (32 * CS_ITEMS);
    K key[CS_ITEMS];
    uint16_t rank[CS_ITEMS];
    // the warp's entries as two halves with counters of their own, ranked side
    // by side: two chains through shared memory instead of one twice as long
    constexpr int HALF = CS_ITEMS / 2;
    uint16_t* cnt = s_cnt + 2 * warp * 256;
#pragma unroll
    for (int s = 0; s < CS_ITEMS; ++s) {
        const int64_t i = base + 32 * s + lane;
        key[s] = i < n ? (K)src.at(i) : (K)0;
    }
#pragma unroll
    for (int s = 0; s < HALF; ++s) {
        int d[2], before[2];
        unsigned peers[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const bool ok = base + 32 * (s + h * HALF) + lane < n;
            d[h] = ok ? dg.of(key[s + h * HALF], p) : 256 + lane;
            peers[h] = same_digit(d[h], ok);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) before[h] = d[h] < 256 ? cnt[h * 256 + d[h]] : 0;
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (d[h] < 256 && lane == 31 - __clz(peers[h]))
                cnt[h * 256 + d[h]] = (uint16_t)(before[h] + __popc(peers[h]));
            rank[s + h * HALF] = (uint16_t)(before[h] + __popc(peers[h] & ((1u << lane) - 1)));
        }
        __syncwarp();
    }
    __syncthreads();
    // thread t: digit t's entries before each half, and in the tile
    uint32_t total = 0;
#pragma unroll
    for (int w = 0; w < 2 * CS_WARPS; ++w) {
        const uint32_t c = s_cnt[w * 256 + t];
        s_cnt[w * 256 + t] = (uint16_t)total;
        total += c;
    }
    unsigned long long* word = status + (int64_t)tile * 256 + t;
    const unsigned long long tag = (unsigned long long)(2 * p + 1) << 48;
    const unsigned long long mask48 = (1ull << 48) - 1;
    store_word(word, (tile == 0 ? tag + (1ull << 48) : tag) | total);
    const uint32_t first = scan256(total, s_warp);
    s_first[t] = first;
    __syncthreads();
#pragma unroll
    for (int s = 0; s < CS_ITEMS; ++s) {
        const int64_t i = base + 32 * s + lane;
        if (i < n) {
            const int d = dg.of(key[s], p);
            const int at = (int)s_first[d] + cnt[(s < HALF ? 0 : 256) + d] + rank[s];
            s_key[at] = key[s];
            if (VAL) s_val[at] = vals[i];
        }
    }
    // digit t's entries in the tiles before
    unsigned long long excl = 0;
    int back = tile - 1, polls = 0;
    while (back >= 0) {
        unsigned long long wd[CS_BACK];
#pragma unroll
        for (int u = 0; u < CS_BACK; ++u)
            wd[u] = back - u >= 0 ? load_word(status + (int64_t)(back - u) * 256 + t) : 0ull;
        bool done = false;
        int u = 0;
#pragma unroll
        for (int q = 0; q < CS_BACK; ++q) {
            if (done || u < q || back - q < 0 || wd[q] < tag) continue;
            excl += wd[q] & mask48;
            done = wd[q] >= tag + (1ull << 48);
            ++u;
        }
        if (done) break;
        back -= u;
        if (u > 0) polls = 0;
        else if (++polls > CS_POLLS || ((polls & 1023) == 0 && (load_word(
                     reinterpret_cast<unsigned long long*>(status) - 1) != 0ull))) {
            // give up: flag it (for the host, and for the other waits) and
            // write nothing
            atomicOr(err, COO_STUCK);
            store_word(status - 1, 1ull);
            s_dead = 1;
            break;
        }
    }
    store_word(word, (tag + (1ull << 48)) | (excl + total));
    s_to[t] = (int64_t)starts[p * 256 + t] + (int64_t)excl - (int64_t)first;
    __syncthreads();
    if (s_dead) return;
    const int64_t left = n - (int64_t)tile * CS_TILE;
    const int here = left < CS_TILE ? (int)left : CS_TILE;
#pragma unroll 4
    for (int x = t; x < here; x += CS_TPB) {
        const K k = s_key[x];
        const int64_t o = s_to[dg.of(k, p)] + x;
        if (o >= 0 && o < n) {
            keys_out[o] = k;
            if (VAL) vals_out[o] = s_val[x];
        }
    }
}

// Runs of equal keys per tile: entries that differ from the one before.
template <class K>
__global__ void __launch_bounds__(CS_TPB)
    k_run_count(int64_t n, const K* __restrict__ keys, int32_t* __restrict__ tile_runs) {
    __shared__ int s_sum;
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    int c = 0;
#pragma unroll 4
    for (int s = 0; s < RUN_ITEMS; ++s) {
        const int64_t i = (int64_t)blockIdx.x * RUN_TILE + s * CS_TPB + threadIdx.x;
        if (i < n) c += i == 0 || keys[i] != keys[i - 1];
    }
    c = __reduce_add_sync(CS_FULL, c);
    if (c_lane() == 0) atomicAdd(&s_sum, c);
    __syncthreads();
    if (threadIdx.x == 0) tile_runs[blockIdx.x] = s_sum;
}

// Rows between two entries that one lane writes the row pointer of; more are
// its warp's (1000 entries in 2^28 rows, call: 143 ms by the lanes, 17 so; 16.8 M
// entries in the first 64 of 2^20 rows: 4.9 and 1.25).
constexpr int ROWS_ALONE = 32;

// The row pointer of the warp's runs that start ROWS_ALONE rows and more after
// the last one (bit s of heads: entry base + 32 s + lane starts a run; out: the
// warp's first). Out of the kernel's way, as few warps have any.
template <class K>
__device__ __noinline__ void far_rows(int64_t base, const K* __restrict__ keys, unsigned heads,
                                      int64_t out, int cb, int32_t* __restrict__ rp) {
    const int lane = c_lane();
    for (int s = 0; s < RUN_ITEMS; ++s) {
        const int64_t i = base + 32 * s + lane;
        const bool head = heads >> s & 1u;
        const unsigned hm = __ballot_sync(CS_FULL, head);
        int32_t row = 0, first = 0;
        if (head) {
            row = (int32_t)(keys[i] >> cb);
            if (i > 0) first = (int32_t)(keys[i - 1] >> cb) + 1;
        }
        const int32_t o = (int32_t)(out + __popc(hm & ((1u << lane) - 1)));
        for (unsigned m = __ballot_sync(CS_FULL, head && row - first >= ROWS_ALONE); m; m &= m - 1) {
            const int j = __ffs(m) - 1;
            const int32_t l = __shfl_sync(CS_FULL, row, j), x = __shfl_sync(CS_FULL, o, j);
            for (int64_t r = (int64_t)__shfl_sync(CS_FULL, first, j) + lane; r <= l; r += 32)
                rp[r] = x;
        }
        out += __popc(hm);
    }
}

// One output entry per run: its column, and its values summed in COO order
// from the first one (no added zero: a lone -0.0 stays). A run that starts a
// new row writes the row pointer of every row since the last run's; the last
// entry those after its own.
template <class K>
__global__ void __launch_bounds__(CS_TPB)
    k_run_write(int64_t n, const K* __restrict__ keys, const float* __restrict__ v,
                const int64_t* __restrict__ tile_off, int cb, int32_t rows, int32_t out_n,
                int32_t* __restrict__ rp, int32_t* __restrict__ out_ci,
                float* __restrict__ out_v) {
    __shared__ int s_warp[CS_WARPS];
    const int lane = c_lane(), warp = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * RUN_TILE + warp * (32 * RUN_ITEMS);
    K key[RUN_ITEMS];
    unsigned heads = 0;
    int mine = 0;
#pragma unroll
    for (int s = 0; s < RUN_ITEMS; ++s) {
        const int64_t i = base + 32 * s + lane;
        key[s] = i < n ? keys[i] : (K)0;
    }
    // the key before the warp's first and the one after its last
    const K edge0 = base > 0 && base <= n ? keys[base - 1] : (K)0;
    const K edge1 = base + 32 * RUN_ITEMS < n ? keys[base + 32 * RUN_ITEMS] : (K)0;
#pragma unroll
    for (int s = 0; s < RUN_ITEMS; ++s) {
        const int64_t i = base + 32 * s + lane;
        K prev = __shfl_up_sync(CS_FULL, key[s], 1);
        const K carry = s > 0 ? __shfl_sync(CS_FULL, key[s > 0 ? s - 1 : 0], 31) : edge0;
        if (lane == 0) prev = carry;
        const bool head = i < n && (i == 0 || key[s] != prev);
        heads |= (unsigned)head << s;
        mine += __popc(__ballot_sync(CS_FULL, head));
    }
    if (lane == 0) s_warp[warp] = mine;
    __syncthreads();
    int64_t out = tile_off[blockIdx.x];
    for (int w = 0; w < warp; ++w) out += s_warp[w];
    const int64_t out0 = out;
    bool far = false;
#pragma unroll
    for (int s = 0; s < RUN_ITEMS; ++s) {
        const int64_t i = base + 32 * s + lane;
        const bool head = heads >> s & 1u;
        const unsigned hm = __ballot_sync(CS_FULL, head);
        K prev = __shfl_up_sync(CS_FULL, key[s], 1), next = __shfl_down_sync(CS_FULL, key[s], 1);
        const K carry0 = s > 0 ? __shfl_sync(CS_FULL, key[s > 0 ? s - 1 : 0], 31) : edge0;
        const K carry1 = s + 1 < RUN_ITEMS
                             ? __shfl_sync(CS_FULL, key[s + 1 < RUN_ITEMS ? s + 1 : 0], 0) : edge1;
        if (lane == 0) prev = carry0;
        if (lane == 31) next = carry1;
        if (head) {
            const int64_t o = out + __popc(hm & ((1u << lane) - 1));
            float acc = v ? v[i] : 1.0f;
            if (next == key[s])
                for (int64_t j = i + 1; j < n && keys[j] == key[s]; ++j) acc += v ? v[j] : 1.0f;
            const int32_t row = (int32_t)(key[s] >> cb);
            out_ci[o] = (int32_t)(key[s] & (((K)1 << cb) - 1));
            out_v[o] = acc;
            const int32_t first = i == 0 ? 0 : (int32_t)(prev >> cb) + 1;
            if (row - first < ROWS_ALONE)
                for (int32_t r = first; r <= row; ++r) rp[r] = (int32_t)o;
            else
                far = true;
        }
        out += __popc(hm);
    }
    if (__any_sync(CS_FULL, far)) far_rows(base, keys, heads, out0, cb, rp);
    if (blockIdx.x == gridDim.x - 1)  // the rows after the last entry's
        for (int64_t r = (int64_t)(keys[n - 1] >> cb) + 1 + threadIdx.x; r <= rows; r += CS_TPB)
            rp[r] = out_n;
}

int bits_for(int64_t x) {  // bits to hold 0 .. x - 1
    int b = 0;
    while (b < 63 && ((int64_t)1 << b) < x) ++b;
    return b;
}

struct Bufs {
    cudaStream_t st;
    void* p[24] = {};
    int n = 0;
    template <class T>
    cudaError_t get(T** out, size_t bytes) {
        void* q = nullptr;
        cudaError_t e = cudaMallocAsync(&q, bytes ? bytes : 16, st);
        if (e == cudaSuccess) p[n++] = q;
        *out = static_cast<T*>(q);
        return e;
    }
    void release() {
        for (int i = 0; i < n; ++i) cudaFreeAsync(p[i], st);
        n = 0;
    }
};

// The list sorted by key: keys and values (null: every value 1) on the device,
// m entries, each tile's first run, and their count in Misc::scan_total.
struct Sorted {
    int64_t m = 0;
    void* keys = nullptr;
    float* vals = nullptr;
    int64_t* tile_off = nullptr;
};

template <class K>
size_t pass_smem(bool val) {
    return CS_TILE * (sizeof(K) + (val ? 4 : 0)) + 2 * 2 * CS_WARPS * 256;
}

template <class K, class Src>
void launch_pass(cudaStream_t s, int64_t n, const Src& src, const float* vals, const Digits& dg,
                 int p, const uint32_t* starts, unsigned long long* status, int32_t* ticket,
                 K* keys_out, float* vals_out, int32_t* err) {
    const unsigned grid = (unsigned)((n + CS_TILE - 1) / CS_TILE);
    if (vals)
        k_coo_pass<K, Src, true><<<grid, CS_TPB, pass_smem<K>(true), s>>>(
            n, src, vals, dg, p, starts, status, ticket, keys_out, vals_out, err);
    else
        k_coo_pass<K, Src, false><<<grid, CS_TPB, pass_smem<K>(false), s>>>(
            n, src, vals, dg, p, starts, status, ticket, keys_out, vals_out, err);
    note_launch(nullptr, 1);
}

template <class K>
void set_pass_attrs() {
    // (per device; a few calls, and only the first on a device changes anything)
    const auto set = [](const void* f, bool val) {
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)pass_smem<K>(val));
    };
    set((const void*)k_coo_pass<K, CooKeys, true>, true);
    set((const void*)k_coo_pass<K, CooKeys, false>, false);
    set((const void*)k_coo_pass<K, ArrayKeys<K>, true>, true);
    set((const void*)k_coo_pass<K, ArrayKeys<K>, false>, false);
}

template <class K>
int sort_list(rvsp_cuda_plan* plan, Bufs& b, int32_t rows, int32_t cols, int64_t n, int cb, int rb,
              const int32_t* d_r, const int32_t* d_c, const float* d_v, int symmetric,
              Sorted* out) {
    cudaStream_t s = plan->stream;
    Misc* misc = plan->misc.as<Misc>();
    cudaError_t e;
    int st;
    const CooKeys list{d_r, d_c, rows, cols, cb, &misc->err};
    int64_t m = n;
    int64_t* mpos = nullptr;
    // expanded count of a symmetric list
    if (symmetric && n > 0) {
        int32_t* flag;
        if ((e = b.get(&mpos, 8 * ((size_t)n + 1))) || (e = b.get(&flag, 4 * (size_t)n)))
            return fail(e, "COO scratch");
        k_offdiag<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, d_r, d_c, flag);
        note_launch(nullptr, 1);
        if ((st = scan_counts(plan, flag, n, mpos, nullptr, &misc->scan_total2))) return st;
        if ((e = cudaMemcpyAsync(&m, &misc->scan_total2, 8, cudaMemcpyDeviceToHost, s)) ||
            (e = cudaStreamSynchronize(s)))
            return fail(e, "symmetric count");
        m += n;
    }
    out->m = m;
    if (m == 0) return RVSP_SUCCESS;
    const int bits = cb + rb;
    Digits dg{(bits + 7) / 8, 0};
    dg.db = dg.passes ? (bits + dg.passes - 1) / dg.passes : 0;  // even digits: fewer, longer runs
    const int64_t tiles = (m + CS_TILE - 1) / CS_TILE, rtiles = (m + RUN_TILE - 1) / RUN_TILE;
    K *k0, *k1;
    float *v0 = nullptr, *v1 = nullptr;
    unsigned long long* work;  // counts, tickets, starts, then the tiles' words after a stop word
    int32_t* runs;
    const size_t fixed = 8 * CS_PASSES * 256 + 4 * CS_PASSES * 256 + 8 * CS_PASSES + 8;
    const size_t work_bytes = fixed + (dg.passes ? 8 * 256 * (size_t)tiles : 0);
    if ((e = b.get(&k0, sizeof(K) * (size_t)m)) || (e = b.get(&k1, sizeof(K) * (size_t)m)) ||
        (d_v && ((e = b.get(&v0, 4 * (size_t)m)) || (e = b.get(&v1, 4 * (size_t)m)))) ||
        (e = b.get(&work, work_bytes)) || (e = b.get(&runs, 4 * (size_t)rtiles)) ||
        (e = b.get(&out->tile_off, 8 * ((size_t)rtiles + 1))))
        return fail(e, "COO scratch");
    unsigned long long* counts = work;
    uint32_t* starts = reinterpret_cast<uint32_t*>(work + CS_PASSES * 256);
    int32_t* tickets = reinterpret_cast<int32_t*>(starts + CS_PASSES * 256);
    unsigned long long* status = reinterpret_cast<unsigned long long*>(tickets + 2 * CS_PASSES) + 1;
    if ((e = cudaMemsetAsync(work, 0, work_bytes, s)) != cudaSuccess) return fail(e, "memset");
    const bool direct = !symmetric && dg.passes > 0;  // the first pass reads the list itself
    if (!direct) {
        k_coo_keys<K><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, list, d_v, symmetric, mpos, k0,
                                                                v0);
        note_launch(nullptr, 1);
    }
    if (dg.passes > 0) {
        set_pass_attrs<K>();
        const unsigned grid = (unsigned)std::min<int64_t>((m + CS_TPB - 1) / CS_TPB, 148 * 6);
        if (direct)
            k_coo_digits<<<grid, CS_TPB, 0, s>>>(m, list, dg, counts);
        else
            k_coo_digits<<<grid, CS_TPB, 0, s>>>(m, ArrayKeys<K>{k0}, dg, counts);
        k_coo_starts<<<dg.passes, 256, 0, s>>>(counts, starts);
        note_launch(nullptr, 2);
    }
    const float* vin = direct ? d_v : v0;
    for (int p = 0; p < dg.passes; ++p) {
        if (direct && p == 0)
            launch_pass<K>(s, m, list, vin, dg, p, starts, status, tickets + p, k1, v1, &misc->err);
        else
            launch_pass<K>(s, m, ArrayKeys<K>{k0}, vin, dg, p, starts, status, tickets + p, k1, v1,
                           &misc->err);
        std::swap(k0, k1);
        std::swap(v0, v1);
        vin = v0;
    }
    out->keys = k0;
    out->vals = v0;
    k_run_count<K><<<(unsigned)rtiles, CS_TPB, 0, s>>>(m, k0, runs);
    note_launch(nullptr, 1);
    return scan_counts(plan, runs, rtiles, out->tile_off, nullptr, &misc->scan_total);
}

thread_local rvsp_cuda_plan_t t_cplan = nullptr;
struct CooReaper {
    ~CooReaper() {
        if (t_cplan) rvsp_cuda_plan_destroy(t_cplan);
        t_cplan = nullptr;
    }
};
thread_local CooReaper t_creaper;

}  // namespace

extern "C" int rvsp_cuda_coo_to_csr(int32_t rows, int32_t cols, int64_t n, const int32_t* coo_row,
                                    const int32_t* coo_col, const float* coo_val, int symmetric,
                                    int device_out, int32_t** row_ptr_out, int32_t** col_idx_out,
                                    float** values_out, int32_t* nnz_out) {
    if (!row_ptr_out || !col_idx_out || !values_out || !nnz_out) return RVSP_ERROR_NULL_POINTER;
    if (n > 0 && (!coo_row || !coo_col)) return RVSP_ERROR_NULL_POINTER;
    if (rows <= 0 || cols <= 0 || n < 0) return RVSP_ERROR_INVALID_ARGUMENT;
    if (symmetric && rows != cols) return RVSP_ERROR_INVALID_ARGUMENT;
    *row_ptr_out = nullptr;
    *col_idx_out = nullptr;
    *values_out = nullptr;
    *nnz_out = 0;
    if (rvsp_cuda_device_count() == 0) return RVSP_ERROR_UNSUPPORTED_BACKEND;
    const int64_t total = symmetric ? 2 * n : n;  // upper bound of the expanded count
    if (total >= INT32_MAX) return RVSP_ERROR_ALLOCATION_FAILED;
    int st;
    if (!t_cplan) {
        if ((st = rvsp_cuda_plan_create(&t_cplan, RVSP_CUDA_ALGO_EXACT))) return st;
    }
    rvsp_cuda_plan_t plan = t_cplan;
    cudaStream_t s = plan->stream;
    keep_pool_memory();
    cudaError_t e;
    if ((e = plan->misc.ensure(sizeof(Misc))) != cudaSuccess) return fail(e, "misc");
    Misc* misc = plan->misc.as<Misc>();
    cudaMemsetAsync(misc, 0, sizeof(Misc), s);
    const bool dev = n > 0 && is_dev(coo_row);
    Bufs b{s};
    auto bail = [&](int code) {
        b.release();
        cudaStreamSynchronize(s);
        return code;
    };
    const int32_t *d_r = coo_row, *d_c = coo_col;
    const float* d_v = coo_val;
    if (n > 0 && !dev) {
        int32_t *tr, *tc;
        float* tv = nullptr;
        if ((e = b.get(&tr, 4 * (size_t)n)) || (e = b.get(&tc, 4 * (size_t)n)) ||
            (coo_val && (e = b.get(&tv, 4 * (size_t)n))))
            return bail(fail(e, "COO staging"));
        cudaMemcpyAsync(tr, coo_row, 4 * (size_t)n, cudaMemcpyHostToDevice, s);
        cudaMemcpyAsync(tc, coo_col, 4 * (size_t)n, cudaMemcpyHostToDevice, s);
        if (coo_val) cudaMemcpyAsync(tv, coo_val, 4 * (size_t)n, cudaMemcpyHostToDevice, s);
        d_r = tr, d_c = tc, d_v = tv;
    }
    const int cb = bits_for(cols), rb = bits_for(rows);
    Sorted so;
    st = cb + rb <= 32
             ? sort_list<uint32_t>(plan, b, rows, cols, n, cb, rb, d_r, d_c, d_v, symmetric, &so)
             : sort_list<uint64_t>(plan, b, rows, cols, n, cb, rb, d_r, d_c, d_v, symmetric, &so);
    if (st) return bail(st);
    const int64_t m = so.m;
    int64_t out_n = 0;
    int32_t bad = 0;
    int32_t *rp, *ci;
    float* v;
    if ((e = cudaMemcpyAsync(&out_n, &misc->scan_total, 8, cudaMemcpyDeviceToHost, s)) ||
        (e = cudaMemcpyAsync(&bad, &misc->err, 4, cudaMemcpyDeviceToHost, s)) ||
        (e = cudaStreamSynchronize(s)))
        return bail(fail(e, "COO sort"));
    if (m == 0) out_n = 0;
    if (bad & COO_STUCK) {
        g_err = "COO sort: a tile's wait ran out";
        return bail(RVSP_ERROR_DEVICE_FAILURE);
    }
    if (bad) {
        g_err = "COO row or column index out of range";
        return bail(RVSP_ERROR_INVALID_ARGUMENT);
    }
    const size_t on = (size_t)(out_n > 0 ? out_n : 1);
    rp = ci = nullptr;
    v = nullptr;
    if ((e = cudaMallocAsync((void**)&rp, 4 * ((size_t)rows + 1), s)) ||
        (e = cudaMallocAsync((void**)&ci, 4 * on, s)) || (e = cudaMallocAsync((void**)&v, 4 * on, s))) {
        if (rp) cudaFreeAsync(rp, s);
        if (ci) cudaFreeAsync(ci, s);
        return bail(fail(e, "CSR alloc"));
    }
    if (m == 0) {
        cudaMemsetAsync(rp, 0, 4 * ((size_t)rows + 1), s);
    } else {
        const unsigned grid = (unsigned)((m + RUN_TILE - 1) / RUN_TILE);
        if (cb + rb <= 32)
            k_run_write<uint32_t><<<grid, CS_TPB, 0, s>>>(m, (const uint32_t*)so.keys, so.vals,
                                                          so.tile_off, cb, rows, (int32_t)out_n,
                                                          rp, ci, v);
        else
            k_run_write<uint64_t><<<grid, CS_TPB, 0, s>>>(m, (const uint64_t*)so.keys, so.vals,
                                                          so.tile_off, cb, rows, (int32_t)out_n,
                                                          rp, ci, v);
        note_launch(nullptr, 1);
    }
    b.release();
    if ((e = cudaGetLastError()) != cudaSuccess) {
        cudaFreeAsync(rp, s);
        cudaFreeAsync(ci, s);
        cudaFreeAsync(v, s);
        cudaStreamSynchronize(s);
        return fail(e, "COO launch");
    }
    if (!device_out) {
        int32_t* hrp = (int32_t*)malloc(4 * ((size_t)rows + 1));
        int32_t* hci = (int32_t*)malloc(4 * on);
        float* hv = (float*)malloc(4 * on);
        if (!hrp || !hci || !hv) {
            free(hrp);
            free(hci);
            free(hv);
            cudaFreeAsync(rp, s);
            cudaFreeAsync(ci, s);
            cudaFreeAsync(v, s);
            cudaStreamSynchronize(s);
            return RVSP_ERROR_ALLOCATION_FAILED;
        }
        cudaMemcpyAsync(hrp, rp, 4 * ((size_t)rows + 1), cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(hci, ci, 4 * (size_t)out_n, cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(hv, v, 4 * (size_t)out_n, cudaMemcpyDeviceToHost, s);
        cudaFreeAsync(rp, s);
        cudaFreeAsync(ci, s);
        cudaFreeAsync(v, s);
        if ((e = cudaStreamSynchronize(s)) != cudaSuccess) {
            free(hrp);
            free(hci);
            free(hv);
            return fail(e, "CSR copy-out");
        }
        rp = hrp, ci = hci, v = hv;
    } else if ((e = cudaStreamSynchronize(s)) != cudaSuccess) {
        return fail(e, "COO to CSR");
    }
    *row_ptr_out = rp;
    *col_idx_out = ci;
    *values_out = v;
    *nnz_out = (int32_t)out_n;
    return RVSP_SUCCESS;
}
