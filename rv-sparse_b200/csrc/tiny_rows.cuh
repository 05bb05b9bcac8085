// Tiny rows (at most 32 products), count and fill: one thread per row.
//
// Each product becomes one word, column << 5 | index in A-row order, which a
// sorting network orders in the thread's registers: no data-dependent loops,
// and equal columns come out together in A-row order, so each run summed left
// to right from +0.0f is the reference's order of additions. A warp's rows are
// staged in C's order and leave as one contiguous range where they are
// neighbours in C, as do the products' positions (pm) that the reuse kernel
// replays.
//
// Bound by issue. Measured (5-point stencil of a 1023 x 1025 grid, 25 products
// a row, device time): COUNT 66 us and FILL with positions 249 us by insertion
// sort and a second walk that searches each product's position; 52 and 145 us
// so. B of more than 2^27 columns keeps that kernel (k_tiny).
#pragma once

#include "spgemm_kernels.cuh"

namespace rvsp {

constexpr int TS_WARPS = 4;
constexpr int TS_LD = 33;  // element x of lane l at x TS_LD + l
constexpr int64_t TS_MAX_COLS = int64_t(1) << 27;

// Batcher's odd-even merge sort of 32 words, ascending, of which the first N
// are not 0xffffffff: the comparators with the others fold away (N = 8, 16, 24,
// 28, 32: 19, 63, 132, 162, 191 remain).
template <int N>
__device__ __forceinline__ void tiny_network(uint32_t (&w)[32]) {
#pragma unroll
    for (int p = 1; p < N; p *= 2)
#pragma unroll
        for (int k = p; k >= 1; k /= 2)
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const int r = i - k % p;  // comparators (i, i + k)
                if (r >= 0 && r % (2 * k) < k && i + k < N && i / (2 * p) == (i + k) / (2 * p)) {
                    const uint32_t lo = min(w[i], w[i + k]), hi = max(w[i], w[i + k]);
                    w[i] = lo;
                    w[i + k] = hi;
                }
            }
}

// Where a warp's rows go.
struct TinyOut {
    const int32_t* c_rp;
    int32_t* c_ci;
    float* c_v;
    int32_t* cnt;
    const int64_t* slot_off;
    uint8_t* pm;  // positions: the warp's are [pm_begin, pm_end) of this word-aligned place
    int pm_begin, pm_end;
};

// The warp's rows (lane's row `row`, n products in words / vals; rows i of the
// list, `live` lanes a prefix), networks of N words.
template <int N, int MODE, bool PM>
__device__ __forceinline__ void tiny_rows(uint32_t* words, float* vals, uint8_t* spos, int row, int n,
                                          bool live, int pm_at, int pm_n, const TinyOut& out,
                                          int32_t* err) {
    const int lane = lane_id();
    uint32_t w[32];
#pragma unroll
    for (int j = 0; j < N; ++j) w[j] = j < n ? words[j * TS_LD + lane] : 0xffffffffu;
    tiny_network<N>(w);
    unsigned heads = 0;
#pragma unroll
    for (int j = 0; j < N; ++j)
        heads |= (unsigned)(j < n && (j == 0 || (w[j] ^ w[j > 0 ? j - 1 : 0]) >= 32u)) << j;
    int m = __popc(heads);
    if (MODE == COUNT) {
        if (live) out.cnt[row] = m;
        return;
    }
    // the warp's place in C: one contiguous range when its rows are neighbours
    const unsigned lives = __ballot_sync(FULL, live);
    const bool prefix = lives && (lives & (lives + 1)) == 0;
    const int last = 31 - __clz(lives);  // -1: none
    int64_t c0 = 0;
    int coff, ctotal;
    bool contig = false;
    if (out.slot_off) {
        if (live) {
            c0 = out.slot_off[row];
            out.cnt[row] = m;
        }
    } else {
        int c1 = 0;
        if (live) {
            c0 = out.c_rp[row];
            c1 = out.c_rp[row + 1];
            if (m != c1 - (int)c0) {  // an operand changed since the count
                atomicOr(err, ERR_STRUCTURE);
                m = min(m, max(c1 - (int)c0, 0));
            }
        }
        const int first = __shfl_sync(FULL, row, 0), end = __shfl_sync(FULL, row, last & 31);
        const int cbase = (int)__shfl_sync(FULL, (long long)c0, 0);
        const int cend = __shfl_sync(FULL, c1, last & 31);
        contig = prefix && end - first == last && cend - cbase <= 32 * TINY_CAP &&
                 __all_sync(FULL, !live || m == c1 - (int)c0);
        coff = (int)c0 - cbase;
        ctotal = cend - cbase;
    }
    if (!contig) {
        const int incl = warp_incl_scan(m);
        coff = incl - m;
        ctotal = __shfl_sync(FULL, incl, 31);
    }
    // columns and positions, then values: each staged over what it was made from
    int32_t* scol = reinterpret_cast<int32_t*>(words);
    const unsigned ends = heads >> 1 | (n > 0 ? 1u << (n - 1) : 0u);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const int d = __popc(heads & ((2u << j) - 1)) - 1;
        if ((heads >> j & 1u) && d < m) scol[coff + d] = (int32_t)(w[j] >> 5);
        if (PM && j < n && (int)(w[j] & 31u) < pm_n) spos[pm_at + (w[j] & 31u)] = (uint8_t)d;
    }
    float o[N];
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const float v = j < n ? vals[(w[j] & 31u) * TS_LD + lane] : 0.0f;
        acc = __fadd_rn(heads >> j & 1u ? 0.0f : acc, v);
        o[j] = acc;
    }
    __syncwarp();
    float* sval = vals + coff;
    const float* send = sval + m;
#pragma unroll
    for (int j = 0; j < N; ++j)
        if ((ends >> j & 1u) && sval < send) *sval++ = o[j];
    sval = vals;
    __syncwarp();
    if (contig) {
        const int64_t cb = __shfl_sync(FULL, (long long)c0, 0);
        for (int e = lane; e < ctotal; e += 32) {
            out.c_ci[cb + e] = scol[e];
            out.c_v[cb + e] = sval[e];
        }
    } else {
        for (int j = 0; j <= last; ++j) {
            const int64_t cj = __shfl_sync(FULL, (long long)c0, j);
            const int nj = __shfl_sync(FULL, m, j), oj = __shfl_sync(FULL, coff, j);
            if (lane < nj) {
                out.c_ci[cj + lane] = scol[oj + lane];
                out.c_v[cj + lane] = sval[oj + lane];
            }
        }
    }
    if (PM) {  // whole words, and the bytes of the first and last one that are this warp's
        const uint32_t* sw = reinterpret_cast<const uint32_t*>(spos);
        for (int e = lane; 4 * e < out.pm_end; e += 32) {
            if (4 * e >= out.pm_begin && 4 * e + 4 <= out.pm_end)
                reinterpret_cast<uint32_t*>(out.pm)[e] = sw[e];
            else
                for (int t = max(4 * e, out.pm_begin); t < min(4 * e + 4, out.pm_end); ++t)
                    out.pm[t] = spos[t];
        }
    }
}

// PM: record the positions (one byte a product, rows starting at list_off[i] -
// list_off[0]).
template <int MODE, bool PM>
__global__ void __launch_bounds__(TS_WARPS * 32, MODE == FILL ? 5 : 12)
    k_tiny_sort(CsrView A, CsrView B, const int32_t* __restrict__ rows, int nrows,
                int32_t* __restrict__ cnt, const int32_t* __restrict__ c_rp,
                int32_t* __restrict__ c_ci, float* __restrict__ c_v,
                const int32_t* __restrict__ list_off, uint8_t* __restrict__ pm,
                int32_t* __restrict__ err, RowCtl ctl) {
    static_assert(MODE == COUNT || MODE == FILL, "");
    __shared__ uint32_t s_words[TS_WARPS][TINY_CAP * TS_LD];
    __shared__ float s_vals[MODE == FILL ? TS_WARPS : 1][MODE == FILL ? TINY_CAP * TS_LD : 1];
    __shared__ uint32_t s_pos[PM ? TS_WARPS : 1][PM ? 8 * TINY_CAP + 1 : 1];
    const int wp = threadIdx.x >> 5, lane = lane_id();
    const int i0 = (blockIdx.x * TS_WARPS + wp) * 32, i = i0 + lane;
    if (i0 >= nrows) return;  // whole warp idle
    uint32_t* words = s_words[wp];
    uint8_t* spos = reinterpret_cast<uint8_t*>(s_pos[PM ? wp : 0]);
    float* vals = s_vals[MODE == FILL ? wp : 0];
    const int row = i < nrows ? rows[i] : 0;
    bool live = i < nrows;
    if (ctl.only && live && !ctl.only[row]) live = false;
    int n = 0;
    if (live) {
        int a0, a1;
        row_range(A, row, &a0, &a1, err);
        tiny_walk<MODE == FILL>(A, B, a0, a1, err, [&](int col, float pv) {
            if (n < TINY_CAP) {
                words[n * TS_LD + lane] = (uint32_t)col << 5 | (uint32_t)n;
                if (MODE == FILL) vals[n * TS_LD + lane] = pv;
                ++n;
            }
        });
    }
    TinyOut out{c_rp, c_ci, c_v, cnt, ctl.slot_off, nullptr, 0, 0};
    int pm_at = 0, pm_n = 0;
    if (PM) {
        const int b0 = list_off[i0], b1 = list_off[min(i0 + 32, nrows)];
        const int at = b0 - list_off[0];
        out.pm = pm + (at & ~3);
        out.pm_begin = at & 3;
        out.pm_end = out.pm_begin + min(b1 - b0, 32 * TINY_CAP);
        if (i < nrows) {
            pm_at = out.pm_begin + list_off[i] - b0;
            pm_n = min(list_off[i + 1] - list_off[i], out.pm_end - pm_at);
        }
    }
    const int most = __reduce_max_sync(FULL, n);
#define TINY_ROWS(N) \
    tiny_rows<N, MODE, PM>(words, vals, spos, row, n, live, pm_at, pm_n, out, err)
    if (most <= 8)
        TINY_ROWS(8);
    else if (most <= 16)
        TINY_ROWS(16);
    else if (most <= 24)
        TINY_ROWS(24);
    else if (most <= 28)
        TINY_ROWS(28);
    else
        TINY_ROWS(32);
#undef TINY_ROWS
}

}  // namespace rvsp
