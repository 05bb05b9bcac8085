// Heavy rows by segment lists. A work item is a (row, column chunk) pair and a
// segment the part of one B row that falls in one chunk. Instead of visiting
// every A entry of the row for every chunk and looking up whether its B row
// reaches it (on R-MAT 2^20 four visits in five find nothing), the analysis
// lists each item's segments once, in A-row order, and count, fill and reuse
// walk the lists.
//
//   k_row_starts, k_chunk_runs, k_row_runs
//                 the chunk runs of every B row: {chunk, first position}, one
//                 array in B's order, and each row's part of it
//   k_heavy_rows  per heavy row: its chunks, units (runs of UNIT A entries)
//                 and cells (chunk, unit)
//   k_alist_count, k_alist_fill
//                 a warp per unit: each cell's number of segments, then the
//                 segments behind the cells' scanned offsets (cells of a chunk
//                 are consecutive, so a chunk's list keeps A-row order over all
//                 its units)
//   k_heavy_items the items and where each one's list starts
//   k_heavy_work  the order and grouping in which FILL and REUSE take them
//   k_heavy_list  the products: a warp per item or group of items
//
// Measured (B200; device time, the lookup kernel k_heavy first): R-MAT 2^17,
// COUNT 5.4 -> 2.8 ms, FILL 11.3 -> 5.8 ms; one 2^31-product row panel of R-MAT
// 2^20, learned FILL 42.9 -> 17.5 ms; reuse of R-MAT 2^16, 4.5 -> 2.2 ms; the
// lists themselves and the items take 0.8 ms of the first and 4.0 ms of the
// second (the lookups' tables took 0.3 and 1.5). FILL is bound by the latency
// of short work on 28 resident warps an SM and by the size of its code: every
// path that is added costs all others (a third step in flight 12 %, a second
// way to combine equal columns 3 %). COUNT is bound by issue. Where the lists
// would take longer than the lookups, k_heavy runs instead (lists_pay).
#pragma once

#include "spgemm_kernels.cuh"

namespace rvsp {

constexpr int LIST_MAX_CHUNKS = 2048;  // chunks of B: a unit's counters stay in shared memory
constexpr int ALIST_WARPS = 4;
// Warps of a CTA of k_heavy_list: FILL and REUSE 28 (72 registers a thread, one
// CTA an SM), COUNT 24 (40 registers, two; R-MAT 2^17 and tall-skinny 2M x
// 100k, calls: 10.46 and 6.65 ms at 32 registers with spills, 10.15 and 6.66
// so, 10.27 and 6.72 at 56).
constexpr int list_max_warps(int mode) { return mode == COUNT ? 24 : 28; }
constexpr int COUNT_GROUP_SEGS = 256;  // segments of the chunks one warp counts together
constexpr int LIST_LONG = 64;          // segments this long are walked on their own

// A segment: its first position in B and (A entry - row start) << cw_log2 |
// (entries - 1), one word each, so rows of up to 2^(32 - cw_log2) entries.
struct HeavyLists {
    const int64_t* item_seg;   // [items + 1] first segment of each item
    const int2* seg;
    const int32_t* item_prod;  // products of each item
    const int2* work;          // FILL and REUSE: {first item, items} a warp takes together
    const int64_t* nwork;
};

// FILL and REUSE: a row's items go in groups of up to SPARSE_COLS columns; a
// group of at most GROUP_PRODUCTS products is one warp's.
constexpr int SPARSE_COLS = 16384;
constexpr int GROUP_PRODUCTS = 2048;
__host__ __device__ constexpr int group_items(int cw_log2) {
    return SPARSE_COLS >> cw_log2 > 32 ? 32 : SPARSE_COLS >> cw_log2 < 1 ? 1 : SPARSE_COLS >> cw_log2;
}

// One bit per B entry, set where a row starts.
__global__ void k_row_starts(CsrView B, uint32_t* __restrict__ bits, int32_t* __restrict__ err) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= B.rows) return;
    int bs, be;
    row_range(B, k, &bs, &be, err);
    if (be > bs) atomicOr(&bits[bs >> 5], 1u << (bs & 31));
}

// Chunk runs of B, by entry (long and short rows alike): an entry starts a run
// when it starts a row or its chunk differs from the entry before. COUNT
// leaves each tile's number of runs, FILL writes {chunk, position} and, per 32
// entries, the runs before them and the starts among them (words, for
// k_row_runs). Entries outside every row (before the first row's start, past
// the last one's end) are never a run. COUNT also sets *irregular where a row
// is not strictly ascending or leaves B's columns: the lists hold each chunk
// of a row once, as one range of distinct columns, so such a B takes the
// lookups instead.
constexpr int RUNS_TPB = 256;
constexpr int RUNS_STEPS = 8;
constexpr int RUNS_TILE = RUNS_TPB * RUNS_STEPS;

template <int MODE>
__global__ void __launch_bounds__(RUNS_TPB)
    k_chunk_runs(CsrView B, int cw_log2, const uint32_t* __restrict__ row_bits,
                 int32_t* __restrict__ tile_cnt, const int64_t* __restrict__ tile_off,
                 int2* __restrict__ runs, int2* __restrict__ words,
                 int32_t* __restrict__ irregular) {
    __shared__ int s_warp[RUNS_TPB / 32];
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * RUNS_TILE + warp * (32 * RUNS_STEPS);
    const int first = max(B.rp[0], 0), end = min(B.rp[B.rows], B.nnz);
    int c[RUNS_STEPS];  // columns
    unsigned m[RUNS_STEPS];
    int n = 0;
    bool bad = false;
#pragma unroll
    for (int s = 0; s < RUNS_STEPS; ++s) {
        const int64_t q = base + 32 * s + lane;
        c[s] = q >= first && q < end ? B.ci[q] : 0;
        if ((unsigned)c[s] >= (unsigned)B.cols) {
            bad = true;
            c[s] = 0;
        }
    }
    const int edge = base > first && base <= end ? B.ci[base - 1] : 0;
#pragma unroll
    for (int s = 0; s < RUNS_STEPS; ++s) {
        const int64_t q = base + 32 * s + lane;
        int prev = __shfl_up_sync(FULL, c[s], 1);
        const int carry = s > 0 ? __shfl_sync(FULL, c[s > 0 ? s - 1 : 0], 31) : edge;
        if (lane == 0) prev = carry;
        const bool in = q >= first && q < end;
        const bool row = in && (row_bits[q >> 5] >> lane & 1u);
        const bool start = row || (in && (c[s] ^ prev) >> cw_log2 != 0);
        bad |= in && !row && c[s] <= prev;
        m[s] = __ballot_sync(FULL, start);
        n += __popc(m[s]);
    }
    if (MODE == COUNT && bad) atomicOr(irregular, 1);
    if (lane == 0) s_warp[warp] = n;
    __syncthreads();
    if (MODE == COUNT) {
        if (threadIdx.x == 0) {
            int t = 0;
            for (int w = 0; w < RUNS_TPB / 32; ++w) t += s_warp[w];
            tile_cnt[blockIdx.x] = t;
        }
        return;
    }
    int out = (int)tile_off[blockIdx.x];
    for (int w = 0; w < warp; ++w) out += s_warp[w];
#pragma unroll
    for (int s = 0; s < RUNS_STEPS; ++s) {
        const int64_t q = base + 32 * s + lane;
        if (lane == 0 && q <= B.nnz) words[q >> 5] = make_int2(out, (int)m[s]);
        if (m[s] >> lane & 1u) {
            const int at = out + __popc(m[s] & ((1u << lane) - 1));
            if (at < B.nnz) runs[at] = make_int2(c[s] >> cw_log2, (int)q);
        }
        out += __popc(m[s]);
    }
}

// Each B row's runs [x, y) and end position z (w unused); a row whose
// structure is out of range reads as empty.
__global__ void k_row_runs(CsrView B, const int2* __restrict__ words, int4* __restrict__ out,
                           int32_t* __restrict__ err) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= B.rows) return;
    int bs, be;
    row_range(B, k, &bs, &be, err);
    int x = 0, y = 0;
    if (be > bs) {
        const int2 a = words[bs >> 5], b = words[be >> 5];
        x = a.x + __popc((unsigned)a.y & ((1u << (bs & 31)) - 1));
        y = b.x + __popc((unsigned)b.y & ((1u << (be & 31)) - 1));
    }
    out[k] = make_int4(x, y, be, 0);
}

__global__ void k_heavy_rows(CsrView A, const int32_t* __restrict__ rows, int nh,
                             const int32_t* __restrict__ nchunks, int32_t* __restrict__ chunks,
                             int32_t* __restrict__ units, int32_t* __restrict__ cells,
                             int32_t* __restrict__ longest, int32_t* __restrict__ err) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= nh) return;
    int a0, a1;
    row_range(A, rows[h], &a0, &a1, err);
    const int n = nchunks[rows[h]], u = (a1 - a0 + HEAVY_UNIT - 1) / HEAVY_UNIT;
    chunks[h] = n;
    units[h] = u;
    cells[h] = n * u;
    atomicMax(longest, a1 - a0);
}

// Largest h in [0, n) with first[h] <= x (first ascending, first[0] <= x).
__device__ __forceinline__ int unit_row(const int32_t* __restrict__ first, int n, int x) {
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (first[mid] <= x) lo = mid; else hi = mid;
    }
    return lo;
}

// A warp's unit: its row, entries [a0, a1), cells cell + c nsub for chunk c of
// [clo, clo + nch). False when there is none (or an operand changed while it
// is analysed, which must not lead outside the cells).
struct ListUnit {
    int r0, a0, a1, clo, nch, nsub;
    int64_t cell;
};

__device__ __forceinline__ bool list_unit(const CsrView& A, const int32_t* rows, int nh, int nunits,
                                          const int32_t* unit0, const int32_t* units,
                                          const int64_t* cell0, int64_t ncells,
                                          const int32_t* chunk_lo, const int32_t* nchunks,
                                          int most, int32_t* err, ListUnit* out) {
    const int u = blockIdx.x * ALIST_WARPS + (threadIdx.x >> 5);
    if (u >= nunits) return false;
    const int h = unit_row(unit0, nh, u);
    const int row = rows[h], sub = u - unit0[h];
    row_range(A, row, &out->r0, &out->a1, err);
    out->nsub = units[h];
    out->clo = chunk_lo[row];
    out->nch = min(nchunks[row], most);
    out->cell = cell0[h] + sub;
    if (sub >= out->nsub || cell0[h] + (int64_t)out->nch * out->nsub > ncells) return false;
    out->a0 = min(out->r0 + sub * HEAVY_UNIT, out->a1);
    out->a1 = min(out->a1, out->a0 + HEAVY_UNIT);
    return true;
}

// Segments and products per cell, a unit a warp: counters of the row's chunks
// in shared memory (segments << 24 | products: a unit's share of a chunk is at
// most HEAVY_UNIT segments of 8192 columns), the lanes taking the runs of one
// B row at a time (distinct chunks, so no two lanes meet), the next entry's
// runs loading meanwhile.
static_assert(HEAVY_UNIT < 256 && (HEAVY_UNIT << HEAVY_CW_LOG2_MAX) < (1 << 24), "");

__global__ void __launch_bounds__(ALIST_WARPS * 32)
    k_alist_count(CsrView A, CsrView B, const int32_t* __restrict__ rows, int nh, int nunits,
                  const int32_t* __restrict__ unit0, const int32_t* __restrict__ units,
                  const int64_t* __restrict__ cell0, int64_t ncells,
                  const int32_t* __restrict__ chunk_lo, const int32_t* __restrict__ nchunks,
                  const int4* __restrict__ brow, const int2* __restrict__ runs, int cw_log2,
                  int32_t* __restrict__ cell_cnt, int32_t* __restrict__ cell_prod,
                  int32_t* __restrict__ err, int32_t* __restrict__ irregular, int stride) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = lane_id();
    ListUnit L;
    if (!list_unit(A, rows, nh, nunits, unit0, units, cell0, ncells, chunk_lo, nchunks, stride, err,
                   &L))
        return;
    uint32_t* cur = reinterpret_cast<uint32_t*>(smem) + warp * stride;
    for (int c = lane; c < L.nch; c += 32) cur[c] = 0u;
    __syncwarp();
    for (int base = L.a0; base < L.a1; base += 32) {
        const int j = base + lane;
        int4 br = make_int4(0, 0, 0, 0);
        if (j < L.a1) {
            const int k = A.ci[j];
            if ((unsigned)k < (unsigned)B.rows) br = brow[k];
            else atomicOr(err, ERR_STRUCTURE);
        }
        const int ne = min(32, L.a1 - base);
        int2 next = make_int2(0, 0);
        int after = 0;
        {  // the first entry's runs
            const int x = __shfl_sync(FULL, br.x, 0) + lane, xe = __shfl_sync(FULL, br.y, 0);
            if (x < xe) {
                next = runs[x];
                if (x + 1 < xe) after = runs[x + 1].y;
            }
        }
        for (int e = 0; e < ne; ++e) {
            const int x0 = __shfl_sync(FULL, br.x, e), xe = __shfl_sync(FULL, br.y, e);
            const int end = __shfl_sync(FULL, br.z, e);
            int2 s = next;
            int t = after;
            if (e + 1 < ne) {
                const int x = __shfl_sync(FULL, br.x, (e + 1) & 31) + lane;
                const int ye = __shfl_sync(FULL, br.y, (e + 1) & 31);
                if (x < ye) {
                    next = runs[x];
                    if (x + 1 < ye) after = runs[x + 1].y;
                }
            }
            for (int b = x0; b < xe; b += 32) {
                const int x = b + lane;
                if (x < xe) {
                    if (b > x0) {
                        s = runs[x];
                        if (x + 1 < xe) t = runs[x + 1].y;
                    }
                    if (x + 1 >= xe) t = end;
                    const int c = s.x - L.clo;
                    if ((unsigned)c < (unsigned)L.nch)
                        cur[c] += (1u << 24) + (uint32_t)min(max(t - s.y, 1), 1 << cw_log2);
                    else
                        atomicOr(irregular, 1);  // B row not sorted
                }
                __syncwarp();
            }
        }
    }
    for (int c = lane; c < L.nch; c += 32) {
        cell_cnt[L.cell + (int64_t)c * L.nsub] = (int32_t)(cur[c] >> 24);
        cell_prod[L.cell + (int64_t)c * L.nsub] = (int32_t)(cur[c] & 0xffffffu);
    }
}

// The lists, a unit a warp: lane l holds entries l and l + 32 and walks each
// one's runs in step with the chunks, so a chunk's segments leave together,
// in entry order, as one coalesced store. (Dealing one B row at a time to the
// chunks' lists stores every 8-byte segment alone: 5.5..14 ms against 1.9 for
// the 2.5e8 segments of an R-MAT 2^20 row panel, by how many half-written
// sectors the lists in flight kept in L2.)
__global__ void __launch_bounds__(ALIST_WARPS * 32)
    k_alist_fill(CsrView A, CsrView B, const int32_t* __restrict__ rows, int nh, int nunits,
                 const int32_t* __restrict__ unit0, const int32_t* __restrict__ units,
                 const int64_t* __restrict__ cell0, int64_t ncells,
                 const int32_t* __restrict__ chunk_lo, const int32_t* __restrict__ nchunks,
                 const int4* __restrict__ brow, const int2* __restrict__ runs,
                 const int64_t* __restrict__ cell_off, int2* __restrict__ seg, int64_t nsegs,
                 int cw_log2, int32_t* __restrict__ err, int stride) {
    const int lane = lane_id();
    ListUnit L;
    if (!list_unit(A, rows, nh, nunits, unit0, units, cell0, ncells, chunk_lo, nchunks, stride, err,
                   &L))
        return;
    constexpr int NB = HEAVY_UNIT / 32;
    // per entry: the run at hand {chunk, start}, the one after it (a chunk
    // past every chunk and the row's end when there is none), its index
    int2 cur[NB], nxt[NB];
    int at[NB], stop[NB], rend[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = L.a0 + 32 * b + lane;
        int4 br = make_int4(0, 0, 0, 0);
        if (j < L.a1) {
            const int k = A.ci[j];
            if ((unsigned)k < (unsigned)B.rows) br = brow[k];
        }
        at[b] = br.x;
        stop[b] = br.y;
        rend[b] = br.z;
        cur[b] = at[b] < stop[b] ? runs[at[b]] : make_int2(INT_MAX, br.z);
        nxt[b] = at[b] + 1 < stop[b] ? runs[at[b] + 1] : make_int2(INT_MAX, br.z);
        if (at[b] < stop[b] && nxt[b].x <= cur[b].x) atomicOr(err, ERR_STRUCTURE);
    }
    int64_t o = cell_off[L.cell];
    for (int c = 0; c < L.nch; ++c) {
        if (L.nsub > 1) o = cell_off[L.cell + (int64_t)c * L.nsub];
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            const bool hit = cur[b].x == L.clo + c;
            const unsigned m = __ballot_sync(FULL, hit);
            if (hit) {
                const int64_t to = o + __popc(m & ((1u << lane) - 1));
                const int n = min(max(nxt[b].y - cur[b].y, 1), 1 << cw_log2);
                if (to < nsegs)
                    seg[to] = make_int2(cur[b].y,
                                        (int)((uint32_t)(L.a0 + 32 * b + lane - L.r0) << cw_log2 |
                                              (uint32_t)(n - 1)));
                ++at[b];
                cur[b] = nxt[b];
                if (at[b] + 1 < stop[b]) {
                    nxt[b] = runs[at[b] + 1];
                    // a list that would skip a run: an operand changed meanwhile
                    if (nxt[b].x <= cur[b].x) atomicOr(err, ERR_STRUCTURE);
                } else {
                    nxt[b] = make_int2(INT_MAX, rend[b]);
                }
            }
            o += __popc(m);
        }
    }
}

// The heavy rows' items, in list order, a warp per row; where each one's list
// starts, its products, and the row's number of work list entries (item_seg
// null: no lists).
__global__ void __launch_bounds__(256)
    k_heavy_items(const int32_t* __restrict__ a_rp, const int32_t* __restrict__ rows, int nh,
                  const int32_t* __restrict__ item0, const int32_t* __restrict__ chunk_lo,
                  const int32_t* __restrict__ nchunks, const int64_t* __restrict__ cell0,
                  const int32_t* __restrict__ units, const int64_t* __restrict__ cell_off,
                  const int32_t* __restrict__ cell_prod, int64_t ncells, int nitems, int cw_log2,
                  HeavyItem* __restrict__ items, int64_t* __restrict__ item_seg,
                  int32_t* __restrict__ item_prod, int32_t* __restrict__ entries) {
    const int64_t h = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = lane_id();
    if (h >= nh) return;
    const int row = rows[h], n = nchunks[row], lo = chunk_lo[row], first = item0[h];
    const int a0 = a_rp[row];
    const int most = group_items(cw_log2);
    int count = 0;
    for (int c0 = 0; c0 < n; c0 += 32) {
        const int c = c0 + lane;
        int64_t p = 0;
        if (c < n) {
            items[first + c] = HeavyItem{row, lo + c, first, a0};
            if (item_seg) {
                const int64_t x0 = min(cell0[h] + (int64_t)c * units[h], ncells);
                const int64_t x1 = min(x0 + units[h], ncells);
                for (int64_t x = x0; x < x1; ++x) p += cell_prod[x];
                item_seg[first + c] = cell_off[x0];
                item_prod[first + c] = (int32_t)min(p, (int64_t)INT_MAX);
            }
        }
        for (int o = most >> 1; o > 0; o >>= 1) p += __shfl_xor_sync(FULL, p, o);
        count += __popc(__ballot_sync(FULL, c < n && (p > GROUP_PRODUCTS || lane % most == 0)));
    }
    if (lane == 0) entries[h] = count;
    if (item_seg && h == nh - 1 && lane == 0) item_seg[nitems] = cell_off[ncells];
}

// The work list, in row order (big rows of a power-law matrix come early, and
// must not start last).
__global__ void __launch_bounds__(256)
    k_heavy_work(const int32_t* __restrict__ rows, int nh, const int32_t* __restrict__ item0,
                 const int32_t* __restrict__ nchunks, const int32_t* __restrict__ item_prod,
                 const int32_t* __restrict__ entry0, int nitems, int cw_log2,
                 int2* __restrict__ work) {
    const int64_t h = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = lane_id();
    if (h >= nh) return;
    const int n = nchunks[rows[h]], first = item0[h];
    const int most = group_items(cw_log2);
    int at = entry0[h];
    for (int c0 = 0; c0 < n; c0 += 32) {
        const int c = c0 + lane;
        int64_t p = c < n ? item_prod[first + c] : 0;
        for (int o = most >> 1; o > 0; o >>= 1) p += __shfl_xor_sync(FULL, p, o);
        const bool alone = p > GROUP_PRODUCTS;
        const bool entry = c < n && (alone || lane % most == 0);
        const unsigned m = __ballot_sync(FULL, entry);
        const int to = at + __popc(m & ((1u << lane) - 1));
        if (entry && to < nitems)
            work[to] = make_int2(first + c, alone ? 1 : min(most, n - c));
        at += __popc(m);
    }
}

// Marked sums: negated, so that zero bits mean no product yet (FILL needs no
// bitmap of the columns that occur). A sum that starts from +0.0f is never
// -0.0f (rounding to nearest gives -0.0f only for -0.0f + -0.0f), so its
// negation never is +0.0f, and the negation of zero bits plus +0.0f is the
// +0.0f that a sum starts from.
__device__ __forceinline__ float marked_sum(float t) { return __fadd_rn(-t, 0.0f); }
__device__ __forceinline__ float marked(float v) {
    return __uint_as_float(__float_as_uint(v) ^ 0x80000000u);
}

// *sum += pr.
template <bool MARKED>
__device__ __forceinline__ void add_one(float* sum, float pr) {
    *sum = MARKED ? marked(__fadd_rn(marked_sum(*sum), pr)) : __fadd_rn(*sum, pr);
}

// Adds one step's products (lane's pr into acc[at], where in) in lane order;
// starts: the lanes after the first at which a segment starts. A segment's
// columns are distinct, so the segments add one after the other. (Finding and
// combining equal columns, ordered_add, takes longer however many segments
// there are, not least by its size: code here is executed from an instruction
// cache that it fills. R-MAT 2^17 whole, fill: 6.72 ms with ordered_add for two
// segments and more, 6.10 for more than 8, 5.87 without.)
template <bool MARKED>
__device__ __forceinline__ void add_step(float* acc, int at, bool in, float pr, unsigned starts) {
    const int turn = in ? __popc(starts & (0xffffffffu >> (31 - lane_id()))) : -1;
    const int last = __popc(starts);
#pragma unroll 1
    for (int r = 0; r <= last; ++r) {
        if (turn == r) add_one<MARKED>(acc + at, pr);
        __syncwarp();
    }
}

// One step of up to 32 products per half h: lane's column c[h] (relative to
// the chunk), B value b[h] and A value a[h], in[h] where it has one; starts:
// as in add_step.
template <int MODE>
__device__ __forceinline__ void list_add(int c, float a, float b, bool in, unsigned starts, int cw,
                                         float* acc, unsigned* bits, int32_t* err) {
    const bool ok = in && (unsigned)c < (unsigned)cw;
    if (in && !ok) atomicOr(err, ERR_STRUCTURE);  // B row not sorted
    if constexpr (MODE == COUNT) {
        if (ok) atomicOr(&bits[c >> 5], 1u << (c & 31));
    } else {
        const float pr = __fmul_rn(a, b);
        add_step<MODE == FILL>(acc, ok ? c : 0, ok, pr, starts);
    }
}

// The products of up to 32 listed segments (lane l: len entries from B
// position sg.x, A value av), in list order (A-row order). Runs of segments
// shorter than LIST_LONG are walked 32 products at a time over consecutive
// segments: each lane finds its segment from the bits of the segments that
// start within its 32 products; two steps are located and loaded before
// either is accumulated (add_step). Longer segments are walked on their own,
// which needs no finding.
template <int MODE>
__device__ __forceinline__ void list_products(const CsrView& B, int2 sg, int len, float av, int lo,
                                              int cw, float* acc, unsigned* bits, int32_t* err) {
    const int lane = lane_id();
    const unsigned upto = 0xffffffffu >> (31 - lane);
    const int incl = warp_incl_scan(len);
    const int start = incl - len;
    const int off = sg.x - start;
    const unsigned longm = __ballot_sync(FULL, len >= LIST_LONG);
    const int nseg = 32 - __clz(__ballot_sync(FULL, len > 0));  // (a prefix of the lanes)
    for (int e0 = 0; e0 < nseg;) {
        const unsigned rest = longm >> e0 << e0;
        const int e1 = rest ? __ffs(rest) - 1 : nseg;
        if (e1 > e0) {
            const int p0 = __shfl_sync(FULL, start, e0), p1 = __shfl_sync(FULL, incl, e1 - 1);
            const bool mine = lane >= e0 && lane < e1;
            for (int f0 = p0; f0 < p1; f0 += 64) {
                int c[2], q[2];
                float a[2], b[2];
                unsigned starts[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int rel = start - (f0 + 32 * h);
                    const unsigned m =
                        __reduce_or_sync(FULL, mine && (unsigned)rel < 32u ? 1u << rel : 0u);
                    const int e = max(e0 + __popc(__ballot_sync(FULL, mine && rel < 0)) +
                                          __popc(m & upto) - 1, 0);
                    starts[h] = m & ~1u;
                    q[h] = __shfl_sync(FULL, off, e) + f0 + 32 * h + lane;
                    a[h] = MODE != COUNT ? __shfl_sync(FULL, av, e) : 0.0f;
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    c[h] = 0;
                    b[h] = 0.0f;
                    if (f0 + 32 * h + lane < p1) {
                        c[h] = __ldg(B.ci + q[h]) - lo;
                        if (MODE != COUNT) b[h] = __ldg(B.v + q[h]);
                    }
                }
                list_add<MODE>(c[0], a[0], b[0], f0 + lane < p1, starts[0], cw, acc, bits, err);
                if (f0 + 32 < p1)
                    list_add<MODE>(c[1], a[1], b[1], f0 + 32 + lane < p1, starts[1], cw, acc, bits,
                                   err);
            }
            e0 = e1;
        }
        if (e0 < nseg) {  // a long segment
            const int s = __shfl_sync(FULL, sg.x, e0), n = __shfl_sync(FULL, len, e0);
            const float ae = __shfl_sync(FULL, av, e0);
            for (int f0 = lane; f0 - lane < n; f0 += 128) {
                int c[4];
                float b[4];
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    c[h] = -1;
                    b[h] = 0.0f;
                    if (f0 + 32 * h < n) {
                        c[h] = __ldg(B.ci + s + f0 + 32 * h) - lo;
                        if (MODE != COUNT) b[h] = __ldg(B.v + s + f0 + 32 * h);
                    }
                }
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    if (f0 + 32 * h < n) {
                        if ((unsigned)c[h] >= (unsigned)cw) {
                            atomicOr(err, ERR_STRUCTURE);
                        } else {
                            if (MODE == COUNT)
                                atomicOr(&bits[c[h] >> 5], 1u << (c[h] & 31));
                            else
                                add_one<MODE == FILL>(acc + c[h], __fmul_rn(ae, b[h]));
                        }
                    }
                }
            }
            __syncwarp();
            ++e0;
        }
    }
}

// Segment i of a list (none past s1): its B position in sg.x, entries and A
// value. One that does not lie in the operands (an operand changed while its
// lists were built) is flagged and stands in as B's first entry: the walks
// take a list's segments to be its lanes' prefix, none of them empty.
template <int MODE>
__device__ __forceinline__ void list_segment(const CsrView& A, const CsrView& B,
                                             const HeavyLists& L, int64_t i, int64_t s1, int a0,
                                             int cw_log2, int2* sg, int* len, float* av,
                                             int32_t* err) {
    *sg = make_int2(0, 0);
    *len = 0;
    *av = 0.0f;
    if (i < s1) {
        *sg = L.seg[i];
        *len = (sg->y & ((1 << cw_log2) - 1)) + 1;
        const int64_t j = (int64_t)a0 + (int64_t)((uint32_t)sg->y >> cw_log2);
        if (sg->x < 0 || (int64_t)sg->x + *len > B.nnz || j >= A.nnz) {
            atomicOr(err, ERR_STRUCTURE);
            sg->x = 0;
            *len = 1;
        } else if (MODE != COUNT) {
            *av = A.v[j];
        }
    }
}

// A stretch of a row's columns with few products (at most SPARSE_PRODUCTS, of
// neighbouring chunks up to SPARSE_COLS columns): instead of an accumulator
// per column, one per distinct column. The products' columns set bits, a
// column's rank among the bits is its place, products add into their places
// in A-row order, and columns and values leave as coalesced stores. A chunk
// costs the dense path some 500 instructions however few products it has, and
// most chunks of a power-law row have few.
constexpr int SPARSE_STEPS = 12;
constexpr int SPARSE_PRODUCTS = 32 * SPARSE_STEPS;
// bitmap, rank of each 64 columns, segments (later values and columns in C's
// order), the products and their columns
constexpr int SPARSE_BYTES =
    SPARSE_COLS / 8 + SPARSE_COLS / 64 * 2 + 8 * SPARSE_PRODUCTS + 6 * SPARSE_PRODUCTS;

// Warps' shared memory in k_heavy_list: the dense path's, or the sparse one's
// over it, and the sparse path's bits of segment starts.
__host__ __device__ constexpr int list_smem_bytes(int mode, int cw) {
    return mode == COUNT ? heavy_smem_bytes(mode, cw)
                         : (4 * cw > SPARSE_BYTES ? 4 * cw : SPARSE_BYTES) + 64;
}

// Lane 0 of the learned sweep's FILL: where `total` entries of item w go, the
// next place in the row's slot, else in the shared overflow pool, -1 if
// neither has room (the row is then filled again).
__device__ __forceinline__ long long learned_place(int w, int row, int total,
                                                   int32_t* __restrict__ item_cnt,
                                                   int32_t* __restrict__ row_cnt,
                                                   const RowCtl& ctl) {
    item_cnt[w] = total;
    const int off = atomicAdd(&row_cnt[row], total);
    const int64_t t0 = ctl.slot_off[row], cap = ctl.slot_off[row + 1] - t0;
    long long dst = -1;
    if ((int64_t)off + total <= cap) {
        dst = t0 + off;
    } else if (total > 0) {
        const unsigned long long p = atomicAdd(ctl.pool_fill, (unsigned long long)total);
        if ((int64_t)p + total <= ctl.pool_cap) dst = ctl.pool_base + (int64_t)p;
    } else {
        dst = t0;  // an empty stretch needs no room
    }
    ctl.item_off[w] = dst;
    if (dst < 0) ctl.ovf[row] = 1;
    return dst;
}

// FILL, a dense chunk's end: its marked sums leave for C in column order, 32
// columns a step (lanes' places from the ballot of those that are there), and
// the accumulator is left zero. R-MAT 2^17 whole, fill: 7.26 ms with a bitmap
// and a lane writing each of its words' columns, 6.72 so.
__device__ __forceinline__ void list_finish(int w, const HeavyItem& it, int lo, int cw, float* acc,
                                            int32_t* __restrict__ item_cnt,
                                            int32_t* __restrict__ row_cnt,
                                            const int64_t* __restrict__ item_scan,
                                            const int32_t* __restrict__ c_rp,
                                            int32_t* __restrict__ c_ci, float* __restrict__ c_v,
                                            int32_t* __restrict__ err, const RowCtl& ctl) {
    const int lane = lane_id();
    __syncwarp();
    int64_t dst, room;
    if (ctl.item_off) {
        int c = 0;
        for (int x = lane; x < cw >> 2; x += 32) {
            const uint4 t = reinterpret_cast<const uint4*>(acc)[x];
            c += (t.x != 0u) + (t.y != 0u) + (t.z != 0u) + (t.w != 0u);
        }
        c = __reduce_add_sync(FULL, c);
        long long d = 0;
        if (lane == 0) d = learned_place(w, it.row, c, item_cnt, row_cnt, ctl);
        dst = __shfl_sync(FULL, d, 0);
        room = dst >= 0 ? INT64_MAX : 0;
    } else {
        // (counts that disagree with this fill would only come from an
        // operand changed in between: stay inside the row)
        dst = (int64_t)c_rp[it.row] + (item_scan[w] - item_scan[it.first]);
        room = (int64_t)c_rp[it.row + 1] - dst;
    }
    const int m = (int)max(min(room, (int64_t)cw), (int64_t)0);
    int32_t* oc = c_ci + dst;
    float* ov = c_v + dst;
    const unsigned below = (1u << lane) - 1;
    int at = 0;
    constexpr int STEP = 4;  // (cw is a multiple of 512)
    for (int x0 = lane; x0 < cw; x0 += 32 * STEP) {
        float t[STEP];
#pragma unroll
        for (int h = 0; h < STEP; ++h) t[h] = acc[x0 + 32 * h];
#pragma unroll
        for (int h = 0; h < STEP; ++h) {
            acc[x0 + 32 * h] = 0.0f;
            const bool there = __float_as_uint(t[h]) != 0u;
            const unsigned b = __ballot_sync(FULL, there);
            const int pos = at + __popc(b & below);
            if (there && pos < m) {
                oc[pos] = lo + x0 + 32 * h;
                ov[pos] = marked(t[h]);
            }
            at += __popc(b);
        }
    }
    if (!ctl.item_off && at > m && lane == 0) atomicOr(err, ERR_STRUCTURE);
    __syncwarp();
}

// Sparse stretch [lo, lo + width) of `row`, segments [s0, s1): work items w ..
// of the row, where its C entries go as in heavy_finish (the first item's
// place; the others' counts are zero in the learned sweep). Leaves the shared
// memory zeroed.
template <int MODE>
__device__ __forceinline__ void sparse_stretch(
    const CsrView& A, const CsrView& B, const HeavyLists& L, int w, int n_items,
    const HeavyItem& it, int64_t s0, int64_t s1, int lo, int width, int cw_log2,
    unsigned char* mine, uint32_t* heads, int32_t* __restrict__ item_cnt,
    int32_t* __restrict__ row_cnt, const int64_t* __restrict__ item_scan,
    const int32_t* __restrict__ c_rp, int32_t* __restrict__ c_ci, float* __restrict__ c_v,
    int32_t* __restrict__ err, const RowCtl& ctl) {
    const int lane = lane_id();
    const unsigned upto = 0xffffffffu >> (31 - lane);
    uint32_t* bm = reinterpret_cast<uint32_t*>(mine);
    uint16_t* rank64 = reinterpret_cast<uint16_t*>(mine + SPARSE_COLS / 8);
    int2* ent = reinterpret_cast<int2*>(mine + SPARSE_COLS / 8 + SPARSE_COLS / 64 * 2);
    float* acc = reinterpret_cast<float*>(ent);
    uint16_t* cols = reinterpret_cast<uint16_t*>(acc + SPARSE_PRODUCTS);
    float* prod = reinterpret_cast<float*>(ent + SPARSE_PRODUCTS);
    uint16_t* pcol = reinterpret_cast<uint16_t*>(prod + SPARSE_PRODUCTS);
    // the segments, and the products at which they start
    int n = 0, ns = 0;
    for (int64_t base = s0; base < s1; base += 32) {
        int2 sg;
        int len;
        float av;
        list_segment<MODE>(A, B, L, base + lane, s1, it.a0, cw_log2, &sg, &len, &av, err);
        const int incl = warp_incl_scan(len);
        const int start = n + incl - len;
        const unsigned some = __ballot_sync(FULL, len > 0);
        if (len > 0 && start < SPARSE_PRODUCTS) {
            ent[ns + __popc(some & ((1u << lane) - 1))] =
                make_int2(sg.x - start, __float_as_int(av));
            atomicOr(&heads[start >> 5], 1u << (start & 31));
        }
        ns += __popc(some);
        n += __shfl_sync(FULL, incl, 31);
        if (n > SPARSE_PRODUCTS) {
            if (lane == 0) atomicOr(err, ERR_STRUCTURE);
            n = SPARSE_PRODUCTS;
            break;
        }
    }
    __syncwarp();
    // (loops kept small: unrolled over the steps, the code outgrows the
    // instruction cache and the warps wait for it)
    int before = -1;
#pragma unroll 2
    for (int s = 0; 32 * s < n; ++s) {
        const unsigned h = heads[s];
        const int p = 32 * s + lane;
        if (p < n) {
            const int2 e = ent[before + __popc(h & upto)];
            const int c = __ldg(B.ci + e.x + p) - lo;
            prod[p] = __fmul_rn(__int_as_float(e.y), __ldg(B.v + e.x + p));
            const bool ok = (unsigned)c < (unsigned)width;
            if (!ok) atomicOr(err, ERR_STRUCTURE);  // B row not sorted
            pcol[p] = (uint16_t)(ok ? c : 0);
            if (ok) atomicOr(&bm[c >> 5], 1u << (c & 31));
        }
        before += __popc(h);
    }
    __syncwarp();
    // rank of every 64 columns: each lane counts SPARSE_COLS / 32 columns
    constexpr int PER = SPARSE_COLS / 32 / 128;  // 16-byte words a lane
    int pc[PER * 2], own = 0;
    const uint4* b4 = reinterpret_cast<const uint4*>(bm) + lane * PER;
#pragma unroll
    for (int x = 0; x < PER; ++x) {
        const uint4 v = b4[x];
        pc[2 * x] = __popc(v.x) + __popc(v.y);
        pc[2 * x + 1] = __popc(v.z) + __popc(v.w);
        own += pc[2 * x] + pc[2 * x + 1];
    }
    const int incl = warp_incl_scan(own);
    const int total = __shfl_sync(FULL, incl, 31);
    int run = incl - own;
#pragma unroll
    for (int x = 0; x < PER * 2; ++x) {
        rank64[lane * PER * 2 + x] = (uint16_t)run;
        run += pc[x];
    }
    // where the entries go
    long long dst = 0;
    if (MODE == FILL && ctl.item_off) {
        if (lane == 0) dst = learned_place(w, it.row, total, item_cnt, row_cnt, ctl);
        if (lane > 0 && lane < n_items) {
            item_cnt[w + lane] = 0;
            ctl.item_off[w + lane] = ctl.slot_off[it.row];
        }
    } else {
        dst = (int64_t)c_rp[it.row] + (item_scan[w] - item_scan[it.first]);
    }
    for (int x = lane; x < (n + 3) >> 2; x += 32)
        reinterpret_cast<float4*>(acc)[x] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncwarp();
#pragma unroll 1
    for (int s = 0; 32 * s < n; ++s) {
        const int p = 32 * s + lane;
        const bool in = p < n;
        int r = 0;
        float pr = 0.0f;
        if (in) {
            const int c = pcol[p];
            pr = prod[p];
            const uint2 b2 = *reinterpret_cast<const uint2*>(bm + (c >> 6) * 2);
            const unsigned below = (1u << (c & 31)) - 1;
            const bool upper = c & 32;
            r = rank64[c >> 6] + __popc(upper ? b2.x : b2.x & below) +
                (upper ? __popc(b2.y & below) : 0);
            cols[r] = (uint16_t)c;
        }
        add_step<false>(acc, r, in, pr, heads[s] & ~1u);
    }
    dst = __shfl_sync(FULL, dst, 0);
    // (counts that disagree with this fill would only come from an operand
    // changed in between: stay inside the row)
    const int64_t room = ctl.item_off ? (dst >= 0 ? INT64_MAX : 0) : (int64_t)c_rp[it.row + 1] - dst;
    const int m = (int)min((int64_t)total, max(room, (int64_t)0));
    if (!ctl.item_off && m < total && lane == 0) atomicOr(err, ERR_STRUCTURE);
    for (int x = lane; x < m; x += 32) {
        if (MODE == FILL) c_ci[dst + x] = lo + cols[x];
        c_v[dst + x] = acc[x];
    }
    __syncwarp();
    // zeroed for the next item
    uint4* z = reinterpret_cast<uint4*>(mine);
    for (int x = lane; x < SPARSE_BYTES / 16; x += 32) z[x] = make_uint4(0u, 0u, 0u, 0u);
    if (lane < 16) heads[lane] = 0u;
    __syncwarp();
}

// Entries drawn as draw_batched does, except at the list's end: a single index
// past it (`limit`) does not end the warp, since the batch in flight may be the
// CTA's last and would be left to the one warp that fetched it (16,000 items on
// 592 CTAs of 16 warps, count: 6.3 ms, most of it with one warp a CTA at work,
// against 1.0). The warp waits until the fetch, 1 us of its CTA's own warp, is
// there; were it not after DRAW_POLLS the warp would leave, and the fetching
// warp take the batch alone. Called by lane 0; returns the entry drawn, limit
// or more at the end. What a draw past its batch does (draw_past; -1: draw
// again) is kept out of the kernel's code: inlined it cost the loops 1 %.
constexpr int DRAW_POLLS = 1 << 12;
__device__ __noinline__ long long draw_past(unsigned long long* s_q, int32_t* queue, long long batch,
                                            long long limit, long long c) {
    if (c == batch) {
        const int nb = atomicAdd(queue, (int)batch);
        atomicExch(s_q, ((unsigned long long)(unsigned)nb << 32) | 1ull);
        return nb;
    }
    const long long single = atomicAdd(queue, 1);
    if (single < limit) return single;
    for (int polls = 0; polls < DRAW_POLLS; ++polls) {
        const unsigned long long v = *(volatile unsigned long long*)s_q;
        if ((long long)(v & 0xffffffffull) <= batch) return (long long)(v >> 32) < limit ? -1 : limit;
        __nanosleep(64);
    }
    return limit;
}
__device__ __forceinline__ long long draw_entry(unsigned long long* s_q, int32_t* queue,
                                                long long batch, long long limit) {
    long long w;
    do {
        const unsigned long long o = atomicAdd(s_q, 1ull);
        const long long c = (long long)(o & 0xffffffffull);
        w = c < batch ? (long long)(o >> 32) + c : draw_past(s_q, queue, batch, limit, c);
    } while (w < 0);
    return w;
}

// Heavy rows, items drawn in CTA batches by a grid that fills the GPU once, as
// in k_heavy. COUNT: one warp per item, or per group of neighbouring items with
// few segments. FILL and REUSE: the work list's entries; a warp takes its
// chunks in stretches of at most SPARSE_PRODUCTS products (sparse_stretch), a
// chunk beyond that through the dense accumulator.
template <int MODE>
__global__ void __launch_bounds__(list_max_warps(MODE) * 32, MODE == COUNT ? 2 : 0)
    k_heavy_list(CsrView A, CsrView B, const HeavyItem* __restrict__ items, int nitems,
                 HeavyLists L, int32_t* __restrict__ item_cnt, int32_t* __restrict__ row_cnt,
                 const int64_t* __restrict__ item_scan, const int32_t* __restrict__ c_rp,
                 int32_t* __restrict__ c_ci, float* __restrict__ c_v, int32_t* __restrict__ err,
                 RowCtl ctl, int cw_log2, int32_t* __restrict__ queue) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int cw = 1 << cw_log2;
    const int nw = cw >> 5;
    const int warp = threadIdx.x >> 5, lane = lane_id();
    const int bytes = list_smem_bytes(MODE, cw);
    unsigned char* mine = smem + warp * bytes;
    float* acc = reinterpret_cast<float*>(mine);
    unsigned* bits = reinterpret_cast<unsigned*>(mine);  // (COUNT)
    for (int x = lane; x < bytes / 16; x += 32)
        reinterpret_cast<float4*>(mine)[x] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncwarp();
    const int limit = MODE == COUNT ? nitems : (int)min(*L.nwork, (int64_t)nitems);
    // (a launch of fewer entries than two a warp spreads them over all CTAs)
    const int warps = blockDim.x >> 5;
    const long long batch = min(max((limit + (long long)gridDim.x - 1) / gridDim.x, 1ll), 2ll * warps);
    unsigned long long* s_q = reinterpret_cast<unsigned long long*>(smem + warps * bytes);
    if (threadIdx.x == 0) *s_q = (unsigned long long)batch;
    __syncthreads();
    for (;;) {
        long long wq = 0;
        if (lane == 0) wq = draw_entry(s_q, queue, batch, limit);
        wq = __shfl_sync(FULL, wq, 0);
        if (wq >= limit) break;
        const int2 wk = MODE == COUNT ? make_int2((int)wq, 1) : L.work[wq];
        const int w = wk.x;
        const HeavyItem it = items[w];
        const int row = it.row;
        if (ctl.only && !ctl.only[row]) continue;
        int span = 1;
        if constexpr (MODE == COUNT) {
            // a row's neighbouring chunks are counted together when they are
            // few segments (one walk fills the lanes better); a long list is
            // left to a warp a chunk (a hub row's group would run alone)
            const int g = w - (w - it.first) % HEAVY_COUNT_SPAN;
            const bool same = lane > 0 && lane < HEAVY_COUNT_SPAN && g + lane < nitems &&
                              items[g + lane].first == it.first;
            const int n = __ffs(~(__ballot_sync(FULL, same) | 1u)) - 1;
            if (L.item_seg[g + n] - L.item_seg[g] <= COUNT_GROUP_SEGS) {
                if (w != g) continue;
                span = n;
            }
        }
        if constexpr (MODE == COUNT) {
            const int64_t s0 = L.item_seg[w], s1 = L.item_seg[w + span];
            for (int64_t base = s0; base < s1; base += 32) {
                int2 sg;
                int len;
                float av;
                list_segment<MODE>(A, B, L, base + lane, s1, it.a0, cw_log2, &sg, &len, &av, err);
                list_products<MODE>(B, sg, len, av, it.chunk << cw_log2, span << cw_log2, acc, bits,
                                    err);
            }
            __syncwarp();
            for (int h = 0; h < span; ++h) {
                int c = 0;
                for (int x = lane; x < nw; x += 32) {
                    c += __popc(bits[h * nw + x]);
                    bits[h * nw + x] = 0u;
                }
                c = __reduce_add_sync(FULL, c);
                if (lane == 0) {
                    item_cnt[w + h] = c;
                    if (c && row_cnt) atomicAdd(&row_cnt[row], c);
                }
            }
            __syncwarp();
        } else {
            uint32_t* heads = reinterpret_cast<uint32_t*>(mine + bytes - 64);
            const int last = wk.y;
            const int prod_l = lane < last ? L.item_prod[w + lane] : 0;
            for (int k = 0; k < last;) {
                const int item = w + k;
                // as many chunks as stay few products
                int m = 1, p = __shfl_sync(FULL, prod_l, k);
                while (k + m < last) {
                    const int q = __shfl_sync(FULL, prod_l, k + m);
                    if (p + q > SPARSE_PRODUCTS) break;
                    p += q;
                    ++m;
                }
                const int lo = (it.chunk + k) << cw_log2;
                const int64_t s0 = L.item_seg[item], s1 = L.item_seg[item + m];
                if (p <= SPARSE_PRODUCTS && (m << cw_log2) <= SPARSE_COLS) {
                    sparse_stretch<MODE>(A, B, L, item, m, it, s0, s1, lo, m << cw_log2, cw_log2,
                                         mine, heads, item_cnt, row_cnt, item_scan, c_rp, c_ci, c_v,
                                         err, ctl);
                } else {
                    for (int64_t base = s0; base < s1; base += 32) {
                        int2 sg;
                        int len;
                        float av;
                        list_segment<MODE>(A, B, L, base + lane, s1, it.a0, cw_log2, &sg, &len, &av,
                                           err);
                        list_products<MODE>(B, sg, len, av, lo, cw, acc, bits, err);
                    }
                    if (MODE == FILL) {
                        const HeavyItem mineit{it.row, it.chunk + k, it.first, it.a0};
                        list_finish(item, mineit, lo, cw, acc, item_cnt, row_cnt, item_scan, c_rp,
                                    c_ci, c_v, err, ctl);
                    } else {
                        // REUSE: the chunk's entries of C, in order, and back to zero
                        __syncwarp();
                        const int64_t r0 = c_rp[row], r1 = c_rp[row + 1];
                        const int64_t o = r0 + (item_scan[item] - item_scan[it.first]);
                        const int64_t e = min(o + item_cnt[item], r1);
                        for (int64_t q = o + lane; q < e; q += 32) {
                            const int col = c_ci[q] - lo;
                            c_v[q] = (unsigned)col < (unsigned)cw ? acc[col] : 0.0f;
                        }
                        __syncwarp();
                        float4* a4 = reinterpret_cast<float4*>(acc);
                        for (int x = lane; x < (cw >> 2); x += 32)
                            a4[x] = make_float4(0.f, 0.f, 0.f, 0.f);
                        __syncwarp();
                    }
                }
                k += m;
            }
        }
    }
}

}  // namespace rvsp
