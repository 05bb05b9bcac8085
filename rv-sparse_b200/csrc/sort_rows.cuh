// Medium rows of up to 1024 products: one warp per row, the row's products
// sorted by column in registers.
//
// Expand, sort, compress. Every product becomes one 32-bit word,
// column << log2(CAP) | index in A-row order; a warp holds CAP = 32 E words,
// E per lane, and sorts them with a bitonic network (compare-exchanges inside
// a lane, shuffles between lanes: no shared memory, no serial chain, E
// independent operations per layer). Equal columns come out together in A-row
// order, so each run summed left to right from +0.0f is the reference's order
// of additions (accum_scalar_f32.c:69) and the values are bit-identical.
//
// Why not the shared-memory table (k_warp): its radix passes and hash probes
// are serial chains through shared memory, and its 12 bytes a slot leave few
// warps to hide them. Measured (B200, device time of the launches): 4096^2 x 16
// a row, FILL 30 -> 12.6 us, COUNT 24 -> 7.4 us; 2M x 100k tall-skinny, rows of
// 65..1024 products, FILL 5.0 -> 2.7 ms, COUNT 2.4 -> 1.7 ms.
#pragma once

#include "spgemm_kernels.cuh"

namespace rvsp {

constexpr int SORT_WARPS = 4;  // rows (warps) per CTA

// Shared memory of one warp: a bit per product (set where an A entry's
// products start), then the A entries {B position - first index, A value} while
// the products are gathered, overlaid afterwards by the products' values and
// the sorted words (padded by one word in 32: a lane stores E consecutive
// words, and the padding spreads the lanes over the banks).
template <int E>
__host__ __device__ constexpr int sort_warp_bytes() {
    return 4 * E + 8 * 32 * E + 4 * E;
}

template <int E>
__device__ __forceinline__ void cross_lane(uint32_t (&k)[E], int mask, bool upper, bool flip) {
    if (flip) {  // partner of word j is word E-1-j of lane ^ mask
#pragma unroll
        for (int j = 0; j < (E + 1) / 2; ++j) {
            const uint32_t a = __shfl_xor_sync(FULL, k[E - 1 - j], mask);
            if (E - 1 - j != j) {
                const uint32_t b = __shfl_xor_sync(FULL, k[j], mask);
                k[E - 1 - j] = upper ? max(k[E - 1 - j], b) : min(k[E - 1 - j], b);
            }
            k[j] = upper ? max(k[j], a) : min(k[j], a);
        }
    } else {
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const uint32_t a = __shfl_xor_sync(FULL, k[j], mask);
            k[j] = upper ? max(k[j], a) : min(k[j], a);
        }
    }
}

// The warp's 32 E words ascending: word j of lane l ends as the (l E + j)-th.
// Bitonic merges in their all-ascending form: a merge starts by comparing
// each word with its mirror image in the block, so no later step depends on
// the block's direction.
template <int E>
__device__ __forceinline__ void warp_bitonic_sort(uint32_t (&k)[E]) {
    const int lane = lane_id();
#pragma unroll
    for (int size = 2; size <= 32 * E; size <<= 1) {
        if (size <= E) {
#pragma unroll
            for (int j = 0; j < E; ++j) {
                const int p = (j & ~(size - 1)) + (size - 1 - (j & (size - 1)));
                if (p > j) {
                    const uint32_t lo = min(k[j], k[p]), hi = max(k[j], k[p]);
                    k[j] = lo;
                    k[p] = hi;
                }
            }
        } else {
            cross_lane<E>(k, size / E - 1, (lane & (size / E / 2)) != 0, true);
        }
#pragma unroll
        for (int stride = size / 4; stride >= 1; stride >>= 1) {
            if (stride < E) {
#pragma unroll
                for (int j = 0; j < E; ++j) {
                    if ((j & stride) == 0) {
                        const uint32_t lo = min(k[j], k[j | stride]), hi = max(k[j], k[j | stride]);
                        k[j] = lo;
                        k[j | stride] = hi;
                    }
                }
            } else {
                cross_lane<E>(k, stride / E, (lane & (stride / E)) != 0, false);
            }
        }
    }
}

// The rows of one sort bin (at most 32 E products each; rows with more, which
// only an operand changed since the analysis can have, flag ERR_STRUCTURE).
// COUNT writes the row's distinct columns to cnt; FILL writes its sorted
// columns and values (in the learned sweep, ctl.slot_off, into the row's slot,
// with the count to cnt, or -1 when it passes the slot) and, with pm, every
// product's position in the row. Columns must fit 32 - log2(32 E) bits
// (sort_cols_fit).
template <int E, int MODE>
__global__ void __launch_bounds__(SORT_WARPS * 32)
    k_sort(CsrView A, CsrView B, const int32_t* __restrict__ rows, int nrows,
           int32_t* __restrict__ cnt, const int32_t* __restrict__ c_rp,
           int32_t* __restrict__ c_ci, float* __restrict__ c_v,
           const int32_t* __restrict__ list_off, uint16_t* __restrict__ pm,
           int32_t* __restrict__ err, RowCtl ctl) {
    static_assert(MODE == COUNT || MODE == FILL, "");
    constexpr int CAP = 32 * E;
    constexpr int IB = __builtin_ctz(CAP);
    extern __shared__ __align__(16) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = lane_id();
    const int w = blockIdx.x * SORT_WARPS + warp;
    if (w >= nrows) return;
    const int row = rows[w];
    if (ctl.only && !ctl.only[row]) return;
    unsigned char* mine = smem + warp * sort_warp_bytes<E>();
    uint32_t* heads = reinterpret_cast<uint32_t*>(mine);
    int2* ent = reinterpret_cast<int2*>(mine + 4 * E);
    float* vals = reinterpret_cast<float*>(mine + 4 * E);
    uint32_t* sorted = reinterpret_cast<uint32_t*>(vals + CAP);
    if (lane < E) heads[lane] = 0u;
    int a0, a1;
    row_range(A, row, &a0, &a1, err);
    __syncwarp();
    // the row's non-empty entries, in order, and where their products start
    int n = 0, entries = 0;
    for (int base = a0; base < a1; base += 32) {
        const int j = base + lane;
        int bs = 0, bl = 0;
        float av = 0.0f;
        if (j < a1) {
            int be;
            row_range(B, A.ci[j], &bs, &be, err);
            bl = min(be - bs, CAP + 1);
            if (MODE == FILL) av = A.v[j];
        }
        const int incl = warp_incl_scan(bl);
        const int start = n + incl - bl;
        const unsigned some = __ballot_sync(FULL, bl > 0);
        if (bl > 0 && start < CAP) {
            ent[entries + __popc(some & ((1u << lane) - 1))] =
                make_int2(bs - start, __float_as_int(av));
            atomicOr(&heads[start >> 5], 1u << (start & 31));
        }
        entries += __popc(some);
        n += __shfl_sync(FULL, incl, 31);
        if (n > CAP) {
            if (lane == 0) atomicOr(err, ERR_STRUCTURE);
            n = CAP;
            break;
        }
    }
    __syncwarp();
    // product p = 32 s + lane: its entry is the number of starts up to p
    uint32_t k[E];
    float v[MODE == FILL ? E : 1];
    const unsigned upto = 0xffffffffu >> (31 - lane);
    int before = -1;
    bool bad = false;
#pragma unroll
    for (int s = 0; s < E; ++s) {
        const unsigned h = heads[s];
        const int p = 32 * s + lane;
        k[s] = 0xffffffffu;
        if (MODE == FILL) v[s] = 0.0f;
        if (p < n) {
            const int2 e = ent[before + __popc(h & upto)];
            const int q = e.x + p;
            const uint32_t col = (uint32_t)__ldg(B.ci + q);
            if (MODE == FILL) v[s] = __fmul_rn(__int_as_float(e.y), __ldg(B.v + q));
            bad |= col >= (uint32_t)B.cols;
            k[s] = MODE == FILL ? (col << IB) | (uint32_t)p : col;
        }
        before += __popc(h);
    }
    if (bad) atomicOr(err, ERR_STRUCTURE);
    if (MODE == FILL) {
        __syncwarp();  // every lane has read the entries
#pragma unroll
        for (int s = 0; s < E; ++s) vals[32 * s + lane] = v[s];
    }
    warp_bitonic_sort<E>(k);
    if (MODE == COUNT || ctl.slot_off) {
        // distinct columns: words that differ from the one before them
        constexpr int SH = MODE == FILL ? IB : 0;
        const uint32_t last = __shfl_up_sync(FULL, k[E - 1], 1);
        int c = 0;
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const uint32_t prev = j > 0 ? k[j > 0 ? j - 1 : 0] : last;
            const bool first = j == 0 && lane == 0;
            c += lane * E + j < n && (first || (prev >> SH) != (k[j] >> SH));
        }
        c = __reduce_add_sync(FULL, c);
        if (MODE == COUNT) {
            if (lane == 0) cnt[row] = c;
            return;
        }
        const int64_t room = ctl.slot_off[row + 1] - ctl.slot_off[row];
        if (lane == 0) cnt[row] = c > room ? -1 : c;
        if (c > room) return;
    }
    if constexpr (MODE == FILL) {
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const int x = lane * E + j;
            sorted[x + (x >> 5)] = k[j];
        }
        __syncwarp();
        const int64_t o = ctl.slot_off ? ctl.slot_off[row] : (int64_t)c_rp[row];
        const int room = ctl.slot_off ? CAP : c_rp[row + 1] - c_rp[row];
        uint16_t* pp = pm ? pm + (list_off[w] - list_off[0]) : nullptr;
        int out = 0;
        for (int b0 = 0; b0 < n; b0 += 32) {
            const int x = b0 + lane;
            const uint32_t wd = sorted[x + (x >> 5)];
            const uint32_t pv = x > 0 ? sorted[(x - 1) + ((x - 1) >> 5)] : ~wd;
            const bool head = x < n && (pv >> IB) != (wd >> IB);
            const unsigned hm = __ballot_sync(FULL, head);
            const int d = out + __popc(hm & upto) - 1;  // the run's place in the row
            if (pp && x < n) pp[wd & (CAP - 1)] = (uint16_t)d;
            if (head) {
                float sum = __fadd_rn(0.0f, vals[wd & (CAP - 1)]);
                for (int y = x + 1; y < n; ++y) {
                    const uint32_t wy = sorted[y + (y >> 5)];
                    if ((wy >> IB) != (wd >> IB)) break;
                    sum = __fadd_rn(sum, vals[wy & (CAP - 1)]);
                }
                if (d < room) {
                    c_ci[o + d] = (int32_t)(wd >> IB);
                    c_v[o + d] = sum;
                }
            }
            out += __popc(hm);
        }
        if (!ctl.slot_off && out != room && lane == 0) atomicOr(err, ERR_STRUCTURE);
    }
}

}  // namespace rvsp
