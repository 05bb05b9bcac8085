// Medium rows of up to 2048 products: the row's products sorted by column in
// registers.
//
// Expand, sort, compress. Every product becomes one word, column <<
// log2(CAP) | index in A-row order, and its value goes to shared memory at
// that index. The words are sorted by a bitonic network: E words a thread,
// compare-exchanges inside a thread, shuffles between a warp's lanes, shared
// memory only between the warps of a large row. Equal columns come out
// together in A-row order, so each run summed left to right from +0.0f is the
// reference's order of additions (accum_scalar_f32.c:69) and the values are
// bit-identical.
//
// Why not the shared-memory table (k_warp): its radix passes and hash probes
// are serial chains through shared memory, and its 12 bytes a slot leave few
// warps to hide them. Bound now by instruction issue (ncu: issue active 52-78 %
// of peak; a 256-word row takes 1,360 instructions). Measured (B200, device
// time): 4096^2 x 16 a row, FILL 30 -> 11 us, COUNT 24 -> 7.6 us; 2M x 100k
// tall-skinny, rows of 33..2048 products, FILL 7.1 -> 3.3 ms, COUNT 3.2 -> 2.1
// ms; 128 batched products, FILL 22.2 -> 9.1 ms. Tried and dropped: the same
// rows by one counting pass over column buckets (more instructions: the
// in-bucket loops cost more than the network's layers), 32 words a thread in
// one warp for 1024 products (1015 us against 902 us with two warps on the
// tall-skinny product: 114 registers and code past the instruction cache).
#pragma once

#include "spgemm_kernels.cuh"

namespace rvsp {

constexpr int SORT_CTA_ROWS = 4;  // one-warp rows per CTA

// The value types of k_sort. arg() is what an A entry's products need of it,
// one word beside the entry's position; entries whose sum is zero are kept
// (KEEP_ZERO, the FP32 path) or dropped (the reference's FP64 and INT8
// kernels, csr_scalar_f64.c:49-272 and csr_scalar_i8.c:24-196).
struct F32Values {
    using In = float;
    using Out = float;
    static constexpr bool KEEP_ZERO = true;
    static __device__ __forceinline__ int arg(const float* a, int j) { return __float_as_int(a[j]); }
    static __device__ __forceinline__ float mul(const float*, int arg, float b) {
        return __fmul_rn(__int_as_float(arg), b);
    }
    static __device__ __forceinline__ float add(float x, float y) { return __fadd_rn(x, y); }
    static __device__ __forceinline__ float read(const float* p) { return __ldg(p); }
};
struct F64Values {
    using In = double;
    using Out = double;
    static constexpr bool KEEP_ZERO = false;
    static __device__ __forceinline__ int arg(const double*, int j) { return j; }
    static __device__ __forceinline__ double mul(const double* a, int j, double b) {
        return __dmul_rn(__ldg(a + j), b);
    }
    static __device__ __forceinline__ double add(double x, double y) { return __dadd_rn(x, y); }
    static __device__ __forceinline__ double read(const double* p) { return __ldg(p); }
};
struct I8Values {
    using In = int8_t;
    using Out = int32_t;
    static constexpr bool KEEP_ZERO = false;
    static __device__ __forceinline__ int arg(const int8_t* a, int j) { return a[j]; }
    static __device__ __forceinline__ int32_t mul(const int8_t*, int a, int8_t b) {
        return (int32_t)((uint32_t)a * (uint32_t)(int32_t)b);
    }
    static __device__ __forceinline__ int32_t add(int32_t x, int32_t y) {
        return (int32_t)((uint32_t)x + (uint32_t)y);
    }
    static __device__ __forceinline__ int8_t read(const int8_t* p) { return *p; }
};

// Threads of one row: NW warps, CAP = 32 NW E words.
template <int E, int NW, class V = F32Values>
struct SortShape {
    static constexpr int T = 32 * NW;
    static constexpr int CAP = T * E;
    static constexpr int WORDS = CAP / 32;
    static constexpr int ROWS = NW == 1 ? SORT_CTA_ROWS : 1;  // rows of a CTA
    static constexpr int PAD = CAP + WORDS;                   // padded array
    // Shared words of a row: a bit per product (set where an A entry's
    // products start) and, for rows of several warps, the starts before each
    // such word, the threads' open runs and counters; the A entries {B
    // position - first index, A value} while the products are gathered,
    // overlaid afterwards by the row's columns and values in C's order; the
    // products' values.
    static constexpr int OW = sizeof(typename V::Out) / 4;  // words of a value
    static constexpr int EXTRA = NW == 1 ? 0 : WORDS + OW * T + 2 * NW + 2;
    static constexpr int BYTES = 4 * (WORDS + EXTRA + (1 + OW) * PAD + OW * CAP);
    static_assert((WORDS + EXTRA) % 2 == 0 && PAD % 2 == 0 && BYTES % 8 == 0, "");
};

// Padded index: one word in 32 is left out, so lanes a power of two words
// apart use different banks.
__device__ __forceinline__ int pad32(int x) { return x + (x >> 5); }

// The row's CAP words ascending, as the floats of the same bits (finite and
// not negative, so they order like the words): word j of thread t ends as the
// (t E + j)-th. Bitonic merges in their all-ascending form: a merge starts by
// comparing each word with its mirror image in the block, so no later step
// depends on the block's direction.
//
// Between lanes, the lane that keeps the larger word holds it negated: its
// partner's word arrives with the other sign, and min(own, -partner's) is the
// right choice on both sides. One min a word and step, against min, max and
// select; the sign changes between steps are multiplications by +-1, which
// run on the FMA pipe beside the ALU that the mins saturate.
template <int E, int NW, int SIZE, int STRIDE>
__device__ __forceinline__ void sort_layer(float (&f)[E], float& sign, int t, float* xbuf) {
    constexpr bool FLIP = STRIDE == SIZE / 2;
    if constexpr (STRIDE < E) {
        if constexpr (STRIDE * 2 == E && SIZE > E) {
#pragma unroll
            for (int j = 0; j < E; ++j) f[j] *= sign;
            sign = 1.0f;
        }
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const int p = j ^ (FLIP ? SIZE - 1 : STRIDE);
            if (p > j) {
                const float lo = fminf(f[j], f[p]), hi = fmaxf(f[j], f[p]);
                f[j] = lo;
                f[p] = hi;
            }
        }
    } else if constexpr (STRIDE < 32 * E) {
        constexpr int MASK = FLIP ? SIZE / E - 1 : STRIDE / E;
        const float want = (t & (STRIDE / E)) ? -1.0f : 1.0f;
        const float m = sign * want;
        sign = want;
#pragma unroll
        for (int j = 0; j < E; ++j) f[j] *= m;
        if constexpr (FLIP) {
#pragma unroll
            for (int j = 0; j < E / 2; ++j) {
                const float a = __shfl_xor_sync(FULL, f[E - 1 - j], MASK);
                const float b = __shfl_xor_sync(FULL, f[j], MASK);
                f[j] = fminf(f[j], -a);
                f[E - 1 - j] = fminf(f[E - 1 - j], -b);
            }
        } else {
#pragma unroll
            for (int j = 0; j < E; ++j) f[j] = fminf(f[j], -__shfl_xor_sync(FULL, f[j], MASK));
        }
    } else {  // between warps
        constexpr int MASK = FLIP ? SIZE - 1 : STRIDE;
        const bool upper = (t & (STRIDE / E)) != 0;
#pragma unroll
        for (int j = 0; j < E; ++j) xbuf[pad32(t * E + j)] = f[j];
        __syncthreads();
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const float a = xbuf[pad32((t * E + j) ^ MASK)];
            f[j] = upper ? fmaxf(f[j], a) : fminf(f[j], a);
        }
        __syncthreads();
    }
    if constexpr (STRIDE > 1) sort_layer<E, NW, SIZE, STRIDE / 2>(f, sign, t, xbuf);
}

template <int E, int NW, int SIZE = 2>
__device__ __forceinline__ void sort_words(float (&f)[E], int t, float* xbuf) {
    static_assert(E >= 2, "");
    float sign = 1.0f;  // the words' sign in this lane
    sort_layer<E, NW, SIZE, SIZE / 2>(f, sign, t, xbuf);
    if constexpr (SIZE < SortShape<E, NW>::CAP) sort_words<E, NW, SIZE * 2>(f, t, xbuf);
}

// The rows of one sort bin (at most CAP products each; rows with more, which
// only an operand changed since the analysis can have, flag ERR_STRUCTURE).
// COUNT writes the row's distinct columns to cnt; FILL writes its sorted
// columns and values (in the learned sweep, ctl.slot_off, into the row's slot,
// with the count to cnt, or -1 when it passes the slot) and, with pm, every
// product's position in the row. Words must stay below the bits of infinity
// (sort_cols_fit).
template <int E, int NW, int MODE, class V>
__global__ void __launch_bounds__(SortShape<E, NW, V>::T * SortShape<E, NW, V>::ROWS)
    k_sort(CsrView A, CsrView B, const typename V::In* __restrict__ a_v,
           const typename V::In* __restrict__ b_v, const int32_t* __restrict__ rows, int nrows,
           int32_t* __restrict__ cnt, const int32_t* __restrict__ c_rp,
           int32_t* __restrict__ c_ci, typename V::Out* __restrict__ c_v,
           const int32_t* __restrict__ list_off, uint16_t* __restrict__ pm,
           int32_t* __restrict__ err, RowCtl ctl) {
    static_assert(MODE == COUNT || MODE == FILL, "");
    using S = SortShape<E, NW, V>;
    using Out = typename V::Out;
    constexpr int CAP = S::CAP, T = S::T, WORDS = S::WORDS;
    constexpr int IB = __builtin_ctz(CAP);
    constexpr uint32_t SAME = MODE == FILL ? CAP : 1;  // words of one column differ by less
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = lane_id();
    const int wi = NW == 1 ? 0 : threadIdx.x >> 5;  // warp of the row
    const int t = NW == 1 ? lane : threadIdx.x;     // thread of the row
    const int slot = NW == 1 ? threadIdx.x >> 5 : 0;
    const int w = blockIdx.x * S::ROWS + slot;
    if (w >= nrows) return;
    const int row = rows[w];
    if (ctl.only && !ctl.only[row]) return;
    uint32_t* heads = reinterpret_cast<uint32_t*>(smem + slot * S::BYTES);
    int* pre = reinterpret_cast<int*>(heads + WORDS);       // NW > 1: starts before each word
    Out* tails = reinterpret_cast<Out*>(pre + WORDS);       // NW > 1: each thread's open run
    int* red = reinterpret_cast<int*>(tails + T);           // NW > 1: per-warp words, n, total
    int2* ent = reinterpret_cast<int2*>(heads + WORDS + S::EXTRA);
    int32_t* scol = reinterpret_cast<int32_t*>(ent);
    Out* sval = reinterpret_cast<Out*>(scol + S::PAD);
    Out* vals = sval + S::PAD;
    const auto sync = [] {
        if constexpr (NW == 1) __syncwarp();
        else __syncthreads();
    };
    if (t < WORDS) heads[t] = 0u;
    sync();
    // the row's non-empty entries, in order, and where their products start
    int n = 0;
    if (NW == 1 || wi == 0) {
        int a0, a1, entries = 0;
        row_range(A, row, &a0, &a1, err);
        for (int base = a0; base < a1; base += 32) {
            const int j = base + lane;
            int bs = 0, bl = 0, arg = 0;
            if (j < a1) {
                int be;
                row_range(B, A.ci[j], &bs, &be, err);
                bl = min(be - bs, CAP + 1);
                if (MODE == FILL) arg = V::arg(a_v, j);
            }
            const int incl = warp_incl_scan(bl);
            const int start = n + incl - bl;
            const unsigned some = __ballot_sync(FULL, bl > 0);
            if (bl > 0 && start < CAP) {
                ent[entries + __popc(some & ((1u << lane) - 1))] = make_int2(bs - start, arg);
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
        if constexpr (NW > 1) {
            __syncwarp();
            if (lane == 0) red[2 * NW] = n;
            int run = 0;
            for (int x0 = 0; x0 < WORDS; x0 += 32) {
                const int c = __popc(heads[x0 + lane]);
                const int incl = warp_incl_scan(c);
                pre[x0 + lane] = run + incl - c;
                run += __shfl_sync(FULL, incl, 31);
            }
        }
    }
    sync();
    if constexpr (NW > 1) n = red[2 * NW];
    // product p = T s + t: its entry is the number of starts up to p
    float f[E];
    const unsigned upto = 0xffffffffu >> (31 - lane);
    {
        bool bad = false;
        int before = -1;
#pragma unroll
        for (int s = 0; s < E; ++s) {
            const unsigned h = heads[s * NW + wi];
            if constexpr (NW > 1) before = pre[s * NW + wi] - 1;
            const int p = T * s + t;
            f[s] = __int_as_float(0x7f800000);  // +inf: after every word
            if (p < n) {
                const int2 e = ent[before + __popc(h & upto)];
                const int q = e.x + p;
                uint32_t col = (uint32_t)__ldg(B.ci + q);
                if (MODE == FILL) vals[p] = V::mul(a_v, e.y, V::read(b_v + q));
                if (col >= (uint32_t)B.cols) {
                    bad = true;
                    col = 0;
                }
                f[s] = __uint_as_float(MODE == FILL ? col << IB | (uint32_t)p : col);
            }
            before += __popc(h);
        }
        if (bad) atomicOr(err, ERR_STRUCTURE);
    }
    sync();  // every thread has read the entries
    sort_words<E, NW>(f, t, reinterpret_cast<float*>(scol));
    // heads: words whose column differs from the one before (bit j of mask)
    const int mine = min(max(n - t * E, 0), E);  // words this thread holds
    float last = __shfl_up_sync(FULL, f[E - 1], 1);
    if constexpr (NW > 1) {
        if (lane == 31) red[wi] = __float_as_int(f[E - 1]);
        __syncthreads();
        if (lane == 0 && wi > 0) last = __int_as_float(red[wi - 1]);
    }
    unsigned mask = 0;
#pragma unroll
    for (int j = 0; j < E; ++j) {
        const uint32_t x = __float_as_uint(f[j]);
        const uint32_t y = __float_as_uint(j > 0 ? f[j > 0 ? j - 1 : 0] : last);
        mask |= (unsigned)(j < mine && ((j == 0 && t == 0) || (x ^ y) >= SAME)) << j;
    }
    const int own = __popc(mask);
    int base = warp_incl_scan(own);
    int total = __shfl_sync(FULL, base, 31);
    if constexpr (NW > 1) {
        if (lane == 31) red[NW + wi] = base;
        __syncthreads();
        total = 0;
        for (int x = 0; x < NW; ++x) {
            const int c = red[NW + x];
            if (x < wi) base += c;
            total += c;
        }
    }
    base -= own;  // the place of this thread's first head
    if constexpr (MODE == COUNT) {
        if (t == 0) cnt[row] = total;
    } else {
        int64_t o;
        if (ctl.slot_off) {
            o = ctl.slot_off[row];
            const bool over = total > ctl.slot_off[row + 1] - o;
            if (V::KEEP_ZERO && t == 0) cnt[row] = over ? -1 : total;
            if (over) return;
        } else {
            o = c_rp[row];
            if (total != c_rp[row + 1] - c_rp[row]) {  // an operand changed since the count
                if (t == 0) atomicOr(err, ERR_STRUCTURE);
                return;
            }
        }
        // each run summed in order; a thread stores the runs that begin and
        // end in its words
        Out v[E];
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = vals[__float_as_uint(f[j]) & (CAP - 1)];
        const bool lead = mine > 0 && !(mask & 1u);  // its first words belong to a run before
        bool follow = __shfl_down_sync(FULL, (int)lead, 1);  // its last run goes on
        if (lane == 31) follow = false;
        if constexpr (NW > 1) {
            if (lane == 0) red[wi] = lead;
            __syncthreads();
            if (lane == 31 && wi + 1 < NW) follow = red[wi + 1] != 0;
        }
        Out acc = Out(0);
        int d = base - 1;
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const bool head = mask >> j & 1u;
            acc = V::add(head ? Out(0) : acc, v[j]);
            d += head;
            const bool end = j == E - 1 ? !follow : (mask >> (j + 1) & 1u) || j + 1 == mine;
            if (j < mine && end && d >= base) {
                scol[pad32(d)] = (int32_t)(__float_as_uint(f[j]) >> IB);
                sval[pad32(d)] = acc;
            }
        }
        if (pm) {
            uint16_t* pp = pm + (list_off[w] - list_off[0]);
#pragma unroll
            for (int j = 0; j < E; ++j)
                if (j < mine)
                    pp[__float_as_uint(f[j]) & (CAP - 1)] =
                        (uint16_t)(base - 1 + __popc(mask & ((2u << j) - 1)));
        }
        // runs that cross threads, continued from the thread before; once
        // more for every thread a run passes through from end to end (rows of
        // 1500 products in 1, 4 and 16 columns, 50,000 of them, calls: 6.1, 2.8
        // and 1.9 ms; by the table, whose ordered adds wait too, 8.8, 3.7, 3.3)
        const bool through = lead && mask == 0;
        bool any;
        int rounds;
        if constexpr (NW == 1) {
            any = __any_sync(FULL, lead);
            rounds = any ? 1 + __popc(__ballot_sync(FULL, through)) : 0;
        } else {
            any = __syncthreads_or(lead);
            rounds = any ? 1 + __syncthreads_count(through) : 0;
        }
        for (int it = 0; it < rounds; ++it) {
            Out in = __shfl_up_sync(FULL, acc, 1);
            if constexpr (NW > 1) {
                if (lane == 31) tails[wi] = acc;
                __syncthreads();
                if (lane == 0 && wi > 0) in = tails[wi - 1];
                __syncthreads();
            }
            if (lead) {
                Out a = in;
                const int until = mask ? __ffs(mask) - 1 : mine;
                int col = 0;
#pragma unroll
                for (int j = 0; j < E; ++j)
                    if (j < until) a = V::add(a, v[j]);
                col = (int32_t)(__float_as_uint(f[0]) >> IB);
                if (through) acc = a;
                if (!(through && follow)) {
                    scol[pad32(base - 1)] = col;
                    sval[pad32(base - 1)] = a;
                }
            }
        }
        sync();
        if constexpr (V::KEEP_ZERO) {
            for (int x = t; x < total; x += T) {
                c_ci[o + x] = scol[pad32(x)];
                c_v[o + x] = sval[pad32(x)];
            }
        } else if (NW == 1 || wi == 0) {
            // without the zero sums, by one warp; the count is what is left
            int kept = 0;
            for (int x0 = 0; x0 < total; x0 += 32) {
                const int x = x0 + lane;
                const Out s = x < total ? sval[pad32(x)] : Out(0);
                const unsigned m = __ballot_sync(FULL, s != Out(0));
                if (s != Out(0)) {
                    const int64_t to = o + kept + __popc(m & ((1u << lane) - 1));
                    c_ci[to] = scol[pad32(x)];
                    c_v[to] = s;
                }
                kept += __popc(m);
            }
            if (lane == 0) cnt[row] = kept;
        }
    }
}

}  // namespace rvsp
