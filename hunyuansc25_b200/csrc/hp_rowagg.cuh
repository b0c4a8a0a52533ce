// hp_rowagg.cuh — "aggregate a row": gather (key, weight) entries, merge equal
// keys by summing weights, drop an excluded key, and write the unique keys in
// ascending order.  Used by contraction (key = coarse neighbour id, the self
// key dropped) and by the gain table (key = neighbour's part).
//
// Size classes (chosen per row by its entry count; the kernels' files give the bounds):
//   registers   a sorting network over 32-bit words (key and index), by a thread, a few
//               lanes, a warp or a CTA per row (64-bit entries where they do not fit)
//   dense       one CTA, dense accumulator + presence bitmap over the key space,
//               scanned in key order (global scratch per CTA for contraction, shared
//               memory for part keys)
// Every class produces the same canonical row, so the class boundaries are a
// performance choice only.
#pragma once

#include "hp_common.cuh"

namespace hp {

constexpr int32_t KEY_NONE = 0x7fffffff;

// ---- one row per thread, in registers ---------------------------------------
// Entries are packed as key << 32 | weight (padding and dropped keys are
// KEY_NONE) and sorted ascending by a bitonic network over the first NET of XN
// registers (compile-time indices only, so the array stays in registers);
// equal keys are then merged by summing the low halves.
template <int NET, int XN>
__device__ __forceinline__ void sort_regs(unsigned long long (&x)[XN])
{
#pragma unroll
    for (int size = 2; size <= NET; size <<= 1)
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1)
#pragma unroll
            for (int i = 0; i < NET; i++) {
                const int j = i ^ stride;
                if (j > i) {
                    const unsigned long long a = x[i], b = x[j];
                    const unsigned long long lo = a < b ? a : b, hi = a < b ? b : a;
                    if ((i & size) == 0) { x[i] = lo; x[j] = hi; }
                    else { x[i] = hi; x[j] = lo; }
                }
            }
}

constexpr unsigned long long PACK_NONE = (unsigned long long)(uint32_t)KEY_NONE << 32;

// ---- one row per thread or per warp, in 32-bit words ---------------------------
// An entry is packed as key << bits | (its index in the row), so a compare-exchange
// is one min and one max of 32-bit registers, and the weight is fetched by the index
// after the sort.  Padding and dropped keys are WORD_NONE, which sorts last: its key
// part, all ones, must be no key (2^(32 - bits) > number of keys).
constexpr unsigned WORD_NONE = 0xffffffffu;

constexpr int pow2_at_least(int n) { return n <= 1 ? 1 : 2 * pow2_at_least((n + 1) / 2); }

// Ascending bitonic network over the first NET of XN registers of one thread.  The
// first step of every merge compares mirrored positions, so all comparators point
// the same way; NET need not be a power of two: the missing high positions would hold
// WORD_NONE, which such comparators leave in place, so they are left out.
template <int NET, int XN>
__device__ __forceinline__ void sort_words(unsigned (&x)[XN])
{
    constexpr int P = pow2_at_least(NET);
#pragma unroll
    for (int size = 2; size <= P; size <<= 1) {
#pragma unroll
        for (int i = 0; i < NET; i++) {
            const int j = i ^ (size - 1);
            if (j > i && j < NET) {
                const unsigned a = x[i], b = x[j];
                x[i] = min(a, b);
                x[j] = max(a, b);
            }
        }
#pragma unroll
        for (int stride = size >> 2; stride > 0; stride >>= 1)
#pragma unroll
            for (int i = 0; i < NET; i++) {
                const int j = i ^ stride;
                if (j > i && j < NET) {
                    const unsigned a = x[i], b = x[j];
                    x[i] = min(a, b);
                    x[j] = max(a, b);
                }
            }
    }
}

// f(integral constant) with the smallest network size that takes len entries (at most XN).
template <int N> struct NetSize { static constexpr int value = N; };
template <int XN, class F>
__device__ __forceinline__ void by_net_size(unsigned len, F &&f)
{
    if (XN == 8 || len <= 8) f(NetSize<8>{});
    else if (len <= 12) f(NetSize<(XN < 12 ? XN : 12)>{});
    else if (XN == 16 || len <= 16) f(NetSize<(XN < 16 ? XN : 16)>{});
    else if (len <= 20) f(NetSize<(XN < 20 ? XN : 20)>{});
    else if (len <= 24) f(NetSize<(XN < 24 ? XN : 24)>{});
    else f(NetSize<XN>{});
}

// ---- a thread's row staged in shared memory -------------------------------------
// The row's entries are words (key << ROW_IDX | index in the row, a dropped key
// WORD_NONE) with the weights beside them.  The words are sorted in registers, the
// weights of equal keys are summed into the slot of the run's first entry, and the
// unique keys are counted.
constexpr int ROW_IDX = 5;                                    // at most 32 entries
constexpr int32_t ROW_KEY_MAX = (1 << (32 - ROW_IDX)) - 1;    // keys below it fit a word

__device__ __forceinline__ bool same_key(unsigned a, unsigned b) { return (a ^ b) < (1u << ROW_IDX); }

template <int NET, int XN>
__device__ __forceinline__ int sort_staged_row(const unsigned *key, int32_t *wgt, int32_t len, unsigned (&x)[XN])
{
#pragma unroll
    for (int i = 0; i < NET; i++) x[i] = i < len ? key[i] : WORD_NONE;
    sort_words<NET, XN>(x);
    constexpr int Q = NET % 8 == 0 ? 8 : 4;   // weights in flight
    int u = 0;
    int32_t acc = 0;          // weight of the entries after i that have its key
    bool same_next = false;   // entry i + 1 has the key of entry i
#pragma unroll
    for (int b = NET - Q; b >= 0; b -= Q) {
        int32_t w[Q];
#pragma unroll
        for (int q = 0; q < Q; q++) w[q] = wgt[x[b + q] == WORD_NONE ? 0 : x[b + q] & ((1u << ROW_IDX) - 1u)];
#pragma unroll
        for (int q = Q - 1; q >= 0; q--) {
            const int i = b + q;
            const bool same = i > 0 && same_key(x[i], x[i > 0 ? i - 1 : 0]);   // the key of entry i - 1
            const bool valid = x[i] != WORD_NONE;
            acc += w[q];
            if (!same && valid && same_next) wgt[x[i] & ((1u << ROW_IDX) - 1u)] = acc;
            u += valid && !same;
            if (!same) acc = 0;
            same_next = same && valid;
        }
    }
    return u;
}

// The strides below 32 * NR / 2 of a merge over the 32 * NR words of a warp (NR per
// lane), from lane distance m down: m = 16 after a step at 16 * NR across lanes or more.
template <int NR>
__device__ __forceinline__ void warp_merge_words(unsigned (&x)[NR], int m)
{
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (; m > 0; m >>= 1) {
        const bool low = (lane & m) == 0;
#pragma unroll
        for (int r = 0; r < NR; r++) {
            const unsigned a = __shfl_xor_sync(HP_FULL_MASK, x[r], m);
            x[r] = low ? min(x[r], a) : max(x[r], a);
        }
    }
#pragma unroll
    for (int stride = NR >> 1; stride > 0; stride >>= 1)
#pragma unroll
        for (int i = 0; i < NR; i++) {
            const int j = i ^ stride;
            if (j > i) {
                const unsigned a = x[i], b = x[j];
                x[i] = min(a, b);
                x[j] = max(a, b);
            }
        }
}

// The network over NR * L words held by L consecutive lanes of a warp, NR per lane: any
// order in, ascending order out with the group's lane l holding positions l * NR ..
// l * NR + NR - 1.  All lanes of the warp call it; every group of L sorts its own.
template <int NR, int L>
__device__ __forceinline__ void lanes_sort_words(unsigned (&x)[NR])
{
    const int lane = threadIdx.x & 31;
    sort_words<NR, NR>(x);
#pragma unroll 1
    for (int g = 2; g <= L; g <<= 1) {   // merges of g lanes' runs
        const bool low = (lane & (g >> 1)) == 0;
#pragma unroll
        for (int r = 0; r < (NR + 1) / 2; r++) {
            const unsigned a = __shfl_xor_sync(HP_FULL_MASK, x[NR - 1 - r], g - 1);
            const unsigned b = __shfl_xor_sync(HP_FULL_MASK, x[r], g - 1);
            x[r] = low ? min(x[r], a) : max(x[r], a);
            if (NR > 1) x[NR - 1 - r] = low ? min(x[NR - 1 - r], b) : max(x[NR - 1 - r], b);
        }
        warp_merge_words<NR>(x, g >> 2);
    }
}

template <int NR>
__device__ __forceinline__ void warp_sort_words(unsigned (&x)[NR])
{
    lanes_sort_words<NR, 32>(x);
}

// The network over 32 * NR * W words held by a CTA of W warps, thread t holding positions
// t * NR .. t * NR + NR - 1 of the result.  Steps across warps go through buf (33 * NR * W
// words, one pad every 32: a thread's NR consecutive words hit every bank once).
template <int NR, int W>
__device__ __forceinline__ void cta_sort_words(unsigned (&x)[NR], unsigned *buf)
{
    const int t = threadIdx.x, wid = t >> 5;
    warp_sort_words<NR>(x);
#pragma unroll 1
    for (int g = 2; g <= W; g <<= 1) {           // merges of g warps' runs
#pragma unroll 1
        for (int d = g; d >= 2; d >>= 1) {       // mirrored over g warps, then strides of g / 4 .. 1 warps
            const bool mirror = d == g;
            const int other = mirror ? 0 : (d >> 1);
#pragma unroll
            for (int r = 0; r < NR; r++) {
                const int e = t * NR + r;
                buf[e + (e >> 5)] = x[r];
            }
            __syncthreads();
            const bool low = (wid & (d >> 1)) == 0;
#pragma unroll
            for (int r = 0; r < NR; r++) {
                const int e = mirror ? ((t * NR + r) ^ (g * 32 * NR - 1)) : ((t * NR + r) ^ (other * 32 * NR));
                const unsigned a = buf[e + (e >> 5)];
                x[r] = low ? min(x[r], a) : max(x[r], a);
            }
            __syncthreads();
        }
        warp_merge_words<NR>(x, 16);
    }
}

// CTA-wide exclusive scan of one int per thread; returns exclusive value and
// writes the block total to *total.
template <int NT>
__device__ __forceinline__ int block_excl_scan(int v, int *total, int32_t *s_scan)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int incl = warp_incl_scan(v);
    if (lane == 31) s_scan[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        int t = lane < NT / 32 ? s_scan[lane] : 0;
        int ti = warp_incl_scan(t);
        if (lane < NT / 32) s_scan[lane] = ti - t;
        if (lane == NT / 32 - 1) s_scan[NT / 32] = ti;
    }
    __syncthreads();
    int r = s_scan[wid] + incl - v;
    *total = s_scan[NT / 32];
    __syncthreads();
    return r;
}

// Dense aggregation over key space [0, nkeys): dw[nkeys] (zero on entry and on
// exit), bm[(nkeys+31)/32] presence bits (zero on entry and exit).  Entries
// must have been accumulated into dw/bm by the caller (atomics) before the
// barrier that precedes this call.  Writes keys in ascending order.
template <int NT>
__device__ __forceinline__ int dense_extract(int32_t *dw, unsigned *bm, int32_t nkeys,
                                             int32_t *out_k, int32_t *out_w, int32_t *s_scan)
{
    const int nwords = (nkeys + 31) >> 5;
    int running = 0;
    for (int wb = 0; wb < nwords; wb += NT) {
        int wi = wb + threadIdx.x;
        unsigned word = wi < nwords ? bm[wi] : 0u;
        int tot;
        int p = running + block_excl_scan<NT>(__popc(word), &tot, s_scan);
        if (word) {
            bm[wi] = 0u;
            while (word) {
                int b = __ffs(word) - 1;
                word &= word - 1;
                int32_t k = (wi << 5) + b;
                out_k[p] = k;
                out_w[p] = dw[k];
                dw[k] = 0;
                p++;
            }
        }
        running += tot;
    }
    __syncthreads();
    return running;
}

// Two-level variant for large key spaces: bm2[(nwords+31)/32] has one bit per
// non-zero word of bm (set by the accumulating thread that turned the word
// non-zero), so the extraction walks nkeys/1024 words plus the occupied bm
// words instead of all nkeys/32.  dw, bm and bm2 are zero again on exit.
__device__ __forceinline__ void dense_mark2(int32_t *dw, unsigned *bm, unsigned *bm2, int32_t k, int32_t w)
{
    atomicAdd(&dw[k], w);
    const unsigned bit = 1u << (k & 31);
    if (atomicOr(&bm[k >> 5], bit) == 0u) atomicOr(&bm2[k >> 10], 1u << ((k >> 5) & 31));
}

template <int NT>
__device__ __forceinline__ int dense_extract2(int32_t *dw, unsigned *bm, unsigned *bm2, int32_t nkeys,
                                              int32_t *out_k, int32_t *out_w, int32_t *s_scan)
{
    const int nwords = (nkeys + 31) >> 5;
    const int nw2 = (nwords + 31) >> 5;
    int running = 0;
    for (int wb = 0; wb < nw2; wb += NT) {
        const int i2 = wb + threadIdx.x;
        const unsigned top = i2 < nw2 ? bm2[i2] : 0u;
        int cnt = 0;
        for (unsigned t = top; t; t &= t - 1) cnt += __popc(bm[(i2 << 5) + __ffs(t) - 1]);
        int tot;
        int p = running + block_excl_scan<NT>(cnt, &tot, s_scan);
        if (top) {
            bm2[i2] = 0u;
            for (unsigned t = top; t; t &= t - 1) {
                const int wi = (i2 << 5) + __ffs(t) - 1;
                unsigned word = bm[wi];
                bm[wi] = 0u;
                while (word) {
                    const int b = __ffs(word) - 1;
                    word &= word - 1;
                    const int32_t k = (wi << 5) + b;
                    out_k[p] = k;
                    out_w[p] = dw[k];
                    dw[k] = 0;
                    p++;
                }
            }
        }
        running += tot;
    }
    __syncthreads();
    return running;
}


// Stable LSD radix sort of cnt (key, value) pairs by the low key_bits bits of
// the keys (non-negative), by one CTA of NT threads.  Ping-pongs between (K, V)
// and (K2, V2); returns true when the result is in (K2, V2).  Per 8-bit digit: a
// histogram, the digit bases, then chunks of NT items in order, each item placed
// at its digit's base + the same digit's count in earlier warps of the chunk +
// its rank inside its warp (__match_any_sync).  tab: block_sort_ints(NT) ints of
// shared memory; s_scan: NT/32 + 2 ints.
constexpr int block_sort_ints(int nt) { return 256 + (nt / 32) * 256; }

template <int NT>
__device__ bool block_sort_pairs(int32_t *K, int32_t *V, int32_t *K2, int32_t *V2, int32_t cnt, int key_bits,
                                 int32_t *tab, int32_t *s_scan)
{
    constexpr int W = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    int32_t *base = tab, *wc = tab + 256;
    bool flip = false;
    for (int shift = 0; shift < key_bits; shift += 8) {
        const int32_t *ks = flip ? K2 : K, *vs = flip ? V2 : V;
        int32_t *kd = flip ? K : K2, *vd = flip ? V : V2;
        for (int q = tid; q < 256; q += NT) base[q] = 0;
        __syncthreads();
        for (int32_t i = tid; i < cnt; i += NT) atomicAdd(&base[((unsigned)ks[i] >> shift) & 255u], 1);
        __syncthreads();
        const int h = tid < 256 ? base[tid] : 0;
        int tot;
        const int ex = block_excl_scan<NT>(h, &tot, s_scan);   // ends with a barrier
        if (tid < 256) base[tid] = ex;
        for (int32_t c0 = 0; c0 < cnt; c0 += NT) {
            const int32_t i = c0 + tid;
            const bool valid = i < cnt;
            const int32_t key = valid ? ks[i] : 0;
            const unsigned d = valid ? (((unsigned)key >> shift) & 255u) : 256u + lane;
            const unsigned peers = __match_any_sync(HP_FULL_MASK, d);
            const int rank = __popc(peers & lanemask_lt());
            for (int q = tid; q < W * 256; q += NT) wc[q] = 0;
            __syncthreads();
            if (valid && rank == 0) wc[wid * 256 + d] = __popc(peers);
            __syncthreads();
            if (valid) {
                int32_t off = base[d] + rank;
                for (int w = 0; w < wid; w++) off += wc[w * 256 + d];
                kd[off] = key;
                vd[off] = vs[i];
            }
            __syncthreads();
            if (tid < 256) {   // the digit bases move past this chunk
                int32_t c = 0;
                for (int w = 0; w < W; w++) c += wc[w * 256 + tid];
                base[tid] += c;
            }
            __syncthreads();
        }
        flip = !flip;
    }
    __syncthreads();
    return flip;
}

}  // namespace hp
