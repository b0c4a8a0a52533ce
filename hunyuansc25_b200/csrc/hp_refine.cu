// hp_refine.cu — uncoarsening: projection and Jet-style k-way refinement over an
// integer gain table, with exact int64 cut tracking.
//
// Reference behaviour replaced (HunyuanGraph):
//   uncoarsening driver / projection      hunyuangraph_GPU_uncoarsen.h:196-223, 555-587
//   pass loop + best partition            hunyuangraph_GPU_krefine.h:4434-4882
//   gain table (set_gain_offset/val)      :4202-4432, rebuild of neighbours :3632-3726
//   LP: select_dest_part, filter,         :1995-2221
//       afterburner, lock
//   weak rebalance (jetrw)                :3136-3563, gain_bucket :2477-2513
//   strong rebalance (jetrs, cookie cut)  :2515-3135
//   perform_moves + cut change            :3933-4155
// Differences by design: every count/filter is a scan or a block reduction
// instead of atomic append order, bucket order inside a part is (bucket,
// vertex id) via a stable radix sort, the cut is int64, balance is judged
// against integer maximum part weights, and one status read per pass replaces
// the reference's 4-6 blocking reads.
#include <cuda.h>

#include <chrono>
#include <cmath>
#include <cstdlib>

#include "hp_internal.cuh"
#include "hp_mlp.cuh"
#include "hp_rowagg.cuh"

namespace {

// Row classes of refinement (hp_tuning): rows of at most `bigd` entries take a
// thread (or a lane segment), longer rows a warp, and hub rows (more than
// `huged` entries) a CTA or grid-wide chunks.  bigd <= 32, the register
// networks' width.
constexpr int32_t NEG = INT_MIN;

inline unsigned nblk(int64_t n, int b = 256) { return (unsigned)std::max<int64_t>(1, (n + b - 1) / b); }

__global__ void project_kernel(int32_t n, const int32_t *__restrict__ cmap,
                               const int32_t *__restrict__ cwhere, int32_t *__restrict__ where)
{
    hp::pdl_wait();
    int32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n) where[v] = cwhere[cmap[v]];
}

// Gain row of v: (part, connectivity) for every part adjacent to v, ascending
// by part, padded with part -1 up to min(deg, k).  A vertex with deg >= k has a
// dense row instead: entry q is (q, conn to part q), zeros included.  When a neighbour
// moves, a dense row is updated in place by atomics and a sparse one rebuilt; a pass that
// moves much of the level rebuilds both (RebuildRule).
//
// Row capacities min(deg, k); rows longer than bigd go on the big list, rows
// longer than huged (the caller's chunk_deg) also on the long-row list (count
// d_bigcnt[3]), rows longer than hubd (gain_hub_deg) on the hub list (count
// d_bigcnt[4]); d_bigcnt[1] records the longest short row above 8 entries,
// d_bigcnt[2] the longest row above huged.
__global__ void gain_cap_kernel(int32_t n, const int32_t *__restrict__ xadj, int32_t k,
                                int32_t *__restrict__ cap, int32_t *big, int32_t *huge, int32_t *hub,
                                int32_t *d_bigcnt, int32_t bigd, int32_t huged, int32_t hubd)
{
    hp::pdl_wait();
    // no early exit: the list appends and maxima are aggregated per warp
    const int32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    int32_t d = 0;
    if (v < n) {
        d = xadj[v + 1] - xadj[v];
        cap[v] = d < k ? d : k;
    }
    const bool is_big = v < n && d > bigd, is_huge = is_big && d > huged, is_hub = is_big && d > hubd;
    const int32_t pb = hp::warp_append(d_bigcnt, is_big);
    const int32_t ph = hp::warp_append(d_bigcnt + 3, is_huge);
    const int32_t pu = hp::warp_append(d_bigcnt + 4, is_hub);
    if (is_big) big[pb] = v;
    if (is_huge) huge[ph] = v;
    if (is_hub) hub[pu] = v;
    const int32_t hm = hp::warp_max(is_huge ? d : 0);
    const int32_t sm = hp::warp_max(v < n && !is_big && d > 8 ? d : 0);
    if ((threadIdx.x & 31) == 0) {
        if (hm > 0) atomicMax(d_bigcnt + 2, hm);
        if (sm > 0) atomicMax(d_bigcnt + 1, sm);
    }
}

// Degree statistics of a level, computed for every level at the start of
// uncoarsening so that the host chooses each level's kernels without reading
// anything back per level: rows longer than bigd, the longest row of 9..bigd
// entries, the longest row overall, the entries of the rows longer than LOOP_LONG_ROW, and
// the most weighted entries of `range` consecutive rows from a multiple of range on (0: not
// asked for): an entry counts LOOP_UNIT in a row longer than LOOP_LONG_ROW, `weight` in
// others (loop_rows).
struct LevelStat {
    int32_t nbig, small_max, maxdeg, long_entries;
    unsigned long long range_entries;
};
constexpr int32_t LOOP_LONG_ROW = 1024, LOOP_UNIT = 8;

__global__ void __launch_bounds__(256)
level_stats_kernel(int32_t n, const int32_t *__restrict__ xadj, LevelStat *st, int32_t bigd, int32_t range,
                   int32_t weight)
{
    hp::pdl_wait();
    int32_t nbig = 0, smax = 0, dmax = 0, lsum = 0;
    if (range > 0) {   // a warp per range
        const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
        long long rmax = 0;
        for (int64_t v0 = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * range; v0 < n; v0 += nwarps * range) {
            const int64_t v1 = v0 + range < n ? v0 + range : n;
            long long e = 0;
            for (int64_t v = v0 + (threadIdx.x & 31); v < v1; v += 32) {
                const int32_t d = xadj[v + 1] - xadj[v];
                e += (long long)d * (d > LOOP_LONG_ROW ? LOOP_UNIT : weight);
            }
            e = hp::warp_sum64(e);
            rmax = e > rmax ? e : rmax;
        }
        if ((threadIdx.x & 31) == 0 && rmax > 0) atomicMax(&st->range_entries, (unsigned long long)rmax);
    }
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const int32_t d = xadj[v + 1] - xadj[v];
        if (d > bigd) nbig++;
        else if (d > 8) smax = d > smax ? d : smax;
        dmax = d > dmax ? d : dmax;
        lsum += d > LOOP_LONG_ROW ? d : 0;
    }
    nbig = hp::warp_sum(nbig);
    lsum = hp::warp_sum(lsum);
    smax = __reduce_max_sync(HP_FULL_MASK, (unsigned)smax);
    dmax = __reduce_max_sync(HP_FULL_MASK, (unsigned)dmax);
    if ((threadIdx.x & 31) == 0) {
        if (lsum) atomicAdd(&st->long_entries, lsum);
        if (nbig) atomicAdd(&st->nbig, nbig);
        if (smax) atomicMax(&st->small_max, smax);
        if (dmax) atomicMax(&st->maxdeg, dmax);
    }
}

// Full build of the gain rows of at most bigd (<= XN) entries: a tile of GT_TILE
// vertices per CTA, one thread per row.  The tile's entries are staged in shared memory
// with consecutive threads on consecutive entries, every thread sorts and merges its own
// row in registers (sort_staged_row), and the rows are written the same way: sparse rows
// (ascending parts, part -1 padding up to the capacity), or dense ones (entry q = part q)
// where deg >= k.
// A thread that read and wrote its row in place made every access of a warp 32 sectors:
// all levels of RGG 2^24 (k = 1024) 6.3 -> 5.1 ms, of R-MAT scale 22 (with its long rows)
// 7.9 -> 7.1, of the 128^3 grid 0.54 -> 0.41.
constexpr int GT_TILE = 128;

template <int XN>
constexpr size_t gain_tile_smem()
{
    return (sizeof(unsigned) + sizeof(int32_t) + sizeof(uint8_t)) * (size_t)GT_TILE * XN;
}

template <int XN>
__global__ void __launch_bounds__(GT_TILE)
gain_tile_kernel(int32_t n, const int32_t *__restrict__ xadj, const int32_t *__restrict__ adjncy,
                 const int32_t *__restrict__ adjwgt, const int32_t *__restrict__ where,
                 const int32_t *__restrict__ goff, int32_t *__restrict__ gpart, int32_t *__restrict__ gconn,
                 int32_t k, int32_t bigd)
{
    hp::pdl_wait();
    extern __shared__ unsigned gt_words[];                                  // GT_TILE * XN
    int32_t *s_wgt = reinterpret_cast<int32_t *>(gt_words + GT_TILE * XN);   // weights, then run sums
    uint8_t *s_row = reinterpret_cast<uint8_t *>(s_wgt + GT_TILE * XN);      // tile row of each entry
    __shared__ int32_t s_off[GT_TILE];   // staged offset of the row
    __shared__ int32_t s_src[GT_TILE];   // its offset in the adjacency minus the staged one
    __shared__ int32_t s_dst[GT_TILE];   // its offset in the gain table minus the staged one
    __shared__ uint8_t s_cap[GT_TILE];   // its capacity (dense rows: k <= 32)
    __shared__ int32_t s_scan[GT_TILE / 32 + 2];
    const int t = threadIdx.x;
    const int32_t v = blockIdx.x * GT_TILE + t;
    const int32_t b = v < n ? xadj[v] : 0, d = v < n ? xadj[v + 1] - b : 0;
    const int32_t o = v < n ? goff[v] : 0;
    const bool mine = v < n && d <= bigd, dense = d >= k;
    int tin;
    const int off = hp::block_excl_scan<GT_TILE>(mine ? d : 0, &tin, s_scan);
    s_off[t] = off;
    s_src[t] = b - off;
    s_dst[t] = o - off;
    s_cap[t] = (uint8_t)(dense ? k : d);
    if (mine)
        for (int i = 0; i < d; i++) s_row[off + i] = (uint8_t)t;
    __syncthreads();
    for (int f0 = t; f0 < tin; f0 += 8 * GT_TILE) {   // eight entries per thread in flight, then their parts
        int32_t a[8], w[8];
        uint8_t rt[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int f = f0 + q * GT_TILE;
            rt[q] = f < tin ? s_row[f] : 0;
            const int32_t j = s_src[rt[q]] + f;
            a[q] = f < tin ? adjncy[j] : 0;
            w[q] = f < tin ? adjwgt[j] : 0;
        }
        int32_t p[8];
#pragma unroll
        for (int q = 0; q < 8; q++) p[q] = f0 + q * GT_TILE < tin ? where[a[q]] : 0;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int f = f0 + q * GT_TILE;
            if (f >= tin) continue;
            gt_words[f] = ((unsigned)p[q] << hp::ROW_IDX) | (unsigned)(f - s_off[rt[q]]);
            s_wgt[f] = w[q];
        }
    }
    __syncthreads();
    const unsigned wmax = __reduce_max_sync(HP_FULL_MASK, mine ? (unsigned)d : 0u);
    unsigned x[XN];
    hp::by_net_size<XN>(wmax, [&](auto net) {
        constexpr int NET = decltype(net)::value;
        if (!mine) return;
        unsigned *out = gt_words + off;   // the row's own slots (its words are in registers)
        hp::sort_staged_row<NET, XN>(out, s_wgt + off, d, x);
        for (int i = 0; i < d; i++) out[i] = hp::WORD_NONE;
        int r = 0;
#pragma unroll
        for (int i = 0; i < NET; i++) {
            if (x[i] == hp::WORD_NONE || (i > 0 && hp::same_key(x[i], x[i > 0 ? i - 1 : 0]))) continue;
            out[dense ? (int)(x[i] >> hp::ROW_IDX) : r] = x[i];
            r++;
        }
    });
    __syncthreads();
    for (int f = t; f < tin; f += GT_TILE) {
        const int rt = s_row[f], i = f - s_off[rt], cap = s_cap[rt];
        if (i >= cap) continue;
        const unsigned e = gt_words[f];
        const bool none = e == hp::WORD_NONE;
        // an empty slot: padding of a sparse row, a part without connectivity in a dense one
        gpart[s_dst[rt] + f] = none ? (cap == k ? i : -1) : (int32_t)(e >> hp::ROW_IDX);
        gconn[s_dst[rt] + f] = none ? 0 : s_wgt[s_off[rt] + (int)(e & ((1u << hp::ROW_IDX) - 1u))];
    }
}

// Rows of a pass's rebuild.  A pass whose moves touch more than `over` entries of the
// level's adjacency rebuilds every row (apply_moves_kernel then touches none), else
// the rows that the moves queued.
struct RebuildRule {
    const unsigned long long *touch;   // entries of the moved vertices' rows; nullptr: the listed rows
    unsigned long long over;
    __device__ __forceinline__ bool all() const { return touch && *touch > over; }
    // the count of the rows to build, both loads in flight together
    __device__ __forceinline__ int32_t rows(const int32_t *d_count, const int32_t *d_all, bool &a) const
    {
        const int32_t c = *d_count, n = *d_all;
        a = all();
        return a ? n : c;
    }
};

// Rebuild of the listed (dirty) rows of at most S entries (S >= the level's longest
// short row); dirty flags are cleared.  S/4 lanes per row with four entries each, so a
// warp has 128/S rows in flight: the rebuild is bound by its chain of loads (row,
// parts, weights) and exchanges.  The entries are sorted as words (part << ROW_IDX |
// index) by the network of hp::warp_sort_words over the row's lanes, the weights fetched
// by the words' indexes, equal parts summed by a segmented scan.  Rows with deg >= k
// (k <= S here) are written dense.  One entry per lane before: a pass of 41,202 vertices
// (128^3 grid, 16 CTAs) spent 88 us here.
// list == nullptr: every vertex with a row of at most bigd (<= S) entries.
// (warp, nwarps: this warp's index among the nwarps warps sharing the list)
template <int S>
__device__ __forceinline__ void gain_seg_rows(int64_t warp, int64_t nwarps, const int32_t *__restrict__ list,
                                              int32_t cnt, const int32_t *__restrict__ xadj,
                                              const int32_t *__restrict__ adjncy, const int32_t *__restrict__ adjwgt,
                                              const int32_t *__restrict__ where, const int32_t *__restrict__ goff,
                                              int32_t *__restrict__ gpart, int32_t *__restrict__ gconn, int32_t k,
                                              int32_t *__restrict__ dirty, int32_t bigd = 0)
{
    constexpr int L = S / 4, R = 32 / L;   // lanes per row, rows per warp
    const int lane = threadIdx.x & 31, sl = lane & (L - 1);
    for (int64_t i0 = warp * R; i0 < cnt; i0 += nwarps * R) {
        const int64_t i = i0 + lane / L;
        int32_t v = -1, b = 0, d = 0;
        if (i < cnt) {
            v = list ? list[i] : (int32_t)i;
            b = xadj[v];
            d = xadj[v + 1] - b;
            if (list) {
                if (sl == 0) dirty[v] = 0;
            } else if (d > bigd) {
                v = -1;
                d = 0;
            }
        }
        const int32_t o = v >= 0 ? goff[v] : 0;
        int32_t a[4];
#pragma unroll
        for (int q = 0; q < 4; q++) a[q] = sl + q * L < d ? adjncy[b + sl + q * L] : -1;
        unsigned x[4];
#pragma unroll
        for (int q = 0; q < 4; q++)
            x[q] = a[q] >= 0 ? ((unsigned)where[a[q]] << hp::ROW_IDX) | (unsigned)(sl + q * L) : hp::WORD_NONE;
        hp::lanes_sort_words<4, L>(x);   // lane sl: positions 4 sl .. 4 sl + 3
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; q++)
            w[q] = x[q] != hp::WORD_NONE ? (uint32_t)adjwgt[b + (x[q] & ((1u << hp::ROW_IDX) - 1u))] : 0u;
        // w[q]: the weight from entry q to the end of its run -- in the lane, then over
        // the row's lanes (a lane whose entries are all one run passes on what follows it)
        const unsigned nx = __shfl_down_sync(HP_FULL_MASK, x[0], 1, L);
#pragma unroll
        for (int q = 2; q >= 0; q--)
            if (hp::same_key(x[q], x[q + 1])) w[q] += w[q + 1];
        bool open = sl + 1 < L && hp::same_key(x[3], nx);   // the run of entry 3 goes on
        const bool single = hp::same_key(x[0], x[3]);       // (sorted: all four in one run)
        uint32_t head = w[0];           // weight of the lane's first run, as far as scanned
        bool through = single && open;  // it reaches past the lanes scanned so far
        uint32_t carry = 0;             // what follows entry 3 in its run
#pragma unroll
        for (int st = 1; st < L; st <<= 1) {
            const uint32_t h = __shfl_down_sync(HP_FULL_MASK, head, st, L);
            const bool t = __shfl_down_sync(HP_FULL_MASK, (int)through, st, L) != 0;
            if (through) { head += h; through = t; }
        }
        const uint32_t next = __shfl_down_sync(HP_FULL_MASK, head, 1, L);
        if (open) carry = next;
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (carry && hp::same_key(x[q], x[3])) w[q] += carry;
        const unsigned px = __shfl_up_sync(HP_FULL_MASK, x[3], 1, L);
        bool hd[4];
        int u = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const unsigned prev = q > 0 ? x[q > 0 ? q - 1 : 0] : px;
            hd[q] = x[q] != hp::WORD_NONE && ((q == 0 && sl == 0) || !hp::same_key(x[q], prev));
            u += hd[q];
        }
        int incl = u;
#pragma unroll
        for (int st = 1; st < L; st <<= 1) {
            const int t = __shfl_up_sync(HP_FULL_MASK, incl, st, L);
            if (sl >= st) incl += t;
        }
        const int total = __shfl_sync(HP_FULL_MASK, incl, L - 1, L);
        int r = incl - u;
        if (v >= 0 && d >= k) {
            const unsigned mask = (L == 32 ? 0xffffffffu : ((1u << L) - 1u) << (lane & ~(L - 1)));
            for (int32_t q = sl; q < k; q += L) { gpart[o + q] = q; gconn[o + q] = 0; }
            __syncwarp(mask);
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (hd[q]) gconn[o + (x[q] >> hp::ROW_IDX)] = (int32_t)w[q];
        } else if (v >= 0) {
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (hd[q]) {
                    gpart[o + r] = (int32_t)(x[q] >> hp::ROW_IDX);
                    gconn[o + r] = (int32_t)w[q];
                    r++;
                }
            for (int32_t t = total + sl; t < d; t += L) { gpart[o + t] = -1; gconn[o + t] = 0; }
        }
        __syncwarp();
    }
}

template <int S>
__global__ void __launch_bounds__(256)
gain_seg_kernel(const int32_t *__restrict__ list, const int32_t *__restrict__ d_count,
                const int32_t *__restrict__ xadj, const int32_t *__restrict__ adjncy,
                const int32_t *__restrict__ adjwgt, const int32_t *__restrict__ where,
                const int32_t *__restrict__ goff, int32_t *__restrict__ gpart, int32_t *__restrict__ gconn,
                int32_t k, int32_t *__restrict__ dirty, RebuildRule rule, int32_t n, int32_t bigd)
{
    hp::pdl_wait();
    const int32_t cnt = *d_count;
    const bool all = rule.all();
    gain_seg_rows<S>((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5, ((int64_t)gridDim.x * blockDim.x) >> 5,
                     all ? nullptr : list, all ? n : cnt, xadj, adjncy, adjwgt, where, goff, gpart, gconn, k,
                     dirty, bigd);
}

// Gain rows of bigd+1 .. huged entries when k <= warp_dense_k: one warp per
// row with its own dense accumulator and presence bitmap over the k parts in
// shared memory (k + k/32 words per warp), extracted in part order; only warp
// synchronisation.  Longer rows (and any row when k is larger) use
// gain_dense_kernel.
constexpr int GW_WARPS = 8;   // k + k/32 words per warp: 33 KB at k = HP_TUNE_WARP_DENSE_K_MAX

// The rows of one warp: dw (k words) and bm (ceil(k/32) words) are the warp's
// own accumulators, zero on entry and left zero.
__device__ __forceinline__ void gain_bigwarp_rows(int64_t warp, int64_t nwarps, int32_t *dw, unsigned *bm,
                                                  const int32_t *__restrict__ list, int32_t cnt,
                                                  const int32_t *__restrict__ xadj, const int32_t *__restrict__ adjncy,
                                                  const int32_t *__restrict__ adjwgt,
                                                  const int32_t *__restrict__ where, const int32_t *__restrict__ goff,
                                                  int32_t *__restrict__ gpart, int32_t *__restrict__ gconn, int32_t k,
                                                  int32_t *__restrict__ dirty, int32_t bigd, int32_t huged,
                                                  bool in_place = false)
{
    const int lane = threadIdx.x & 31;
    const int nwords = (k + 31) >> 5;
    for (int64_t li = warp; li < cnt; li += nwarps) {
        const int32_t v = list[li];
        const int32_t b = xadj[v], e = xadj[v + 1];
        if (e - b <= bigd || e - b > huged) continue;
        if (dirty && lane == 0) dirty[v] = 0;
        // a row of at least k entries becomes a dense row (entry q = part q):
        // its presence bits are never read
        const bool dense = e - b >= k;
        for (int32_t j = b + lane; j < e; j += 128) {   // four chunks in flight
            int32_t u[4], w[4], q[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const int32_t jj = j + 32 * t;
                u[t] = jj < e ? adjncy[jj] : -1;
                w[t] = jj < e ? adjwgt[jj] : 0;
            }
#pragma unroll
            for (int t = 0; t < 4; t++) q[t] = u[t] >= 0 ? where[u[t]] : -1;   // the four gathers together
#pragma unroll
            for (int t = 0; t < 4; t++) {
                if (q[t] < 0) continue;
                atomicAdd(&dw[q[t]], w[t]);
                if (!dense) atomicOr(&bm[q[t] >> 5], 1u << (q[t] & 31));
            }
        }
        __syncwarp();
        const int32_t o = goff[v], cap = goff[v + 1] - o;
        if (dense) {   // (no presence bits were set; in_place: the parts are there from the level's build)
            for (int32_t q = lane; q < k; q += 32) {
                if (!in_place) gpart[o + q] = q;
                gconn[o + q] = dw[q];
                dw[q] = 0;
            }
            __syncwarp();
            continue;
        }
        int32_t run = 0;
        for (int wb = 0; wb < nwords; wb += 32) {
            const int wi = wb + lane;
            unsigned word = wi < nwords ? bm[wi] : 0u;
            const int c = __popc(word);
            const int incl = hp::warp_incl_scan(c);
            int32_t pos = run + incl - c;
            run += __shfl_sync(HP_FULL_MASK, incl, 31);
            if (word) bm[wi] = 0u;
            while (word) {
                const int bit = __ffs(word) - 1;
                word &= word - 1;
                const int32_t q = (wi << 5) + bit;
                gpart[o + pos] = q;
                gconn[o + pos] = dw[q];
                dw[q] = 0;
                pos++;
            }
        }
        for (int32_t t = run + lane; t < cap; t += 32) { gpart[o + t] = -1; gconn[o + t] = 0; }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(32 * GW_WARPS)
gain_bigwarp_kernel(const int32_t *__restrict__ list, const int32_t *__restrict__ d_count,
                    const int32_t *__restrict__ xadj, const int32_t *__restrict__ adjncy,
                    const int32_t *__restrict__ adjwgt, const int32_t *__restrict__ where,
                    const int32_t *__restrict__ goff, int32_t *__restrict__ gpart,
                    int32_t *__restrict__ gconn, int32_t k, int32_t *__restrict__ dirty, int32_t bigd,
                    int32_t huged, RebuildRule rule, const int32_t *__restrict__ all_list,
                    const int32_t *__restrict__ d_all)
{
    hp::pdl_wait();
    bool all;
    const int32_t cnt = rule.rows(d_count, d_all, all);
    if (all) list = all_list;
    extern __shared__ int32_t gsm[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nwords = (k + 31) >> 5;
    int32_t *dw = gsm + wid * (k + nwords);
    unsigned *bm = (unsigned *)(dw + k);
    for (int i = lane; i < k; i += 32) dw[i] = 0;
    for (int i = lane; i < nwords; i += 32) bm[i] = 0u;
    __syncwarp();
    gain_bigwarp_rows((int64_t)blockIdx.x * GW_WARPS + wid, (int64_t)gridDim.x * GW_WARPS, dw, bm, list, cnt,
                      xadj, adjncy, adjwgt, where, goff, gpart, gconn, k, dirty, bigd, huged, dirty != nullptr);
}

template <int NT>
__global__ void __launch_bounds__(NT)
gain_dense_kernel(const int32_t *__restrict__ list, const int32_t *__restrict__ d_count,
                  const int32_t *__restrict__ xadj, const int32_t *__restrict__ adjncy,
                  const int32_t *__restrict__ adjwgt, const int32_t *__restrict__ where,
                  const int32_t *__restrict__ goff, int32_t *__restrict__ gpart,
                  int32_t *__restrict__ gconn, int32_t k, int32_t *__restrict__ dirty, int32_t bigd,
                  int32_t huged, int32_t warp_dense_k, RebuildRule rule, const int32_t *__restrict__ all_list,
                  const int32_t *__restrict__ d_all)
{
    hp::pdl_wait();
    bool all;
    const int32_t cnt = rule.rows(d_count, d_all, all);
    if (all) list = all_list;
    if (!list || (int32_t)blockIdx.x >= cnt) return;
    extern __shared__ int32_t dsm[];
    __shared__ int32_t s_scan[NT / 32 + 2];
    int32_t *dw = dsm;
    unsigned *bm = (unsigned *)(dsm + k);
    const int nwords = (k + 31) >> 5;
    for (int i = threadIdx.x; i < k; i += NT) dw[i] = 0;
    for (int i = threadIdx.x; i < nwords; i += NT) bm[i] = 0;
    __syncthreads();
    for (int32_t li = blockIdx.x; li < cnt; li += gridDim.x) {
        const int32_t v = list[li];
        const int32_t b = xadj[v], e = xadj[v + 1];
        if (e - b <= bigd) continue;
        if (k <= warp_dense_k && e - b <= huged) continue;   // gain_bigwarp_kernel's rows
        if (dirty && threadIdx.x == 0) dirty[v] = 0;
        // a row of at least k entries becomes a dense row (entry q = part q):
        // its presence bits are never read
        const bool dense = e - b >= k;
        for (int32_t j = b + threadIdx.x; j < e; j += 4 * NT) {   // four entries per thread in flight
            int32_t u[4], w[4], q[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const int32_t jj = j + NT * t;
                u[t] = jj < e ? adjncy[jj] : -1;
                w[t] = jj < e ? adjwgt[jj] : 0;
            }
#pragma unroll
            for (int t = 0; t < 4; t++) q[t] = u[t] >= 0 ? where[u[t]] : -1;
#pragma unroll
            for (int t = 0; t < 4; t++) {
                if (q[t] < 0) continue;
                atomicAdd(&dw[q[t]], w[t]);
                if (!dense) atomicOr(&bm[q[t] >> 5], 1u << (q[t] & 31));
            }
        }
        __syncthreads();
        const int32_t o = goff[v], cap = goff[v + 1] - o;
        if (dense) {
            for (int32_t q = threadIdx.x; q < k; q += NT) {
                if (!dirty) gpart[o + q] = q;
                gconn[o + q] = dw[q];
                dw[q] = 0;
            }
            __syncthreads();
            continue;
        }
        int c = hp::dense_extract<NT>(dw, bm, k, gpart + o, gconn + o, s_scan);
        for (int32_t t = c + threadIdx.x; t < cap; t += NT) { gpart[o + t] = -1; gconn[o + t] = 0; }
        __syncthreads();
    }
}

// Calls f(part, connectivity) for the entries of a gain row up to its padding, in
// order, ROW_BATCH loads of both arrays in flight at a time: a walk that tests every
// entry before it loads the next one pays a memory latency per entry.
constexpr int ROW_BATCH = 4;
template <class F>
__device__ __forceinline__ void row_walk(const int32_t *gpart, const int32_t *gconn, int32_t o, int32_t len, F &&f)
{
    for (int32_t j0 = 0; j0 < len; j0 += ROW_BATCH) {
        int32_t q[ROW_BATCH], c[ROW_BATCH];
#pragma unroll
        for (int t = 0; t < ROW_BATCH; t++) {
            const bool in = j0 + t < len;
            q[t] = in ? gpart[o + j0 + t] : -1;
            c[t] = in ? gconn[o + j0 + t] : 0;
        }
#pragma unroll
        for (int t = 0; t < ROW_BATCH; t++) {
            if (q[t] < 0) return;
            f(q[t], c[t]);
        }
    }
}

// The connectivity to part q in a gain row of len entries (capacity).
__device__ __forceinline__ int32_t row_conn(const int32_t *gp, const int32_t *gc, int32_t len, int32_t q, int32_t k)
{
    if (len == k) return gc[q];   // dense row
    // rows are ascending by part and padded with -1: bisect to a short window
    // (entries before lo are parts below q; entries from hi on are padding or
    // parts >= q), then read the window [lo, hi] at once
    int32_t lo = 0, hi = len;
    while (hi - lo > 7) {
        const int32_t mid = (lo + hi) >> 1;
        const int32_t p = gp[mid];
        if (p >= 0 && p < q) lo = mid + 1;
        else hi = mid;
    }
    int32_t at = -1;
#pragma unroll
    for (int t = 0; t < 8; t++)
        if (lo + t < len && gp[lo + t] == q) at = lo + t;
    return at >= 0 ? gc[at] : 0;
}

// conn(a) - conn(b) in a gain row: the two lookups' loads overlap in dense and in
// short rows.
__device__ __forceinline__ long long row_diff(const int32_t *gp, const int32_t *gc, int32_t len, int32_t a, int32_t b,
                                              int32_t k)
{
    if (len == k) return (long long)gc[a] - gc[b];
    if (len > 12) return (long long)row_conn(gp, gc, len, a, k) - row_conn(gp, gc, len, b, k);
    int32_t ia = -1, ib = -1;
#pragma unroll
    for (int t = 0; t < 12; t++) {
        const int32_t p = t < len ? gp[t] : -1;
        if (p == a) ia = t;   // (a, b >= 0: never the padding)
        if (p == b) ib = t;
    }
    const int32_t ca = ia >= 0 ? gc[ia] : 0, cb = ib >= 0 ? gc[ib] : 0;
    return (long long)ca - cb;
}

__global__ void __launch_bounds__(256)
pw_kernel(int32_t n, const int32_t *__restrict__ where, const int32_t *__restrict__ vwgt,
          unsigned long long *__restrict__ pw, int32_t k)
{
    hp::pdl_wait();
    extern __shared__ unsigned long long spw[];
    const bool use_s = k <= 2048;
    if (use_s) {
        for (int i = threadIdx.x; i < k; i += blockDim.x) spw[i] = 0;
        __syncthreads();
    }
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n;
         v += (int64_t)gridDim.x * blockDim.x) {
        if (use_s) atomicAdd(&spw[where[v]], (unsigned long long)vwgt[v]);
        else atomicAdd(&pw[where[v]], (unsigned long long)vwgt[v]);
    }
    if (use_s) {
        __syncthreads();
        for (int i = threadIdx.x; i < k; i += blockDim.x)
            if (spw[i]) atomicAdd(&pw[i], spw[i]);
    }
}

// 2 x cut from the gain rows.
__global__ void __launch_bounds__(256)
rowcut_kernel(int32_t n, const int32_t *__restrict__ goff, const int32_t *__restrict__ gpart,
              const int32_t *__restrict__ gconn, const int32_t *__restrict__ where,
              unsigned long long *cut2)
{
    hp::pdl_wait();
    const int32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    long long acc = 0;
    int32_t p = 0, o = 0, len = 0;
    if (v < n) {
        p = where[v];
        o = goff[v];
        len = goff[v + 1] - o;
    }
    // rows longer than 32 entries are summed by the whole warp, one at a time
    const bool coop = len > 32;
    if (!coop)
        row_walk(gpart, gconn, o, len, [&](int32_t q, int32_t cq) {
            if (q != p) acc += cq;
        });
    unsigned cm = __ballot_sync(HP_FULL_MASK, coop);
    while (cm) {
        const int src = __ffs(cm) - 1;
        cm &= cm - 1;
        const int32_t so = __shfl_sync(HP_FULL_MASK, o, src), sl = __shfl_sync(HP_FULL_MASK, len, src);
        const int32_t sp = __shfl_sync(HP_FULL_MASK, p, src);
        for (int32_t j = lane; j < sl; j += 32) {
            const int32_t q = gpart[so + j];
            if (q < 0) break;
            if (q != sp) acc += gconn[so + j];
        }
    }
    hp::block_add_to<256>(acc, cut2);
}

// Status of a pass: [0] moves, [1] c1, [2] c2 (as written by kernels),
// [3] max excess (written here).
__global__ void excess_kernel(int32_t k, const unsigned long long *__restrict__ pw,
                              const int64_t *__restrict__ maxp, long long *out)
{
    hp::pdl_wait();
    long long m = LLONG_MIN;
    for (int p = threadIdx.x; p < k; p += blockDim.x) {
        long long e = (long long)pw[p] - maxp[p];
        m = e > m ? e : m;
    }
    m = hp::warp_max64(m);
    __shared__ long long s[32];
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) m = s[w] > m ? s[w] : m;
        *out = m;
    }
}

// One gain row against the own part p: connectivity to p (pc), the best other
// part b (largest connectivity, the first -- lowest -- part among equals; -1
// when no other part has positive connectivity) and bc, the row's total
// connectivity wd and its count np of parts with positive connectivity.
struct RowBest {
    int64_t pc, bc, wd;
    int32_t b, np;
};

// One gain row of more than 32 entries by a whole warp, the result in every lane:
// conn(own), the best other part among those that ok() takes (the first, i.e. lowest,
// of the most connected), the row's weight and its connected parts.  DEPTH loads per
// lane are in flight (ROW_DEEP: a dense row of 256 parts is one batch; walked an entry
// at a time, each load waited for the one before), and the warp reduces by redux.sync:
// the weight and every connectivity are below 2^31.  The launched kernels take ROW_DEEP
// on levels with dense rows of more than 64 parts, where most rows are long (R-MAT scale
// 22, learned: selections 15.8 -> 12.2 ms), and two loads elsewhere: the registers of
// eight cost the short rows' occupancy (RGG 2^24).
constexpr int ROW_DEEP = 8, ROW_FLAT = 2;
template <int DEPTH, class F>
__device__ __forceinline__ RowBest warp_row_best(const int32_t *__restrict__ gpart, const int32_t *__restrict__ gconn,
                                                 int32_t o, int32_t len, int32_t p, int32_t k, F &&ok)
{
    const int lane = threadIdx.x & 31;
    unsigned lpc = 0, lbc = 0, lnp = 0, lwd = 0, lb = 0xffffffffu;
    const bool dense = len == k;   // entry j is part j
    for (int32_t j0 = lane; __any_sync(HP_FULL_MASK, j0 < len); j0 += 32 * DEPTH) {
        int32_t q[DEPTH], c[DEPTH];
#pragma unroll
        for (int i = 0; i < DEPTH; i++) {
            const int32_t j = j0 + 32 * i;
            q[i] = j >= len ? -1 : (dense ? j : gpart[o + j]);
            c[i] = j < len ? gconn[o + j] : 0;
        }
        bool end = false;   // padding runs to the end of the row
#pragma unroll
        for (int i = 0; i < DEPTH; i++) {
            end |= q[i] < 0;
            if (q[i] < 0) continue;
            const unsigned cq = (unsigned)c[i];
            lwd += cq;
            lnp += cq > 0u;
            if (q[i] == p) { lpc = cq; continue; }
            if (cq > lbc && ok(q[i])) { lbc = cq; lb = (unsigned)q[i]; }
        }
        if (__any_sync(HP_FULL_MASK, end)) break;
    }
    RowBest r;
    r.pc = __reduce_add_sync(HP_FULL_MASK, lpc);   // (one lane has it)
    r.np = (int32_t)__reduce_add_sync(HP_FULL_MASK, lnp);
    r.wd = __reduce_add_sync(HP_FULL_MASK, lwd);
    const unsigned m = __reduce_max_sync(HP_FULL_MASK, lbc);
    r.bc = m;
    r.b = (int32_t)__reduce_min_sync(HP_FULL_MASK, lbc == m ? lb : 0xffffffffu);   // none: -1
    return r;
}

// Called by every lane of the warp, each with its own row (len 0 for none).
// Rows of at most 32 entries are walked by their lane; longer rows by the
// whole warp, one row at a time, reduced in the serial walk's order.
__device__ __forceinline__ RowBest row_best(const int32_t *__restrict__ gpart, const int32_t *__restrict__ gconn,
                                            int32_t o, int32_t len, int32_t p, int32_t k)
{
    const int lane = threadIdx.x & 31;
    RowBest r{0, 0, 0, -1, 0};
    const bool coop = len > 32;
    if (!coop)
        row_walk(gpart, gconn, o, len, [&](int32_t q, int32_t cq) {
            r.wd += cq;
            r.np += cq > 0;
            if (q == p) { r.pc = cq; return; }
            if (cq > r.bc) { r.bc = cq; r.b = q; }   // ascending parts: first max = lowest part
        });
    unsigned cm = __ballot_sync(HP_FULL_MASK, coop);
    while (cm) {
        const int src = __ffs(cm) - 1;
        cm &= cm - 1;
        const int32_t so = __shfl_sync(HP_FULL_MASK, o, src), sl = __shfl_sync(HP_FULL_MASK, len, src);
        const int32_t sp = __shfl_sync(HP_FULL_MASK, p, src);
        const RowBest w = warp_row_best<ROW_DEEP>(gpart, gconn, so, sl, sp, k, [](int32_t) { return true; });
        if (lane == src) r = w;
    }
    return r;
}

// The best partition so far, copied by the first proposal kernel of the next
// pass: when the previous pass set the control block's take flag, the partition
// it left is the best so far, and that kernel, which reads where[v] of every
// vertex anyway, stores it into best_where (and block / tile 0 the part weights
// into best_pw) before any move of its own pass is applied.  A pass that ends
// the level needs no copy: where is then either the best (take set) or
// restored from best_where.
struct BestCopy {
    const int32_t *take;
    int32_t *best_where;
    const unsigned long long *pw;
    unsigned long long *best_pw;
    int32_t k;
    __device__ __forceinline__ bool on() const { return *take != 0; }
    __device__ __forceinline__ void parts() const
    {
        for (int32_t q = threadIdx.x; q < k; q += blockDim.x) best_pw[q] = pw[q];
    }
};

// Long gain rows (more than 32 entries) of a CTA, shared by all its warps: the
// rows are queued in shared memory and the warps take them in turn, so that a
// warp with many long rows does not hold the whole CTA at its next barrier
// (the look-back of rb_candidates_kernel, the block sums of the LP selection).
// A row's result does not depend on the warp that walks it.
template <int NT>
struct CoopRows {
    int32_t o[NT], len[NT], p[NT];
    long long pc[NT], bc[NT], wd[NT];
    int32_t b[NT], np[NT];
    int32_t n;
};

// Queues the calling thread's row when it is long; returns its queue slot or -1.
// All NT threads call it; it ends with a barrier.
template <int NT>
__device__ __forceinline__ int coop_queue(CoopRows<NT> &S, bool coop, int32_t o, int32_t len, int32_t p)
{
    if (threadIdx.x == 0) S.n = 0;
    __syncthreads();
    int my = -1;
    if (coop) {
        my = atomicAdd(&S.n, 1);
        S.o[my] = o;
        S.len[my] = len;
        S.p[my] = p;
    }
    __syncthreads();
    return my;
}

// row_best with the CTA's long rows shared by all its warps (CoopRows).  All NT
// threads call it.
template <int NT, int DEPTH>
__device__ __forceinline__ RowBest row_best_cta(CoopRows<NT> &S, const int32_t *__restrict__ gpart,
                                                const int32_t *__restrict__ gconn, int32_t o, int32_t len,
                                                int32_t p, int32_t k)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    RowBest r{0, 0, 0, -1, 0};
    const bool coop = len > 32;
    if (!coop)
        row_walk(gpart, gconn, o, len, [&](int32_t q, int32_t cq) {
            r.wd += cq;
            r.np += cq > 0;
            if (q == p) { r.pc = cq; return; }
            if (cq > r.bc) { r.bc = cq; r.b = q; }   // ascending parts: first max = lowest part
        });
    const int my = coop_queue<NT>(S, coop, o, len, p);
    const int nc = S.n;
    for (int i = wid; i < nc; i += NT / 32) {
        const int32_t so = S.o[i], sl = S.len[i], sp = S.p[i];
        const RowBest w = warp_row_best<DEPTH>(gpart, gconn, so, sl, sp, k, [](int32_t) { return true; });
        if (lane == 0) { S.pc[i] = w.pc; S.bc[i] = w.bc; S.b[i] = w.b; S.wd[i] = w.wd; S.np[i] = w.np; }
    }
    __syncthreads();
    if (my >= 0) { r.pc = S.pc[my]; r.bc = S.bc[my]; r.b = S.b[my]; r.wd = S.wd[my]; r.np = S.np[my]; }
    return r;
}

// ---- LP ------------------------------------------------------------------------
template <int DEPTH>
__global__ void __launch_bounds__(256, DEPTH == ROW_FLAT ? 8 : 5)
lp_select_kernel(int32_t n, const int32_t *__restrict__ goff, const int32_t *__restrict__ gpart,
                 const int32_t *__restrict__ gconn, const int32_t *__restrict__ where,
                 const int8_t *__restrict__ lock, int finest, int32_t *__restrict__ dest,
                 int32_t *__restrict__ pregain, unsigned long long *d_ncand, const int32_t *gate, int32_t k,
                 BestCopy bcp)
{
    hp::pdl_wait();
    if (gate && *gate != 0) return;   // graph mode: the learned kernel runs this pass
    __shared__ CoopRows<256> S;
    const int32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    const bool copy = bcp.on();
    if (copy && blockIdx.x == 0) bcp.parts();
    int cand = 0;
    int32_t p = 0, o = 0, len = 0;
    if (v < n) {
        p = where[v];
        o = goff[v];
        len = goff[v + 1] - o;
        if (copy) bcp.best_where[v] = p;
    }
    const RowBest rb = row_best_cta<256, DEPTH>(S, gpart, gconn, o, len, p, k);
    const int64_t pc = rb.pc, bc = rb.bc;
    const int32_t b = rb.b;
    if (v < n) {
        int32_t g = NEG, d = p;
        if (b >= 0) {
            int64_t thr = finest ? pc / 4 : (3 * pc) / 4;
            if ((bc >= pc || (pc - bc) < thr) && !lock[v]) { g = (int32_t)(bc - pc); d = b; cand = 1; }
        }
        pregain[v] = g;
        dest[v] = d;
    }
    hp::block_add_to<256>(cand, d_ncand);
}

// Learned LP selection: the plain rule first, then the MLP scores every
// candidate (all lanes of a warp run the tensor-core inference together) and
// drops candidates scoring below the threshold.  Dropped candidates stay put;
// under the judge (learned = 3) they keep their plain gain and destination
// with prune[v] = 1, so that the afterburner leaves them out of the learned
// move set but keeps them in the plain set it judges the pass by.  Nothing the
// network says bypasses the exact afterburner.
__global__ void __launch_bounds__(256)
lp_select_learned_kernel(int32_t n, const int32_t *__restrict__ goff, const int32_t *__restrict__ gpart,
                         const int32_t *__restrict__ gconn, const int32_t *__restrict__ where,
                         const int32_t *__restrict__ xadj, const int8_t *__restrict__ lock, int finest,
                         const unsigned long long *__restrict__ pw, const int64_t *__restrict__ maxp,
                         const int64_t *__restrict__ opt, const float *__restrict__ params, float threshold,
                         int32_t *__restrict__ dest, int32_t *__restrict__ pregain, unsigned long long *d_ncand,
                         const int32_t *gate, int32_t k, int8_t *__restrict__ prune,
                         unsigned long long *d_ncandp, const int32_t *judge_flag, BestCopy bcp)
{
    hp::pdl_wait();
    if (gate && *gate != 1) return;   // graph mode: the plain kernel runs this pass
    __shared__ hp::MlpSmem sm;
    __shared__ CoopRows<256> S;
    hp::mlp_load_smem(sm, params);
    __syncthreads();
    const int32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    const bool copy = bcp.on();
    if (copy && blockIdx.x == 0) bcp.parts();
    int cand = 0, candp = 0;
    int8_t pr = 0;
    float f[HP_MLP_IN] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    int32_t g = NEG, d = 0;
    int32_t p = 0, o = 0, len = 0;
    if (v < n) {
        p = where[v];
        o = goff[v];
        len = goff[v + 1] - o;
        if (copy) bcp.best_where[v] = p;
    }
    const RowBest rb = row_best_cta<256, ROW_DEEP>(S, gpart, gconn, o, len, p, k);
    if (v < n) {
        const int64_t pc = rb.pc, bc = rb.bc, wd = rb.wd;
        const int32_t b = rb.b, np = rb.np;
        d = p;
        if (b >= 0) {
            int64_t thr = finest ? pc / 4 : (3 * pc) / 4;
            if ((bc >= pc || (pc - bc) < thr) && !lock[v]) {
                g = (int32_t)(bc - pc);
                d = b;
                cand = 1;
                candp = 1;
                hp::mlp_features(pc, bc, wd, np, xadj[v + 1] - xadj[v], maxp[b] - (int64_t)pw[b], opt[b],
                                 maxp[p] - (int64_t)pw[p], opt[p], finest, f);
            }
        }
    }
    // the warp's tensor-core inference only when one of its vertices is a
    // candidate (the logit is read for candidates alone; the vote is uniform)
    float logit = 0.0f;
    if (__any_sync(HP_FULL_MASK, cand)) logit = hp::mlp_warp_logit(sm, f);
    // under the judge a dropped candidate keeps its plain gain and destination
    const bool judge = *judge_flag != 0;
    if (cand && logit < threshold) {
        cand = 0;
        if (judge) pr = 1;
        else { g = NEG; d = where[v]; }
    }
    if (v < n) {
        pregain[v] = g;
        dest[v] = d;
        if (judge) prune[v] = pr;
    }
    hp::block_add_to<256>(cand, d_ncand);
    if (judge) hp::block_add_to<256>(candp, d_ncandp);
}

// Move log (record mode): features of every LP candidate, its vertex and
// destination; rec_of[v] links the vertex to its record for the afterburner.
__global__ void __launch_bounds__(256)
log_candidates_kernel(int32_t n, const int32_t *__restrict__ goff, const int32_t *__restrict__ gpart,
                      const int32_t *__restrict__ gconn, const int32_t *__restrict__ where,
                      const int32_t *__restrict__ xadj, int finest, const unsigned long long *__restrict__ pw,
                      const int64_t *__restrict__ maxp, const int64_t *__restrict__ opt,
                      const int32_t *__restrict__ dest, const int32_t *__restrict__ pregain,
                      int32_t *__restrict__ rec_of, float *__restrict__ lx, int32_t *__restrict__ lv,
                      int32_t *__restrict__ ld, int32_t *__restrict__ lacc, unsigned long long *lcount, int64_t cap)
{
    hp::pdl_wait();
    int32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    rec_of[v] = -1;
    if (pregain[v] == NEG) return;
    const int32_t p = where[v], b = dest[v];
    int64_t pc = 0, bc = 0, wd = 0;
    int32_t np = 0;
    for (int32_t j = goff[v]; j < goff[v + 1]; j++) {
        int32_t q = gpart[j];
        if (q < 0) break;
        int32_t cq = gconn[j];
        wd += cq;
        np += cq > 0;
        if (q == p) pc = cq;
        if (q == b) bc = cq;
    }
    const unsigned long long r = atomicAdd(lcount, 1ull);
    if ((int64_t)r >= cap) return;
    float f[HP_MLP_IN];
    hp::mlp_features(pc, bc, wd, np, xadj[v + 1] - xadj[v], maxp[b] - (int64_t)pw[b], opt[b],
                     maxp[p] - (int64_t)pw[p], opt[p], finest, f);
    for (int i = 0; i < HP_MLP_IN; i++) lx[r * HP_MLP_IN + i] = f[i];
    lv[r] = v;
    ld[r] = b;
    lacc[r] = 0;
    rec_of[v] = (int32_t)r;
}

__global__ void log_accept_kernel(int32_t n, const int32_t *__restrict__ rec_of, const int8_t *__restrict__ lock,
                                  const unsigned long long *d_ncand, int32_t *__restrict__ lacc)
{
    hp::pdl_wait();
    if (*d_ncand == 0ull) return;
    int32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n && rec_of[v] >= 0) lacc[rec_of[v]] = lock[v];
}

// Label of a record once its level is final: the afterburner accepted the
// move and the vertex ends the level in that destination.
__global__ void log_label_kernel(int64_t r0, int64_t r1, const int32_t *__restrict__ where,
                                 const int32_t *__restrict__ lv, const int32_t *__restrict__ ld,
                                 const int32_t *__restrict__ lacc, float *__restrict__ ly)
{
    hp::pdl_wait();
    int64_t r = r0 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r < r1) ly[r] = (lacc[r] && where[lv[r]] == ld[r]) ? 1.f : 0.f;
}

// Where a pass's moves go: the move list and count, the old part per move, and
// the cut-change sum c1 (conn(to) - conn(from) of every move, read from the mover's
// own gain row before any move applies).  The kernels that decide the moves append
// them through move_append and add the c1 terms per block, so no separate pass
// over the moves precedes their application.  The terms come from the gains the
// selection left in pregain: an LP candidate's is its term; a weak rebalance
// candidate's too (an undersized destination taken for want of a connected one has
// connectivity 0: it would have been connected otherwise); a strong one's is
// -conn(from), to which the destination's connectivity is added (goff .. k).
struct MoveSink {
    int32_t *moves, *oldp;
    unsigned long long *d_nmoves, *d_c1;
    unsigned long long *d_touch;   // adjacency entries of the moved vertices (nullptr: not needed)
    const int32_t *goff, *gpart, *gconn, *xadj;
    int32_t k;
};

// Appends the move of v out of part p.
__device__ __forceinline__ void move_append(const MoveSink &ms, int32_t v, int32_t p)
{
    const unsigned long long i = atomicAdd(ms.d_nmoves, 1ull);
    ms.moves[i] = v;
    ms.oldp[i] = p;
}

// The block's sums over its moves (256 threads).
__device__ __forceinline__ void sink_sums(const MoveSink &ms, long long c1, long long touch)
{
    if (ms.d_touch) hp::block_add2_to<256>(c1, ms.d_c1, touch, ms.d_touch);
    else hp::block_add_to<256>(c1, ms.d_c1);
}

__device__ __forceinline__ long long ab_change(int32_t v, int32_t g, int32_t p, int32_t b,
                                               int32_t u, int32_t w, const int32_t *pregain,
                                               const int32_t *dest, const int32_t *where)
{
    int32_t gu = pregain[u];
    long long ch = 0;
    if (gu > g || (gu == g && u < v)) {
        int32_t du = dest[u], wu = where[u];
        if (du == p) ch -= w;
        else if (du == b) ch += w;
        if (wu == p) ch += w;
        else if (wu == b) ch -= w;
    }
    return ch;
}

// The plain refiner as the judge of a learned LP pass.  In such a pass the
// selection keeps the plain rule's candidates and marks the ones the MLP dropped
// (prune); the afterburner scores every candidate twice in one walk of its row --
// against the higher-priority plain candidates and against the learned ones only
// -- applies the learned decision (lock, moves) and keeps the plain one in accp.
// The vertices that either decision moves are listed (list, *d_n), and
// judge_off_kernel / judge_delta_kernel add both move sets' exact cut changes
// over their rows.  flag: the control block's learned_pass, so the plain
// refiner's passes (and every pass of a plain run) skip all of it.
struct Judge {
    const int32_t *flag;
    const int8_t *prune;
    int8_t *accp;
    int32_t *list, *d_n;
    const unsigned long long *d_ncandp;   // plain candidates of the pass
};

// ab_change of one entry into the plain sum and, when judging, into the sum
// over the learned candidates (a neighbour the MLP dropped stays put there).
__device__ __forceinline__ void ab_change2(int32_t v, int32_t g, int32_t p, int32_t b, int32_t u, int32_t w,
                                           const int32_t *pregain, const int32_t *dest, const int32_t *where,
                                           const int8_t *prune, bool judge, long long &chp, long long &chl)
{
    const long long c = ab_change(v, g, p, b, u, w, pregain, dest, where);
    chp += c;
    if (judge && c != 0 && !prune[u]) chl += c;
}

// ab_row_sum into both sums (chl only when judging).
__device__ __forceinline__ void ab_row_sum2(int32_t v, int32_t g, int32_t p, int32_t b, int32_t j0, int32_t e,
                                            int32_t stride, const int32_t *__restrict__ adjncy,
                                            const int32_t *__restrict__ adjwgt, const int32_t *pregain,
                                            const int32_t *dest, const int32_t *where, const int8_t *prune,
                                            bool judge, long long &chp, long long &chl)
{
    for (int32_t j = j0; j < e; j += 4 * stride) {
        int32_t u[4], w[4], gu[4], du[4], wu[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int32_t jj = j + q * stride;
            const bool in = jj < e;
            u[q] = in ? adjncy[jj] : v;
            w[q] = in ? adjwgt[jj] : 0;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            gu[q] = pregain[u[q]];
            du[q] = dest[u[q]];
            wu[q] = where[u[q]];
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (u[q] == v) continue;   // no entry (rows have no self loops)
            if (gu[q] > g || (gu[q] == g && u[q] < v)) {
                long long c = 0;
                if (du[q] == p) c -= w[q];
                else if (du[q] == b) c += w[q];
                if (wu[q] == p) c += w[q];
                else if (wu[q] == b) c -= w[q];
                chp += c;
                if (judge && c != 0 && !prune[u[q]]) chl += c;
            }
        }
    }
}

// Entries of a short row whose loads are in flight together.  An entry's neighbour was
// looked up before the next entry was loaded: RGG 2^24, a pass of 8,816,196 vertices
// 429 -> 412 us, 4,735,944 252 -> 246.
constexpr int AB_BATCH = 4;

__global__ void __launch_bounds__(256)
afterburner_small_kernel(int32_t n, const int32_t *__restrict__ xadj, const int32_t *__restrict__ adjncy,
                         const int32_t *__restrict__ adjwgt, const int32_t *__restrict__ where,
                         const int32_t *__restrict__ dest, const int32_t *__restrict__ pregain,
                         int8_t *__restrict__ lock, const unsigned long long *d_ncand, MoveSink ms, int32_t bigd,
                         Judge J)
{
    hp::pdl_wait();
    const bool judge = *J.flag != 0;
    if (*d_ncand == 0ull && !(judge && *J.d_ncandp != 0ull)) return;
    const int32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    long long c1 = 0, touch = 0;
    bool listed = false;
    if (v < n) {
        const int32_t b0 = xadj[v], e0 = xadj[v + 1];
        if (e0 - b0 <= bigd) {
            const int32_t g = pregain[v];
            int8_t sel = 0, selp = 0;
            int32_t p = 0, b = 0;
            if (g != NEG) {
                p = where[v];
                b = dest[v];
                long long chp = 0, chl = 0;
                for (int32_t j0 = b0; j0 < e0; j0 += AB_BATCH) {   // the row, then the gains, in flight together
                    int32_t u[AB_BATCH], w[AB_BATCH], gu[AB_BATCH];
#pragma unroll
                    for (int q = 0; q < AB_BATCH; q++) {
                        const bool in = j0 + q < e0;
                        u[q] = in ? adjncy[j0 + q] : v;
                        w[q] = in ? adjwgt[j0 + q] : 0;
                    }
#pragma unroll
                    for (int q = 0; q < AB_BATCH; q++) gu[q] = u[q] != v ? pregain[u[q]] : NEG;
#pragma unroll
                    for (int q = 0; q < AB_BATCH; q++)
                        if (gu[q] > g || (gu[q] == g && u[q] < v))
                            ab_change2(v, g, p, b, u[q], w[q], pregain, dest, where, J.prune, judge, chp, chl);
                }
                selp = ((long long)g + chp >= 0);
                sel = judge ? (int8_t)(!J.prune[v] && (long long)g + chl >= 0) : selp;
            }
            lock[v] = sel;
            if (judge) {
                J.accp[v] = selp;
                listed = sel || selp;
            }
            if (sel) {
                move_append(ms, v, p);
                c1 = g;
                touch = e0 - b0;
            }
        }
    }
    if (judge) {
        const int32_t pos = hp::warp_append(J.d_n, listed);
        if (listed) J.list[pos] = v;
    }
    sink_sums(ms, c1, touch);
}

__global__ void __launch_bounds__(256)
afterburner_big_kernel(const int32_t *__restrict__ big, const int32_t *__restrict__ d_bigcnt,
                       const int32_t *__restrict__ xadj, const int32_t *__restrict__ adjncy,
                       const int32_t *__restrict__ adjwgt, const int32_t *__restrict__ where,
                       const int32_t *__restrict__ dest, const int32_t *__restrict__ pregain,
                       int8_t *__restrict__ lock, const unsigned long long *d_ncand, MoveSink ms,
                       int32_t chunkd, Judge J)
{
    hp::pdl_wait();
    const bool judge = *J.flag != 0;
    if (*d_ncand == 0ull && !(judge && *J.d_ncandp != 0ull)) return;
    const int lane = threadIdx.x & 31;
    const int32_t cnt = *d_bigcnt;
    long long c1 = 0, touch = 0;
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; i < cnt;
         i += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int32_t v = big[i];
        if (xadj[v + 1] - xadj[v] > chunkd) continue;   // chunked over the grid
        const int32_t g = pregain[v];
        int8_t sel = 0, selp = 0;
        int32_t p = 0, b = 0;
        if (g != NEG) {
            p = where[v];
            b = dest[v];
            long long chp = 0, chl = 0;
            ab_row_sum2(v, g, p, b, xadj[v] + lane, xadj[v + 1], 32, adjncy, adjwgt, pregain, dest, where, J.prune,
                        judge, chp, chl);
            chp = hp::warp_sum64(chp);
            selp = ((long long)g + chp >= 0);
            if (judge) {
                chl = hp::warp_sum64(chl);
                sel = (int8_t)(!J.prune[v] && (long long)g + chl >= 0);
            } else {
                sel = selp;
            }
        }
        if (lane == 0) {
            lock[v] = sel;
            if (judge) {
                J.accp[v] = selp;
                if (sel || selp) J.list[atomicAdd(J.d_n, 1)] = v;
            }
            if (sel) {
                move_append(ms, v, p);
                c1 += g;
                touch += xadj[v + 1] - xadj[v];
            }
        }
    }
    sink_sums(ms, c1, touch);
}

// ---- long rows (longer than chunk_deg): chunk plans ------------------------------
// The afterburner and move application of rows longer than the tuning's
// chunk_deg are cut into chunks of HUB_CHUNK entries dealt over the whole grid,
// so that no warp walks a long row alone.  A plan per pass selects the rows that
// have work (afterburner: candidates; moves: moved rows) and writes each one's
// vertex, its item (list position or move index) and the exclusive prefix of
// the chunk counts, so that a chunk finds its row by a binary search.  The plan
// is one pass of persistent CTAs over tiles of PLAN_TILE items with two epoch
// look-back chains (selected rows: tile words [0, half); chunks: [half, 2 half)).
constexpr int HUB_CHUNK = 512;
constexpr int PLAN_THREADS = 256, PLAN_ITEMS = 4, PLAN_TILE = PLAN_THREADS * PLAN_ITEMS;

template <bool MOVES>
__global__ void __launch_bounds__(PLAN_THREADS)
hub_plan_kernel(const int32_t *__restrict__ items, const int32_t *__restrict__ d_nitems,
                const int32_t *__restrict__ moves, const int32_t *__restrict__ pregain,
                const int32_t *__restrict__ xadj, int32_t *__restrict__ plan_v, int32_t *__restrict__ plan_item,
                int32_t *__restrict__ plan_off, int32_t *__restrict__ d_plan, unsigned long long *tile_status,
                int64_t half, hp::LbCtl *lb, unsigned *status)
{
    hp::pdl_wait();
    __shared__ int32_t s_scan[PLAN_THREADS / 32 + 2];
    __shared__ int32_t s_excl[2];
    const unsigned epoch = hp::lb_epoch(lb);
    const int32_t ni = *d_nitems;
    for (;;) {
        const int64_t tile = hp::lb_next(lb);
        const int64_t base = tile * PLAN_TILE;
        if (base > ni) break;   // the tile holding index ni (it writes the totals) was the last
        const int64_t t0 = base + (int64_t)threadIdx.x * PLAN_ITEMS;
        int32_t v[PLAN_ITEMS], c[PLAN_ITEMS];
        int32_t ns = 0, nc = 0;
#pragma unroll
        for (int q = 0; q < PLAN_ITEMS; q++) {
            const int64_t t = t0 + q;
            v[q] = -1;
            c[q] = 0;
            if (t < ni) {
                const int32_t vv = MOVES ? moves[items[t]] : items[t];
                if (MOVES || pregain[vv] != NEG) {
                    v[q] = vv;
                    c[q] = (xadj[vv + 1] - xadj[vv] + HUB_CHUNK - 1) / HUB_CHUNK;
                }
            }
            ns += v[q] >= 0;
            nc += c[q];
        }
        int ts, tc;
        int32_t ps = hp::block_excl_scan<PLAN_THREADS>(ns, &ts, s_scan);
        int32_t pc = hp::block_excl_scan<PLAN_THREADS>(nc, &tc, s_scan);
        if (threadIdx.x < 32) {
            const int32_t ex = hp::lookback_epoch(tile_status, tile, ts, epoch, status);
            if (threadIdx.x == 0) s_excl[0] = ex;
        } else if (threadIdx.x < 64) {
            const int32_t ex = hp::lookback_epoch(tile_status + half, tile, tc, epoch, status);
            if (threadIdx.x == 32) s_excl[1] = ex;
        }
        __syncthreads();
        ps += s_excl[0];
        pc += s_excl[1];
#pragma unroll
        for (int q = 0; q < PLAN_ITEMS; q++) {
            if (v[q] >= 0) {
                plan_v[ps] = v[q];
                plan_item[ps] = MOVES ? items[t0 + q] : (int32_t)(t0 + q);
                plan_off[ps] = pc;
                ps++;
            }
            pc += c[q];
        }
        if (ni >= base && ni < base + PLAN_TILE && threadIdx.x == 0) {
            d_plan[0] = s_excl[0] + ts;
            d_plan[1] = s_excl[1] + tc;
        }
    }
    hp::lb_end(lb);
}

// chunk gc -> selected hub j (the last j with plan_off[j] <= gc)
__device__ __forceinline__ int32_t plan_find(const int32_t *__restrict__ plan_off, int32_t nsel, int64_t gc)
{
    int32_t lo = 0, hi = nsel - 1;
    while (lo < hi) {
        const int32_t mid = (lo + hi + 1) >> 1;
        if (plan_off[mid] <= gc) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Afterburner of the candidate hubs: every chunk adds its part of the change to
// the hub's accumulator (ab_acc, indexed by hub-list position, zero on entry;
// ab_acc2 the learned candidates' sum when judging);
// afterburner_huge_final_kernel then decides from the full sums.
__global__ void __launch_bounds__(HUB_CHUNK)
afterburner_huge_kernel(const int32_t *__restrict__ plan_v, const int32_t *__restrict__ plan_item,
                        const int32_t *__restrict__ plan_off, const int32_t *__restrict__ d_plan,
                        const int32_t *__restrict__ xadj, const int32_t *__restrict__ adjncy,
                        const int32_t *__restrict__ adjwgt, const int32_t *__restrict__ where,
                        const int32_t *__restrict__ dest, const int32_t *__restrict__ pregain,
                        const unsigned long long *d_ncand, unsigned long long *__restrict__ ab_acc,
                        unsigned long long *__restrict__ ab_acc2, Judge J)
{
    hp::pdl_wait();
    const bool judge = *J.flag != 0;
    if (*d_ncand == 0ull && !(judge && *J.d_ncandp != 0ull)) return;
    const int lane = threadIdx.x & 31;
    const int32_t nsel = d_plan[0], nch = d_plan[1];
    for (int64_t gc = blockIdx.x; gc < nch; gc += gridDim.x) {
        const int32_t jp = plan_find(plan_off, nsel, gc);
        const int32_t v = plan_v[jp];
        const int32_t g = pregain[v], p = where[v], b = dest[v];
        const int32_t e0 = xadj[v + 1];
        const int32_t j = xadj[v] + (int32_t)(gc - plan_off[jp]) * HUB_CHUNK + threadIdx.x;
        long long cp = 0, cl = 0;
        if (j < e0) ab_change2(v, g, p, b, adjncy[j], adjwgt[j], pregain, dest, where, J.prune, judge, cp, cl);
        cp = hp::warp_sum64(cp);
        if (judge) cl = hp::warp_sum64(cl);
        if (lane == 0 && cp != 0) atomicAdd(&ab_acc[plan_item[jp]], (unsigned long long)cp);
        if (lane == 0 && cl != 0) atomicAdd(&ab_acc2[plan_item[jp]], (unsigned long long)cl);
    }
}

__global__ void afterburner_huge_final_kernel(const int32_t *__restrict__ huge, const int32_t *__restrict__ d_nhuge,
                                              const int32_t *__restrict__ pregain, const unsigned long long *d_ncand,
                                              unsigned long long *__restrict__ ab_acc,
                                              unsigned long long *__restrict__ ab_acc2, int8_t *__restrict__ lock,
                                              const int32_t *__restrict__ where, const int32_t *__restrict__ dest,
                                              MoveSink ms, Judge J)
{
    hp::pdl_wait();
    const bool judge = *J.flag != 0;
    if (*d_ncand == 0ull && !(judge && *J.d_ncandp != 0ull)) return;
    const int32_t nh = *d_nhuge;
    long long c1 = 0, touch = 0;
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nh; i += gridDim.x * blockDim.x) {
        const int32_t v = huge[i];
        const int32_t g = pregain[v];
        const long long totp = (long long)ab_acc[i];
        ab_acc[i] = 0ull;
        const int8_t selp = (g != NEG) && ((long long)g + totp >= 0);
        int8_t sel = selp;
        if (judge) {
            const long long totl = (long long)ab_acc2[i];
            ab_acc2[i] = 0ull;
            sel = (g != NEG) && !J.prune[v] && ((long long)g + totl >= 0);
            J.accp[v] = selp;
            if (sel || selp) J.list[atomicAdd(J.d_n, 1)] = v;
        }
        lock[v] = sel;
        if (sel) {
            move_append(ms, v, where[v]);
            c1 += g;
            if (ms.d_touch) touch += ms.xadj[v + 1] - ms.xadj[v];
        }
    }
    sink_sums(ms, c1, touch);
}

// ---- the judge's exact cut changes ---------------------------------------------------
// Over the listed vertices' entries (tiles of JD_TILE, owner rows from the
// prefix): twice the exact cut decrease of the plain move set (accp) into
// sums[0] and of the learned one (lock) into sums[1].  An entry (v, u, w) of a
// moved v counts w ([p_v != p_u] - [d_v != new p_u]), twice when u stays put
// and once when u moves too (then its row counts the edge again).
constexpr int JD_THREADS = 256, JD_ITEMS = 8, JD_TILE = JD_THREADS * JD_ITEMS;

// One entry (v, u, w) of a listed vertex v (part pv, destination dv; apv / alv:
// v moves in the plain / learned set) into the two sums.
__device__ __forceinline__ void judge_entry(int32_t pv, int32_t dv, bool apv, bool alv, int32_t u, int32_t w,
                                            const int32_t *where, const int32_t *dest, const int8_t *accp,
                                            const int8_t *lock, long long &sp, long long &sl)
{
    const int32_t pu = where[u];
    const bool apu = accp[u] != 0, alu = lock[u] != 0;
    const int32_t du = (apu || alu) ? dest[u] : pu;
    const long long before = pv != pu;
    if (apv) sp += (long long)w * (before - (dv != (apu ? du : pu))) * (apu ? 1 : 2);
    if (alv) sl += (long long)w * (before - (dv != (alu ? du : pu))) * (alu ? 1 : 2);
}

__global__ void __launch_bounds__(JD_THREADS)
judge_delta_kernel(const int32_t *flag, const int32_t *__restrict__ list, const int32_t *d_n,
                   const int32_t *__restrict__ off, const int32_t *__restrict__ xadj,
                   const int32_t *__restrict__ adjncy, const int32_t *__restrict__ adjwgt,
                   const int32_t *__restrict__ where, const int32_t *__restrict__ dest,
                   const int8_t *__restrict__ accp, const int8_t *__restrict__ lock, unsigned long long *sums)
{
    hp::pdl_wait();
    __shared__ int32_t owner[JD_TILE];
    __shared__ int32_t s_warp[JD_THREADS / 32];
    __shared__ int32_t s_v0;
    if (*flag == 0) return;
    const int32_t cnt = *d_n;
    if (cnt <= 0) return;
    const int64_t tot = off[cnt];
    long long sp = 0, sl = 0;
    for (int64_t tb = (int64_t)blockIdx.x * JD_TILE; tb < tot; tb += (int64_t)gridDim.x * JD_TILE) {
        const int64_t te = tb + JD_TILE < tot ? tb + JD_TILE : tot;
        hp::tile_owners<JD_THREADS, JD_ITEMS>(off, cnt, tb, te, owner, s_warp, &s_v0);
        for (int64_t t = tb + threadIdx.x; t < te; t += JD_THREADS) {
            const int32_t i = owner[t - tb];
            const int32_t v = list[i];
            const int32_t j = xadj[v] + (int32_t)(t - off[i]);
            judge_entry(where[v], dest[v], accp[v] != 0, lock[v] != 0, adjncy[j], adjwgt[j], where, dest, accp, lock,
                        sp, sl);
        }
        __syncthreads();   // owner[] is rebuilt for the next tile
    }
    hp::block_add_to<JD_THREADS>(sp, &sums[0]);
    hp::block_add_to<JD_THREADS>(sl, &sums[1]);
}

// ---- applying moves -------------------------------------------------------------
// Effect of one move on its neighbours' gain rows.  A vertex's own row does
// not depend on its own part: only neighbours' rows change.  Dense neighbour
// rows (deg >= k) take the change in place; a sparse neighbour is queued once
// (atomicExch on its dirty flag) on the small or big rebuild list.
// o and cap: the neighbour's gain-row offset and capacity (goff[u], goff[u+1] - o),
// loaded by the caller.
__device__ __forceinline__ void touch_neighbour(bool valid, int32_t u, int32_t w, int32_t o, int32_t cap, int32_t p,
                                                int32_t d, const int32_t *__restrict__ xadj,
                                                int32_t *__restrict__ gconn, int32_t *__restrict__ dirty,
                                                int32_t *__restrict__ small_l, int32_t *__restrict__ big_l,
                                                int32_t *counts, int32_t k, int32_t bigd)
{
    // all 32 lanes call (valid marks the lanes with a neighbour); list appends
    // take one counter atomic per warp and list (ballot ranks inside the warp)
    bool sm = false, bg = false;
    if (valid) {
        if (cap == k) {
            atomicAdd(&gconn[o + p], -w);
            atomicAdd(&gconn[o + d], w);
        } else if (__ldcg(&dirty[u]) == 0 && atomicExch(&dirty[u], 1) == 0) {
            // (a row already queued in this pass is skipped without an atomic;
            // flags only go from 0 to 1 inside the kernel)
            if (xadj[u + 1] - xadj[u] > bigd) bg = true;
            else sm = true;
        }
    }
    const unsigned lt = hp::lanemask_lt();
    const unsigned ms = __ballot_sync(HP_FULL_MASK, sm), mb = __ballot_sync(HP_FULL_MASK, bg);
    const int lane = threadIdx.x & 31;
    int32_t bs = 0, bb = 0;
    if (lane == 0) {
        if (ms) bs = atomicAdd(&counts[0], __popc(ms));
        if (mb) bb = atomicAdd(&counts[1], __popc(mb));
    }
    bs = __shfl_sync(HP_FULL_MASK, bs, 0);
    bb = __shfl_sync(HP_FULL_MASK, bb, 0);
    if (sm) small_l[bs + __popc(ms & lt)] = u;
    if (bg) big_l[bb + __popc(mb & lt)] = u;
}

// One warp per move (warp, nwarps: this warp among those sharing the moves).
__device__ __forceinline__ void apply_moves_rows(int64_t warp, int64_t nwarps, const int32_t *__restrict__ moves,
                                                 int64_t nm, int32_t *__restrict__ where,
                                                 const int32_t *__restrict__ dest, const int32_t *__restrict__ vwgt,
                                                 unsigned long long *__restrict__ pw, const int32_t *__restrict__ xadj,
                                                 const int32_t *__restrict__ adjncy,
                                                 const int32_t *__restrict__ adjwgt, const int32_t *__restrict__ goff,
                                                 int32_t *__restrict__ gconn, int32_t *__restrict__ dirty,
                                                 int32_t *__restrict__ small_l, int32_t *__restrict__ big_l,
                                                 int32_t *counts, int32_t k, int32_t *__restrict__ huge_mv,
                                                 int32_t *__restrict__ d_nhuge, int32_t bigd, int32_t chunkd)
{
    const int lane = threadIdx.x & 31;
    for (int64_t i = warp; i < nm; i += nwarps) {
        const int32_t v = moves[i];
        const int32_t p = where[v], d = dest[v];
        __syncwarp();
        if (lane == 0) {
            const unsigned long long w = (unsigned long long)vwgt[v];
            atomicAdd(&pw[d], w);
            atomicAdd(&pw[p], (unsigned long long)(-(long long)w));
        }
        const int32_t b = xadj[v], e = xadj[v + 1];
        if (e - b > chunkd) {
            // neighbours of a hub are touched by apply_moves_huge_kernel, spread
            // over the whole grid (it reads the old part from oldp)
            if (lane == 0) {
                huge_mv[atomicAdd(d_nhuge, 1)] = (int32_t)i;
                where[v] = d;
            }
            continue;
        }
        // four chunks of 32 entries at a time: row loads, then the neighbours'
        // gain-row offsets, are in flight together
        for (int32_t j0 = b; j0 < e; j0 += 128) {
            int32_t u[4], w[4], o[4], cap[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int32_t j = j0 + 32 * q + lane;
                const bool valid = j < e;
                u[q] = valid ? adjncy[j] : -1;
                w[q] = valid ? adjwgt[j] : 0;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                o[q] = u[q] >= 0 ? goff[u[q]] : 0;
                cap[q] = u[q] >= 0 ? goff[u[q] + 1] - o[q] : 0;
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
                touch_neighbour(u[q] >= 0, u[q], w[q], o[q], cap[q], p, d, xadj, gconn, dirty, small_l, big_l, counts,
                                k, bigd);
        }
        if (lane == 0) where[v] = d;   // the move itself (every lane has read where[v])
    }
}

__global__ void __launch_bounds__(256)
apply_moves_kernel(const int32_t *__restrict__ moves, const unsigned long long *d_nmoves,
                   int32_t *__restrict__ where, const int32_t *__restrict__ dest,
                   const int32_t *__restrict__ vwgt, unsigned long long *__restrict__ pw,
                   const int32_t *__restrict__ xadj, const int32_t *__restrict__ adjncy,
                   const int32_t *__restrict__ adjwgt, const int32_t *__restrict__ goff,
                   int32_t *__restrict__ gconn, int32_t *__restrict__ dirty, int32_t *__restrict__ small_l,
                   int32_t *__restrict__ big_l, int32_t *counts, int32_t k, int32_t *__restrict__ huge_mv,
                   int32_t *__restrict__ d_nhuge, int32_t bigd, int32_t chunkd, RebuildRule rule)
{
    hp::pdl_wait();
    const int64_t nm = (int64_t)*d_nmoves;
    if (rule.all()) {   // the rebuild takes every row: only the moves themselves
        for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nm; i += (int64_t)gridDim.x * blockDim.x) {
            const int32_t v = moves[i];
            const int32_t p = where[v], d = dest[v];
            const unsigned long long w = (unsigned long long)vwgt[v];
            atomicAdd(&pw[d], w);
            atomicAdd(&pw[p], (unsigned long long)(-(long long)w));
            where[v] = d;
        }
        return;
    }
    apply_moves_rows((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5, ((int64_t)gridDim.x * blockDim.x) >> 5,
                     moves, nm, where, dest, vwgt, pw, xadj, adjncy, adjwgt, goff, gconn, dirty,
                     small_l, big_l, counts, k, huge_mv, d_nhuge, bigd, chunkd);
}

// Neighbours of the moved hubs (queued by apply_moves_kernel, planned by
// hub_plan_kernel<true>): chunks of HUB_CHUNK entries over the whole grid.  A
// hub's old part comes from oldp (the hub itself is already committed).
__global__ void __launch_bounds__(HUB_CHUNK)
apply_moves_huge_kernel(const int32_t *__restrict__ plan_v, const int32_t *__restrict__ plan_item,
                        const int32_t *__restrict__ plan_off, const int32_t *__restrict__ d_plan,
                        const int32_t *__restrict__ oldp, const int32_t *__restrict__ dest,
                        const int32_t *__restrict__ xadj, const int32_t *__restrict__ adjncy,
                        const int32_t *__restrict__ adjwgt, const int32_t *__restrict__ goff,
                        int32_t *__restrict__ gconn, int32_t *__restrict__ dirty, int32_t *__restrict__ small_l,
                        int32_t *__restrict__ big_l, int32_t *counts, int32_t k, int32_t bigd)
{
    hp::pdl_wait();
    const int32_t nsel = d_plan[0], nch = d_plan[1];
    for (int64_t gc = blockIdx.x; gc < nch; gc += gridDim.x) {
        const int32_t jp = plan_find(plan_off, nsel, gc);
        const int32_t v = plan_v[jp];
        const int32_t p = oldp[plan_item[jp]], d = dest[v];
        const int32_t e = xadj[v + 1];
        const int32_t j = xadj[v] + (int32_t)(gc - plan_off[jp]) * HUB_CHUNK + threadIdx.x;
        const bool valid = j < e;
        const int32_t u = valid ? adjncy[j] : 0;
        const int32_t o = valid ? goff[u] : 0, cap = valid ? goff[u + 1] - o : 0;
        touch_neighbour(valid, u, valid ? adjwgt[j] : 0, o, cap, p, d, xadj, gconn, dirty, small_l, big_l, counts, k,
                        bigd);
    }
}

// ---- rebalancing ------------------------------------------------------------------
// Undersized parts (pw < max(0.99 maxp, maxp - 100)) in part order; one CTA.
__device__ __forceinline__ void undersized_block(int32_t k, const unsigned long long *__restrict__ pw,
                                                 const int64_t *__restrict__ maxp, int32_t *__restrict__ und,
                                                 int32_t *d_nu, int32_t *s_scan /* 1024/32 + 2 */)
{
    int running = 0;
    for (int base = 0; base < k; base += 1024) {
        int p = base + threadIdx.x;
        int f = 0;
        if (p < k) {
            int64_t md = (maxp[p] * 99) / 100;
            if (md < maxp[p] - 100) md = maxp[p] - 100;
            f = (int64_t)pw[p] < md;
        }
        int tot;
        int pos = running + hp::block_excl_scan<1024>(f, &tot, s_scan);
        if (f) und[pos] = p;
        running += tot;
    }
    if (threadIdx.x == 0) *d_nu = running;
}

// Rebalance candidates of a pass in one ordered pass over the vertices, tiles
// of RB_TILE in launch order with an epoch look-back: the key (part * 64 + gain
// bucket) of every candidate, compacted in vertex order into K/V, the count
// into *d_cnt, and dest[v] for every vertex (the proposed part, or its own).
//   weak  (jetrw, hunyuangraph_GPU_krefine.h:3381-3563): v in an overweight part
//         with 2 vwgt < 3 (pw - opt); destination = most connected part that
//         is not overweight (first max in part order), else an undersized part
//         (und[v % nu]); gain = conn(dest) - conn(own)
//   strong (jetrs, :2774-3135): v in an overweight part with vwgt < 2 (pw - opt);
//         loss = -conn(own)
constexpr int RB_TILE = 256;
constexpr int RB_COOP = 32;   // weak rebalance: longer gain rows are walked by a warp

template <bool STRONG, int DEPTH>
__global__ void __launch_bounds__(RB_TILE)
rb_candidates_kernel(int32_t n, const int32_t *__restrict__ where, const int32_t *__restrict__ vwgt,
                     const unsigned long long *__restrict__ pw, const int64_t *__restrict__ maxp,
                     const int64_t *__restrict__ opt, const int32_t *__restrict__ goff,
                     const int32_t *__restrict__ gpart, const int32_t *__restrict__ gconn,
                     const int32_t *__restrict__ und, const int32_t *__restrict__ d_nu, int32_t k,
                     int32_t *__restrict__ K, int32_t *__restrict__ V, int32_t *__restrict__ dest,
                     int32_t *__restrict__ d_cnt, unsigned long long *tile_status, hp::LbCtl *lb, unsigned *status,
                     const int8_t *__restrict__ ufl, int32_t *__restrict__ pregain, BestCopy bcp)
{
    hp::pdl_wait();
    __shared__ int32_t s_scan[RB_TILE / 32 + 2];
    __shared__ int32_t s_excl;
    __shared__ CoopRows<RB_TILE> S;
    int64_t tile;
    unsigned epoch;
    hp::lb_begin(lb, &tile, &epoch);
    const int64_t v64 = tile * RB_TILE + threadIdx.x;
    const int lane = threadIdx.x & 31;
    int32_t kk = -1;
    const bool in = v64 < n;
    const int32_t v = in ? (int32_t)v64 : 0;
    int32_t p = 0;
    bool cand = false;   // in an overweight part and light enough to leave it
    const bool copy = bcp.on();
    if (copy && tile == 0) bcp.parts();
    if (in) {
        p = where[v];
        if (copy) bcp.best_where[v] = p;
        const int64_t pwp = (int64_t)pw[p];
        cand = STRONG ? (pwp > maxp[p] && (int64_t)vwgt[v] < 2 * (pwp - opt[p]))
                      : (pwp > maxp[p] && 2 * (int64_t)vwgt[v] < 3 * (pwp - opt[p]));
    }
    const int32_t o = cand ? goff[v] : 0, len = cand ? goff[v + 1] - o : 0;
    int32_t d = p, gain = 0;
    if (!STRONG) {
        // best underweight part by connectivity (first, i.e. lowest part, among
        // equals) and the connectivity to the own part; rows of more than
        // RB_COOP entries are walked by a whole warp, any warp of the CTA
        int64_t pc = 0, bc = 0;
        int32_t b = -1;
        const bool coop = cand && len > RB_COOP;
        if (cand && !coop) {
            row_walk(gpart, gconn, o, len, [&](int32_t q, int32_t cq) {
                if (q == p) pc = cq;
                if (cq > bc && ufl[q]) { bc = cq; b = q; }
            });
        }
        // the CTA's long rows, shared by all its warps
        const int my = coop_queue<RB_TILE>(S, coop, o, len, p);
        const int nc = S.n;
        for (int i = threadIdx.x >> 5; i < nc; i += RB_TILE / 32) {
            const int32_t so = S.o[i], sl = S.len[i], sp = S.p[i];
            const RowBest w = warp_row_best<DEPTH>(gpart, gconn, so, sl, sp, k, [&](int32_t q) { return ufl[q] != 0; });
            if (lane == 0) { S.pc[i] = w.pc; S.bc[i] = w.bc; S.b[i] = w.b; }
        }
        __syncthreads();
        if (my >= 0) { pc = S.pc[my]; bc = S.bc[my]; b = S.b[my]; }
        if (cand) {
            int64_t g = 0;
            bool ok = true;
            if (b >= 0) g = bc - pc;
            else {
                const int32_t nu = *d_nu;
                if (nu == 0) ok = false;
                else { b = und[v % nu]; g = -pc; }
            }
            if (ok) { d = b; gain = (int32_t)g; kk = p * 64 + hp::gain_bucket(gain, vwgt[v]); }
        }
    } else if (cand) {
        gain = -row_conn(gpart + o, gconn + o, len, p, k);
        kk = p * 64 + hp::gain_bucket(gain, vwgt[v]);
    }
    if (in) dest[v] = d;
    if (kk >= 0) pregain[v] = gain;   // the move's c1 term (MoveSink)
    int tot;
    const int local = hp::block_excl_scan<RB_TILE>(kk >= 0 ? 1 : 0, &tot, s_scan);
    if (threadIdx.x < 32) {
        const int32_t ex = hp::lookback_epoch(tile_status, tile, tot, epoch, status);
        if (threadIdx.x == 0) s_excl = ex;
    }
    __syncthreads();
    if (kk >= 0) {
        const int32_t pos = s_excl + local;
        K[pos] = kk;
        V[pos] = (int32_t)v64;
    }
    if (tile == gridDim.x - 1 && threadIdx.x == 0) *d_cnt = s_excl + tot;
    hp::lb_end(lb);
}

// Over the sorted candidates: pre[i] = weight of the candidates before i in
// the sorted order (pre[cnt] = total), and pstart, the index of every part's first
// candidate, from the sorted keys.  Tiles of RK_TILE items in
// launch order with an epoch look-back, taken by a fixed grid of persistent
// CTAs until the tile holding index cnt, so the work follows the count on
// the device, not n.
constexpr int RK_THREADS = 256, RK_ITEMS = 4, RK_TILE = RK_THREADS * RK_ITEMS;

__global__ void __launch_bounds__(RK_THREADS)
rb_rank_kernel(const int32_t *__restrict__ K, const int32_t *__restrict__ V, const int32_t *__restrict__ d_cnt,
               const int32_t *__restrict__ vwgt, int32_t *__restrict__ pre, int32_t *__restrict__ pstart,
               unsigned long long *tile_status, hp::LbCtl *lb, unsigned *status)
{
    hp::pdl_wait();
    __shared__ int32_t s_scan[RK_THREADS / 32 + 2];
    __shared__ int32_t s_excl;
    const unsigned epoch = hp::lb_epoch(lb);
    const int32_t cnt = *d_cnt;
    for (;;) {
        const int64_t tile = hp::lb_next(lb);
        const int64_t base = tile * RK_TILE;
        if (base > cnt) break;   // the tile holding index cnt was the last one
        const int64_t i0 = base + (int64_t)threadIdx.x * RK_ITEMS;
        int32_t w[RK_ITEMS];
        int32_t sum = 0;
#pragma unroll
        for (int q = 0; q < RK_ITEMS; q++) {
            w[q] = i0 + q < cnt ? vwgt[V[i0 + q]] : 0;
            sum += w[q];
        }
        int tot;
        int32_t run = hp::block_excl_scan<RK_THREADS>(sum, &tot, s_scan);
        if (threadIdx.x < 32) {
            const int32_t ex = hp::lookback_epoch(tile_status, tile, tot, epoch, status);
            if (threadIdx.x == 0) s_excl = ex;
        }
        __syncthreads();
        run += s_excl;
#pragma unroll
        for (int q = 0; q < RK_ITEMS; q++) {
            const int64_t i = i0 + q;
            if (i <= cnt) pre[i] = run;
            run += w[q];
            if (i < cnt) {
                const int32_t p = K[i] >> 6;
                if (i == 0 || (K[i - 1] >> 6) != p) pstart[p] = (int32_t)i;
            }
        }
    }
    hp::lb_end(lb);
}

// The judge's list: exclusive prefix of the row lengths of the listed vertices
// (off[i]; off[cnt] = all their entries), in tiles of RK_TILE with an epoch
// look-back, by persistent CTAs until the tile holding index cnt.
__global__ void __launch_bounds__(RK_THREADS)
judge_off_kernel(const int32_t *flag, const int32_t *__restrict__ list, const int32_t *d_n,
                 const int32_t *__restrict__ xadj, int32_t *__restrict__ off, unsigned long long *tile_status,
                 hp::LbCtl *lb, unsigned *status)
{
    hp::pdl_wait();
    __shared__ int32_t s_scan[RK_THREADS / 32 + 2];
    __shared__ int32_t s_excl;
    const unsigned epoch = hp::lb_epoch(lb);
    const int32_t cnt = *flag != 0 ? *d_n : -1;   // -1: not judging, no tile
    for (;;) {
        const int64_t tile = hp::lb_next(lb);
        const int64_t base = tile * RK_TILE;
        if (base > cnt) break;   // the tile holding index cnt was the last one
        const int64_t i0 = base + (int64_t)threadIdx.x * RK_ITEMS;
        int32_t d[RK_ITEMS];
        int32_t sum = 0;
#pragma unroll
        for (int q = 0; q < RK_ITEMS; q++) {
            const int64_t i = i0 + q;
            d[q] = 0;
            if (i < cnt) {
                const int32_t v = list[i];
                d[q] = xadj[v + 1] - xadj[v];
            }
            sum += d[q];
        }
        int tot;
        int32_t run = hp::block_excl_scan<RK_THREADS>(sum, &tot, s_scan);
        if (threadIdx.x < 32) {
            const int32_t ex = hp::lookback_epoch(tile_status, tile, tot, epoch, status);
            if (threadIdx.x == 0) s_excl = ex;
        }
        __syncthreads();
        run += s_excl;
#pragma unroll
        for (int q = 0; q < RK_ITEMS; q++) {
            if (i0 + q <= cnt) off[i0 + q] = run;
            run += d[q];
        }
    }
    hp::lb_end(lb);
}

__global__ void rw_select_kernel(const int32_t *__restrict__ K, const int32_t *__restrict__ V,
                                 const int32_t *__restrict__ d_cnt, const int32_t *__restrict__ pre,
                                 const int32_t *__restrict__ pstart,
                                 const unsigned long long *__restrict__ pw,
                                 const int64_t *__restrict__ maxp, const int32_t *__restrict__ pregain, MoveSink ms)
{
    hp::pdl_wait();
    const int32_t cnt = *d_cnt;
    long long c1 = 0, touch = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < cnt;
         i += (int64_t)gridDim.x * blockDim.x) {
        int32_t p = K[i] >> 6;
        int64_t before = (int64_t)pre[i] - pre[pstart[p]];
        if (before < (int64_t)pw[p] - maxp[p]) {
            const int32_t v = V[i];
            move_append(ms, v, p);
            c1 += pregain[v];
            if (ms.d_touch) touch += ms.xadj[v + 1] - ms.xadj[v];
        }
    }
    sink_sums(ms, c1, touch);
}

// Strong rebalance: the evicted prefix of every overweight part (up to the first
// candidate where the weight before it reaches the part's excess: the candidates
// whose weight before them is less) compacted in sorted order -- P[j] = i and sp[j] = weight of
// the evicted candidates before j (sp[np] = total), *d_np = np -- in one pass
// with two epoch look-back chains (count: tile words [0, half); weight: words
// [half, 2 half)); persistent CTAs as in rb_rank_kernel.
__global__ void __launch_bounds__(RK_THREADS)
rs_evict_kernel(const int32_t *__restrict__ K, const int32_t *__restrict__ V, const int32_t *__restrict__ d_cnt,
                const int32_t *__restrict__ pre, const int32_t *__restrict__ pstart,
                const unsigned long long *__restrict__ pw, const int64_t *__restrict__ maxp,
                const int32_t *__restrict__ vwgt, int32_t *__restrict__ P,
                int32_t *__restrict__ sp, int32_t *__restrict__ d_np, unsigned long long *tile_status,
                int64_t half, hp::LbCtl *lb, unsigned *status)
{
    hp::pdl_wait();
    __shared__ int32_t s_scan[RK_THREADS / 32 + 2];
    __shared__ int32_t s_excl[2];
    const unsigned epoch = hp::lb_epoch(lb);
    const int32_t cnt = *d_cnt;
    for (;;) {
        const int64_t tile = hp::lb_next(lb);
        const int64_t base = tile * RK_TILE;
        if (base > cnt) break;   // the tile holding index cnt was the last one
        const int64_t i0 = base + (int64_t)threadIdx.x * RK_ITEMS;
        int32_t w[RK_ITEMS];
        bool f[RK_ITEMS];
        int32_t nf = 0, sw = 0;
#pragma unroll
        for (int q = 0; q < RK_ITEMS; q++) {
            const int64_t i = i0 + q;
            f[q] = false;
            if (i < cnt) {
                const int32_t p = K[i] >> 6;
                f[q] = (int64_t)pre[i] - pre[pstart[p]] < (int64_t)pw[p] - maxp[p];
            }
            w[q] = f[q] ? vwgt[V[i]] : 0;
            nf += f[q];
            sw += w[q];
        }
        int tc, tw;
        int32_t pos = hp::block_excl_scan<RK_THREADS>(nf, &tc, s_scan);
        int32_t run = hp::block_excl_scan<RK_THREADS>(sw, &tw, s_scan);
        if (threadIdx.x < 32) {
            const int32_t ex = hp::lookback_epoch(tile_status, tile, tc, epoch, status);
            if (threadIdx.x == 0) s_excl[0] = ex;
        } else if (threadIdx.x < 64) {
            const int32_t ex = hp::lookback_epoch(tile_status + half, tile, tw, epoch, status);
            if (threadIdx.x == 32) s_excl[1] = ex;
        }
        __syncthreads();
        pos += s_excl[0];
        run += s_excl[1];
#pragma unroll
        for (int q = 0; q < RK_ITEMS; q++) {
            if (f[q]) {
                P[pos] = (int32_t)(i0 + q);
                sp[pos] = run;
                pos++;
            }
            run += w[q];
        }
        if (cnt >= base && cnt < base + RK_TILE && threadIdx.x == 0) {
            *d_np = s_excl[0] + tc;
            sp[s_excl[0] + tc] = s_excl[1] + tw;
        }
    }
    hp::lb_end(lb);
}

// Sequential cookie cutter over the parts (one warp), as in the reference
// (hunyuangraph_GPU_krefine.h:3075): part p takes the evicted range starting
// at the previous end whose weight is closest to its room maxp[p] - pw[p].
// Rooms are read 32 parts at a time; a part without room keeps an empty range
// (the rule gives end = start there); otherwise the end is searched first among
// the 32 entries after the start (one coalesced read), then 32-ary over the rest.
// Once the start reaches np the remaining parts all get the empty range [np, np).
// The whole CTA first stages sp[0..np] in shared memory when it fits
// (COOKIE_SMEM_INTS entries), then warp 0 walks the parts; every search then
// waits on shared memory instead of L2.
constexpr int COOKIE_SMEM_INTS = 50 * 1024;

__device__ void cookie_cut_warp(int32_t k, const unsigned long long *__restrict__ pw,
                                const int64_t *__restrict__ maxp, const int32_t *sp, int32_t np,
                                int32_t *__restrict__ es, int32_t *__restrict__ ee);

__global__ void __launch_bounds__(1024)
cookie_cutter_kernel(int32_t k, const unsigned long long *__restrict__ pw, const int64_t *__restrict__ maxp,
                     const int32_t *__restrict__ sp_g, const int32_t *__restrict__ d_np, int32_t *__restrict__ es,
                     int32_t *__restrict__ ee)
{
    hp::pdl_wait();
    extern __shared__ int32_t sp_s[];
    const int32_t np = *d_np;
    const bool staged = np + 1 <= COOKIE_SMEM_INTS;
    if (staged)
        for (int32_t i = threadIdx.x; i <= np; i += blockDim.x) sp_s[i] = sp_g[i];
    __syncthreads();
    if (threadIdx.x >= 32) return;
    cookie_cut_warp(k, pw, maxp, staged ? sp_s : sp_g, np, es, ee);
}

// The walk itself, by one full warp.
__device__ void cookie_cut_warp(int32_t k, const unsigned long long *__restrict__ pw,
                                const int64_t *__restrict__ maxp, const int32_t *sp, int32_t np,
                                int32_t *__restrict__ es, int32_t *__restrict__ ee)
{
    // The parts form one dependent chain (each starts where the one before ended), so the
    // number of its steps and their latency are what counts: parts that take nothing are
    // skipped 32 at a time, the 32 prefix weights after the window's start wb and the
    // chain's own prefix stay in registers, in 32 bits (weights total below 2^31, a room
    // is clamped to 2^31), and the ranges are stored 32 parts at a time.  RGG 2^24,
    // k = 1024: a pass of the 8,517-vertex level 166 -> 61 us, of 1,942 vertices 102 -> 48.
    const int lane = threadIdx.x & 31;
    const unsigned total = (unsigned)sp[np];
    int32_t st = 0, wb = 0;
    unsigned cur = (unsigned)sp[0];   // sp[st]
    // positions past np count as reached: the answer is then np
    auto window = [&](int32_t b) -> unsigned {
        const int32_t pos = b + 1 + lane;
        return pos <= np ? (unsigned)sp[pos] : 0xffffffffu;
    };
    unsigned w = window(0);
    for (int32_t p0 = 0; p0 < k; p0 += 32) {
        const int32_t pl = p0 + lane;
        const int64_t room64 = pl < k ? maxp[pl] - (int64_t)pw[pl] : 0;
        const unsigned my_room = room64 <= 0 ? 0u : (unsigned)min(room64, (int64_t)1 << 31);
        const int cnt = min(32, k - p0);
        int32_t my_s = np, my_e = np;   // (parts after the list is used up: empty at np)
        int q = 0;
        while (q < cnt && st < np) {
            // the next part that takes something: the first whose room is nearer to the
            // first vertex's weight w1 than to nothing (the parts before it end where
            // they start, at st)
            if (st - wb >= 32) { wb = st; w = window(wb); }
            const unsigned w1 = __shfl_sync(HP_FULL_MASK, w, st - wb) - cur;
            const unsigned t = __ballot_sync(HP_FULL_MASK, lane >= q && lane < cnt && my_room > 0u &&
                                                               (w1 < my_room || w1 - my_room < my_room));
            const int nq = t ? __ffs(t) - 1 : cnt;
            if (lane >= q && lane < nq) { my_s = st; my_e = st; }
            q = nq;
            if (q == cnt) break;
            const unsigned room = __shfl_sync(HP_FULL_MASK, my_room, q);
            int32_t end = st;
            unsigned vend = cur;
            {
                // e: the first position after st with sp[e] >= find, else np
                const unsigned find = cur + room;
                unsigned m = __ballot_sync(HP_FULL_MASK, w >= find);
                if (m == 0u) {
                    wb = st;
                    w = window(wb);
                    m = __ballot_sync(HP_FULL_MASK, w >= find);
                }
                if (m == 0u) {   // beyond the 32 positions after st (sp[st + 32] < find)
                    int32_t lo = st + 32, hi = np;   // sp[lo] < find; the answer is in (lo, hi]
                    while (hi - lo > 32) {
                        const int64_t span = hi - lo;
                        const int32_t pos = lo + (int32_t)((span * (lane + 1)) / 32);
                        const unsigned g = __ballot_sync(HP_FULL_MASK, (unsigned)sp[pos] >= find);
                        if (g == 0u) { lo = np; break; }
                        const int f = __ffs(g) - 1;
                        hi = __shfl_sync(HP_FULL_MASK, pos, f);
                        if (f > 0) lo = __shfl_sync(HP_FULL_MASK, pos, f - 1);
                    }
                    wb = lo < np ? lo : np - 1;
                    w = window(wb);
                    m = __ballot_sync(HP_FULL_MASK, w >= find);
                }
                // (m == 0: np is the last position of the window)
                const int f = m ? __ffs(m) - 1 : 31;
                const int32_t e = min(wb + 1 + f, np);
                const unsigned vw = __shfl_sync(HP_FULL_MASK, w, e - wb - 1);
                const unsigned vb = __shfl_sync(HP_FULL_MASK, w, e - wb - 2 >= 0 ? e - wb - 2 : 0);
                const unsigned ve = e == np ? total : vw;
                const unsigned vs = e - 1 == st ? cur : (e - 1 == wb ? (unsigned)sp[wb] : vb);
                const unsigned dh = ve >= find ? ve - find : find - ve, dl = find - vs;
                end = dh < dl ? e : e - 1;
                vend = dh < dl ? ve : vs;
            }
            if (lane == q) { my_s = st; my_e = end; }
            st = end;
            cur = vend;
            q++;
        }
        if (pl < k) { es[pl] = my_s; ee[pl] = my_e; }
    }
}

__global__ void rs_assign_kernel(int32_t k, const int32_t *__restrict__ P, const int32_t *__restrict__ d_np,
                                 const int32_t *__restrict__ V, const int32_t *__restrict__ es,
                                 const int32_t *__restrict__ ee, const int32_t *__restrict__ where,
                                 int32_t *__restrict__ dest, const int32_t *__restrict__ pregain, MoveSink ms)
{
    hp::pdl_wait();
    const int32_t np = *d_np;
    long long c1 = 0, touch = 0;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < np;
         j += (int64_t)gridDim.x * blockDim.x) {
        // last part with es[p] <= j
        int32_t lo = 0, hi = k - 1;
        while (lo < hi) {
            int32_t mid = (lo + hi + 1) / 2;
            if (es[mid] <= j) lo = mid; else hi = mid - 1;
        }
        const int32_t p = lo;
        const int32_t v = V[P[j]];
        const int32_t from = where[v];
        if (j < ee[p] && p != from) {
            dest[v] = p;
            move_append(ms, v, from);
            if (ms.d_touch) touch += ms.xadj[v + 1] - ms.xadj[v];
            const int32_t o = ms.goff[v], len = ms.goff[v + 1] - o;
            c1 += (long long)row_conn(ms.gpart + o, ms.gconn + o, len, p, ms.k) + pregain[v];
        }
    }
    sink_sums(ms, c1, touch);
}


// ---------------------------------------------------------------------------------
struct RefineBufs {
    int32_t *goff, *gpart, *gconn, *big, *dest, *pregain, *moves, *oldp, *dirty;
    int32_t *small_l, *big_l, *best_where, *huge_mv, *huge;
    int32_t *hub;     // rows longer than gain_hub_deg (the dense gain build's rows when k <= warp_dense_k)
    int32_t *recof;   // move log: a vertex's record (record mode)
    int32_t *plan_v, *plan_item, *plan_off, *plan_cnt;   // chunk plan of the current step
    int64_t nhub_cap;   // capacity of the long-row list and the plan (rows longer than chunk_deg)
    unsigned long long *ab_acc;   // afterburner sums of the hub rows (zero between passes)
    int8_t *lock;
    int8_t *prune, *accp;                  // the judge of a learned pass (Judge)
    int32_t *jlist, *joff;                 // its listed vertices and their row prefix
    unsigned long long *ab_acc2;           // learned-candidate sums of the hub rows
    int32_t *K, *V, *K2, *V2, *pre, *P, *sp;
    int32_t *pstart, *und, *es, *ee;
    int8_t *ufl;   // per part: pw < maxp (a weak pass's destination rule), set by ctl_begin
    unsigned long long *pw;
    const int64_t *opt, *maxp;
    int32_t small_max;  // longest row of at most bigd entries (picks the gain kernel's network)
    bool huge_rows;     // the level has rows longer than huged
    bool dense_rows;    // the level has rows of at least k entries
    bool deep_rows;     // and k above 64: most gain rows are long (ROW_DEEP)
};

// scalar slots used by refinement
// Slots below S_PASS_END are reset at the start of every pass (S_NCANDP .. S_JL:
// the judge of a learned pass -- plain candidates, listed vertices, twice the
// plain and the learned exact cut decrease); S_BIGCNT (the
// level's list of rows longer than 32) lives above it and persists.
// S_BIGCNT (slots 16-18) holds the big-row count, the longest short row, the
// longest row above huged, the long-row count and the hub-row count.
enum { S_NMOVES = 0, S_C1 = 1, S_C2 = 2, S_EXCESS = 3, S_NCAND = 4, S_CUT2 = 5, S_DIRTY = 6,
       S_HUGEMV = 7, S_LISTCNT = 8, S_NU = 9, S_NP = 10, S_NCANDP = 11, S_JN = 12, S_JP = 13, S_JL = 14, S_TOUCH = 15,
       S_PASS_END = 16, S_BIGCNT = 16, S_DONE = 20 };

// hub_list: the level's rows longer than gain_hub_deg, which a full dense build walks
// instead of all long rows when k <= warp_dense_k (the others are gain_bigwarp_kernel's)
int build_rows(hp_context *c, HpLevel &g, RefineBufs &B, int32_t k, const int32_t *small_list,
               const int32_t *d_small_cnt, const int32_t *big_list, const int32_t *d_big_cnt,
               bool any_big, int32_t *dirty, const int32_t *hub_list, const int32_t *d_hub_cnt,
               const RebuildRule &rule = RebuildRule{nullptr, 0})
{
    const hp_tuning &tn = c->tune;
    if (small_list) {
        // rebuild of dirty rows: segments of S lanes per row (latency of a warp
        // per row, 32/S rows per warp)
        const unsigned grid = (unsigned)(c->sm_count * tn.grid_ctas_per_sm);
        if (B.small_max <= 8)
            HP_LAUNCH(c, gain_seg_kernel<8>, grid, 256, 0, small_list, d_small_cnt, g.xadj, g.adjncy, g.adjwgt,
                      g.where, B.goff, B.gpart, B.gconn, k, dirty, rule, g.n, tn.gain_thread_deg);
        else if (B.small_max <= 16)
            HP_LAUNCH(c, gain_seg_kernel<16>, grid, 256, 0, small_list, d_small_cnt, g.xadj, g.adjncy, g.adjwgt,
                      g.where, B.goff, B.gpart, B.gconn, k, dirty, rule, g.n, tn.gain_thread_deg);
        else
            HP_LAUNCH(c, gain_seg_kernel<32>, grid, 256, 0, small_list, d_small_cnt, g.xadj, g.adjncy, g.adjwgt,
                      g.where, B.goff, B.gpart, B.gconn, k, dirty, rule, g.n, tn.gain_thread_deg);
    } else {
        // full build of the level
        const unsigned grid = (unsigned)std::max<int64_t>(1, ((int64_t)g.n + GT_TILE - 1) / GT_TILE);
        auto build = [&](auto kernel, size_t smem) -> int {
            HP_LAUNCH(c, kernel, grid, GT_TILE, smem, g.n, g.xadj, g.adjncy, g.adjwgt, g.where, B.goff, B.gpart,
                      B.gconn, k, tn.gain_thread_deg);
            return HP_OK;
        };
        if (B.small_max <= 8) HP_TRY(build(gain_tile_kernel<8>, gain_tile_smem<8>()));
        else if (B.small_max <= 16) HP_TRY(build(gain_tile_kernel<16>, gain_tile_smem<16>()));
        else HP_TRY(build(gain_tile_kernel<32>, gain_tile_smem<32>()));
    }
    if (any_big) {
        // eight CTAs per SM in flight (where their accumulators fit): the rows are bound by
        // gather latency (R-MAT scale 22, all levels: four and two CTAs 9.7 ms, eight 7.9)
        const size_t smem = sizeof(int32_t) * (size_t)k + sizeof(unsigned) * (size_t)((k + 31) / 32);
        const int32_t *d_all = (const int32_t *)&c->d_scal[S_BIGCNT];
        if (k <= tn.warp_dense_k)
            HP_LAUNCH(c, gain_bigwarp_kernel, (unsigned)(c->sm_count * 8), 32 * GW_WARPS, GW_WARPS * smem, big_list,
                      d_big_cnt, g.xadj, g.adjncy, g.adjwgt, g.where, B.goff, B.gpart, B.gconn, k, dirty,
                      tn.gain_thread_deg, tn.gain_hub_deg, rule, B.big, d_all);
        // hub rows: every such row in a full build (of a level or after a pass); among the
        // queued rows only sparse ones (deg < k) exist, and only when k > gain_hub_deg
        const bool hubs = k <= tn.warp_dense_k;
        const int32_t *list = big_list, *d_cnt = d_big_cnt;
        if (hubs && !dirty) { list = hub_list; d_cnt = d_hub_cnt; }
        else if (hubs && k <= tn.gain_hub_deg) list = nullptr;
        if (!hubs || B.huge_rows)
            HP_LAUNCH(c, gain_dense_kernel<256>, (unsigned)(c->sm_count * 8), 256, smem, list, d_cnt, g.xadj, g.adjncy,
                      g.adjwgt, g.where, B.goff, B.gpart, B.gconn, k, dirty, tn.gain_thread_deg, tn.gain_hub_deg,
                      tn.warp_dense_k, rule, hubs ? hub_list : B.big, hubs ? d_hub_cnt : d_all);
    }
    return HP_OK;
}

int key_bits_for(int32_t k)
{
    int64_t maxkey = (int64_t)k * 64;
    int bits = 0;
    while ((1ll << bits) < maxkey) bits++;
    return (bits + 7) / 8 * 8;
}

// Persistent grid of the rank/evict kernels: at most the tiles a count of n
// can need, at most grid_ctas_per_sm CTAs per SM (they take tiles until the
// device count).
unsigned rank_grid(const hp_context *c, int64_t tiles)
{
    return (unsigned)std::min<int64_t>(tiles, (int64_t)c->sm_count * c->tune.grid_ctas_per_sm);
}

// Persistent grid of a chunk plan over at most cap items (the tile holding
// index cap included).
unsigned plan_grid(const hp_context *c, int64_t cap)
{
    return rank_grid(c, cap / PLAN_TILE + 1);
}

// Candidates of the pass (rb_candidates_kernel, K/V in vertex order) -> stable
// radix sort by key -> prefix weights and part bounds (rb_rank_kernel).
// Returns the arrays holding the sorted pairs.
template <bool STRONG>
int rank_candidates(hp_context *c, HpLevel &g, RefineBufs &B, int32_t k, int32_t **Ks, int32_t **Vs,
                    const BestCopy &bcp)
{
    const int32_t n = g.n;
    unsigned long long *sc = c->d_scal;
    int32_t *d_cnt = (int32_t *)&sc[S_LISTCNT];
    const int64_t ct = ((int64_t)n + RB_TILE - 1) / RB_TILE;
    const int64_t rt = ((int64_t)n + RK_TILE) / RK_TILE;   // a tile holds index cnt <= n
    if (ct > c->lb_cap || 2 * rt > c->lb_cap) return HP_ERR_INTERNAL;
    auto launch = [&](auto kernel) -> int {
        HP_LAUNCH(c, kernel, (unsigned)ct, RB_TILE, 0, n, g.where, g.vwgt, B.pw, B.maxp, B.opt, B.goff, B.gpart,
                  B.gconn, B.und, (const int32_t *)&sc[S_NU], k, B.K, B.V, B.dest, d_cnt, c->lb_status, c->lb_ctl,
                  c->d_status, B.ufl, B.pregain, bcp);
        return HP_OK;
    };
    HP_TRY(B.deep_rows ? launch(rb_candidates_kernel<STRONG, ROW_DEEP>)
                       : launch(rb_candidates_kernel<STRONG, ROW_FLAT>));
    bool in_tmp = false;
    HP_TRY(hp_sort_pairs(c, B.K, B.V, B.K2, B.V2, n, d_cnt, key_bits_for(k), &in_tmp));
    *Ks = in_tmp ? B.K2 : B.K;
    *Vs = in_tmp ? B.V2 : B.V;
    HP_LAUNCH(c, rb_rank_kernel, rank_grid(c, rt), RK_THREADS, 0, *Ks, *Vs, d_cnt, g.vwgt, B.pre, B.pstart,
              c->lb_status, c->lb_ctl, c->d_status);
    return HP_OK;
}

MoveSink move_sink(hp_context *c, const HpLevel &g, const RefineBufs &B, int32_t k)
{
    unsigned long long *sc = c->d_scal;
    return MoveSink{B.moves, B.oldp, &sc[S_NMOVES], &sc[S_C1], B.dense_rows ? &sc[S_TOUCH] : nullptr, B.goff, B.gpart, B.gconn, g.xadj, k};
}

// The undersized-part list of a weak pass is built by ctl_begin_kernel.
int weak_rebalance(hp_context *c, HpLevel &g, RefineBufs &B, int32_t k, const BestCopy &bcp)
{
    unsigned long long *sc = c->d_scal;
    int32_t *Ks, *Vs;
    HP_TRY(rank_candidates<false>(c, g, B, k, &Ks, &Vs, bcp));
    HP_LAUNCH(c, rw_select_kernel, (unsigned)(c->sm_count * 8), 256, 0, Ks, Vs,
              (const int32_t *)&sc[S_LISTCNT], B.pre, B.pstart, B.pw, B.maxp, B.pregain, move_sink(c, g, B, k));
    return HP_OK;
}

int strong_rebalance(hp_context *c, HpLevel &g, RefineBufs &B, int32_t k, const BestCopy &bcp)
{
    const int32_t n = g.n;
    unsigned long long *sc = c->d_scal;
    int32_t *Ks, *Vs;
    HP_TRY(rank_candidates<true>(c, g, B, k, &Ks, &Vs, bcp));
    const unsigned pg = (unsigned)(c->sm_count * 8);
    const int32_t *d_cnt = (const int32_t *)&sc[S_LISTCNT];
    int32_t *d_np = (int32_t *)&sc[S_NP];
    const int64_t rt = ((int64_t)n + RK_TILE) / RK_TILE;
    HP_LAUNCH(c, rs_evict_kernel, rank_grid(c, rt), RK_THREADS, 0, Ks, Vs, d_cnt, B.pre, B.pstart, B.pw,
              B.maxp, g.vwgt, B.P, B.sp, d_np,
              c->lb_status, c->lb_cap / 2, c->lb_ctl, c->d_status);
    HP_LAUNCH(c, cookie_cutter_kernel, 1, 1024, sizeof(int32_t) * COOKIE_SMEM_INTS, k, B.pw, B.maxp, B.sp, d_np,
              B.es, B.ee);
    HP_LAUNCH(c, rs_assign_kernel, pg, 256, 0, k, B.P, d_np, Vs, B.es, B.ee, g.where, B.dest, B.pregain,
              move_sink(c, g, B, k));
    return HP_OK;
}

// ---- pass control ------------------------------------------------------------------
// The pass loop's bookkeeping (exact cut, best partition, patience, stall rule,
// next mode) lives in device memory and is advanced by one-thread kernels.  The
// same rule therefore drives both loops: the eager loop reads the block after
// every pass, the CUDA-graph loop lets the block set its own WHILE and SWITCH
// conditions.  Passes per level are capped (a bound on the device-side loop).
constexpr int32_t HP_MAX_REFINE_PASSES = 1 << 14;

struct RefineCtl {
    long long cut, excess, best_cut, best_excess, cut_before, cut_start, last_moves;
    int32_t count, bal, passes, lp_idle;
    int32_t learned_active, learned_pass, mode, best_current;
    int32_t take, cont, patience, last_mode;
    int32_t mode_passes[4];
    int32_t gain_entries, pad;   // G of the level (for the profiler's byte counts)
    int32_t judge_mode;          // hp_options.learned = 3: the plain refiner judges every learned pass
    int32_t judge_pass;          // the current pass is a learned LP pass under that judge
};

__device__ void ctl_prepare(RefineCtl *s)
{
    s->passes++;
    s->mode = s->excess <= 0 ? 0 : (s->bal < 2 ? 1 : 2);
    s->learned_pass = (s->excess <= 0 && s->learned_active) ? 1 : 0;
    s->judge_pass = s->learned_pass && s->judge_mode;
    s->cut_before = s->cut;
    s->bal = s->mode == 0 ? 0 : s->bal + 1;
    s->mode_passes[s->mode]++;
}

__device__ int ctl_advance(RefineCtl *s, long long m, long long c1, long long c2, long long nmoves, long long ncand,
                           long long jp2);

// The level's starting cut: the coarser level's best cut when there is one (a
// projection keeps the cut exactly: every coarse edge weight is the sum of
// the fine edges between its two clusters, and edges inside a cluster are
// never cut), else the cut summed from the gain rows (rowcut_kernel).
__device__ void ctl_init_state(RefineCtl *s, long long cut, long long excess, int32_t patience, int32_t learned,
                               int32_t gain_total, int32_t judge)
{
    s->gain_entries = gain_total;
    s->cut = cut;
    s->excess = excess;
    s->cut_start = s->cut;
    s->best_cut = s->cut;
    s->best_excess = s->excess;
    s->best_current = 1;
    s->count = 0;
    s->bal = 0;
    s->passes = 0;
    s->lp_idle = 0;
    s->learned_active = learned;
    s->learned_pass = 0;
    s->judge_mode = learned && judge;
    s->judge_pass = 0;
    s->take = 0;
    s->last_moves = 0;
    s->last_mode = -1;
    s->patience = patience;
    s->mode = 0;
    for (int i = 0; i < 4; i++) s->mode_passes[i] = 0;
    s->cont = s->count <= patience;   // while (count++ <= patience)
    s->count++;
    if (s->cont) ctl_prepare(s);
}

__global__ void ctl_init_kernel(RefineCtl *s, const unsigned long long *sc, int32_t patience, int32_t learned,
                                const int32_t *gain_total, const RefineCtl *coarser, int32_t judge)
{
    hp::pdl_wait();
    ctl_init_state(s, coarser ? coarser->best_cut : (long long)sc[S_CUT2] / 2, (long long)sc[S_EXCESS], patience,
                   learned, *gain_total, judge);
}

// End of a pass: the exact cut change, the learned fallback, the stall rule, the
// best partition and the loop condition, in the order of the host loop they replace.
// End of a pass: the after-move half of the exact cut change (c2: the moved
// vertices' gain rows, rebuilt, at the old and new parts; c1 came with the moves),
// then the control step, run by the last CTA to finish (a ticket on *done,
// reset by that CTA): the max excess over the parts (max_p pw[p] - maxp[p]) and,
// by thread 0, the control block's advance and the graph loop's condition.
// One launch instead of a cut-change kernel and a one-CTA control kernel.
__global__ void __launch_bounds__(256)
pass_end_kernel(const int32_t *__restrict__ moves, const unsigned long long *d_nmoves,
                const int32_t *__restrict__ goff, const int32_t *__restrict__ gpart,
                const int32_t *__restrict__ gconn, const int32_t *__restrict__ where,
                const int32_t *__restrict__ oldp, int32_t k, RefineCtl *s, unsigned long long *sc,
                cudaGraphConditionalHandle hloop, int graph, const unsigned long long *__restrict__ pw,
                const int64_t *__restrict__ maxp, unsigned *status, unsigned *done)
{
    hp::pdl_wait();
    __shared__ bool s_last;
    __shared__ long long s_max[256 / 32];
    const int64_t nm = (int64_t)*d_nmoves;
    long long acc = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nm; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t v = moves[i];
        const int32_t o = goff[v], len = goff[v + 1] - o;
        acc += row_diff(gpart + o, gconn + o, len, where[v], oldp[i], k);
    }
    hp::block_add_to<256>(acc, &sc[S_C2]);   // ends with a barrier
    if (threadIdx.x == 0) {
        __threadfence();   // this CTA's sum is visible before its ticket
        s_last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    long long m = LLONG_MIN;
    for (int p = threadIdx.x; p < k; p += blockDim.x) {
        const long long e = (long long)pw[p] - maxp[p];
        m = e > m ? e : m;
    }
    m = hp::warp_max64(m);
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < (int)(blockDim.x >> 5); w++) m = s_max[w] > m ? s_max[w] : m;
    *done = 0u;
    volatile unsigned long long *vs = sc;
    sc[S_EXCESS] = (unsigned long long)m;
    const long long c1 = (long long)vs[S_C1], c2 = (long long)vs[S_C2];
    // the judge's sum over the learned moves is the applied pass's exact change
    if (s->judge_pass && (long long)vs[S_JL] != c1 + c2) atomicOr(status, HP_STATUS_OVERFLOW);
    const int cont = ctl_advance(s, m, c1, c2, (long long)vs[S_NMOVES], (long long)vs[S_NCAND], (long long)vs[S_JP]);
    if (graph) cudaGraphSetConditional(hloop, cont ? 1u : 0u);
}

// The control step of a pass end (one thread): new excess m, the cut-change
// sums c1 and c2, the pass's moves and LP candidates.  Returns the loop condition.
__device__ int ctl_advance(RefineCtl *s, long long m, long long c1, long long c2, long long nmoves, long long ncand,
                           long long jp2)
{
    s->excess = m;
    s->cut -= (c1 + c2) / 2;
    s->last_moves = nmoves;
    s->last_mode = s->mode;
    // The plain refiner takes over for the rest of the level as soon as a
    // learned pass does not lower the cut, and under the judge (learned = 3) as
    // soon as it lowers the cut less than the plain pass would have on the same
    // state: c1 + c2 and jp2 are twice the exact cut decrease of the learned and
    // of the plain moves.
    bool handed = false;
    if (s->learned_pass && (c1 + c2 <= 0 || (s->judge_pass && c1 + c2 < jp2))) {
        s->learned_active = 0;
        handed = true;
    }
    const int mode = s->mode;
    // A pass that changed nothing (no moves, no lock change) is repeated
    // identically by every later pass and can never improve the best
    // partition: stop now; the result is the same as running on.  Under the
    // judge a learned pass that handed over is not such a pass: the plain pass
    // after it differs.
    const bool stalled = !(handed && s->judge_mode) && nmoves == 0 &&
                         (mode == 2 || (mode == 0 && (ncand == 0 || s->lp_idle)));
    s->lp_idle = (mode == 0 && nmoves == 0) ? 1 : 0;
    int take = 0;
    if (s->best_excess > 0 && s->excess < s->best_excess) {
        take = 1;
        s->count = 0;
    } else if (s->cut < s->best_cut && (s->excess <= 0 || s->excess <= s->best_excess)) {
        if (1000 * s->cut < 999 * s->best_cut) s->count = 0;
        take = 1;
    }
    if (take) {
        s->best_cut = s->cut;
        s->best_excess = s->excess;
    }
    s->best_current = take;
    s->take = take;
    int cont = 0;
    if (!stalled) {
        cont = s->count <= s->patience;
        s->count++;
    }
    if (s->passes >= HP_MAX_REFINE_PASSES) cont = 0;
    s->cont = cont;
    if (cont) ctl_prepare(s);
    return cont;
}

// Start of a pass (one CTA of 1024 threads): clear the per-pass scalar slots,
// in the graph loop select the proposal body (0 LP, 1 weak rebalance, 2 strong
// rebalance), and for a weak pass build the undersized-part list.
__global__ void __launch_bounds__(1024)
ctl_begin_kernel(const RefineCtl *s, unsigned long long *sc, cudaGraphConditionalHandle hmode, int graph, int32_t k,
                 const unsigned long long *__restrict__ pw, const int64_t *__restrict__ maxp,
                 int32_t *__restrict__ und, int8_t *__restrict__ ufl)
{
    hp::pdl_wait();
    __shared__ int32_t s_scan[1024 / 32 + 2];
    if (threadIdx.x < S_PASS_END) sc[threadIdx.x] = 0;
    const int mode = s->mode;
    if (graph && threadIdx.x == 0) cudaGraphSetConditional(hmode, (unsigned)mode);
    __syncthreads();
    if (mode == 1) {
        undersized_block(k, pw, maxp, und, (int32_t *)&sc[S_NU], s_scan);
        for (int32_t q = threadIdx.x; q < k; q += blockDim.x) ufl[q] = (int64_t)pw[q] < maxp[q];
    }
}

__global__ void restore_best_kernel(const RefineCtl *s, int32_t n, const int32_t *__restrict__ best_where,
                                    int32_t *__restrict__ where)
{
    hp::pdl_wait();
    if (s->best_current) return;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride) where[i] = best_where[i];
}

// ---- profile-only byte counts -------------------------------------------------------
// The data-dependent terms of the refinement classes' algorithmic byte models
// (rows walked, candidates, moves, dirty rows), counted on the device in
// profiled eager passes into the class counters (hp_prof_counter) after the
// class's launches, so that the counting is not timed with them.  Neighbour
// gathers are not counted (compulsory-traffic model, as for every class).

// Bytes a gain-row walk reads: a dense row (k entries, longer than 32 and so
// walked by a warp with the part ids implied) reads k connectivities; any
// other row its (part, conn) pairs up to and including the first padding slot.
__device__ __forceinline__ long long row_walk_bytes(const int32_t *__restrict__ gpart, int32_t o, int32_t len,
                                                    int32_t k)
{
    if (len > 32 && len == k) return 4ll * k;
    int32_t f = 0;
    while (f < len && gpart[o + f] >= 0) f++;
    return 8ll * (f < len ? f + 1 : f);
}

// LP: every row's walk by the selection, and each candidate's adjacency row
// (adjncy + adjwgt) and destination read by the afterburner.
__global__ void __launch_bounds__(256)
lp_bytes_kernel(int32_t n, const int32_t *__restrict__ goff, const int32_t *__restrict__ gpart,
                const int32_t *__restrict__ xadj, const int32_t *__restrict__ pregain, int32_t k,
                unsigned long long *acc)
{
    hp::pdl_wait();
    long long b = 0;
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        b += row_walk_bytes(gpart, goff[v], goff[v + 1] - goff[v], k);
        if (pregain[v] != NEG) b += 8ll * (xadj[v + 1] - xadj[v]) + 4;
    }
    hp::block_add_to<256>(b, acc);
}

// Rebuild of the dirty rows: xadj, goff and the list entry, the adjacency row,
// the rewritten gain row (8 bytes per slot) and the dirty flag's reset.
__global__ void __launch_bounds__(256)
rebuild_bytes_kernel(const int32_t *__restrict__ small_l, const int32_t *__restrict__ d_nsmall,
                     const int32_t *__restrict__ big_l, const int32_t *__restrict__ d_nbig,
                     const int32_t *__restrict__ xadj, const int32_t *__restrict__ goff, RebuildRule rule, int32_t n,
                     unsigned long long *acc)
{
    hp::pdl_wait();
    const int32_t ns = *d_nsmall, nb = *d_nbig;
    long long b = 0;
    // every row: xadj, goff and the parts, the adjacency, the gain rows
    if (rule.all() && blockIdx.x == 0 && threadIdx.x == 0) b = 12ll * n + 8ll * xadj[n] + 8ll * goff[n];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (int64_t)ns + nb;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t v = i < ns ? small_l[i] : big_l[i - ns];
        b += 24 + 8ll * (xadj[v + 1] - xadj[v]) + 8ll * (goff[v + 1] - goff[v]);
    }
    hp::block_add_to<256>(b, acc);
}

// Rebalance proposals (counted before the moves apply, with the part weights
// the proposal saw): where and dest of every vertex; vertex weight, goff and
// the gain-row walk of every vertex of an overweight part; per candidate its
// key/value write, 20 bytes per radix pass (digit histogram read, pair
// scatter) and the rank/select (or evict) reads of the sorted pairs.
__global__ void __launch_bounds__(256)
rebalance_bytes_kernel(int32_t n, const int32_t *__restrict__ where, const unsigned long long *__restrict__ pw,
                       const int64_t *__restrict__ maxp, const int32_t *__restrict__ goff,
                       const int32_t *__restrict__ gpart, int32_t k, const int32_t *__restrict__ d_cnt,
                       int32_t radix_passes, unsigned long long *acc)
{
    hp::pdl_wait();
    long long b = 0;
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const int32_t p = where[v];
        b += 8;
        if ((int64_t)pw[p] > maxp[p]) b += 12 + row_walk_bytes(gpart, goff[v], goff[v + 1] - goff[v], k);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) b += (long long)(*d_cnt) * (32 + 20ll * radix_passes);
    hp::block_add_to<256>(b, acc);
}

// Move application: per move its list entries (vertex, old part), destination,
// vertex weight, xadj, adjacency row and where write, then the exact cut
// change's goff read and walk of the mover's gain row; once per pass the
// control step's part weights and bounds, and the best-partition copy when
// the pass was the best so far.
__global__ void __launch_bounds__(256)
apply_bytes_kernel(const int32_t *__restrict__ moves, const unsigned long long *__restrict__ d_nmoves,
                   const int32_t *__restrict__ xadj, const int32_t *__restrict__ goff,
                   const int32_t *__restrict__ gpart, int32_t k, int32_t n, const RefineCtl *ctl,
                   unsigned long long *acc)
{
    hp::pdl_wait();
    const int64_t nm = (int64_t)*d_nmoves;
    long long b = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nm; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t v = moves[i];
        b += 36 + 8ll * (xadj[v + 1] - xadj[v]) + row_walk_bytes(gpart, goff[v], goff[v + 1] - goff[v], k);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) b += 16ll * k + (ctl->take ? 8ll * n + 16ll * k : 0);
    hp::block_add_to<256>(b, acc);
}

struct PassCfg {
    int32_t k;
    bool finest, any_big, recording, huge_rows;   // huge_rows: rows longer than chunk_deg exist
    bool judged;                                  // learned = 3: learned passes are judged
    bool huge_moves;                              // rows longer than apply_chunk_deg exist
    RefineCtl *ctl;
    unsigned long long *best_pw;
};

BestCopy best_copy(const RefineBufs &B, const PassCfg &P)
{
    return BestCopy{&P.ctl->take, B.best_where, B.pw, P.best_pw, P.k};
}

// Proposal phase of one pass.  Eager mode launches the LP selection kernel the
// host chose; graph mode launches both when the MLP is loaded, gated by the
// control block's learned_pass flag.
int pass_propose(hp_context *c, HpLevel &g, RefineBufs &B, const PassCfg &P, int mode, bool learned_pass,
                 bool both_lp)
{
    const int32_t n = g.n, k = P.k;
    unsigned long long *sc = c->d_scal;
    int32_t *d_bigcnt = (int32_t *)&sc[S_BIGCNT];
    const unsigned pg = (unsigned)(c->sm_count * c->tune.grid_ctas_per_sm);
    const int32_t *gate = both_lp ? &P.ctl->learned_pass : nullptr;
    if (mode == 0) {
        const int ltok = hp_prof_begin(c);
        const Judge J{&P.ctl->judge_pass, B.prune, B.accp, B.jlist, (int32_t *)&sc[S_JN], &sc[S_NCANDP]};
        const bool judging = P.judged && (both_lp || learned_pass);
        if (both_lp || learned_pass)
            HP_LAUNCH(c, lp_select_learned_kernel, nblk(n), 256, 0, n, B.goff, B.gpart, B.gconn, g.where, g.xadj,
                      B.lock, P.finest ? 1 : 0, B.pw, B.maxp, B.opt, c->mlp_params, c->mlp_threshold, B.dest,
                      B.pregain, &sc[S_NCAND], gate, k, B.prune, &sc[S_NCANDP], J.flag, best_copy(B, P));
        if (both_lp || !learned_pass) {
            auto launch = [&](auto kernel) -> int {
                HP_LAUNCH(c, kernel, nblk(n), 256, 0, n, B.goff, B.gpart, B.gconn, g.where, B.lock,
                      P.finest ? 1 : 0, B.dest, B.pregain, &sc[S_NCAND], gate, k, best_copy(B, P));
                return HP_OK;
            };
            HP_TRY(B.deep_rows ? launch(lp_select_kernel<ROW_DEEP>) : launch(lp_select_kernel<ROW_FLAT>));
        }
        if (P.recording)
            HP_LAUNCH(c, log_candidates_kernel, nblk(n), 256, 0, n, B.goff, B.gpart, B.gconn, g.where, g.xadj,
                      P.finest ? 1 : 0, B.pw, B.maxp, B.opt, B.dest, B.pregain, B.recof, c->log_x, c->log_v,
                      c->log_d, c->log_acc, c->log_count, c->log_cap);
        HP_LAUNCH(c, afterburner_small_kernel, nblk(n), 256, 0, n, g.xadj, g.adjncy, g.adjwgt, g.where, B.dest,
                  B.pregain, B.lock, &sc[S_NCAND], move_sink(c, g, B, k), c->tune.gain_thread_deg, J);
        if (P.any_big)
            HP_LAUNCH(c, afterburner_big_kernel, pg, 256, 0, B.big, d_bigcnt, g.xadj, g.adjncy, g.adjwgt, g.where,
                      B.dest, B.pregain, B.lock, &sc[S_NCAND], move_sink(c, g, B, k), c->tune.chunk_deg, J);
        if (P.huge_rows) {
            const int32_t *d_nhuge = d_bigcnt + 3;
            HP_LAUNCH(c, hub_plan_kernel<false>, plan_grid(c, B.nhub_cap), PLAN_THREADS, 0, B.huge, d_nhuge, B.moves,
                      B.pregain, g.xadj, B.plan_v, B.plan_item, B.plan_off, B.plan_cnt, c->lb_status, c->lb_cap / 2,
                      c->lb_ctl, c->d_status);
            HP_LAUNCH(c, afterburner_huge_kernel, (unsigned)(4 * c->sm_count), HUB_CHUNK, 0, B.plan_v, B.plan_item,
                      B.plan_off, B.plan_cnt, g.xadj, g.adjncy, g.adjwgt, g.where, B.dest, B.pregain, &sc[S_NCAND],
                      B.ab_acc, B.ab_acc2, J);
            HP_LAUNCH(c, afterburner_huge_final_kernel, (unsigned)c->sm_count, 256, 0, B.huge, d_nhuge, B.pregain,
                      &sc[S_NCAND], B.ab_acc, B.ab_acc2, B.lock, g.where, B.dest, move_sink(c, g, B, k), J);
        }
        if (judging) {   // the plain refiner's exact cut change on the same state (learned passes only)
            const int64_t rt = ((int64_t)n + RK_TILE) / RK_TILE;   // a tile holds index cnt <= n
            if (rt > c->lb_cap) return HP_ERR_INTERNAL;
            HP_LAUNCH(c, judge_off_kernel, rank_grid(c, rt), RK_THREADS, 0, J.flag, B.jlist, J.d_n, g.xadj, B.joff,
                      c->lb_status, c->lb_ctl, c->d_status);
            HP_LAUNCH(c, judge_delta_kernel, pg, JD_THREADS, 0, J.flag, B.jlist, J.d_n, B.joff, g.xadj, g.adjncy,
                      g.adjwgt, g.where, B.dest, B.accp, B.lock, &sc[S_JP]);
        }
        if (P.recording)
            HP_LAUNCH(c, log_accept_kernel, nblk(n), 256, 0, n, B.recof, B.lock, &sc[S_NCAND], c->log_acc);
        // fixed terms -- selection: goff, where, lock in, dest and pregain out;
        // afterburner: xadj, pregain in, lock out.  The rows walked and the
        // candidates' adjacency rows are counted on the device.
        hp_prof_end(c, ltok, HP_PROF_LP, 8 * ((int64_t)n + 1) + 18 * (int64_t)n);
        if (unsigned long long *cnt = hp_prof_counter(c, HP_PROF_LP))
            HP_LAUNCH(c, lp_bytes_kernel, std::min(nblk(n), pg), 256, 0, n, B.goff, B.gpart, g.xadj, B.pregain, k,
                      cnt);
    } else {
        const int btok = hp_prof_begin(c);
        if (mode == 1) HP_TRY(weak_rebalance(c, g, B, k, best_copy(B, P)));
        else HP_TRY(strong_rebalance(c, g, B, k, best_copy(B, P)));
        hp_prof_end(c, btok, HP_PROF_REBALANCE, 0);
        if (unsigned long long *cnt = hp_prof_counter(c, HP_PROF_REBALANCE))
            HP_LAUNCH(c, rebalance_bytes_kernel, std::min(nblk(n), pg), 256, 0, n, g.where, B.pw, B.maxp, B.goff,
                      B.gpart, k, (const int32_t *)&sc[S_LISTCNT], key_bits_for(k) / 8, cnt);
    }
    return HP_OK;
}

// When a pass rebuilds every gain row: on a level with dense rows, its moves touch more
// than an eighth of the adjacency.  Touching an entry costs a gather of the neighbour's
// row offset and, where the neighbour's row is dense, two scattered atomics; the full
// build reads every entry once, in order, and adds in shared memory.  R-MAT scale 22,
// k = 256, learned: moves and rebuilds 22.8 ms a call without the rule, 14.3 at an
// eighth, 14.5 at a quarter, 15.4 at a sixteenth.  Levels without dense rows touch by
// flags alone, and their passes are too short for the extra sum.
constexpr int64_t REBUILD_SHARE = 8;
RebuildRule rebuild_rule(hp_context *c, const HpLevel &g, const RefineBufs &B)
{
    return RebuildRule{B.dense_rows ? &c->d_scal[S_TOUCH] : nullptr, (unsigned long long)(g.m / REBUILD_SHARE)};
}

// Apply phase of one pass: simultaneous moves, exact cut change from the gain
// rows before and after, gain-row maintenance, balance, then the control step.
int pass_apply(hp_context *c, HpLevel &g, RefineBufs &B, const PassCfg &P, cudaGraphConditionalHandle hloop,
               int graph)
{
    const int32_t n = g.n, k = P.k;
    unsigned long long *sc = c->d_scal;
    const unsigned pg = (unsigned)(c->sm_count * c->tune.grid_ctas_per_sm);
    const unsigned mg = std::min(nblk(n), pg);   // grid-stride over the device move count
    // (the proposal kernels appended the moves with their old parts, c1 and their entries)
    const RebuildRule rule = rebuild_rule(c, g, B);
    int atok = hp_prof_begin(c);
    HP_LAUNCH(c, apply_moves_kernel, pg, 256, 0, B.moves, &sc[S_NMOVES], g.where, B.dest, g.vwgt, B.pw, g.xadj,
              g.adjncy, g.adjwgt, B.goff, B.gconn, B.dirty, B.small_l, B.big_l, (int32_t *)&sc[S_DIRTY], k,
              B.huge_mv, (int32_t *)&sc[S_HUGEMV], c->tune.gain_thread_deg, c->tune.apply_chunk_deg, rule);
    if (P.huge_moves) {
        HP_LAUNCH(c, hub_plan_kernel<true>, plan_grid(c, B.nhub_cap), PLAN_THREADS, 0, B.huge_mv,
                  (const int32_t *)&sc[S_HUGEMV], B.moves, B.pregain, g.xadj, B.plan_v, B.plan_item, B.plan_off,
                  B.plan_cnt, c->lb_status, c->lb_cap / 2, c->lb_ctl, c->d_status);
        HP_LAUNCH(c, apply_moves_huge_kernel, (unsigned)(4 * c->sm_count), HUB_CHUNK, 0, B.plan_v, B.plan_item,
                  B.plan_off, B.plan_cnt, B.oldp, B.dest, g.xadj, g.adjncy, g.adjwgt, B.goff, B.gconn, B.dirty,
                  B.small_l, B.big_l, (int32_t *)&sc[S_DIRTY], k, c->tune.gain_thread_deg);
    }
    hp_prof_end(c, atok, HP_PROF_APPLY, 0);
    const int rtok = hp_prof_begin(c);
    HP_TRY(build_rows(c, g, B, k, B.small_l, (const int32_t *)&sc[S_DIRTY], B.big_l,
                      ((const int32_t *)&sc[S_DIRTY]) + 1, P.any_big, B.dirty, B.hub,
                      (const int32_t *)&sc[S_BIGCNT] + 4, rule));
    hp_prof_end(c, rtok, HP_PROF_REBUILD, 0);
    if (unsigned long long *cnt = hp_prof_counter(c, HP_PROF_REBUILD))
        HP_LAUNCH(c, rebuild_bytes_kernel, pg, 256, 0, B.small_l, (const int32_t *)&sc[S_DIRTY], B.big_l,
                  ((const int32_t *)&sc[S_DIRTY]) + 1, g.xadj, B.goff, rule, n, cnt);
    atok = hp_prof_begin(c);
    HP_LAUNCH(c, pass_end_kernel, mg, 256, 0, B.moves, &sc[S_NMOVES], B.goff, B.gpart, B.gconn, g.where, B.oldp, k,
              P.ctl, sc, hloop, graph, B.pw, B.maxp, c->d_status, (unsigned *)&sc[S_DONE]);
    hp_prof_end(c, atok, HP_PROF_APPLY, 0);
    if (unsigned long long *cnt = hp_prof_counter(c, HP_PROF_APPLY))
        HP_LAUNCH(c, apply_bytes_kernel, mg, 256, 0, B.moves, &sc[S_NMOVES], g.xadj, B.goff, B.gpart, k, n, P.ctl,
                  cnt);
    return HP_OK;
}

// ---- small levels: every pass of the level in one cluster of CTAs --------------------
// A level of at most cluster_level_n() vertices runs its whole pass loop inside one
// thread-block cluster of up to CL_MAX CTAs of CL_THREADS threads.  The phases are
// those of the multi-kernel pass, in the same order and by the same rules -- LP
// selection and afterburner, weak or strong rebalance (candidates, stable radix
// sort, ranks, selection or eviction and cookie cutter), simultaneous moves,
// gain-row maintenance, the exact cut change, the control step and the best
// partition -- separated by the hardware's cluster barrier instead of kernel
// boundaries.  Every warp of the cluster owns one contiguous range of vertices
// (then of sorted candidates), so ordered results need one exchange of the CTAs'
// totals through distributed shared memory, and rows walked by a whole warp are
// spread over all of them.  The control block and the part weights are kept by
// every CTA alike.  Gain rows, candidates and moves equal the multi-kernel pass's,
// so the level's result is identical; what goes away is about fifteen dependent
// launches per pass, which on these levels cost more than the work.
// Per level and pass, one CTA or the launched kernels before, a cluster now: 128^3 grid
// (k = 64) 2,817 vertices 100 -> 47 us, 8,854 93 -> 58, 25,181 85 -> 62; 256^2 grid
// (k = 8) 10,870 vertices 62 -> 28 us, 65,536 63 -> 36.  Fewer than about 512 vertices
// per CTA buy nothing: the passes are chains of L2 latencies and barriers.
constexpr int CL_THREADS = 1024;
constexpr int CL_WARPS = CL_THREADS / 32;
constexpr int CL_MAX = 16;                 // CTAs of a cluster (above 8: non-portable size)
constexpr int CL_SORT_INTS = CL_WARPS * 256;
constexpr size_t CL_COOKIE_BYTES = 100 * 1024;   // staged prefix weights of the cookie cutter
constexpr int CL_KMAX = HP_TUNE_WARP_DENSE_K_MAX;

struct SmallLevel {
    int32_t n, k, finest, bigd, small_max, key_bits, learned_mlp;
    int32_t patience, judge;    // the control block's init (the level's setup runs in the kernel)
    int32_t cookie_cap;         // prefix weights that fit the dynamic shared memory
    const RefineCtl *coarser;   // the coarser level's control block (its best cut), or nullptr
    float mlp_threshold;
    const int32_t *xadj, *adjncy, *adjwgt, *vwgt;
    int32_t *where;
    int32_t *goff;
    int32_t *gpart, *gconn;
    int32_t *dest, *pregain, *moves, *oldp, *dirty, *small_l, *big_l, *best_where;
    int32_t *K, *V, *K2, *V2, *pre, *P, *sp;
    int32_t *pbase, *es, *ee;
    int32_t *counts;        // 2 sets of 4: moves, dirty short rows, dirty long rows
    int8_t *lock;
    int8_t *prune, *accp;   // the judge of a learned pass
    unsigned long long *pw, *best_pw;
    const int64_t *opt, *maxp;
    const float *mlp_params;
    RefineCtl *ctl;
    unsigned *status;
    // the grid variant's barrier counter (zero at launch) and exchange arrays
    unsigned *bar;
    unsigned spin_limit;
    long long *gx;          // 2 x CTAs x 3
    int32_t *ghist;         // CTAs x 256
};

// Dynamic shared memory: the largest of the phases' needs (sort tables; the staged
// prefix weights of the cookie cutter, at most n + 1; the warps' dense gain-row
// accumulators; the part weights of the setup).
size_t small_level_smem(int32_t n, int32_t k)
{
    const size_t sort = sizeof(int32_t) * CL_SORT_INTS;
    const size_t cookie = std::min(sizeof(int32_t) * ((size_t)n + 1), CL_COOKIE_BYTES);
    const size_t rows = sizeof(int32_t) * CL_WARPS * ((size_t)k + (k + 31) / 32);
    return std::max(sort, std::max(cookie, rows));
}

// CTAs of a level's cluster, a power of two: CL_PER_CTA vertices and CL_ENT_PER_CTA
// adjacency entries each.
constexpr int32_t CL_PER_CTA = 512;
constexpr int64_t CL_ENT_PER_CTA = 8192;
int cluster_ctas(const hp_context *c, int32_t n, int64_t m)
{
    int q = 1;
    while (q < c->max_cluster && ((int64_t)q * CL_PER_CTA < n || q * CL_ENT_PER_CTA < m)) q *= 2;
    return q;
}

// The largest level a cluster takes: small_level_n vertices per CTA, at most CL_LEVEL_MAX,
// and at most CL_DEG entries per vertex of that bound.  Above CL_LEVEL_MAX the same loop
// over the whole GPU has cheaper passes.  Cluster / cooperative launch, us per pass:
// RGG (k = 100, 12 entries a vertex) 32,768 vertices 39 / 44, 49,152 46 / 45, 65,536
// 47 / 46, 81,920 52 / 44, 131,072 68 / 47; 3-D grid (k = 64, 5.8 entries) 32,768 34 / 44,
// 64,000 43 / 47, 81,356 48 / 48, 97,336 50 / 47, 130,050 57 / 49; 2-D grid (k = 8,
// 4 entries) 65,536 35 / 39, 81,796 37 / 40, 98,596 42 / 40, 131,044 44 / 35.
constexpr int32_t CL_LEVEL_MAX = 65536;
constexpr int64_t CL_DEG = 16;
int32_t cluster_level_n(const hp_context *c)
{
    return (int32_t)std::min<int64_t>((int64_t)c->tune.small_level_n * c->max_cluster, CL_LEVEL_MAX);
}

// Whether a level may be a cluster's by its size.
bool cluster_size(const hp_context *c, const HpLevel &g, int32_t k)
{
    const int32_t n = cluster_level_n(c);
    return g.n <= n && k <= CL_KMAX && g.m <= CL_DEG * n;
}

// ... and by its rows: a warp of the loop walks the rows of its own range of vertices and
// a moved vertex's row, so a hub row, or many long rows side by side (the low ids of a
// power-law graph), hold the cluster at its barriers, where the launched passes spread
// rows over the grid.  The entries in a range at which both take the same time:
//   rows above LOOP_LONG_ROW (grids of 19,600 and 59,536 vertices with 1 to 64 hubs,
//   k = 8 to 256; us per pass cluster / launched): 8,192 43-58 / 53-69, 16,384 42-103 /
//   58-77, 32,768 44-140 / 57-86, 65,536 60-254 / 63-90;
//   rows below it (R-MAT, 8,000 to 65,536 vertices), where every gain row of more than 32
//   parts is a warp's turn: about 32,000 for k = 8 (31,111 76 / 82, 36,033 97 / 83),
//   24,000 for 16 (18,187 81 / 78, 26,784 69 / 75), 16,000 for 32 (16,240 80 / 72, 15,410
//   70 / 74), 12,000 for 64 (11,628 77 / 85, 14,306 93 / 87), 9,500 for 200 (8,758 91 / 83,
//   15,410 127 / 95): so an entry counts sqrt(k) / 5.6 there, at most 1.75.
// Hubs spread over the warps count by all their entries (us per pass): 32,768 41-67 / 60-85,
// 65,536 42-92 / 57-86, 131,072 56-155 / 69-101, 262,144 73-145 / 75-100.  The smallest
// levels keep the cluster whatever their rows (3,969 vertices, 30,400 entries in a warp's
// range, k = 256: 81 / 122).
constexpr int64_t LOOP_WARP_ENTRIES = 16384;
constexpr int32_t LOOP_LONG_ENTRIES = 98304;
int32_t loop_weight(int32_t k)
{
    return (int32_t)std::lround(LOOP_UNIT * std::min(1.75, std::sqrt((double)k) / 5.6));
}
constexpr int32_t LOOP_ANY_ROWS_N = 4096;
bool loop_rows(const HpLevel &g, const LevelStat &ls)
{
    return (g.n <= LOOP_ANY_ROWS_N && g.m <= CL_DEG * LOOP_ANY_ROWS_N) ||
           ((int64_t)ls.range_entries <= LOOP_UNIT * LOOP_WARP_ENTRIES && ls.long_entries <= LOOP_LONG_ENTRIES);
}

// Levels above that run their passes in one cooperative launch over the whole GPU, a CTA
// per SM: the same loop with a barrier through global memory (about 2.5 us against the
// cluster's 1) and 148 SMs.  Against launched passes (a graph), us per pass: 3-D grid
// (k = 64) 130,050 vertices 49 / 54, 1,000,000 74 / 94, 2,097,152 113 / 129, 8,000,000
// 295 / 326; RGG (k = 100) 131,072 47 / 57, 1,000,000 95 / 116, 2,097,152 144 / 172,
// 4,500,000 258 / 291.  It was not slower at any size, and saves the host half a
// millisecond a level for the graph.  GRID_LEVEL_MAX is no crossing: it bounds how long a
// launch that needs every SM keeps the other streams of the device out (about 3 ms for
// the twenty passes of a level), which launched passes let in between their kernels.
// A longer row than GRID_DEG_MAX would hold the one warp that walks it.
constexpr int32_t GRID_LEVEL_MAX = 1 << 21;
constexpr int32_t GRID_DEG_MAX = 1024;

__device__ __forceinline__ unsigned cl_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ unsigned cl_size()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}

// All threads of the cluster; writes before it (global and shared, this CTA's and
// remote) are visible after it.
__device__ __forceinline__ void cl_sync()
{
    // (not the .aligned forms: a warp may reach this diverged, and its parts would then
    // arrive as if each were the whole warp)
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release;\n"
                 "barrier.cluster.wait.acquire;" ::: "memory");
}

// The address of CTA `rank`'s copy of a shared-memory object.
__device__ __forceinline__ unsigned cl_map(const void *p, unsigned rank)
{
    unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}

__device__ __forceinline__ void cl_st64(unsigned addr, long long v)
{
    asm volatile("st.shared::cluster.s64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}

__device__ __forceinline__ int32_t cl_ld32(unsigned addr)
{
    int32_t v;
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

// The barrier of the grid variant (a cooperative launch: every CTA is resident): an
// arrival counter that only grows, *gen its value when the last barrier completed.
// Writes before it are visible after it.  The wait is bounded by `limit`: on expiry it sets
// HP_STATUS_SPIN_TIMEOUT and returns false in every thread of the CTA, which then
// leaves the kernel (as the CTAs that wait for it will).
__device__ __forceinline__ bool grid_sync(unsigned *bar, unsigned *gen, unsigned *status, unsigned limit)
{
    __shared__ bool s_ok;
    *gen += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(bar, 1u);
        unsigned seen = 0, spins = 0;
        for (;;) {
            asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
            if ((int)(seen - *gen) >= 0) break;
            if (++spins > limit) {
                atomicOr(status, HP_STATUS_SPIN_TIMEOUT);
                break;
            }
            if (spins > 64) __nanosleep(32);
        }
        __threadfence();
        s_ok = (int)(seen - *gen) >= 0;
    }
    __syncthreads();
    return s_ok;
}

// Exchange of the CTAs' sums through the barrier.  Two buffers in turn: a CTA
// writes a buffer again only two barriers later, when every CTA has read it.
// A cluster's CTAs write into each other's shared memory; a grid's go through
// global memory, read by one warp of every CTA.
struct ClXch {
    long long x[2][CL_MAX][3];
    long long w[CL_WARPS][3];
    long long tot[4];
};

template <bool GRID>
struct ClTeam {
    unsigned rank, nct;
    unsigned gen;       // grid: the barrier's count so far
    const SmallLevel &a;
    ClXch &X;
    __device__ __forceinline__ ClTeam(const SmallLevel &a_, ClXch &X_) : gen(0), a(a_), X(X_)
    {
        rank = GRID ? blockIdx.x : cl_rank();
        nct = GRID ? gridDim.x : cl_size();
    }
    // All threads of the team; false: the wait expired and the kernel ends.
    __device__ __forceinline__ bool sync()
    {
        if (GRID) return grid_sync(a.bar, &gen, a.status, a.spin_limit);
        cl_sync();
        return true;
    }
    __device__ __forceinline__ void put(int buf, int i, long long v)   // (the first warp, the same v in its lanes)
    {
        const int lane = threadIdx.x & 31;
        if (GRID) {
            if (lane == 0) a.gx[((size_t)buf * nct + rank) * 3 + i] = v;
        } else if (lane < (int)nct) {
            cl_st64(cl_map(&X.x[buf][rank][i], lane), v);
        }
    }
    // Sums of N (at most 3) values over all threads of the team; every thread gets
    // them.  Everything written before the call is visible after it.
    template <int N>
    __device__ __forceinline__ bool sum(long long (&v)[N], int buf)
    {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const long long s = hp::warp_sum64(v[i]);
            if (lane == 0) X.w[wid][i] = s;
        }
        __syncthreads();
        if (wid == 0) {
#pragma unroll
            for (int i = 0; i < N; i++) put(buf, i, hp::warp_sum64(X.w[lane][i]));
        }
        if (!sync()) return false;
        if (GRID) {
            if (wid == 0) {
#pragma unroll
                for (int i = 0; i < N; i++) {
                    long long s = 0;
                    for (unsigned r = lane; r < nct; r += 32) s += __ldcg(&a.gx[((size_t)buf * nct + r) * 3 + i]);
                    s = hp::warp_sum64(s);
                    if (lane == 0) X.tot[i] = s;
                }
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < N; i++) v[i] = X.tot[i];
            return true;
        }
#pragma unroll
        for (int i = 0; i < N; i++) {
            long long s = 0;
            for (unsigned r = 0; r < nct; r++) s += X.x[buf][r][i];
            v[i] = s;
        }
        return true;
    }
    // Exclusive prefix over the team's warps (rank, then warp order) of two values
    // per warp (the same in all its lanes), and their totals.
    __device__ __forceinline__ bool warp_scan2(int32_t va, int32_t vb, int32_t *ea, int32_t *eb, int32_t *ta,
                                               int32_t *tb, int buf)
    {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        if (lane == 0) { X.w[wid][0] = va; X.w[wid][1] = vb; }
        __syncthreads();
        if (wid == 0) {
            const int qa = (int)X.w[lane][0], qb = (int)X.w[lane][1];
            const int ia = hp::warp_incl_scan(qa), ib = hp::warp_incl_scan(qb);
            X.w[lane][0] = ia - qa;
            X.w[lane][1] = ib - qb;
            put(buf, 0, __shfl_sync(HP_FULL_MASK, ia, 31));
            put(buf, 1, __shfl_sync(HP_FULL_MASK, ib, 31));
        }
        if (!sync()) return false;
        int32_t pa = (int32_t)X.w[wid][0], pb = (int32_t)X.w[wid][1], xa = 0, xb = 0;
        if (GRID) {
            if (wid == 0) {
                int32_t la = 0, lb = 0;   // the CTAs before this one
                for (unsigned r = lane; r < nct; r += 32) {
                    const int32_t qa = (int32_t)__ldcg(&a.gx[((size_t)buf * nct + r) * 3]);
                    const int32_t qb = (int32_t)__ldcg(&a.gx[((size_t)buf * nct + r) * 3 + 1]);
                    if (r < rank) { la += qa; lb += qb; }
                    xa += qa;
                    xb += qb;
                }
                la = hp::warp_sum(la); lb = hp::warp_sum(lb);
                xa = hp::warp_sum(xa); xb = hp::warp_sum(xb);
                if (lane == 0) { X.tot[0] = la; X.tot[1] = lb; X.tot[2] = xa; X.tot[3] = xb; }
            }
            __syncthreads();
            pa += (int32_t)X.tot[0];
            pb += (int32_t)X.tot[1];
            xa = (int32_t)X.tot[2];
            xb = (int32_t)X.tot[3];
            __syncthreads();   // (the totals and the warps' prefixes are read)
        } else {
            for (unsigned r = 0; r < nct; r++) {
                const int32_t qa = (int32_t)X.x[buf][r][0], qb = (int32_t)X.x[buf][r][1];
                if (r < rank) { pa += qa; pb += qb; }
                xa += qa;
                xb += qb;
            }
        }
        *ea = pa;
        *eb = pb;
        *ta = xa;
        *tb = xb;
        return true;
    }
};

// The gain rows of the listed vertices (short rows by lane segments, long rows by a
// warp's dense accumulator in shared memory).
__device__ __forceinline__ void cl_rebuild(const SmallLevel &a, int gw, int tw, int32_t ns, int32_t nb, int32_t *dyn)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (ns > 0) {
        if (a.small_max <= 8)
            gain_seg_rows<8>(gw, tw, a.small_l, ns, a.xadj, a.adjncy, a.adjwgt, a.where, a.goff, a.gpart, a.gconn,
                             a.k, a.dirty);
        else if (a.small_max <= 16)
            gain_seg_rows<16>(gw, tw, a.small_l, ns, a.xadj, a.adjncy, a.adjwgt, a.where, a.goff, a.gpart, a.gconn,
                              a.k, a.dirty);
        else
            gain_seg_rows<32>(gw, tw, a.small_l, ns, a.xadj, a.adjncy, a.adjwgt, a.where, a.goff, a.gpart, a.gconn,
                              a.k, a.dirty);
    }
    if (nb > 0) {
        const int nw = (a.k + 31) >> 5;
        int32_t *dw = dyn + (size_t)wid * (a.k + nw);
        unsigned *bm = (unsigned *)(dw + a.k);
        for (int i = lane; i < a.k; i += 32) dw[i] = 0;
        for (int i = lane; i < nw; i += 32) bm[i] = 0u;
        __syncwarp();
        gain_bigwarp_rows(gw, tw, dw, bm, a.big_l, nb, a.xadj, a.adjncy, a.adjwgt, a.where, a.goff, a.gpart, a.gconn,
                          a.k, a.dirty, a.bigd, INT_MAX);
    }
}

// GRID: the CTAs of a cooperative launch instead of a cluster (grid_level).
template <bool GRID>
__global__ void __launch_bounds__(CL_THREADS, 1)
refine_loop_kernel(const __grid_constant__ SmallLevel a)
{
    hp::pdl_wait();
    extern __shared__ __align__(16) int32_t cl_dyn[];
    __shared__ hp::MlpSmem s_mlp;
    __shared__ ClXch X;
    __shared__ RefineCtl s_ctl;
    __shared__ long long s_pw[CL_KMAX];      // part weights (of the current partition)
    __shared__ int32_t s_part[CL_KMAX];      // weak: the undersized parts; strong: the parts' evicted ranges
    __shared__ int8_t s_ufl[CL_KMAX];        // weak: pw < maxp
    __shared__ int32_t s_hist[256], s_base[256];
    __shared__ int32_t s_group[2][GRID ? CL_THREADS : 1];   // digit counts before this CTA and in all, by group
    __shared__ int32_t s_scan[CL_WARPS + 2];
    __shared__ int32_t s_nu;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const unsigned lt = hp::lanemask_lt();
    ClTeam<GRID> team(a, X);
    const unsigned rank = team.rank, nct = team.nct;
    const int tw = (int)nct * CL_WARPS, gw = (int)rank * CL_WARPS + wid;
    const int gt = (int)nct * CL_THREADS, gtid = (int)rank * CL_THREADS + tid;
    const int32_t n = a.n, k = a.k;
    const int32_t vpw = (n + tw - 1) / tw;   // the warp's vertices [vb, ve)
    const int32_t vb = min(n, gw * vpw), ve = min(n, vb + vpw);
    int buf = 0;                             // exchange buffer (uniform over the cluster)
    // no CTA writes another's shared memory before that CTA runs: being placed together
    // does not mean having started
    if (!GRID && !team.sync()) return;
    if (a.learned_mlp) hp::mlp_load_smem(s_mlp, a.mlp_params);
    // ---- the level's setup, as the launches of the multi-kernel levels:
    // gain-row capacities min(deg, k) and offsets, cleared locks and dirty
    // flags, the rows' lists by length, part weights, the full gain-row build,
    // the starting cut (the coarser level's best cut, else summed from the
    // rows), the excess, the best-partition copy and the control block
    {
        int32_t *spw = cl_dyn;   // this CTA's share of the part weights (each total below 2^31)
        for (int32_t q = tid; q < k; q += CL_THREADS) spw[q] = 0;
        if (rank == 0) {
            for (int32_t q = tid; q < k; q += CL_THREADS) a.pw[q] = 0ull;
            if (tid < 8) a.counts[tid] = 0;
        }
        __syncthreads();
        int32_t caps = 0;
        for (int32_t v = vb + lane; v < ve; v += 32) {
            const int32_t d = a.xadj[v + 1] - a.xadj[v], p = a.where[v];
            caps += d < k ? d : k;
            a.lock[v] = 0;
            a.dirty[v] = 0;
            a.best_where[v] = p;
            atomicAdd(&spw[p], a.vwgt[v]);
        }
        caps = hp::warp_sum(caps);
        int32_t run, e1, total, t1;
        if (!team.warp_scan2(caps, 0, &run, &e1, &total, &t1, buf)) return;
        buf ^= 1;
        for (int32_t v0 = vb; v0 < ve; v0 += 32) {
            const int32_t v = v0 + lane;
            const bool in = v < ve;
            const int32_t d = in ? a.xadj[v + 1] - a.xadj[v] : 0;
            const int32_t cap = d < k ? d : k, incl = hp::warp_incl_scan(cap);
            if (in) a.goff[v] = run + incl - cap;
            run += __shfl_sync(HP_FULL_MASK, incl, 31);
            const bool sh = in && d <= a.bigd, lg = in && d > a.bigd;
            const int32_t ps = hp::warp_append(&a.counts[1], sh), pl = hp::warp_append(&a.counts[2], lg);
            if (sh) a.small_l[ps] = v;
            if (lg) a.big_l[pl] = v;
        }
        if (gtid == 0) a.goff[n] = total;
        for (int32_t q = tid; q < k; q += CL_THREADS)
            if (spw[q]) atomicAdd(&a.pw[q], (unsigned long long)spw[q]);
        if (!team.sync()) return;
        const int32_t ns = __ldcg(&a.counts[1]), nb = __ldcg(&a.counts[2]);
        cl_rebuild(a, gw, tw, ns, nb, cl_dyn);
        if (!team.sync()) return;
        if (rank == 0 && tid < 4) a.counts[tid] = 0;   // (the first pass's; barriers follow before its use)
        long long cut[1] = {0};
        if (!a.coarser) {   // the coarsest level: the cut from the gain rows
            for (int32_t v = vb + lane; v < ve; v += 32) {
                const int32_t p = a.where[v], o = a.goff[v], len = a.goff[v + 1] - o;
                row_walk(a.gpart, a.gconn, o, len, [&](int32_t q, int32_t cq) {
                    if (q != p) cut[0] += cq;
                });
            }
        }
        if (!team.sum(cut, buf)) return;
        buf ^= 1;
        long long m = LLONG_MIN;
        for (int32_t q = tid; q < k; q += CL_THREADS) {
            const long long w = (long long)__ldcg(&a.pw[q]), e = w - a.maxp[q];
            s_pw[q] = w;
            s_ufl[q] = e < 0;
            if (rank == 0) a.best_pw[q] = (unsigned long long)w;
            m = e > m ? e : m;
        }
        m = hp::warp_max64(m);
        if (lane == 0) X.w[wid][0] = m;
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < CL_WARPS; w++) m = X.w[w][0] > m ? X.w[w][0] : m;
            ctl_init_state(&s_ctl, a.coarser ? a.coarser->best_cut : cut[0] / 2, m, a.patience, a.learned_mlp, total,
                           a.judge);
        }
    }
    __syncthreads();
    // the control step ends the loop; the pass cap bounds it as well
    for (int32_t guard = 0; guard <= HP_MAX_REFINE_PASSES; guard++) {
        if (!s_ctl.cont) break;
        const int mode = s_ctl.mode;
        int32_t *cn = a.counts + 4 * (guard & 1);   // this pass's counters (zero; the other set is cleared below)
        long long ncand = 0, jp2 = 0, jl2 = 0;
        bool judged = false;
        long long c1 = 0;   // conn(to) - conn(from) over the moves, before any applies
        if (mode == 0) {
            // ---- LP selection (plain or learned), as lp_select[_learned]_kernel
            const bool lrn = a.learned_mlp && s_ctl.learned_pass;
            const bool jdg = lrn && s_ctl.judge_pass;
            long long my[2] = {0, 0};
            for (int32_t v0 = vb; v0 < ve; v0 += 32) {
                const int32_t v = v0 + lane;
                const bool in = v < ve;
                int32_t p = 0, o = 0, len = 0;
                if (in) {
                    p = a.where[v];
                    o = a.goff[v];
                    len = a.goff[v + 1] - o;
                }
                const RowBest rb = row_best(a.gpart, a.gconn, o, len, p, k);
                int cand = 0;
                int32_t g = NEG, d = p;
                float f[HP_MLP_IN] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                if (in && rb.b >= 0) {
                    const int64_t thr = a.finest ? rb.pc / 4 : (3 * rb.pc) / 4;
                    if ((rb.bc >= rb.pc || (rb.pc - rb.bc) < thr) && !a.lock[v]) {
                        g = (int32_t)(rb.bc - rb.pc);
                        d = rb.b;
                        cand = 1;
                        if (lrn)
                            hp::mlp_features(rb.pc, rb.bc, rb.wd, rb.np, a.xadj[v + 1] - a.xadj[v],
                                             a.maxp[d] - (int64_t)s_pw[d], a.opt[d], a.maxp[p] - (int64_t)s_pw[p],
                                             a.opt[p], a.finest, f);
                    }
                }
                int8_t pr = 0;   // dropped by the MLP: keeps the plain gain and destination for the judge
                my[1] += cand;
                if (lrn && __any_sync(HP_FULL_MASK, cand)) {   // a warp without candidates needs no scores
                    const float logit = hp::mlp_warp_logit(s_mlp, f);
                    if (cand && logit < a.mlp_threshold) {
                        cand = 0;
                        if (jdg) pr = 1;
                        else { g = NEG; d = p; }
                    }
                }
                if (in) {
                    a.pregain[v] = g;
                    a.dest[v] = d;
                    if (jdg) a.prune[v] = pr;
                }
                my[0] += cand;
            }
            if (!team.sum(my, buf)) return;   // (barrier: every selection is visible)
            buf ^= 1;
            ncand = my[0];
            judged = jdg;
            if (ncand > 0 || (jdg && my[1] > 0)) {
                // ---- afterburner: every candidate re-scored against the
                // higher-priority neighbours; locks and moves
                for (int32_t v0 = vb; v0 < ve; v0 += 32) {
                    const int32_t v = v0 + lane;
                    const bool in = v < ve;
                    const int32_t g = in ? a.pregain[v] : NEG;
                    const bool act = g != NEG;
                    const int32_t ro = act ? a.xadj[v] : 0, rl = act ? a.xadj[v + 1] - ro : 0;
                    const int32_t pp = act ? a.where[v] : 0, bb = act ? a.dest[v] : 0;
                    long long chp = 0, chl = 0;
                    const bool coop = rl > 32;
                    if (act && !coop)
                        ab_row_sum2(v, g, pp, bb, ro, ro + rl, 1, a.adjncy, a.adjwgt, a.pregain, a.dest, a.where,
                                    a.prune, jdg, chp, chl);
                    unsigned cm = __ballot_sync(HP_FULL_MASK, coop);
                    while (cm) {
                        const int src = __ffs(cm) - 1;
                        cm &= cm - 1;
                        const int32_t sv = __shfl_sync(HP_FULL_MASK, v, src), sg = __shfl_sync(HP_FULL_MASK, g, src);
                        const int32_t sp_ = __shfl_sync(HP_FULL_MASK, pp, src), sb = __shfl_sync(HP_FULL_MASK, bb, src);
                        const int32_t so = __shfl_sync(HP_FULL_MASK, ro, src), sl = __shfl_sync(HP_FULL_MASK, rl, src);
                        long long cp = 0, cl = 0;
                        ab_row_sum2(sv, sg, sp_, sb, so + lane, so + sl, 32, a.adjncy, a.adjwgt, a.pregain, a.dest,
                                    a.where, a.prune, jdg, cp, cl);
                        cp = hp::warp_sum64(cp);
                        if (jdg) cl = hp::warp_sum64(cl);
                        if (lane == src) { chp = cp; chl = cl; }
                    }
                    const bool selp = act && ((long long)g + chp >= 0);
                    const bool sel = jdg ? (act && !a.prune[v] && (long long)g + chl >= 0) : selp;
                    if (in) {
                        a.lock[v] = (int8_t)sel;
                        if (jdg) a.accp[v] = (int8_t)selp;
                    }
                    const int32_t pos = hp::warp_append(&cn[0], sel);
                    if (sel) {
                        a.moves[pos] = v;
                        a.oldp[pos] = pp;
                        c1 += g;   // the gain is conn(dest) - conn(own)
                    }
                }
                if (jdg) {
                    // ---- the judge: exact cut decrease of the plain and the
                    // learned move sets on this state, as judge_delta_kernel
                    if (!team.sync()) return;   // every lock / accp is visible
                    long long sj[2] = {0, 0};
                    for (int32_t v0 = vb; v0 < ve; v0 += 32) {
                        const int32_t v = v0 + lane;
                        const bool in = v < ve;
                        const bool mp = in && a.accp[v] != 0, ml = in && a.lock[v] != 0;
                        const bool act = mp || ml;
                        const int32_t ro = act ? a.xadj[v] : 0, rl = act ? a.xadj[v + 1] - ro : 0;
                        const int32_t pv = act ? a.where[v] : 0, dv = act ? a.dest[v] : 0;
                        const bool coop = rl > 32;
                        if (act && !coop)
                            for (int32_t j = ro; j < ro + rl; j++)
                                judge_entry(pv, dv, mp, ml, a.adjncy[j], a.adjwgt[j], a.where, a.dest, a.accp, a.lock,
                                            sj[0], sj[1]);
                        unsigned cm = __ballot_sync(HP_FULL_MASK, coop);
                        while (cm) {
                            const int src = __ffs(cm) - 1;
                            cm &= cm - 1;
                            const int32_t so = __shfl_sync(HP_FULL_MASK, ro, src), sn = __shfl_sync(HP_FULL_MASK, rl, src);
                            const int32_t spv = __shfl_sync(HP_FULL_MASK, pv, src), sdv = __shfl_sync(HP_FULL_MASK, dv, src);
                            const bool smp = __shfl_sync(HP_FULL_MASK, (int)mp, src) != 0;
                            const bool sml = __shfl_sync(HP_FULL_MASK, (int)ml, src) != 0;
                            for (int32_t j = so + lane; j < so + sn; j += 32)
                                judge_entry(spv, sdv, smp, sml, a.adjncy[j], a.adjwgt[j], a.where, a.dest, a.accp,
                                            a.lock, sj[0], sj[1]);
                        }
                    }
                    if (!team.sum(sj, buf)) return;
                    buf ^= 1;
                    jp2 = sj[0];
                    jl2 = sj[1];
                }
            }
        } else {
            // ---- rebalance, as rb_candidates / sort / rb_rank / rw_select or
            // rs_evict / cookie_cutter / rs_assign
            const bool strong = mode == 2;
            if (!strong) {   // undersized parts (pw < max(0.99 maxp, maxp - 100)) in part order; k <= CL_THREADS
                int f = 0;
                if (tid < k) {
                    const int64_t mp = a.maxp[tid];
                    int64_t md = (mp * 99) / 100;
                    if (md < mp - 100) md = mp - 100;
                    f = s_pw[tid] < md;
                }
                int tot;
                const int pos = hp::block_excl_scan<CL_THREADS>(f, &tot, s_scan);
                if (f) s_part[pos] = tid;
                if (tid == 0) s_nu = tot;
                __syncthreads();
            }
            // candidates, by each warp in vertex order at the front of its own range
            int32_t cw = 0;
            for (int32_t v0 = vb; v0 < ve; v0 += 32) {
                const int32_t v = v0 + lane;
                const bool in = v < ve;
                int32_t p = 0, vw = 0;
                bool cand = false;
                if (in) {
                    p = a.where[v];
                    vw = a.vwgt[v];
                    const int64_t pwp = s_pw[p], over = pwp - a.opt[p];
                    cand = pwp > a.maxp[p] && (strong ? (int64_t)vw < 2 * over : 2 * (int64_t)vw < 3 * over);
                }
                const int32_t o = cand ? a.goff[v] : 0, len = cand ? a.goff[v + 1] - o : 0;
                int32_t d = p, kk = -1, gain = 0;
                if (!strong) {
                    int64_t pc = 0, bc = 0;
                    int32_t b = -1;
                    const bool coop = cand && len > RB_COOP;
                    if (cand && !coop)
                        row_walk(a.gpart, a.gconn, o, len, [&](int32_t q, int32_t cq) {
                            if (q == p) pc = cq;
                            if (cq > bc && s_ufl[q]) { bc = cq; b = q; }
                        });
                    unsigned cm = __ballot_sync(HP_FULL_MASK, coop);
                    while (cm) {
                        const int src = __ffs(cm) - 1;
                        cm &= cm - 1;
                        const int32_t so = __shfl_sync(HP_FULL_MASK, o, src), sl = __shfl_sync(HP_FULL_MASK, len, src);
                        const int32_t sp_ = __shfl_sync(HP_FULL_MASK, p, src);
                        const RowBest w = warp_row_best<ROW_DEEP>(a.gpart, a.gconn, so, sl, sp_, k, [&](int32_t q) { return s_ufl[q] != 0; });
                        if (lane == src) { pc = w.pc; bc = w.bc; b = w.b; }
                    }
                    if (cand) {
                        bool ok = true;
                        if (b >= 0) gain = (int32_t)(bc - pc);
                        else if (s_nu == 0) ok = false;
                        else { b = s_part[v % s_nu]; gain = (int32_t)-pc; }   // (no connectivity to an undersized part)
                        if (ok) { d = b; kk = p * 64 + hp::gain_bucket(gain, vw); }
                    }
                } else if (cand) {
                    gain = -row_conn(a.gpart + o, a.gconn + o, len, p, k);
                    kk = p * 64 + hp::gain_bucket(gain, vw);
                }
                const unsigned m = __ballot_sync(HP_FULL_MASK, kk >= 0);
                if (kk >= 0) {
                    const int32_t pos = vb + cw + __popc(m & lt);
                    a.K[pos] = kk;
                    a.V[pos] = v;
                    a.dest[v] = d;
                    a.pregain[v] = gain;   // weak: conn(dest) - conn(own)
                }
                cw += __popc(m);
            }
            __syncwarp();
            // stable radix sort by key, digits of at most 8 bits: per-warp digit counts, their
            // prefix over the CTA's warps, the CTAs' totals read through the cluster
            int32_t *ks = a.K, *vs = a.V, *kd = a.K2, *vd = a.V2;
            int32_t ib = vb, ie = vb + cw, cnt = 0;   // the warp's items
            int32_t *wc = cl_dyn + wid * 256;
            const int passes = (a.key_bits + 7) / 8, dbits = (a.key_bits + passes - 1) / passes, bins = 1 << dbits;
            for (int shift = 0; shift < a.key_bits; shift += dbits) {
                for (int q = lane; q < bins; q += 32) wc[q] = 0;
                __syncwarp();
                for (int32_t i = ib + lane; i < ie; i += 32) atomicAdd(&wc[((unsigned)ks[i] >> shift) & (bins - 1)], 1);
                __syncthreads();
                if (tid < bins) {
                    int32_t s = 0;
#pragma unroll 8
                    for (int w = 0; w < CL_WARPS; w++) {
                        const int32_t t = cl_dyn[w * 256 + tid];
                        cl_dyn[w * 256 + tid] = s;
                        s += t;
                    }
                    if (GRID) a.ghist[(size_t)rank * 256 + tid] = s;
                    else s_hist[tid] = s;
                }
                if (!team.sync()) return;
                int32_t before = 0, all = 0;
                if (GRID) {   // a group of threads per set of CTAs, a thread per digit
                    const int groups = CL_THREADS >> dbits, per = ((int)nct + groups - 1) / groups;
                    const int dg = tid & (bins - 1), r0 = (tid >> dbits) * per, r1 = min((int)nct, r0 + per);
                    int32_t bg = 0, ag = 0;
#pragma unroll 10
                    for (int r = r0; r < r1; r++) {
                        const int32_t t = __ldcg(&a.ghist[(size_t)r * 256 + dg]);
                        if (r < (int)rank) bg += t;
                        ag += t;
                    }
                    s_group[0][tid] = bg;
                    s_group[1][tid] = ag;
                    __syncthreads();
                    if (tid < bins)
                        for (int g = 0; g < groups; g++) {
                            before += s_group[0][(g << dbits) + tid];
                            all += s_group[1][(g << dbits) + tid];
                        }
                } else if (tid < bins) {
                    for (unsigned r = 0; r < nct; r++) {
                        const int32_t t = cl_ld32(cl_map(&s_hist[tid], r));
                        if (r < rank) before += t;
                        all += t;
                    }
                }
                const int ex = hp::block_excl_scan<CL_THREADS>(all, &cnt, s_scan);
                if (tid < bins) s_base[tid] = ex + before;
                __syncthreads();
                for (int32_t i0 = ib; i0 < ie; i0 += 32) {
                    const int32_t i = i0 + lane;
                    const bool valid = i < ie;
                    const int32_t key = valid ? ks[i] : 0, val = valid ? vs[i] : 0;
                    const unsigned dg = valid ? (((unsigned)key >> shift) & (bins - 1)) : 256u + lane;
                    const unsigned peers = __match_any_sync(HP_FULL_MASK, dg);
                    const int rk = __popc(peers & lt);
                    if (valid) {
                        const int32_t pos = s_base[dg] + wc[dg] + rk;
                        kd[pos] = key;
                        vd[pos] = val;
                    }
                    __syncwarp();
                    if (valid && rk == 0) wc[dg] += __popc(peers);
                    __syncwarp();
                }
                if (!team.sync()) return;
                int32_t *t = ks; ks = kd; kd = t;
                t = vs; vs = vd; vd = t;
                const int32_t ipw = (cnt + tw - 1) / tw;
                ib = min(cnt, gw * ipw);
                ie = min(cnt, ib + ipw);
            }
            // prefix weights in sorted order; pbase[p]: the prefix at part p's first candidate
            int32_t wsum = 0;
            for (int32_t i = ib + lane; i < ie; i += 32) wsum += a.vwgt[vs[i]];
            wsum = hp::warp_sum(wsum);
            int32_t run, e1, t0, t1;
            if (!team.warp_scan2(wsum, 0, &run, &e1, &t0, &t1, buf)) return;
            buf ^= 1;
            for (int32_t i0 = ib; i0 < ie; i0 += 32) {
                const int32_t i = i0 + lane;
                const bool valid = i < ie;
                const int32_t w = valid ? a.vwgt[vs[i]] : 0, incl = hp::warp_incl_scan(w);
                if (valid) {
                    const int32_t p = ks[i] >> 6, pr = run + incl - w;
                    a.pre[i] = pr;
                    if (i == 0 || (ks[i - 1] >> 6) != p) a.pbase[p] = pr;
                }
                run += __shfl_sync(HP_FULL_MASK, incl, 31);
            }
            if (!team.sync()) return;
            // a candidate leaves its part when the part's candidates before it weigh
            // less than the part's excess (weak: the moves; strong: the evicted prefix,
            // whose end is the first candidate where that weight reaches the excess)
            int32_t nf = 0, fw = 0;
            for (int32_t i0 = ib; i0 < ie; i0 += 32) {
                const int32_t i = i0 + lane;
                int32_t p = 0, v = 0;
                bool sel = false;
                if (i < ie) {
                    p = ks[i] >> 6;
                    v = vs[i];
                    sel = (int64_t)a.pre[i] - a.pbase[p] < s_pw[p] - a.maxp[p];
                }
                if (!strong) {
                    const int32_t pos = hp::warp_append(&cn[0], sel);
                    if (sel) {
                        a.moves[pos] = v;
                        a.oldp[pos] = p;
                        c1 += a.pregain[v];
                    }
                } else {
                    nf += sel;
                    fw += sel ? a.vwgt[v] : 0;
                }
            }
            if (strong) {
                nf = hp::warp_sum(nf);
                fw = hp::warp_sum(fw);
                int32_t pc, pr, np, wt;
                if (!team.warp_scan2(nf, fw, &pc, &pr, &np, &wt, buf)) return;
                buf ^= 1;
                // the evicted vertices in sorted order and their prefix weights (rs_evict_kernel)
                for (int32_t i0 = ib; i0 < ie; i0 += 32) {
                    const int32_t i = i0 + lane;
                    bool sel = false;
                    int32_t v = 0, w = 0;
                    if (i < ie) {
                        const int32_t p = ks[i] >> 6;
                        v = vs[i];
                        sel = (int64_t)a.pre[i] - a.pbase[p] < s_pw[p] - a.maxp[p];
                        w = sel ? a.vwgt[v] : 0;
                    }
                    const unsigned m = __ballot_sync(HP_FULL_MASK, sel);
                    const int32_t incl = hp::warp_incl_scan(w);
                    if (sel) {
                        a.P[pc + __popc(m & lt)] = v;
                        a.sp[pc + __popc(m & lt)] = pr + incl - w;
                    }
                    pc += __popc(m);
                    pr += __shfl_sync(HP_FULL_MASK, incl, 31);
                }
                if (gtid == 0) a.sp[np] = wt;
                if (!team.sync()) return;
                if (rank == 0) {   // the cookie cutter, on staged prefix weights when they fit
                    const bool staged = np + 1 <= a.cookie_cap;
                    if (staged)
                        for (int32_t i = tid; i <= np; i += CL_THREADS) cl_dyn[i] = a.sp[i];
                    __syncthreads();
                    if (wid == 0)
                        cookie_cut_warp(k, (const unsigned long long *)s_pw, a.maxp, staged ? cl_dyn : a.sp, np, a.es,
                                        a.ee);
                }
                if (!team.sync()) return;
                for (int32_t q = tid; q < k; q += CL_THREADS) s_part[q] = a.es[q];
                __syncthreads();
                for (int32_t j0 = gw * 32; j0 < np; j0 += tw * 32) {   // rs_assign_kernel
                    const int32_t j = j0 + lane;
                    bool sel = false;
                    int32_t v = 0, lo = 0, from = 0;
                    if (j < np) {
                        int32_t hi = k - 1;   // last part with es[p] <= j
                        while (lo < hi) {
                            const int32_t mid = (lo + hi + 1) / 2;
                            if (s_part[mid] <= j) lo = mid; else hi = mid - 1;
                        }
                        v = a.P[j];
                        from = a.where[v];
                        sel = j < a.ee[lo] && lo != from;
                    }
                    const int32_t pos = hp::warp_append(&cn[0], sel);
                    if (sel) {
                        a.dest[v] = lo;
                        a.moves[pos] = v;
                        a.oldp[pos] = from;
                        const int32_t o = a.goff[v], len = a.goff[v + 1] - o;
                        c1 += (long long)row_conn(a.gpart + o, a.gconn + o, len, lo, k) + a.pregain[v];
                    }
                }
            }
        }
        if (!team.sync()) return;   // the moves are complete
        // ---- apply: moves, gain-row maintenance, cut change after
        const int32_t nmoves = __ldcg(&cn[0]);
        if (nmoves > 0) {
            apply_moves_rows(gw, tw, a.moves, nmoves, a.where, a.dest, a.vwgt, a.pw, a.xadj, a.adjncy, a.adjwgt,
                             a.goff, a.gconn, a.dirty, a.small_l, a.big_l, &cn[1], k, nullptr, nullptr, a.bigd,
                             INT_MAX);
            if (!team.sync()) return;
            cl_rebuild(a, gw, tw, __ldcg(&cn[1]), __ldcg(&cn[2]), cl_dyn);
        }
        if (rank == 0 && tid < 4) a.counts[4 * ((guard & 1) ^ 1) + tid] = 0;   // the next pass's set
        long long c[2] = {c1, 0};
        if (nmoves > 0) {
            if (!team.sync()) return;
            for (int32_t i = gtid; i < nmoves; i += gt) {
                const int32_t v = a.moves[i];
                const int32_t o = a.goff[v], len = a.goff[v + 1] - o;
                c[1] += row_diff(a.gpart + o, a.gconn + o, len, a.where[v], a.oldp[i], k);
            }
        }
        long long m = LLONG_MIN;
        for (int32_t q = tid; q < k; q += CL_THREADS) {
            const long long w = (long long)__ldcg(&a.pw[q]), e = w - a.maxp[q];
            s_pw[q] = w;
            s_ufl[q] = e < 0;
            m = e > m ? e : m;
        }
        m = hp::warp_max64(m);
        if (!team.sum(c, buf)) return;
        buf ^= 1;
        if (lane == 0) X.w[wid][2] = m;
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < CL_WARPS; w++) m = X.w[w][2] > m ? X.w[w][2] : m;
            // the judge's sum over the learned moves is the applied pass's exact change
            if (rank == 0 && judged && jl2 != c[0] + c[1]) atomicOr(a.status, HP_STATUS_OVERFLOW);
            ctl_advance(&s_ctl, m, c[0], c[1], nmoves, ncand, jp2);
        }
        __syncthreads();
        if (s_ctl.take) {
            for (int32_t v = vb + lane; v < ve; v += 32) a.best_where[v] = a.where[v];
            if (rank == 0)
                for (int32_t q = tid; q < k; q += CL_THREADS) a.best_pw[q] = (unsigned long long)s_pw[q];
        }
    }
    if (!s_ctl.best_current)
        for (int32_t v = vb + lane; v < ve; v += 32) a.where[v] = a.best_where[v];
    if (gtid == 0) *a.ctl = s_ctl;
}

// Graph-capture helper: records the launches of body() into `graph`.  The capture
// is always ended, also when body() fails.
template <class F>
int capture_into(hp_context *c, cudaGraph_t graph, F &&body)
{
    HP_CUDA(cudaStreamBeginCaptureToGraph(c->stream, graph, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    // event records cannot sit in conditional bodies: the kernel-class profiler
    // skips the captured launches (eager calls time them)
    c->prof_suspended = true;
    const int rc = body();
    c->prof_suspended = false;
    cudaGraph_t out = nullptr;
    const cudaError_t e = cudaStreamEndCapture(c->stream, &out);
    if (rc != HP_OK) {
        cudaGetLastError();
        return rc;
    }
    if (e != cudaSuccess) {
        fprintf(stderr, "hp: graph capture failed: %s\n", cudaGetErrorString(e));
        return HP_ERR_CUDA;
    }
    return HP_OK;
}

struct GraphHold {
    cudaGraph_t g = nullptr;
    cudaGraphExec_t x = nullptr;
    ~GraphHold()
    {
        if (x) cudaGraphExecDestroy(x);
        if (g) cudaGraphDestroy(g);
    }
};

// The pass graphs of one uncoarsening.  Destroying a graph that is still
// running waits for it, so they go to the context's reaper thread, which
// releases them once the stream has passed their launches (also on error paths).
struct GraphKeep {
    hp_context *c = nullptr;
    std::vector<std::pair<cudaGraph_t, cudaGraphExec_t>> items;
    ~GraphKeep() { hp_graph_retire(c, std::move(items)); }
};

// The level's pass loop as one CUDA graph:
//   WHILE (cont) { ctl_begin; SWITCH (mode) { LP | weak | strong }; apply; pass_end }
// pass_end sets the WHILE condition, ctl_begin the SWITCH value; nothing returns to
// the host between passes.  Launch accounting: kernels per body x passes per mode,
// read back from the control block.
// host milliseconds per step of run_passes_graph (HP_DEBUG_LEVELS diagnostics):
// create+handles, body capture, mode captures, instantiate, launch, destroy
double g_graph_host_ms[6];

int run_passes_graph(hp_context *c, HpLevel &g, RefineBufs &B, const PassCfg &P, bool both_lp, int *n_common,
                     int n_mode[3], GraphKeep *keep)
{
    using clk = std::chrono::steady_clock;
    auto tick = [](clk::time_point &t, int slot) {
        const auto now = clk::now();
        g_graph_host_ms[slot] += std::chrono::duration<double, std::milli>(now - t).count();
        t = now;
    };
    auto t = clk::now();
    GraphHold H;
    HP_CUDA(cudaGraphCreate(&H.g, 0));
    cudaGraphConditionalHandle hloop;
    HP_CUDA(cudaGraphConditionalHandleCreate(&hloop, H.g, 1, cudaGraphCondAssignDefault));
    cudaGraphNodeParams wp = {};
    wp.type = cudaGraphNodeTypeConditional;
    wp.conditional.handle = hloop;
    wp.conditional.type = cudaGraphCondTypeWhile;
    wp.conditional.size = 1;
    cudaGraphNode_t wnode;
    HP_CUDA(cudaGraphAddNode(&wnode, H.g, nullptr, 0, &wp));
    cudaGraph_t body = wp.conditional.phGraph_out[0];
    cudaGraphConditionalHandle hmode;
    HP_CUDA(cudaGraphConditionalHandleCreate(&hmode, body, 0, 0));
    cudaGraph_t mode_body[3] = {nullptr, nullptr, nullptr};
    tick(t, 0);
    const int l0 = c->launches;
    HP_TRY(capture_into(c, body, [&]() -> int {
        HP_LAUNCH(c, ctl_begin_kernel, 1, 1024, 0, P.ctl, c->d_scal, hmode, 1, P.k, B.pw, B.maxp, B.und, B.ufl);
        cudaStreamCaptureStatus cs;
        cudaGraph_t capg = nullptr;
        const cudaGraphNode_t *deps = nullptr;
        size_t ndeps = 0;
        HP_CUDA(cudaStreamGetCaptureInfo(c->stream, &cs, nullptr, &capg, &deps, &ndeps));
        cudaGraphNodeParams sp = {};
        sp.type = cudaGraphNodeTypeConditional;
        sp.conditional.handle = hmode;
        sp.conditional.type = cudaGraphCondTypeSwitch;
        sp.conditional.size = 3;
        cudaGraphNode_t snode;
        HP_CUDA(cudaGraphAddNode(&snode, capg, deps, ndeps, &sp));
        for (int i = 0; i < 3; i++) mode_body[i] = sp.conditional.phGraph_out[i];
        HP_CUDA(cudaStreamUpdateCaptureDependencies(c->stream, &snode, 1, cudaStreamSetCaptureDependencies));
        return pass_apply(c, g, B, P, hloop, 1);
    }));
    *n_common = c->launches - l0;
    tick(t, 1);
    for (int m = 0; m < 3; m++) {
        const int l1 = c->launches;
        HP_TRY(capture_into(c, mode_body[m], [&]() -> int { return pass_propose(c, g, B, P, m, false, both_lp); }));
        n_mode[m] = c->launches - l1;
    }
    c->launches = l0;
    tick(t, 2);
    HP_CUDA(cudaGraphInstantiate(&H.x, H.g, 0));
    tick(t, 3);
    HP_CUDA(cudaGraphLaunch(H.x, c->stream));
    tick(t, 4);
    keep->items.emplace_back(H.g, H.x);   // released after the stream has finished
    H.g = nullptr;
    H.x = nullptr;
    tick(t, 5);
    return HP_OK;
}

// Enqueues the refinement of one level; nothing is read back unless the eager
// loop, the kernel-class profiler or the move log needs it.  The level's control
// block (ctl) holds its cuts and pass count when the stream reaches the end.
// CUDA-graph pass loop unless the caller asked for eager launches, the move log
// or the per-pass debug log is on, or the stream is the legacy one.
bool graph_loop(const hp_context *c)
{
    const bool recording = c->opt.learned == 2 && c->log_x != nullptr;
    return !c->opt.eager && c->tune.graph_passes && !recording && getenv("HP_DEBUG_PASSES") == nullptr &&
           c->opt.refine_patience >= 0 &&
           c->stream != nullptr && c->stream != cudaStreamLegacy;
}

// Kernels per pass body of a graphed level (for the launch count, resolved
// with the control block's pass counts once the stream has finished).
struct LevelLaunches {
    bool graph = false;
    int n_common = 0, n_mode[3] = {0, 0, 0};
    int gain_tok = -1;   // profiler interval of the level's gain build (bytes completed at the end)
};

// Cooperative launches of one device, from any context and thread, follow one another:
// each takes every SM, and two that were half resident would wait for each other.  The
// event of the latest one belongs to the context that launched it, which takes itself out
// when it is destroyed.  A context that the caller left behind at a device reset has
// another CUDA context's id: its event is gone, and so is its launch.
struct CoopOrder {
    std::mutex mu;
    const hp_context *last = nullptr;
};

CoopOrder &coop_order(int device)
{
    static CoopOrder order[64];
    return order[device & 63];
}

// Launches the level's loop on `ctas` CTAs.  *refused: the device does not place them all
// at once (its SMs are shared out since the context was made); nothing was launched, and
// the level takes launched passes.
int coop_launch(hp_context *c, int ctas, size_t smem, const SmallLevel &a, bool *refused)
{
    CoopOrder &o = coop_order(c->device);
    std::lock_guard<std::mutex> lk(o.mu);
    if (o.last && o.last->cuda_ctx == c->cuda_ctx) HP_CUDA(cudaStreamWaitEvent(c->stream, o.last->coop_ev, 0));
    const cudaError_t e = c->refuse_coop ? cudaErrorCooperativeLaunchTooLarge :
                                           hp_launch_coop(c, refine_loop_kernel<true>, (unsigned)ctas, CL_THREADS, smem, a);
    *refused = e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources;
    if (*refused) {
        cudaGetLastError();
        return HP_OK;
    }
    HP_CUDA(e);
    c->launches++;
    HP_CUDA(cudaEventRecord(c->coop_ev, c->stream));
    o.last = c;
    return HP_OK;
}

// Levels above a cluster's that run their pass loop in one cooperative launch over the
// whole GPU: see GRID_LEVEL_MAX.  Not under the eager loop (the batch workers' contexts
// share the GPU, and a cooperative launch waits for all of it).
bool grid_size(const hp_context *c, const HpLevel &g, int32_t k)
{
    return c->grid_ctas > 0 && c->tune.small_level_n > 0 && !c->opt.eager && g.n <= GRID_LEVEL_MAX && k <= CL_KMAX &&
           g.m <= CL_DEG * (int64_t)g.n;
}

// Vertices per warp of the loop kernel that may take the level (LevelStat::range_entries).
int32_t loop_range(const hp_context *c, const HpLevel &g, int32_t k)
{
    const int64_t warps = CL_WARPS * (int64_t)(cluster_size(c, g, k) ? cluster_ctas(c, g.n, g.m) :
                                               grid_size(c, g, k) ? c->grid_ctas : 0);
    return warps > 0 ? (int32_t)((g.n + warps - 1) / warps) : 0;
}

int refine_level(hp_context *c, HpLevel &g, int32_t k, bool finest, const int64_t *d_opt,
                 const int64_t *d_maxp, const LevelStat &ls, RefineCtl *ctl, const RefineCtl *coarser,
                 LevelLaunches *ll, GraphKeep *keep)
{
    const int32_t n = g.n;
    if (n == 0) return HP_OK;
    const size_t mark = c->hi;
    RefineBufs B{};
    B.opt = d_opt;
    B.maxp = d_maxp;
    int32_t **n_arrays[] = {&B.goff, &B.big, &B.dest, &B.pregain, &B.moves, &B.oldp, &B.dirty,
                            &B.small_l, &B.big_l, &B.best_where, &B.K, &B.V, &B.K2, &B.V2, &B.pre,
                            &B.P, &B.sp, &B.huge_mv, &B.huge, &B.recof};
    for (auto pp : n_arrays) *pp = ralloc_t<int32_t>(c, (int64_t)n + 1);
    int32_t **k_arrays[] = {&B.pstart, &B.und, &B.es, &B.ee};
    for (auto pp : k_arrays) *pp = ralloc_t<int32_t>(c, k);
    B.lock = ralloc_t<int8_t>(c, n);
    B.prune = ralloc_t<int8_t>(c, n);
    B.accp = ralloc_t<int8_t>(c, n);
    B.jlist = ralloc_t<int32_t>(c, (int64_t)n + 1);
    B.joff = ralloc_t<int32_t>(c, (int64_t)n + 2);
    B.ufl = ralloc_t<int8_t>(c, k);
    B.pw = ralloc_t<unsigned long long>(c, k);
    unsigned long long *best_pw = ralloc_t<unsigned long long>(c, k);
    // at most m / (t + 1) rows are longer than t: the long-row lists of the
    // afterburner (t = chunk_deg) and of the moves (t = apply_chunk_deg) share
    // the chunk-plan buffers
    const int32_t huged = c->tune.gain_hub_deg, chunkd = c->tune.chunk_deg, mchunkd = c->tune.apply_chunk_deg;
    const int64_t nhub_cap =
        std::min<int64_t>((int64_t)n, g.m / ((int64_t)std::min(chunkd, mchunkd) + 1)) + 1;
    if (2 * (nhub_cap / PLAN_TILE + 1) > c->lb_cap) return HP_ERR_INTERNAL;
    B.nhub_cap = nhub_cap;
    B.ab_acc = ralloc_t<unsigned long long>(c, nhub_cap);
    B.ab_acc2 = ralloc_t<unsigned long long>(c, nhub_cap);
    // at most m / (huged + 1) rows are longer than huged
    B.hub = ralloc_t<int32_t>(c, std::min<int64_t>((int64_t)n, g.m / ((int64_t)huged + 1)) + 1);
    B.plan_v = ralloc_t<int32_t>(c, nhub_cap);
    B.plan_item = ralloc_t<int32_t>(c, nhub_cap);
    B.plan_off = ralloc_t<int32_t>(c, nhub_cap);
    B.plan_cnt = ralloc_t<int32_t>(c, 2);
    HP_CHECK_OOM(c);
    // learned LP proposals (opt.learned = 1, or 3 with the plain refiner as the
    // judge of every learned pass) until a learned pass fails to
    // improve the exact cut; then the plain rule for the rest of the level
    const bool learned = (c->opt.learned == 1 || c->opt.learned == 3) && c->mlp_ready && c->learned_skewed;
    const bool judged = learned && c->opt.learned == 3;
    const bool recording = c->opt.learned == 2 && c->log_x != nullptr;
    const int patience = c->opt.refine_patience;
    const bool dbg = getenv("HP_DEBUG_PASSES") != nullptr;
    // small levels: the whole pass loop in one cluster (same rule, same result), in
    // either loop mode unless the per-pass move log or pass log is on
    const bool loop = !recording && !dbg && loop_rows(g, ls);
    const bool small_level = loop && cluster_size(c, g, k);
    const bool grid_level = loop && !cluster_size(c, g, k) && !learned && ls.maxdeg <= GRID_DEG_MAX &&
                            grid_size(c, g, k);
    const size_t loop_mark = c->hi;
    if (small_level || grid_level) {
        // the level's setup (gain rows, part weights, cut, control block) runs
        // inside the kernel: no launch per setup step
        B.gpart = ralloc_t<int32_t>(c, std::max<int64_t>(g.m, 1));
        B.gconn = ralloc_t<int32_t>(c, std::max<int64_t>(g.m, 1));
        B.small_max = ls.small_max;
        HP_CHECK_OOM(c);
        SmallLevel a{};
        a.n = n;
        a.k = k;
        a.finest = finest ? 1 : 0;
        a.bigd = c->tune.gain_thread_deg;
        a.small_max = B.small_max;
        a.key_bits = key_bits_for(k);
        a.learned_mlp = learned ? 1 : 0;
        a.patience = patience;
        a.judge = judged ? 1 : 0;
        a.coarser = coarser;
        a.mlp_threshold = c->mlp_threshold;
        a.xadj = g.xadj;
        a.adjncy = g.adjncy;
        a.adjwgt = g.adjwgt;
        a.vwgt = g.vwgt;
        a.where = g.where;
        a.goff = B.goff;
        a.gpart = B.gpart;
        a.gconn = B.gconn;
        a.dest = B.dest;
        a.pregain = B.pregain;
        a.moves = B.moves;
        a.oldp = B.oldp;
        a.dirty = B.dirty;
        a.small_l = B.small_l;
        a.big_l = B.big_l;
        a.best_where = B.best_where;
        a.K = B.K;
        a.V = B.V;
        a.K2 = B.K2;
        a.V2 = B.V2;
        a.pre = B.pre;
        a.P = B.P;
        a.sp = B.sp;
        a.pbase = B.pstart;
        a.counts = (int32_t *)c->d_scal;
        a.es = B.es;
        a.ee = B.ee;
        a.lock = B.lock;
        a.prune = B.prune;
        a.accp = B.accp;
        a.status = c->d_status;
        a.pw = B.pw;
        a.best_pw = best_pw;
        a.opt = B.opt;
        a.maxp = B.maxp;
        a.mlp_params = c->mlp_params;
        a.ctl = ctl;
        const size_t smem = small_level_smem(n, k);
        a.cookie_cap = (int32_t)(smem / sizeof(int32_t));
        if (grid_level) {
            const int ctas = c->grid_ctas;
            a.bar = ralloc_t<unsigned>(c, 1);
            a.gx = ralloc_t<long long>(c, 2 * 3 * (int64_t)ctas);
            a.ghist = ralloc_t<int32_t>(c, 256 * (int64_t)ctas);
            HP_CHECK_OOM(c);
            // (hp_test_grid_expiry: one arrival short, so the first barrier never completes)
            a.spin_limit = c->grid_short ? 1u << 14 : HP_SPIN_LIMIT;
            HP_CUDA(cudaMemsetAsync(a.bar, c->grid_short ? 0xff : 0, sizeof(unsigned), c->stream));
            HP_CUDA(cudaMemsetAsync(c->d_scal, 0, sizeof(unsigned long long) * S_PASS_END, c->stream));
            bool refused = false;
            HP_TRY(coop_launch(c, ctas, smem, a, &refused));
            if (!refused) {
                c->hi = mark;
                return HP_OK;
            }
            c->hi = loop_mark;   // (what the loop took)
        } else {
            const int ctas = cluster_ctas(c, n, g.m);
            HP_LAUNCH_CLUSTER(c, refine_loop_kernel<false>, ctas, ctas, CL_THREADS, smem, a);
            c->hi = mark;
            return HP_OK;
        }
    }
    unsigned long long *sc = c->d_scal;
    HP_CUDA(cudaMemsetAsync(sc, 0, sizeof(unsigned long long) * (S_DONE + 1), c->stream));
    int32_t *d_bigcnt = (int32_t *)&sc[S_BIGCNT];
    HP_LAUNCH(c, gain_cap_kernel, nblk(n), 256, 0, n, g.xadj, k, B.goff, B.big, B.huge, B.hub, d_bigcnt,
              c->tune.gain_thread_deg, chunkd, huged);
    if (ls.maxdeg > chunkd) {
        HP_CUDA(cudaMemsetAsync(B.ab_acc, 0, sizeof(unsigned long long) * (size_t)nhub_cap, c->stream));
        HP_CUDA(cudaMemsetAsync(B.ab_acc2, 0, sizeof(unsigned long long) * (size_t)nhub_cap, c->stream));
    }
    HP_TRY(hp_scan_excl(c, B.goff, B.goff, n));
    // the gain rows take G = sum min(deg, k) <= m entries: allocated for m, so
    // that no count is read back (the gain-build class completes its byte
    // count with G from the control block at the end of uncoarsening)
    B.small_max = ls.small_max;
    B.huge_rows = ls.maxdeg > huged;
    B.dense_rows = ls.maxdeg >= k;
    B.deep_rows = B.dense_rows && k > 64;
    B.gpart = ralloc_t<int32_t>(c, std::max<int64_t>(g.m, 1));
    B.gconn = ralloc_t<int32_t>(c, std::max<int64_t>(g.m, 1));
    HP_CHECK_OOM(c);
    const bool any_big = ls.nbig > 0;
    int tok = hp_prof_begin(c);
    HP_TRY(build_rows(c, g, B, k, nullptr, nullptr, B.big, d_bigcnt, any_big, nullptr, B.hub, d_bigcnt + 4));
    // xadj, adjncy, adjwgt, where (own), goff in; gain rows (8 G) out
    hp_prof_end(c, tok, HP_PROF_GAIN, 4 * ((int64_t)n + 1) + 8 * g.m + 4 * (int64_t)n + 4 * ((int64_t)n + 1));
    ll->gain_tok = tok;
    HP_CUDA(cudaMemsetAsync(B.pw, 0, sizeof(unsigned long long) * (size_t)k, c->stream));
    HP_CUDA(cudaMemsetAsync(B.lock, 0, (size_t)n, c->stream));
    HP_CUDA(cudaMemsetAsync(B.dirty, 0, sizeof(int32_t) * (size_t)n, c->stream));
    HP_LAUNCH(c, pw_kernel, (unsigned)std::min<int64_t>(nblk(n), c->sm_count * 8), 256,
              k <= 2048 ? sizeof(unsigned long long) * k : 0, n, g.where, g.vwgt, B.pw, k);
    if (!coarser)   // the coarsest level; the others start from the coarser level's best cut
        HP_LAUNCH(c, rowcut_kernel, nblk(n), 256, 0, n, B.goff, B.gpart, B.gconn, g.where, &sc[S_CUT2]);
    HP_LAUNCH(c, excess_kernel, 1, 1024, 0, k, B.pw, B.maxp, (long long *)&sc[S_EXCESS]);
    HP_CUDA(cudaMemcpyAsync(B.best_where, g.where, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, c->stream));
    HP_CUDA(cudaMemcpyAsync(best_pw, B.pw, sizeof(unsigned long long) * k, cudaMemcpyDeviceToDevice, c->stream));

    HP_LAUNCH(c, ctl_init_kernel, 1, 1, 0, ctl, (const unsigned long long *)sc, patience, learned ? 1 : 0,
              (const int32_t *)(B.goff + n), coarser, judged ? 1 : 0);
    int64_t log_r0 = 0;
    if (recording) {
        unsigned long long lc = 0;
        HP_TRY(hp_read_scalars(c, c->log_count, sizeof(lc), &lc));
        log_r0 = (int64_t)std::min<unsigned long long>(lc, (unsigned long long)c->log_cap);
    }
    PassCfg P{k, finest, any_big, recording, ls.maxdeg > chunkd, judged, ls.maxdeg > mchunkd, ctl, best_pw};
    const bool use_graph = graph_loop(c);
    RefineCtl h{};
    if (use_graph) {
        ll->graph = true;
        HP_TRY(run_passes_graph(c, g, B, P, learned, &ll->n_common, ll->n_mode, keep));
        HP_LAUNCH(c, restore_best_kernel, std::min<unsigned>(nblk(n), (unsigned)(c->sm_count * 4)), 256, 0, ctl, n,
                  B.best_where, g.where);
    } else {
        HP_TRY(hp_read_scalars(c, ctl, sizeof(h), &h));
        while (h.cont) {
            HP_LAUNCH(c, ctl_begin_kernel, 1, 1024, 0, ctl, sc, cudaGraphConditionalHandle{}, 0, k, B.pw, B.maxp,
                      B.und, B.ufl);
            HP_TRY(pass_propose(c, g, B, P, h.mode, h.learned_pass != 0, false));
            HP_TRY(pass_apply(c, g, B, P, 0, 0));
            HP_TRY(hp_read_scalars(c, ctl, sizeof(h), &h));
            if (dbg)
                fprintf(stderr, "gpu pass n=%d pass=%d mode=%d moves=%lld cut=%lld excess=%lld\n", n,
                        h.passes - (h.cont ? 1 : 0), h.last_mode, h.last_moves, h.cut, h.excess);
        }
        HP_LAUNCH(c, restore_best_kernel, std::min<unsigned>(nblk(n), (unsigned)(c->sm_count * 4)), 256, 0, ctl, n,
                  B.best_where, g.where);
    }
    if (recording) {
        unsigned long long lc = 0;
        HP_TRY(hp_read_scalars(c, c->log_count, sizeof(lc), &lc));
        const int64_t r1 = (int64_t)std::min<unsigned long long>(lc, (unsigned long long)c->log_cap);
        if (r1 > log_r0)
            HP_LAUNCH(c, log_label_kernel, nblk(r1 - log_r0), 256, 0, log_r0, r1, g.where, c->log_v, c->log_d,
                      c->log_acc, c->log_y);
    }
    c->hi = mark;
    return HP_OK;
}

}  // namespace

int hp_refine_init(hp_context *c)
{
    HP_CUDA(cudaFuncSetAttribute(cookie_cutter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(int32_t) * COOKIE_SMEM_INTS)));
    const int bytes = HP_MAX_PARTS * 4 + (HP_MAX_PARTS / 32) * 4;
    HP_CUDA(cudaFuncSetAttribute(gain_dense_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    const size_t smem = small_level_smem(CL_LEVEL_MAX, CL_KMAX);
    HP_CUDA(cudaFuncSetAttribute(refine_loop_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    HP_CUDA(cudaFuncSetAttribute(refine_loop_kernel<false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    // the CTAs of a cooperative launch of the grid variant: one per SM
    HP_CUDA(cudaFuncSetAttribute(refine_loop_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0, coop = 0;
    HP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, refine_loop_kernel<true>, CL_THREADS, smem));
    HP_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device));
    using GetId = CUresult (*)(CUcontext, unsigned long long *);
    void *get_id = nullptr;
    cudaDriverEntryPointQueryResult found;
    HP_CUDA(cudaGetDriverEntryPoint("cuCtxGetId", &get_id, cudaEnableDefault, &found));
    const bool id = found == cudaDriverEntryPointSuccess && ((GetId)get_id)(nullptr, &c->cuda_ctx) == CUDA_SUCCESS;
    HP_CUDA(cudaEventCreateWithFlags(&c->coop_ev, cudaEventDisableTiming));
    c->grid_ctas = id && coop && per_sm > 0 && c->device < 64 ? c->sm_count : 0;
    // the largest cluster the device can place
    c->max_cluster = 1;
    for (int q = CL_MAX; q > 1; q /= 2) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(q);
        cfg.blockDim = dim3(CL_THREADS);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)q;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, refine_loop_kernel<false>, &cfg) == cudaSuccess && fit > 0) {
            c->max_cluster = q;
            break;
        }
        cudaGetLastError();
    }
    return HP_OK;
}

void hp_refine_close(hp_context *c)
{
    {
        CoopOrder &o = coop_order(c->device);
        std::lock_guard<std::mutex> lk(o.mu);
        if (o.last == c) o.last = nullptr;
    }
    if (c->coop_ev) cudaEventDestroy(c->coop_ev);
}

int hp_uncoarsen(hp_context *c, int32_t nparts, const int64_t *h_opt, const int64_t *h_maxp)
{
    const int L = (int)c->levels.size() - 1;
    int64_t *d_opt = lalloc_t<int64_t>(c, nparts);
    int64_t *d_maxp = lalloc_t<int64_t>(c, nparts);
    LevelStat *d_ls = lalloc_t<LevelStat>(c, L + 1);
    RefineCtl *d_ctl = lalloc_t<RefineCtl>(c, L + 1);
    HP_CHECK_OOM(c);
    HP_CUDA(cudaMemcpyAsync(d_opt, h_opt, sizeof(int64_t) * nparts, cudaMemcpyHostToDevice, c->stream));
    HP_CUDA(cudaMemcpyAsync(d_maxp, h_maxp, sizeof(int64_t) * nparts, cudaMemcpyHostToDevice, c->stream));
    // every level's degree statistics in one read: afterwards the levels are
    // enqueued without waiting, so the host builds level l-1's pass graph while
    // the device runs level l
    HP_CUDA(cudaMemsetAsync(d_ls, 0, sizeof(LevelStat) * (size_t)(L + 1), c->stream));
    HP_CUDA(cudaMemsetAsync(d_ctl, 0, sizeof(RefineCtl) * (size_t)(L + 1), c->stream));
    for (int l = 0; l <= L; l++)
        if (c->levels[l].n > 0)
            HP_LAUNCH(c, level_stats_kernel, std::min<unsigned>(nblk(c->levels[l].n), (unsigned)(c->sm_count * 8)),
                      256, 0, c->levels[l].n, c->levels[l].xadj, d_ls + l, c->tune.gain_thread_deg,
                      loop_range(c, c->levels[l], nparts), loop_weight(nparts));
    std::vector<LevelStat> ls(L + 1);
    HP_CUDA(cudaMemcpyAsync(ls.data(), d_ls, sizeof(LevelStat) * (size_t)(L + 1), cudaMemcpyDeviceToHost,
                            c->stream));
    HP_CUDA(cudaStreamSynchronize(c->stream));
    // The learned move proposals run on inputs whose degree distribution is as
    // skewed as the power-law graphs the network was trained for and validated on
    // (largest degree at least HP_LEARNED_SKEW times the mean degree; R-MAT scale
    // 22: 10^4; the 3-D grid and the RGG: 1-3); on the others the plain refiner
    // runs, as it would after a hand-over.
    {
        const HpLevel &g0 = c->levels[0];
        const int64_t mean0 = std::max<int64_t>(1, g0.m / std::max<int64_t>(1, g0.n));
        c->learned_skewed = (int64_t)ls[0].maxdeg >= HP_LEARNED_SKEW * mean0;
    }
    std::vector<LevelLaunches> ll(L + 1);
    GraphKeep keep;
    keep.c = c;
    const bool trace = c->opt.trace != 0;
    // HP_DEBUG_LEVELS: per-level size, passes, device time, host enqueue time and
    // whether the device had gone idle before the level was enqueued (stderr,
    // printed after the last level so that nothing is serialised)
    const bool dbg_levels = getenv("HP_DEBUG_LEVELS") != nullptr;
    std::vector<cudaEvent_t> lev;
    std::vector<double> host_ms(L + 1, 0.0);
    std::vector<int> idle(L + 1, 0);
    if (dbg_levels) {
        lev.resize(2 * (L + 1));
        for (auto &e : lev) HP_CUDA(cudaEventCreate(&e));
    }
    for (int l = L; l >= 0; l--) {
        HpLevel &g = c->levels[l];
        const auto t0 = std::chrono::steady_clock::now();
        if (dbg_levels) {
            idle[l] = cudaStreamQuery(c->stream) == cudaSuccess;
            HP_CUDA(cudaEventRecord(lev[2 * l], c->stream));
        }
        if (l < L)
            HP_LAUNCH(c, project_kernel, nblk(g.n), 256, 0, g.n, g.cmap, c->levels[l + 1].where, g.where);
        if (trace) {
            g.where_start = lalloc_t<int32_t>(c, g.n);
            g.where_final = lalloc_t<int32_t>(c, g.n);
            HP_CHECK_OOM(c);
            HP_CUDA(cudaMemcpyAsync(g.where_start, g.where, sizeof(int32_t) * g.n, cudaMemcpyDeviceToDevice, c->stream));
        }
        HP_TRY(refine_level(c, g, nparts, l == 0, d_opt, d_maxp, ls[l], d_ctl + l,
                            l < L && c->levels[l + 1].n > 0 ? d_ctl + l + 1 : nullptr, &ll[l], &keep));
        if (dbg_levels) {
            HP_CUDA(cudaEventRecord(lev[2 * l + 1], c->stream));
            host_ms[l] = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        }
        if (trace)
            HP_CUDA(cudaMemcpyAsync(g.where_final, g.where, sizeof(int32_t) * g.n, cudaMemcpyDeviceToDevice, c->stream));
    }
    // results of every level: cuts and pass counts from the control blocks
    std::vector<RefineCtl> hc(L + 1);
    HP_CUDA(cudaMemcpyAsync(hc.data(), d_ctl, sizeof(RefineCtl) * (size_t)(L + 1), cudaMemcpyDeviceToHost,
                            c->stream));
    HP_CUDA(cudaStreamSynchronize(c->stream));
    if (dbg_levels) {
        for (int l = L; l >= 0; l--) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, lev[2 * l], lev[2 * l + 1]);
            fprintf(stderr, "gpu level %d n=%d m=%lld passes=%d ms=%.3f host_ms=%.3f idle_before=%d\n", l,
                    c->levels[l].n, (long long)c->levels[l].m, hc[l].passes, ms, host_ms[l], idle[l]);
        }
        for (auto e : lev) cudaEventDestroy(e);
        fprintf(stderr, "graph host ms: create %.3f body %.3f modes %.3f instantiate %.3f launch %.3f destroy %.3f\n",
                g_graph_host_ms[0], g_graph_host_ms[1], g_graph_host_ms[2], g_graph_host_ms[3], g_graph_host_ms[4],
                g_graph_host_ms[5]);
        for (double &x : g_graph_host_ms) x = 0.0;
    }
    int total_passes = 0;
    for (int l = 0; l <= L; l++) {
        HpLevel &g = c->levels[l];
        g.cut_start = g.n > 0 ? hc[l].cut_start : 0;
        g.cut_final = g.n > 0 ? hc[l].best_cut : 0;
        total_passes += hc[l].passes;
        hp_prof_add_bytes(c, ll[l].gain_tok, 8 * (int64_t)hc[l].gain_entries);
        if (ll[l].graph)   // the graph's own launch + its kernels per pass
            c->launches += 1 + hc[l].passes * ll[l].n_common + hc[l].mode_passes[0] * ll[l].n_mode[0] +
                           hc[l].mode_passes[1] * ll[l].n_mode[1] + hc[l].mode_passes[2] * ll[l].n_mode[2];
    }
    c->stats.refine_passes = total_passes;
    return hp_check_status(c);
}
