// hp_initpart.cu — initial k-way partition of the coarsest graph by batched
// recursive bisection.
//
// Reference behaviour replaced (HunyuanGraph):
//   hunyuangraph_gpu_initialpartition        hunyuangraph_GPU_initialpartition.h:4405-4498
//   hunyuangraph_gpu_RecursiveBisection      :3913-4386  (one recursion call per
//     subgraph, each with its own launches and device->host reads)
//   per-warp BFS growth + 2-way FM           :2426, :3035 (curand start sampling)
//   hunyuangraph_gpu_SplitGraph_intersect    hunyuangraph_GPU_splitgraph.h:802-945
//   CPU growth / FM the trials follow        hunyuangraph_CPU_initialpartition.h:36-145,
//                                            hunyuangraph_CPU_2wayrefine.h:77-245
// Here every subgraph of one recursion depth lives in one "forest" CSR and a
// depth costs a fixed handful of launches: trials (one thread per start vertex
// of every subgraph), best-trial selection (one CTA per subgraph), and a
// scan-based split that builds the next depth's forest.  Start vertices are
// evenly spaced instead of random, FM's priority queue is ordered by
// (gain desc, vertex asc), so every trial is reproducible.
#include <algorithm>
#include <vector>

#include "hp_internal.cuh"
#include "hp_rowagg.cuh"

// Shared memory for the trial states of one CTA (<= 227 KB per CTA on B200).
#define HP_TRIAL_SMEM (200 * 1024)

namespace {

struct SubInfo {
    int32_t vbeg, n;
    int32_t tbeg, ntr;
    int64_t tv, want1, onemin, onemax;
    int64_t slab_off;
};

// One BFS-growth + FM bisection trial per group of G threads: a warp, or a CTA of
// TC_THREADS on large or dense subgraphs.  Trial state lives in shared memory
// when the largest subgraph of the depth fits (SMEM), else in a global slab.
//
// FM without a heap: the reference's priority queues
// (hunyuangraph_CPU_2wayrefine.h:117-225, hunyuangraph_priorityqueue.h) only
// ever hold the boundary vertices that have not moved in the pass, keyed by
// ed[v]-id[v] (every insert/update/delete keeps that invariant), so popping side
// `from` is an argmax of (ed-id desc, v asc) over them, which is exact and
// needs no heap maintenance on dense coarse graphs.  A vertex is on the boundary
// exactly when ed > 0, or when it has no neighbours, in every state the
// reference's insert and delete rules reach.  So the state keeps per vertex
//   ed     the external weight, gain = ed - id,
//   pop    gain while the vertex may be popped, INT_MIN otherwise,
//   side, moved,
// and the pop reads one 16-byte load of pop[] and one 4-byte load of side[] per
// four vertices, all independent, where reading a boundary flag, then the moved
// mark, the side and the two weights chained four shared-memory latencies per
// vertex.  A trial is one dependent chain of moves on an otherwise idle SM, so
// its latency per move is its cost; the argmax across lanes is two redux.sync.
// The whole initial partition, before and after: 128^3 grid, k = 64 (510 vertices)
// 3.8 -> 1.7 ms; R-MAT scale 20, k = 256 (900 vertices of 286 entries) 8.8 -> 3.7 ms;
// RGG 2^24, k = 1024 (1,934 vertices) 8.6 -> 3.7 ms.
struct TrialState {
    int8_t *side, *mark;              // mark: visited (growth), then moved (FM)
    int32_t *pop, *gain, *ed, *list;  // list: the growth's queue, then the pass's moves
};

__host__ __device__ inline int32_t pad4(int32_t n) { return (n + 3) & ~3; }

__host__ __device__ inline int64_t state_bytes(int32_t n)
{
    return (((int64_t)2 * pad4(n) + 15) & ~(int64_t)15) + (int64_t)16 * pad4(n);
}

__device__ __forceinline__ TrialState carve(char *p, int32_t n)
{
    const int32_t np = pad4(n);
    TrialState t;
    t.side = (int8_t *)p;
    t.mark = t.side + np;
    int32_t *ip = (int32_t *)(p + (((int64_t)2 * np + 15) & ~(int64_t)15));   // (16-byte aligned)
    t.pop = ip;
    t.gain = ip + np;
    t.ed = ip + 2 * np;
    t.list = ip + 3 * np;
    return t;
}

constexpr int TC_THREADS = 256;   // a CTA per trial
constexpr int64_t TC_DEG = 64;    // ... also where the rows are at least this long on average
constexpr int TW_WARPS = 4;       // a warp per trial: trials per CTA at most

template <int G>
__device__ __forceinline__ void trial_sync()
{
    if (G == 32) __syncwarp();
    else __syncthreads();
}

constexpr int GROW_DEPTH = 4;

// BFS growth of side 0 by one warp (hunyuangraph_CPU_initialpartition.h:66-120);
// returns the weight of side 0.  Once every vertex is visited a row adds nothing
// to the queue and is not read.
__device__ __forceinline__ int64_t trial_grow(const TrialState &T, int32_t n, const int32_t *__restrict__ xadj,
                                              const int32_t *__restrict__ fadj, const int32_t *__restrict__ vwgt,
                                              int32_t start, int64_t tv, int64_t onemin, int64_t onemax)
{
    const int lane = threadIdx.x & 31;
    int64_t pw0 = 0, pw1 = tv;
    for (int32_t v = lane; v < n; v += 32) { T.side[v] = 1; T.mark[v] = 0; }
    __syncwarp();
    int32_t first = 0, last = 1, nleft = n - 1, next_unvis = 0;
    bool drain = false;
    if (lane == 0) { T.list[0] = start; T.mark[start] = 1; }
    __syncwarp();
    for (;;) {
        if (first == last) {
            if (nleft == 0 || drain) break;
            // lowest unvisited vertex
            for (;;) {
                const int32_t v = next_unvis + lane;
                const bool un = v < n && !T.mark[v];
                const unsigned m = __ballot_sync(HP_FULL_MASK, un);
                if (m) { next_unvis += __ffs(m) - 1; break; }
                next_unvis += 32;
            }
            if (lane == 0) { T.list[0] = next_unvis; T.mark[next_unvis] = 1; }
            __syncwarp();
            first = 0; last = 1; nleft--;
        }
        const int32_t i = T.list[first++];
        const int32_t wi = vwgt[i];
        if (pw0 > 0 && pw1 - wi < onemin) { drain = true; continue; }
        if (lane == 0) T.side[i] = 0;
        pw0 += wi; pw1 -= wi;
        if (pw1 <= onemax) break;
        drain = false;
        // GROW_DEPTH chunks of 32 entries in flight, taken in row order
        const int32_t e = xadj[i + 1];
        for (int32_t j0 = xadj[i]; j0 < e && nleft > 0; j0 += 32 * GROW_DEPTH) {
            int32_t k[GROW_DEPTH];
#pragma unroll
            for (int q = 0; q < GROW_DEPTH; q++) {
                const int32_t j = j0 + 32 * q + lane;
                k[q] = j < e ? fadj[j] : -1;
            }
#pragma unroll
            for (int q = 0; q < GROW_DEPTH; q++) {
                if (j0 + 32 * q >= e) break;
                const bool un = k[q] >= 0 && !T.mark[k[q]];
                const unsigned m = __ballot_sync(HP_FULL_MASK, un);
                if (un) { T.list[last + __popc(m & hp::lanemask_lt())] = k[q]; T.mark[k[q]] = 1; }
                last += __popc(m);
                nleft -= __popc(m);
                __syncwarp();
            }
        }
    }
    __syncwarp();
    return pw0;
}

// The trial's FM neighbour update after h moved to `to` (all G threads).
template <int G>
__device__ __forceinline__ void trial_relax(const TrialState &T, int t, int32_t b, int32_t e, int to,
                                            const int32_t *__restrict__ fadj, const int32_t *__restrict__ fwgt)
{
#pragma unroll 2
    for (int32_t j = b + t; j < e; j += G) {
        const int32_t k = fadj[j], w = fwgt[j];
        const int32_t kw = (to == T.side[k]) ? w : -w;
        const int32_t ned = T.ed[k] - kw, ng = T.gain[k] - kw - kw;
        T.ed[k] = ned;
        T.gain[k] = ng;
        T.pop[k] = (!T.mark[k] && ned > 0) ? ng : INT_MIN;
    }
}

template <int G, bool SMEM>
__global__ void __launch_bounds__(G == 32 ? 32 * TW_WARPS : G)
trial_kernel(const SubInfo *__restrict__ subs, const int32_t *__restrict__ trial_sub, int32_t ntrials,
             const int32_t *__restrict__ fxadj, const int32_t *__restrict__ fadj, const int32_t *__restrict__ fwgt,
             const int32_t *__restrict__ fvwgt, char *slab_base, int32_t starts, int32_t fm_passes, int64_t *tr_cut,
             int64_t *tr_viol, int64_t smem_per_trial)
{
    hp::pdl_wait();
    extern __shared__ __align__(16) char tsm[];
    constexpr int W = G / 32;
    __shared__ int2 s_pop[2][W];        // (key, vertex) of each warp's best, double buffered (G > 32)
    __shared__ long long s_cut[W];
    __shared__ long long s_pw0;
    const int lane = threadIdx.x & 31, t = threadIdx.x % G, grp = threadIdx.x / G, wid = t >> 5;
    const int32_t tr = blockIdx.x * (blockDim.x / G) + grp;
    if (tr >= ntrials) return;   // the whole group
    const SubInfo S = subs[trial_sub[tr]];
    const int32_t lt = tr - S.tbeg;
    const int32_t n = S.n, np = pad4(n);
    const int32_t *xadj = fxadj + S.vbeg;   // global edge offsets, local neighbour ids
    const int32_t *vwgt = fvwgt + S.vbeg;
    char *gbase = slab_base + S.slab_off + (int64_t)lt * state_bytes(n);
    const TrialState T = carve(SMEM ? tsm + (int64_t)grp * smem_per_trial : gbase, n);
    const int32_t start = (n <= starts) ? lt : (int32_t)(((int64_t)lt * n) / starts);
    const int64_t tv = S.tv, want1 = S.want1, onemin = S.onemin, onemax = S.onemax;

    int64_t pw0 = 0;
    if (wid == 0) {
        pw0 = trial_grow(T, n, xadj, fadj, vwgt, start, tv, onemin, onemax);
        if (G > 32 && lane == 0) s_pw0 = pw0;
    }
    trial_sync<G>();
    if (G > 32) pw0 = s_pw0;
    int64_t pw1 = tv - pw0;

    // ---- 2-way FM (hunyuangraph_CPU_2wayrefine.h:24-245)
    long long cut2 = 0;
    const int32_t m = xadj[n] - xadj[0];
    auto init_vertex = [&](int32_t v, int32_t id, int32_t ed, bool isolated) {
        T.ed[v] = ed;
        T.gain[v] = ed - id;
        T.pop[v] = (ed > 0 || isolated) ? ed - id : INT_MIN;
        T.mark[v] = 0;
        cut2 += ed;
    };
    if (m >= 16 * n) {   // long rows: a warp per vertex, the row coalesced
        for (int32_t v = wid; v < n; v += W) {
            int32_t id = 0, ed = 0;
            const int8_t sv = T.side[v];
            const int32_t b = xadj[v], e = xadj[v + 1];
#pragma unroll 4
            for (int32_t j = b + lane; j < e; j += 32) {
                const int32_t w = fwgt[j];
                if (T.side[fadj[j]] == sv) id += w;
                else ed += w;
            }
            id = hp::warp_sum(id);
            ed = hp::warp_sum(ed);
            if (lane == 0) init_vertex(v, id, ed, b == e);
        }
    } else {
        for (int32_t v = t; v < n; v += G) {
            int32_t id = 0, ed = 0;
            const int8_t sv = T.side[v];
            const int32_t b = xadj[v], e = xadj[v + 1];
#pragma unroll 4
            for (int32_t j = b; j < e; j++) {
                const int32_t w = fwgt[j];
                if (T.side[fadj[j]] == sv) id += w;
                else ed += w;
            }
            init_vertex(v, id, ed, b == e);
        }
    }
    for (int32_t v = n + t; v < np; v += G) { T.pop[v] = INT_MIN; T.side[v] = 0; }
    cut2 = hp::warp_sum64(cut2);
    if (G > 32) {
        if (lane == 0) s_cut[wid] = cut2;
        __syncthreads();
        cut2 = 0;
#pragma unroll
        for (int w = 0; w < W; w++) cut2 += s_cut[w];
    } else {
        __syncwarp();
    }
    int64_t cut = cut2 / 2;
    const int64_t tpw0 = tv - want1, tpw1 = want1;
    int64_t limit = n / 100;
    if (limit < 15) limit = 15;
    if (limit > 100) limit = 100;
    int64_t avgvwgt = (pw0 + pw1) / 20;
    if (n > 0 && 2 * (pw0 + pw1) / n < avgvwgt) avgvwgt = 2 * (pw0 + pw1) / n;
    const int64_t origdiff = hp::iabs64(tpw0 - pw0);

    for (int32_t pass = 0; pass < fm_passes; pass++) {
        int64_t mincutorder = -1;
        int64_t newcut = cut, mincut = cut, initcut = cut;
        int64_t mindiff = hp::iabs64(tpw0 - pw0);
        int32_t nswaps;
        for (nswaps = 0; nswaps < n; nswaps++) {
            const int from = (tpw0 - pw0 < tpw1 - pw1) ? 0 : 1;
            const int to = 1 - from;
            // pop: argmax (gain desc, v asc) over the poppable vertices of side `from`
            int32_t bk = INT_MIN, bh = INT_MAX;
#pragma unroll 2
            for (int32_t v = 4 * t; v < np; v += 4 * G) {   // ascending v per thread
                const int4 k4 = *reinterpret_cast<const int4 *>(T.pop + v);
                const char4 s4 = *reinterpret_cast<const char4 *>(T.side + v);
                if (s4.x == from && k4.x > bk) { bk = k4.x; bh = v; }
                if (s4.y == from && k4.y > bk) { bk = k4.y; bh = v + 1; }
                if (s4.z == from && k4.z > bk) { bk = k4.z; bh = v + 2; }
                if (s4.w == from && k4.w > bk) { bk = k4.w; bh = v + 3; }
            }
            int32_t key = __reduce_max_sync(HP_FULL_MASK, bk);
            int32_t h = __reduce_min_sync(HP_FULL_MASK, bk == key ? bh : INT_MAX);
            if (G > 32) {
                // two buffers: a warp a round ahead does not overwrite what is still read
                int2 *sp = s_pop[nswaps & 1];
                if (lane == 0) sp[wid] = make_int2(key, h);
                __syncthreads();
                key = INT_MIN; h = INT_MAX;
#pragma unroll
                for (int w = 0; w < W; w++) {
                    const int2 o = sp[w];
                    if (o.x > key || (o.x == key && o.y < h)) { key = o.x; h = o.y; }
                }
            }
            if (key == INT_MIN) break;
            const int32_t gain = key, wh = vwgt[h], b = xadj[h], e = xadj[h + 1];
            newcut -= gain;
            if (to == 0) { pw0 += wh; pw1 -= wh; } else { pw1 += wh; pw0 -= wh; }
            if ((newcut < mincut && hp::iabs64(tpw0 - pw0) <= origdiff + avgvwgt) ||
                (newcut == mincut && hp::iabs64(tpw0 - pw0) < mindiff)) {
                mincut = newcut;
                mindiff = hp::iabs64(tpw0 - pw0);
                mincutorder = nswaps;
            } else if (nswaps - mincutorder > limit) {
                newcut += gain;
                if (to == 0) { pw0 -= wh; pw1 += wh; } else { pw1 -= wh; pw0 += wh; }
                break;
            }
            // (h is not its own neighbour: its entries and its neighbours' are disjoint)
            if (t == 0) {
                T.side[h] = (int8_t)to;
                T.mark[h] = 1;
                T.list[nswaps] = h;
                T.ed[h] -= gain;
                T.gain[h] = -gain;
                T.pop[h] = INT_MIN;
            }
            trial_relax<G>(T, t, b, e, to, fadj, fwgt);
            trial_sync<G>();
        }
        trial_sync<G>();
        for (int32_t i = t; i < nswaps; i += G) {
            const int32_t h = T.list[i];
            T.mark[h] = 0;
            T.pop[h] = (T.ed[h] > 0 || xadj[h] == xadj[h + 1]) ? T.gain[h] : INT_MIN;
        }
        trial_sync<G>();
        // undo the moves after the best prefix, last first
        nswaps--;
        int32_t h = nswaps > mincutorder ? T.list[nswaps] : 0;
        int to = nswaps > mincutorder ? 1 - T.side[h] : 0;
        trial_sync<G>();   // every thread has read side[h]
        while (nswaps > mincutorder) {
            const int32_t b = xadj[h], e = xadj[h + 1];
            if (t == 0) {
                const int32_t g = -T.gain[h], ed = T.ed[h] + g;
                T.side[h] = (int8_t)to;
                T.ed[h] = ed;
                T.gain[h] = g;
                T.pop[h] = (ed > 0 || b == e) ? g : INT_MIN;
            }
            const int32_t wh = vwgt[h];
            if (to == 0) { pw0 += wh; pw1 -= wh; } else { pw1 += wh; pw0 -= wh; }
            trial_relax<G>(T, t, b, e, to, fadj, fwgt);
            // the next vertex: its side is not written before the barrier
            nswaps--;
            if (nswaps > mincutorder) {
                h = T.list[nswaps];
                to = 1 - T.side[h];
            }
            trial_sync<G>();
        }
        cut = mincut;
        if (mincutorder <= 0 || mincut == initcut) break;
    }
    int64_t viol = 0;
    if (pw1 > onemax) viol += pw1 - onemax;
    if (pw1 < onemin) viol += onemin - pw1;
    // the trial's sides go to the global slab for the selection kernel
    if (SMEM)
        for (int32_t v = t; v < n; v += G) gbase[v] = T.side[v];
    if (t == 0) { tr_cut[tr] = cut; tr_viol[tr] = viol; }
}

// Best trial of every subgraph: min (violation, cut, trial index); copies its
// sides into side[] and reports the side-0 vertex count and weight.
__global__ void __launch_bounds__(256)
select_kernel(const SubInfo *__restrict__ subs, const int64_t *__restrict__ tr_cut,
              const int64_t *__restrict__ tr_viol, const char *slab_base,
              const int32_t *__restrict__ fvwgt, int32_t *__restrict__ side,
              int64_t *__restrict__ res /* per sub: n0, tv0 */)
{
    hp::pdl_wait();
    __shared__ long long s_v[8], s_c[8];
    __shared__ int s_t[8];
    __shared__ int s_best;
    const SubInfo S = subs[blockIdx.x];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    long long bv = LLONG_MAX, bc = LLONG_MAX;
    int bt = INT_MAX;
    for (int t = threadIdx.x; t < S.ntr; t += blockDim.x) {
        long long v = tr_viol[S.tbeg + t], c = tr_cut[S.tbeg + t];
        if (v < bv || (v == bv && (c < bc || (c == bc && t < bt)))) { bv = v; bc = c; bt = t; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        long long ov = __shfl_xor_sync(HP_FULL_MASK, bv, o);
        long long oc = __shfl_xor_sync(HP_FULL_MASK, bc, o);
        int ot = __shfl_xor_sync(HP_FULL_MASK, bt, o);
        if (ov < bv || (ov == bv && (oc < bc || (oc == bc && ot < bt)))) { bv = ov; bc = oc; bt = ot; }
    }
    if (lane == 0) { s_v[wid] = bv; s_c[wid] = bc; s_t[wid] = bt; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); w++)
            if (s_v[w] < bv || (s_v[w] == bv && (s_c[w] < bc || (s_c[w] == bc && s_t[w] < bt)))) {
                bv = s_v[w]; bc = s_c[w]; bt = s_t[w];
            }
        s_best = bt;
    }
    __syncthreads();
    const int8_t *w = (const int8_t *)(slab_base + S.slab_off + (int64_t)s_best * state_bytes(S.n));
    long long n0 = 0, tv0 = 0;
    for (int i = threadIdx.x; i < S.n; i += blockDim.x) {
        int sd = w[i];
        side[S.vbeg + i] = sd;
        if (sd == 0) { n0++; tv0 += fvwgt[S.vbeg + i]; }
    }
    __shared__ unsigned long long s_acc[2];
    if (threadIdx.x == 0) { s_acc[0] = 0; s_acc[1] = 0; }
    __syncthreads();
    hp::block_add_to<256>(n0, &s_acc[0]);
    __syncthreads();
    hp::block_add_to<256>(tv0, &s_acc[1]);
    __syncthreads();
    if (threadIdx.x == 0) { res[2 * blockIdx.x] = (int64_t)s_acc[0]; res[2 * blockIdx.x + 1] = (int64_t)s_acc[1]; }
}

struct ChildMap {
    int32_t newbeg[2];   // first new vertex id of each side, -1 = side not carried on
    int32_t fpart[2];    // part of a final (single-part) side, -1 otherwise
};

__global__ void __launch_bounds__(256)
sub_of_kernel(const SubInfo *__restrict__ subs, int32_t *__restrict__ sub_of,
              int32_t *__restrict__ flag0)
{
    hp::pdl_wait();
    const SubInfo S = subs[blockIdx.x];
    for (int i = threadIdx.x; i < S.n; i += blockDim.x) sub_of[S.vbeg + i] = blockIdx.x;
    (void)flag0;
}

__global__ void __launch_bounds__(256)
side_flag_kernel(int32_t nf, const int32_t *__restrict__ side, int32_t *__restrict__ f0)
{
    hp::pdl_wait();
    int32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < nf) f0[v] = side[v] == 0;
}

// New id of every forest vertex and its degree inside its side; final sides
// write the output partition directly.
__global__ void __launch_bounds__(256)
split_count_kernel(int32_t nf, const SubInfo *__restrict__ subs, const int32_t *__restrict__ sub_of,
                   const ChildMap *__restrict__ cm, const int32_t *__restrict__ side,
                   const int32_t *__restrict__ p0, const int32_t *__restrict__ fxadj,
                   const int32_t *__restrict__ fadj, const int32_t *__restrict__ label,
                   int32_t *__restrict__ newid, int32_t *__restrict__ ndeg, int32_t *__restrict__ where_out)
{
    hp::pdl_wait();
    int32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nf) return;
    const int32_t s = sub_of[v];
    const SubInfo S = subs[s];
    const int sd = side[v];
    const ChildMap C = cm[s];
    if (C.fpart[sd] >= 0) where_out[label[v]] = C.fpart[sd];
    if (C.newbeg[sd] < 0) { newid[v] = -1; return; }
    int32_t r0 = p0[v] - p0[S.vbeg];
    int32_t rank = sd == 0 ? r0 : (v - S.vbeg) - r0;
    int32_t nid = C.newbeg[sd] + rank;
    newid[v] = nid;
    int32_t d = 0;
    for (int32_t j = fxadj[v]; j < fxadj[v + 1]; j++) d += side[S.vbeg + fadj[j]] == sd;
    ndeg[nid] = d;
}

__global__ void __launch_bounds__(256)
split_write_kernel(int32_t nf, const SubInfo *__restrict__ subs, const int32_t *__restrict__ sub_of,
                   const ChildMap *__restrict__ cm, const int32_t *__restrict__ side,
                   const int32_t *__restrict__ newid, const int32_t *__restrict__ fxadj,
                   const int32_t *__restrict__ fadj, const int32_t *__restrict__ fwgt,
                   const int32_t *__restrict__ fvwgt, const int32_t *__restrict__ label,
                   const int32_t *__restrict__ nxadj, int32_t *__restrict__ nadj,
                   int32_t *__restrict__ nwgt, int32_t *__restrict__ nvwgt, int32_t *__restrict__ nlabel)
{
    hp::pdl_wait();
    int32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nf) return;
    const int32_t nid = newid[v];
    if (nid < 0) return;
    const int32_t s = sub_of[v];
    const SubInfo S = subs[s];
    const int sd = side[v];
    const int32_t nb = cm[s].newbeg[sd];
    nvwgt[nid] = fvwgt[v];
    nlabel[nid] = label[v];
    int32_t e = nxadj[nid];
    for (int32_t j = fxadj[v]; j < fxadj[v + 1]; j++) {
        int32_t u = S.vbeg + fadj[j];
        if (side[u] != sd) continue;
        nadj[e] = newid[u] - nb;
        nwgt[e] = fwgt[j];
        e++;
    }
}

__global__ void assign_all_kernel(int32_t n, int32_t *where, int32_t value)
{
    hp::pdl_wait();
    int32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n) where[v] = value;
}

__global__ void copy_kernel(int64_t n, const int32_t *src, int32_t *dst)
{
    hp::pdl_wait();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = src[i];
}

struct HostSub {
    int32_t vbeg, n;
    int32_t k, fpart;
    int64_t tv;
};

inline unsigned nblk(int64_t n, int b = 256) { return (unsigned)std::max<int64_t>(1, (n + b - 1) / b); }

}  // namespace

int hp_initpart_init()
{
    HP_CUDA(cudaFuncSetAttribute(trial_kernel<32, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)HP_TRIAL_SMEM));
    HP_CUDA(cudaFuncSetAttribute(trial_kernel<TC_THREADS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)HP_TRIAL_SMEM));
    return HP_OK;
}

int hp_initial_partition(hp_context *c, HpLevel &g, int32_t nparts, const int64_t *h_tw,
                         int64_t ub2_fx, int32_t *d_where)
{
    const int32_t n = g.n;
    if (n == 0) return HP_OK;
    if (nparts == 1) {
        HP_LAUNCH(c, assign_all_kernel, nblk(n), 256, 0, n, d_where, 0);
        return HP_OK;
    }
    const int32_t starts = std::max(1, c->opt.init_starts);
    const int32_t fm_passes = std::max(0, c->opt.fm_passes);
    const size_t mark = c->hi;

    // forest of depth 0 = the coarsest graph itself (labels = ids)
    int32_t nf = n;
    int64_t mf = g.m;
    int32_t *fxadj = ralloc_t<int32_t>(c, nf + 1), *fadj = ralloc_t<int32_t>(c, mf);
    int32_t *fwgt = ralloc_t<int32_t>(c, mf), *fvwgt = ralloc_t<int32_t>(c, nf);
    int32_t *flabel = ralloc_t<int32_t>(c, nf);
    // ping-pong forest
    int32_t *gxadj = ralloc_t<int32_t>(c, nf + 1), *gadj = ralloc_t<int32_t>(c, mf);
    int32_t *gwgt = ralloc_t<int32_t>(c, mf), *gvwgt = ralloc_t<int32_t>(c, nf);
    int32_t *glabel = ralloc_t<int32_t>(c, nf);
    int32_t *side = ralloc_t<int32_t>(c, nf), *p0 = ralloc_t<int32_t>(c, nf + 1);
    int32_t *sub_of = ralloc_t<int32_t>(c, nf), *newid = ralloc_t<int32_t>(c, nf);
    int32_t *ndeg = ralloc_t<int32_t>(c, nf + 1);
    HP_CHECK_OOM(c);
    HP_LAUNCH(c, copy_kernel, nblk(nf + 1), 256, 0, (int64_t)nf + 1, g.xadj, fxadj);
    HP_LAUNCH(c, copy_kernel, nblk(mf), 256, 0, mf, g.adjncy, fadj);
    HP_LAUNCH(c, copy_kernel, nblk(mf), 256, 0, mf, g.adjwgt, fwgt);
    HP_LAUNCH(c, copy_kernel, nblk(nf), 256, 0, (int64_t)nf, g.vwgt, fvwgt);
    HP_TRY(hp_iota_i32(c, flabel, nf));

    // total vertex weight of the coarsest graph
    std::vector<int32_t> hv(nf);
    HP_CUDA(cudaMemcpyAsync(hv.data(), g.vwgt, sizeof(int32_t) * (size_t)nf, cudaMemcpyDeviceToHost, c->stream));
    HP_CUDA(cudaStreamSynchronize(c->stream));
    int64_t tv0 = 0;
    for (int32_t v = 0; v < nf; v++) tv0 += hv[v];

    std::vector<HostSub> subs{{0, nf, nparts, 0, tv0}};
    while (!subs.empty()) {
        const int ns = (int)subs.size();
        std::vector<SubInfo> info(ns);
        std::vector<int32_t> trial_sub;
        int64_t slab_total = 0;
        int32_t tcount = 0;
        for (int s = 0; s < ns; s++) {
            const HostSub &H = subs[s];
            SubInfo &I = info[s];
            const int32_t kl = H.k >> 1;
            int64_t wl = 0, wr = 0;
            for (int32_t p = 0; p < kl; p++) wl += h_tw[H.fpart + p];
            for (int32_t p = kl; p < H.k; p++) wr += h_tw[H.fpart + p];
            I.vbeg = H.vbeg; I.n = H.n; I.tv = H.tv;
            I.want1 = (wl + wr) > 0 ? (H.tv * wr) / (wl + wr) : H.tv / 2;
            I.onemax = (I.want1 * ub2_fx) >> 16;
            I.onemin = (I.want1 << 16) / ub2_fx;
            I.ntr = H.n <= starts ? H.n : starts;
            I.tbeg = tcount;
            I.slab_off = slab_total;
            slab_total += (int64_t)I.ntr * state_bytes(H.n);
            for (int32_t t = 0; t < I.ntr; t++) trial_sub.push_back(s);
            tcount += I.ntr;
        }
        const size_t dmark = c->hi;
        SubInfo *d_info = ralloc_t<SubInfo>(c, ns);
        int32_t *d_tsub = ralloc_t<int32_t>(c, tcount);
        int64_t *d_cut = ralloc_t<int64_t>(c, tcount), *d_viol = ralloc_t<int64_t>(c, tcount);
        char *slab = (char *)hp_ralloc(c, (size_t)slab_total);
        int64_t *d_res = ralloc_t<int64_t>(c, 2 * (int64_t)ns);
        ChildMap *d_cm = ralloc_t<ChildMap>(c, ns);
        HP_CHECK_OOM(c);
        HP_CUDA(cudaMemcpyAsync(d_info, info.data(), sizeof(SubInfo) * ns, cudaMemcpyHostToDevice, c->stream));
        HP_CUDA(cudaMemcpyAsync(d_tsub, trial_sub.data(), sizeof(int32_t) * tcount, cudaMemcpyHostToDevice, c->stream));
        // trial state in shared memory when the largest subgraph fits
        int32_t maxn = 0;
        for (const HostSub &H : subs) maxn = std::max(maxn, H.n);
        const int64_t per = (state_bytes(maxn) + 15) & ~(int64_t)15;
        const bool smem = per <= HP_TRIAL_SMEM;
        const int wpb = smem ? (int)std::min<int64_t>(TW_WARPS, HP_TRIAL_SMEM / per) : TW_WARPS;
        const int tok = hp_prof_begin(c);
        // a CTA per trial (same trial, same result) on large subgraphs, and on dense
        // ones, whose moves read long rows: rows of deg0 entries on average in the
        // whole graph, shrinking with the subgraph as in a dense one (R-MAT, 900
        // vertices of 286 entries, 512 as the vertex bound: 6.3 ms with warps at the
        // depths below it, 3.7 ms with CTAs)
        const int64_t deg0 = g.m / n, deg = deg0 * maxn / n;
        const bool cta = maxn >= c->tune.trial_cta_n || deg >= TC_DEG;
        const unsigned tgrid = cta ? (unsigned)tcount : nblk(tcount, wpb);
        const unsigned tblock = cta ? TC_THREADS : 32 * wpb;
        const size_t tsmem = !smem ? 0 : cta ? (size_t)per : (size_t)(per * wpb);
#define HP_TRIAL_LAUNCH(K)                                                                              \
    HP_LAUNCH(c, K, tgrid, tblock, tsmem, d_info, d_tsub, tcount, fxadj, fadj, fwgt, fvwgt, slab, starts, \
              fm_passes, d_cut, d_viol, per)
        if (cta && smem) HP_TRIAL_LAUNCH((trial_kernel<TC_THREADS, true>));
        else if (cta) HP_TRIAL_LAUNCH((trial_kernel<TC_THREADS, false>));
        else if (smem) HP_TRIAL_LAUNCH((trial_kernel<32, true>));
        else HP_TRIAL_LAUNCH((trial_kernel<32, false>));
#undef HP_TRIAL_LAUNCH
        hp_prof_end(c, tok, HP_PROF_INIT, 0);
        HP_LAUNCH(c, select_kernel, (unsigned)ns, 256, 0, d_info, d_cut, d_viol, slab, fvwgt, side, d_res);
        std::vector<int64_t> res(2 * ns);
        HP_CUDA(cudaMemcpyAsync(res.data(), d_res, sizeof(int64_t) * 2 * ns, cudaMemcpyDeviceToHost, c->stream));
        HP_CUDA(cudaStreamSynchronize(c->stream));

        // children
        std::vector<ChildMap> cm(ns);
        std::vector<HostSub> next;
        int32_t nnew = 0;
        for (int s = 0; s < ns; s++) {
            const HostSub &H = subs[s];
            const int32_t kl = H.k >> 1;
            const int32_t cn[2] = {(int32_t)res[2 * s], H.n - (int32_t)res[2 * s]};
            const int64_t ctv[2] = {res[2 * s + 1], H.tv - res[2 * s + 1]};
            const int32_t ck[2] = {kl, H.k - kl};
            const int32_t cf[2] = {H.fpart, H.fpart + kl};
            for (int sd = 0; sd < 2; sd++) {
                cm[s].fpart[sd] = ck[sd] == 1 ? cf[sd] : -1;
                if (ck[sd] >= 2 && cn[sd] > 0) {
                    cm[s].newbeg[sd] = nnew;
                    next.push_back({nnew, cn[sd], ck[sd], cf[sd], ctv[sd]});
                    nnew += cn[sd];
                } else {
                    cm[s].newbeg[sd] = -1;
                }
            }
        }
        HP_CUDA(cudaMemcpyAsync(d_cm, cm.data(), sizeof(ChildMap) * ns, cudaMemcpyHostToDevice, c->stream));
        HP_LAUNCH(c, sub_of_kernel, (unsigned)ns, 256, 0, d_info, sub_of, (int32_t *)nullptr);
        HP_LAUNCH(c, side_flag_kernel, nblk(nf), 256, 0, nf, side, p0);
        HP_TRY(hp_scan_excl(c, p0, p0, nf));
        HP_LAUNCH(c, split_count_kernel, nblk(nf), 256, 0, nf, d_info, sub_of, d_cm, side, p0, fxadj,
                  fadj, flabel, newid, ndeg, d_where);
        if (nnew > 0) {
            HP_TRY(hp_scan_excl(c, ndeg, gxadj, nnew));
            HP_LAUNCH(c, split_write_kernel, nblk(nf), 256, 0, nf, d_info, sub_of, d_cm, side, newid,
                      fxadj, fadj, fwgt, fvwgt, flabel, gxadj, gadj, gwgt, gvwgt, glabel);
        }
        HP_CUDA(cudaStreamSynchronize(c->stream));
        c->hi = dmark;
        std::swap(fxadj, gxadj); std::swap(fadj, gadj); std::swap(fwgt, gwgt);
        std::swap(fvwgt, gvwgt); std::swap(flabel, glabel);
        nf = nnew;
        subs.swap(next);
    }
    HP_TRY(hp_check_status(c));
    c->hi = mark;
    return HP_OK;
}
