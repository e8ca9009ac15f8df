// Iteration passes of a solve, split by what a pass couples.
//
// cfr_solve_kernel gives a subgame to one thread block, which walks the nodes of the tree one after another: the
// time of a pass is that walk (about 7 us an internal node and sweep), and a batch of few subgames leaves most of the
// chip idle.  Two facts allow a pass without the walk:
//
//   * What couples the hands of a row (the sums that normalise beliefs, the per-card sums behind "the other
//     player's policy as this hand sees it", the showdown) needs the node's own beliefs only.  A player's reach
//     at a node is the product of the current policies along the path, so all nodes can be worked on at once.
//   * What couples the nodes (value backup, regrets, next policy, average policy) is elementwise in the hand.
//
// So a pass is split_rows_kernel, one block per internal node of the whole batch, followed by split_up_kernel,
// where the warps of a block own a slice of the hands of one subgame and go up the tree level by level, a warp a node.  A solve whose leaves are valued by the caller's model has the model between the two.
// There is no top-down sweep: the row kernel multiplies along the path (3 to 5 rows that are in L2), and does the
// same with the average policy of the pass before, by which the average-policy mix weights.
//
// Arithmetic and results are those of cfr.cu, bit for bit: same operations in the same order, also in the fp64 sums.
//
// Measured on a B200, a pass in the general kernel / here (the iteration passes by the library's timer, over their number):
// one subgame of 57 nodes 0.32 / 0.034 ms, 37 of 96 nodes 1.15 / 0.155 ms, 192 flop subgames of 77 nodes (largest 271)
// 1.4 / 0.39 ms.  The row kernel takes 6.3 us an SM and node with two blocks resident; shared-memory wavefronts (0.59 of
// their peak on 192 river subgames, mostly the gathers of the per-card sums and of the showdown tables) and the barriers
// between its phases bound it, with half of the issue slots used.  The up kernel is bound by memory at large batches
// (2.55 ms on 4096 subgames of 54 nodes, 0.9 of the copy bandwidth over the 15 GB it moves) and by the latency of a warp's walk at
// small ones (DRAM at 0.44 of its peak on 192 river subgames).
#include "cfr_split.cuh"

#include "cfr_dev.cuh"
#include "exactdiv.cuh"
#include "showdown.cuh"

namespace p2b {

int sm_count();

namespace {

// An internal node, as both kernels read it.
struct SplitItem {  // 64 bytes
    int32_t subgame;
    int32_t node_begin;
    uint16_t node, first_child;
    uint8_t n_children, to_act;
    uint8_t n_path[2];    // nodes on the path from the root where the acting / the other player chose
    uint16_t path[kSplitMaxDepth];  // these nodes, top-down: first the acting player's, then the other's
    uint8_t kind[kCfrMaxChildren];  // NodeKind of the children
    uint8_t first_sd;     // slot of the first showdown child, kNoChild: none
    uint8_t pad[7];
};
static_assert(sizeof(SplitItem) == 64, "SplitItem is four 16-byte vectors");
constexpr uint8_t kNoChild = 0xFF;

struct SplitLevels {  // of one subgame
    int32_t item_begin;
    int32_t n_levels;
    uint16_t begin[kSplitMaxDepth + 2];  // items of level d: item_begin + begin[d] .. begin[d + 1]
};
static_assert(sizeof(SplitLevels) % 4 == 0, "");

// Work rows of a node, next to one another: one address serves them all.
enum RecRow {
    kRecPolicy = 0,  // current policy
    kRecSeen = 1,    // the policy as each hand of the player who does not choose sees it
    kRecWeight = 2,  // regret weights of the acting player's hands (internal nodes)
    kRecValue = 3,   // values of player 0, then of player 1 (internal nodes and showdown leaves)
    kRecReach = 5,   // the acting player's reach under the current policy and under the old average policy (internal
    kRecOldReach = 6,  // nodes, passes that mix)
    kRecActing = 2,  // final pass: beliefs of the acting player
    kRecBelief = 5,  // final pass: beliefs of player 0, then of player 1; later the best-response values of the second sweep
    kRecRows = 7
};
constexpr int kRec = kRecRows * P2B_HPAD;  // floats from a node's record to the next

struct SplitWork {
    int32_t* total;       // [4] number of items
    SplitItem* items;     // [rows]
    SplitLevels* levels;  // [B], in queue order
    float* rec;           // [rows][kRecRows][HPAD]
};

constexpr long long kItemFloats = sizeof(SplitItem) / 4;
constexpr long long kLevelFloats = sizeof(SplitLevels) / 4;
__host__ __device__ inline long long round4(long long x) { return (x + 3) / 4 * 4; }

SplitWork carve(float* scratch, int num_subgames, long long rows) {
    SplitWork w;
    w.total = reinterpret_cast<int32_t*>(scratch);
    float* at = scratch + 4;
    w.items = reinterpret_cast<SplitItem*>(at);
    at += rows * kItemFloats;
    w.levels = reinterpret_cast<SplitLevels*>(at);
    at += round4(num_subgames * kLevelFloats);
    w.rec = at;
    return w;
}

// Whether the solve has been refused (work_counter[1]).  A kernel that nothing runs beside has its block agree on it, as other
// blocks of the same kernel may set the word.  The two kernels of a pass, which may start before the one ahead of them has
// ended, read it thread by thread: no kernel that they can meet writes it, a wait that runs out is noted in a word of its own
// (gave_up), which the record check of the next call and the final pass carry over.
__device__ __forceinline__ bool refused(const CfrParams& p) { return p.work_counter[1] != 0; }
__device__ __forceinline__ bool block_refused(const CfrParams& p) {
    return __syncthreads_or(threadIdx.x == 0 && *reinterpret_cast<const volatile int32_t*>(p.work_counter + 1) != 0) != 0;
}
__device__ __forceinline__ int32_t* gave_up(const CfrParams& p) { return p.work_counter + kGaveUp; }
__device__ __forceinline__ void report_gave_up(const CfrParams& p) {  // one thread of a kernel that has started after the others' end
    if (blockIdx.x == 0 && threadIdx.x == 0 && *gave_up(p) != 0) atomicMax(p.work_counter + 1, *gave_up(p));
}

// ---- work lists -------------------------------------------------------------------------------
// The items of a batch follow the queue order, those of a subgame the node order, which is breadth-first.

// Where the items of each subgame begin (levels[].item_begin), by one block: a thread adds up a run of subgames, the block the
// threads' sums.
constexpr int kBeginThreads = 1024;
__global__ void __launch_bounds__(kBeginThreads) split_begin_kernel(const CfrParams p, const SplitWork w) {
    __shared__ int s_warp[kBeginThreads / 32];
    if (block_refused(p)) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int run = (p.num_subgames + kBeginThreads - 1) / kBeginThreads;
    const int first = min(tid * run, p.num_subgames), last = min(first + run, p.num_subgames);
    auto items = [&](int q) { return p.subgames[p.queue_order ? p.queue_order[q] : q].n_internal; };
    int mine = 0;
#pragma unroll 8
    for (int q = first; q < last; ++q) mine += items(q);
    int upto = mine;
    for (int d = 1; d < 32; d <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, upto, d);
        if (lane >= d) upto += x;
    }
    if (lane == 31) s_warp[warp] = upto;
    __syncthreads();
    int at = upto - mine;
    for (int x = 0; x < warp; ++x) at += s_warp[x];
#pragma unroll 8
    for (int q = first; q < last; ++q) {
        w.levels[q].item_begin = at;
        at += items(q);
    }
}

// One block per subgame, one thread per node.  `begun`: split_begin_kernel has run; else every block adds up the subgames
// before its own.
__global__ void __launch_bounds__(kCfrMaxNodes) split_items_kernel(const CfrParams p, const SplitWork w, bool begun) {
    __shared__ int s_before, s_depth[kSplitMaxDepth + 1], s_bad;
    const int q = blockIdx.x, i = threadIdx.x;
    if (i == 0) s_before = s_bad = 0;
    if (i <= kSplitMaxDepth) s_depth[i] = 0;
    if (block_refused(p)) {  // the record check refused the batch
        if (q == 0 && i == 0) w.total[0] = 0;
        return;
    }
    const int s = p.queue_order ? p.queue_order[q] : q;
    if (begun) {
        if (i == 0) s_before = w.levels[q].item_begin;
    } else {
        int before = 0;
        for (int r = i; r < q; r += kCfrMaxNodes) before += p.subgames[p.queue_order ? p.queue_order[r] : r].n_internal;
        for (int d = 16; d > 0; d >>= 1) before += __shfl_xor_sync(0xffffffffu, before, d);
        if ((i & 31) == 0) atomicAdd(&s_before, before);
    }
    __syncthreads();
    const SubgameRec sg = p.subgames[s];
    const NodeRecPacked* nodes = p.nodes + sg.node_begin;
    if (i < sg.n_nodes) {
        const NodeRec nd = load_node(nodes + i);
        if (nd.kind == kInternal) {
            SplitItem it{};
            it.subgame = s;
            it.node_begin = sg.node_begin;
            it.node = (uint16_t)i;
            it.first_child = nd.first_child;
            it.n_children = nd.n_children;
            it.to_act = nd.to_act;
            uint16_t up[kSplitMaxDepth];
            uint8_t who[kSplitMaxDepth];
            int depth = 0, x = i;
            while (x > 0 && depth < kSplitMaxDepth) {
                const NodeRec me = load_node(nodes + x);
                if (me.parent >= x) break;  // a parent comes before its children
                up[depth] = (uint16_t)x;
                who[depth] = load_node(nodes + me.parent).to_act;
                x = me.parent;
                ++depth;
            }
            if (x != 0) s_bad = 1;
            int n = 0;
            for (int side = 0; side < 2; ++side) {
                const int pl = side == 0 ? nd.to_act : 1 - nd.to_act;
                int m = 0;
                for (int e = depth - 1; e >= 0; --e)
                    if (who[e] == pl) {
                        it.path[n++] = up[e];
                        ++m;
                    }
                it.n_path[side] = (uint8_t)m;
            }
            it.first_sd = kNoChild;
            for (int c = nd.n_children - 1; c >= 0; --c) {
                it.kind[c] = load_node(nodes + nd.first_child + c).kind;
                if (it.kind[c] == kShowdownLeaf) it.first_sd = (uint8_t)c;
            }
            atomicAdd(&s_depth[depth], 1);
            w.items[s_before + nd.internal_idx] = it;
        }
    }
    __syncthreads();
    if (i == 0) {
        SplitLevels lv{};
        lv.item_begin = s_before;
        int n = 0;
        for (int d = 0; d <= kSplitMaxDepth; ++d) {
            lv.begin[d] = (uint16_t)n;
            n += s_depth[d];
            if (s_depth[d] > 0) lv.n_levels = d + 1;
        }
        lv.begin[kSplitMaxDepth + 1] = (uint16_t)n;
        w.levels[q] = lv;
        if (q == (int)gridDim.x - 1) w.total[0] = s_before + sg.n_internal;
        if (s_bad) atomicMax(p.work_counter + 1, s + 1);  // a tree deeper than the caller said
    }
}

// ---- hands of a thread --------------------------------------------------------------------------
template <int VPT>
__device__ __forceinline__ FV<VPT> ldc(const float* p) {  // VPT consecutive hands
    FV<VPT> r;
    if constexpr (VPT == 2) {
        const float2 t = *reinterpret_cast<const float2*>(p);
        r.v[0] = t.x;
        r.v[1] = t.y;
    } else {
        r.v[0] = *p;
    }
    return r;
}
template <int VPT>
__device__ __forceinline__ void stc(float* p, const FV<VPT>& r) {
    if constexpr (VPT == 2) *reinterpret_cast<float2*>(p) = make_float2(r.v[0], r.v[1]);
    else *p = r.v[0];
}

template <int N>
struct Count {
    static constexpr int value = N;
};
// body(Count<k>) for the run-time child count k, uniform over the warp
template <int MAXK, typename Body>
__device__ __forceinline__ void with_children(int k, Body&& body) {
    switch (k) {
        case 1: body(Count<1>{}); break;
        case 2: body(Count<2>{}); break;
        case 3: body(Count<3>{}); break;
        case 4: body(Count<4>{}); break;
        case 5: body(Count<5>{}); break;
        case 6: body(Count<6>{}); break;
        default:
            if constexpr (MAXK > 6) {
                if (k == 7) body(Count<7>{});
                else body(Count<8>{});
            }
            break;
    }
}

// Regret matching over K siblings (cfr_evaluator.py:1168-1185): R -> policy.
template <int VPT, int K>
__device__ __forceinline__ void regret_matching(FV<VPT> (&R)[K]) {
    constexpr float invk = 1.0f / (float)K;
    FV<VPT> sum;
    Divisor d[VPT];
    bool ok = true;
#pragma unroll
    for (int i = 0; i < VPT; ++i) sum.v[i] = 0.0f;
#pragma unroll
    for (int c = 0; c < K; ++c)
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            R[c].v[i] = fmaxf(R[c].v[i], 0.0f);
            sum.v[i] = __fadd_rn(sum.v[i], R[c].v[i]);
        }
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        d[i] = make_divisor(fmaxf(sum.v[i], 1e-8f));
        ok = ok && d[i].ok;
    }
    DivGuard g = guard_begin(ok);
    FV<VPT> q[K];
#pragma unroll
    for (int c = 0; c < K; ++c)
#pragma unroll
        for (int i = 0; i < VPT; ++i) q[c].v[i] = div_g<true>(R[c].v[i], d[i].y, d[i].r, g);
    if (__builtin_expect(guard_bad(g), 0)) {
#pragma unroll
        for (int c = 0; c < K; ++c)
#pragma unroll
            for (int i = 0; i < VPT; ++i) q[c].v[i] = __fdiv_rn(R[c].v[i], d[i].y);
    }
#pragma unroll
    for (int c = 0; c < K; ++c)
#pragma unroll
        for (int i = 0; i < VPT; ++i) R[c].v[i] = sum.v[i] > 1e-8f ? q[c].v[i] : invk;
}

// Product of the rows of the nodes on a path (`stride` floats from node to node), times the mask, in path order.
template <int VPT>
__device__ __forceinline__ FV<VPT> path_product(const float* base, int stride, const uint16_t* path, int n, FV<VPT> r) {
#pragma unroll 2
    for (int e = 0; e < n; ++e) {
        const FV<VPT> x = ldc<VPT>(base + (unsigned)path[e] * (unsigned)stride);
#pragma unroll
        for (int i = 0; i < VPT; ++i) r.v[i] = __fmul_rn(r.v[i], x.v[i]);
    }
    return r;
}

// The root's row of the pass becomes what the node beliefs of the next pass derive from.
__device__ __forceinline__ void advance_root(const CfrParams& p, int s, int h) {
    float* cr = p.carry_roots + (long long)s * 4 * P2B_HPAD + h;
    stc<2>(cr, ldc<2>(cr + 2 * P2B_HPAD));
    stc<2>(cr + P2B_HPAD, ldc<2>(cr + 3 * P2B_HPAD));
}

// Average-policy mix and renormalisation of K siblings (cfr_evaluator.py:1195-1258): A <- mix of A and P, weighted by
// the acting player's reach under the old average policy (rba) and under the current one (ra).
template <int VPT, int K>
__device__ __forceinline__ void mix_average(const IterScalars& sc, const FV<VPT>& ra, const FV<VPT>& rba,
                                            const FV<VPT> (&P)[K], FV<VPT> (&A)[K]) {
    FV<VPT> ro, rn, sum;
    Divisor d[VPT];
    bool ok = true;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        ro.v[i] = __fmul_rn(rba.v[i], sc.mix_old);
        rn.v[i] = __fmul_rn(ra.v[i], sc.mix_new);
        const float den = __fadd_rn(ro.v[i], rn.v[i]);
        const bool weighted = den > 1e-5f;  // else: (numerically) no reach, the plain iteration weights (:1231-1239)
        ro.v[i] = weighted ? ro.v[i] : sc.mix_old;
        rn.v[i] = weighted ? rn.v[i] : sc.mix_new;
        d[i] = make_divisor(weighted ? den : sc.mix_total);
        ok = ok && d[i].ok;
        sum.v[i] = 0.0f;
    }
    {
        DivGuard g = guard_begin(ok);
        FV<VPT> num[K];
#pragma unroll
        for (int c = 0; c < K; ++c)
#pragma unroll
            for (int i = 0; i < VPT; ++i) {
                num[c].v[i] = __fadd_rn(__fmul_rn(ro.v[i], A[c].v[i]), __fmul_rn(rn.v[i], P[c].v[i]));
                A[c].v[i] = div_g<true>(num[c].v[i], d[i].y, d[i].r, g);
            }
        if (__builtin_expect(guard_bad(g), 0)) {
#pragma unroll
            for (int c = 0; c < K; ++c)
#pragma unroll
                for (int i = 0; i < VPT; ++i) A[c].v[i] = __fdiv_rn(num[c].v[i], d[i].y);
        }
    }
#pragma unroll
    for (int c = 0; c < K; ++c)
#pragma unroll
        for (int i = 0; i < VPT; ++i) sum.v[i] = __fadd_rn(sum.v[i], A[c].v[i]);
    ok = true;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        d[i] = make_divisor(sum.v[i]);
        ok = ok && d[i].ok;
    }
    DivGuard g = guard_begin(ok);
    FV<VPT> q[K];
#pragma unroll
    for (int c = 0; c < K; ++c)
#pragma unroll
        for (int i = 0; i < VPT; ++i) q[c].v[i] = div_g<true>(A[c].v[i], d[i].y, d[i].r, g);
    if (__builtin_expect(guard_bad(g), 0)) {
#pragma unroll
        for (int c = 0; c < K; ++c)
#pragma unroll
            for (int i = 0; i < VPT; ++i) q[c].v[i] = __fdiv_rn(A[c].v[i], sum.v[i]);
    }
#pragma unroll
    for (int c = 0; c < K; ++c)
#pragma unroll
        for (int i = 0; i < VPT; ++i)
            if (sum.v[i] > 1e-5f) A[c].v[i] = q[c].v[i];
}

// The two elementwise passes over the nodes that need no values: the first current policy from the regrets (and the root's
// rows moved on to the coming pass), and the average-policy mix alone, for solves whose beliefs are taken under the updated
// average policy.  A warp takes a node for 64 hands, from the deepest level up: the old average policy of a node's ancestors
// is still in place when it is visited.
enum PrepMode { kPrepPolicy = 0, kPrepMix = 1 };

template <int K, int MODE>
__device__ __forceinline__ void prep_node(const CfrParams& p, const SplitWork& w, const SplitItem& it, const FV<2>& mask, int h,
                                          const IterScalars& sc) {
    const long long kids = (long long)(it.node_begin + it.first_child) * P2B_HPAD + h;
    float* rec = w.rec + (long long)(it.node_begin + it.first_child) * kRec + h;  // of the first child
    FV<2> P[K];
    if (MODE == kPrepPolicy) {
#pragma unroll
        for (int c = 0; c < K; ++c) P[c] = ldc<2>(p.regrets + kids + c * P2B_HPAD);
        regret_matching<2, K>(P);
#pragma unroll
        for (int c = 0; c < K; ++c) stc<2>(rec + c * kRec, P[c]);
        return;
    }
    float* A_row = p.policy_avg + kids;
#pragma unroll
    for (int c = 0; c < K; ++c) P[c] = ldc<2>(rec + c * kRec);
    if (sc.do_mix & 1) {
        FV<2> A[K];
#pragma unroll
        for (int c = 0; c < K; ++c) A[c] = ldc<2>(A_row + c * P2B_HPAD);
        const FV<2> ra = path_product<2>(w.rec + (long long)it.node_begin * kRec + h, kRec, it.path, it.n_path[0], mask);
        const FV<2> rba = path_product<2>(p.policy_avg + (long long)it.node_begin * P2B_HPAD + h, P2B_HPAD, it.path,
                                          it.n_path[0], mask);
        mix_average<2, K>(sc, ra, rba, P, A);
#pragma unroll
        for (int c = 0; c < K; ++c) stc<2>(A_row + c * P2B_HPAD, A[c]);
    } else {
#pragma unroll
        for (int c = 0; c < K; ++c) stc<2>(A_row + c * P2B_HPAD, P[c]);
    }
}

constexpr int kPrepWarps = 4;
template <int MAXK, int MODE>
__global__ void __launch_bounds__(32 * kPrepWarps) split_prep_kernel(const CfrParams p, const SplitWork w, int pass) {
    constexpr int kSlices = P2B_HPAD / 64;
    if (block_refused(p)) return;
    const int q = blockIdx.x / kSlices, warp = threadIdx.x >> 5;
    const int h = (blockIdx.x - q * kSlices) * 64 + (threadIdx.x & 31) * 2;
    const int s = p.queue_order ? p.queue_order[q] : q;
    const SubgameRec sg = p.subgames[s];
    const SplitLevels* lv = w.levels + q;
    const SplitItem* items = w.items + lv->item_begin;
    FV<2> mask;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const bool real = h + i < P2B_NUM_HANDS;
        const int hc = real ? h + i : P2B_NUM_HANDS - 1;
        const bool blocked = (((sg.board_mask >> p.combos->c1[hc]) | (sg.board_mask >> p.combos->c2[hc])) & 1ull) != 0;
        mask.v[i] = real && !blocked ? 1.0f : 0.0f;
    }
    const IterScalars sc = p.scalars[pass];
    for (int d = lv->n_levels - 1; d >= 0; --d) {
        for (int x = lv->begin[d] + warp; x < lv->begin[d + 1]; x += kPrepWarps) {
            const SplitItem& it = items[x];
            with_children<MAXK>(it.n_children, [&](auto kc) { prep_node<decltype(kc)::value, MODE>(p, w, it, mask, h, sc); });
        }
        if (MODE == kPrepMix) __syncthreads();
    }
    if (MODE == kPrepPolicy && warp == 0) advance_root(p, s, h);
}

// ---- columns --------------------------------------------------------------------------------------
// The bottom-up half of a pass: value backup (cfr_evaluator.py:1095-1115), average-policy mix and renormalisation
// (:1195-1258), instantaneous regrets (:1117-1165) folded into the discounted update of the next pass (:1346-1368) and
// the policy that follows from it (:1168-1185), all elementwise in the hand.
//
// A warp owns a slice of 64 hands and takes one node at a time.  A node's rows (7 a child, 256 bytes each for the slice) are
// copied into the warp's part of shared memory while the warp works on the node before, so that neither the child loops have
// to be unrolled to have loads in flight nor a register is spent on a row that waits: with the loads in registers and a body
// per child count the kernel ran at 20 warps an SM, half of their stalls on loads and a fifth on instruction fetches.
constexpr int kUpThreads = 256, kUpSlices = 3;  // of a block, at most
enum UpSlot { kUpPolicy = 0, kUpSeen = 1, kUpRegret = 2, kUpSum = 3, kUpAverage = 4, kUpValueA = 5, kUpValueO = 6, kUpSlots = 7 };
constexpr int kUpNodeRows = 3;  // behind the children's rows: regret weights, reach, old average reach
constexpr int kUpRow = 64;      // floats
__host__ __device__ constexpr int up_rows(int children) { return kUpSlots * children + kUpNodeRows; }

__device__ __forceinline__ void async_pair(float* shared, const float* global) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(shared)), "l"(global) : "memory");
}

// The kernels of consecutive passes follow one another without a gap: each lets the next one be scheduled as soon as its own
// blocks run (launch_next), and the next one reads what no pass changes (work lists, records, board tables) before it
// waits for this one's results (previous_done).
__device__ __forceinline__ void launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void previous_done() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

enum UpJob {
    kUpIter = 0,   // second half of an iteration pass
    kUpStart = 1,  // of the start pass: no regrets and sums yet
    kUpFinal = 2,  // of the final pass: values only, the root's too
    kUpBase = 3    // plain expectation under the average policy from the clamped leaf values (:732-735), for the exploitability
};
struct UpPass {  // what a pass does, uniform over the grid
    int job;
    bool update, tracked, mix, mixed, keep_values, keep_policy, sample;
    IterScalars sc, sn;
    Divisor d_pos, d_neg;
};

// Starts the copies of a node's rows, except the values of its internal children, which may not be there yet.
__device__ __forceinline__ void up_stage(const CfrParams& p, const SplitWork& w, const UpPass& u, const SplitItem& it,
                                         const NodeRecPacked* nodes, int h, int leaf0, float* at) {
    const int k = it.n_children, a = it.to_act;
    const long long row = it.node_begin + it.first_child;
    const float* rec = w.rec + row * kRec + h;
    const long long kids = row * P2B_HPAD + h;
    const float *R = p.regrets + kids, *W = p.weight_sums + kids, *A = p.policy_avg + kids;
    float* d = at;
#pragma unroll 1
    for (int c = 0; c < k; ++c) {
        async_pair(d + kUpPolicy * kUpRow, rec + kRecPolicy * P2B_HPAD);
        async_pair(d + kUpSeen * kUpRow, rec + kRecSeen * P2B_HPAD);
        if (u.job == kUpStart) {
            *reinterpret_cast<float2*>(d + kUpRegret * kUpRow) = make_float2(0.0f, 0.0f);
            *reinterpret_cast<float2*>(d + kUpSum * kUpRow) = make_float2(0.0f, 0.0f);
        } else {
            if (u.update) async_pair(d + kUpRegret * kUpRow, R);
            if (u.tracked) async_pair(d + kUpSum * kUpRow, W);
        }
        if (u.mix) async_pair(d + kUpAverage * kUpRow, A);
        const int kind = it.kind[c];
        if (u.job == kUpBase && kind != kInternal) {
            const float* v = p.values_avg + 2 * (row + c) * P2B_HPAD + h;
            async_pair(d + kUpValueA * kUpRow, v + a * P2B_HPAD);
            async_pair(d + kUpValueO * kUpRow, v + (1 - a) * P2B_HPAD);
        } else if (kind == kShowdownLeaf || (kind == kModelLeaf && p.leaf_values)) {
            const float* v = kind == kShowdownLeaf
                                 ? rec + kRecValue * P2B_HPAD
                                 : p.leaf_values + (long long)(leaf0 + nodes[it.first_child + c].internal_idx) * 2 * P2B_HPAD + h;
            async_pair(d + kUpValueA * kUpRow, v + a * P2B_HPAD);
            async_pair(d + kUpValueO * kUpRow, v + (1 - a) * P2B_HPAD);
        } else if (kind != kInternal) {
            const float v0 = kind == kFoldLeaf ? nodes[it.first_child + c].v0 : 0.0f, f = a == 0 ? v0 : -v0;
            *reinterpret_cast<float2*>(d + kUpValueA * kUpRow) = make_float2(f, f);
            *reinterpret_cast<float2*>(d + kUpValueO * kUpRow) = make_float2(-f, -f);
        }
        d += kUpSlots * kUpRow;
        rec += kRec;
        R += P2B_HPAD;
        W += P2B_HPAD;
        A += P2B_HPAD;
    }
    const float* me = w.rec + (long long)(it.node_begin + it.node) * kRec + h;
    if (u.update) async_pair(d, me + kRecWeight * P2B_HPAD);
    if (u.mix) {
        async_pair(d + kUpRow, me + kRecReach * P2B_HPAD);
        async_pair(d + 2 * kUpRow, me + kRecOldReach * P2B_HPAD);
    }
}

__device__ __forceinline__ void up_stage_values(const SplitWork& w, const SplitItem& it, int h, float* at) {
    const float* v = w.rec + (long long)(it.node_begin + it.first_child) * kRec + kRecValue * P2B_HPAD + h;
#pragma unroll 1
    for (int c = 0; c < it.n_children; ++c) {
        if (it.kind[c] == kInternal) {
            async_pair(at + (kUpSlots * c + kUpValueA) * kUpRow, v + c * kRec + it.to_act * P2B_HPAD);
            async_pair(at + (kUpSlots * c + kUpValueO) * kUpRow, v + c * kRec + (1 - it.to_act) * P2B_HPAD);
        }
    }
}

// The warps of a slice tell one another when the values of a level are stored: an mbarrier a level, at which each warp arrives
// once.  What follows the values at a node (average, regrets, next policy) does not hold up the levels above.
__device__ __forceinline__ void level_init(uint64_t* bar, int warps) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(bar)), "r"(warps) : "memory");
}
__device__ __forceinline__ void level_arrive(uint64_t* bar) {  // the whole warp
    __threadfence_block();
    __syncwarp();
    if ((threadIdx.x & 31) == 0)
        asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"((unsigned)__cvta_generic_to_shared(bar)) : "memory");
}
__device__ __forceinline__ bool level_wait(uint64_t* bar, const int32_t* others) {  // false: given up, the sooner if others have
    for (int i = 0; i < (1 << 20); ++i) {
        unsigned done;
        asm volatile(
            "{\n .reg .pred q;\n mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 q, [%1], 0;\n selp.u32 %0, 1, 0, q;\n}"
            : "=r"(done)
            : "r"((unsigned)__cvta_generic_to_shared(bar))
            : "memory");
        if (done) return true;
        if ((i & 1023) == 1023 && *reinterpret_cast<const volatile int32_t*>(others) != 0) break;
    }
    return false;
}

// `stored`: where to arrive once the node's values are stored (null: the warp has another node of this level to come).
__device__ __forceinline__ void up_node(const CfrParams& p, const SplitWork& w, const UpPass& u, const SplitItem& it, int h,
                                        float* at, uint64_t* stored) {
    const int k = it.n_children, a = it.to_act, j = it.node, fc = it.first_child;
    const long long kids = (long long)(it.node_begin + fc) * P2B_HPAD + h;
    const float* node_rows = at + k * kUpSlots * kUpRow;
    auto slot = [&](int c, int which) { return at + (kUpSlots * c + which) * kUpRow; };
    FV<2> acc_a, acc_o;
    acc_a.v[0] = acc_a.v[1] = acc_o.v[0] = acc_o.v[1] = 0.0f;
#pragma unroll 2
    for (int c = 0; c < k; ++c) {
        const FV<2> P = ldc<2>(slot(c, kUpPolicy)), Q = ldc<2>(slot(c, kUpSeen));
        FV<2> Va = ldc<2>(slot(c, kUpValueA)), Vo = ldc<2>(slot(c, kUpValueO));
        if (u.job == kUpBase && it.kind[c] != kInternal) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                Va.v[i] = fminf(fmaxf(Va.v[i], -1.0f), 1.0f);
                Vo.v[i] = fminf(fmaxf(Vo.v[i], -1.0f), 1.0f);
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            acc_a.v[i] = __fadd_rn(acc_a.v[i], __fmul_rn(Va.v[i], P.v[i]));
            acc_o.v[i] = __fadd_rn(acc_o.v[i], __fmul_rn(Vo.v[i], Q.v[i]));
        }
    }
    if (j != 0 || u.job >= kUpFinal) {
        float* v = j == 0 && u.job == kUpBase ? p.carry_roots + (long long)it.subgame * 4 * P2B_HPAD + h
                                              : w.rec + (long long)(it.node_begin + j) * kRec + kRecValue * P2B_HPAD + h;
        stc<2>(v + a * P2B_HPAD, acc_a);
        stc<2>(v + (1 - a) * P2B_HPAD, acc_o);
    }
    if (stored) level_arrive(stored);
    if (u.job >= kUpFinal) return;
    if (u.keep_values) {  // the values of this iteration at the node and at the leaves below it
        float* out = p.values_avg + (long long)it.node_begin * 2 * P2B_HPAD + h;
        stc<2>(out + (2 * j + a) * P2B_HPAD, acc_a);
        stc<2>(out + (2 * j + 1 - a) * P2B_HPAD, acc_o);
#pragma unroll 1
        for (int c = 0; c < k; ++c)
            if (it.kind[c] != kInternal) {
                stc<2>(out + (2 * (fc + c) + a) * P2B_HPAD, ldc<2>(slot(c, kUpValueA)));
                stc<2>(out + (2 * (fc + c) + 1 - a) * P2B_HPAD, ldc<2>(slot(c, kUpValueO)));
            }
    }
    if (u.keep_policy || u.sample) {
#pragma unroll 1
        for (int c = 0; c < k; ++c) {
            const FV<2> P = ldc<2>(slot(c, kUpPolicy));
            if (u.keep_policy) stc<2>(p.policy + kids + c * P2B_HPAD, P);
            if (u.sample) stc<2>(p.policy_sample + kids + c * P2B_HPAD, P);
        }
    }
    float* A_row = p.policy_avg + kids;
    if (u.mix) {
        const FV<2> ra = ldc<2>(node_rows + kUpRow), rba = ldc<2>(node_rows + 2 * kUpRow);
        FV<2> ro, rn, sum;
        Divisor d[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            ro.v[i] = __fmul_rn(rba.v[i], u.sc.mix_old);
            rn.v[i] = __fmul_rn(ra.v[i], u.sc.mix_new);
            const float den = __fadd_rn(ro.v[i], rn.v[i]);
            const bool weighted = den > 1e-5f;  // else: (numerically) no reach, the plain iteration weights (:1231-1239)
            ro.v[i] = weighted ? ro.v[i] : u.sc.mix_old;
            rn.v[i] = weighted ? rn.v[i] : u.sc.mix_new;
            d[i] = make_divisor(weighted ? den : u.sc.mix_total);
            sum.v[i] = 0.0f;
        }
#pragma unroll 2
        for (int c = 0; c < k; ++c) {
            const FV<2> P = ldc<2>(slot(c, kUpPolicy)), A = ldc<2>(slot(c, kUpAverage));
            DivGuard g = guard_begin(d[0].ok && d[1].ok);
            FV<2> num, q;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                num.v[i] = __fadd_rn(__fmul_rn(ro.v[i], A.v[i]), __fmul_rn(rn.v[i], P.v[i]));
                q.v[i] = div_g<true>(num.v[i], d[i].y, d[i].r, g);
            }
            if (__builtin_expect(guard_bad(g), 0)) {
#pragma unroll
                for (int i = 0; i < 2; ++i) q.v[i] = __fdiv_rn(num.v[i], d[i].y);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) sum.v[i] = __fadd_rn(sum.v[i], q.v[i]);
            stc<2>(slot(c, kUpAverage), q);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) d[i] = make_divisor(sum.v[i]);
#pragma unroll 2
        for (int c = 0; c < k; ++c) {
            FV<2> x = ldc<2>(slot(c, kUpAverage)), q;
            DivGuard g = guard_begin(d[0].ok && d[1].ok);
#pragma unroll
            for (int i = 0; i < 2; ++i) q.v[i] = div_g<true>(x.v[i], d[i].y, d[i].r, g);
            if (__builtin_expect(guard_bad(g), 0)) {
#pragma unroll
                for (int i = 0; i < 2; ++i) q.v[i] = __fdiv_rn(x.v[i], sum.v[i]);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
                if (sum.v[i] > 1e-5f) x.v[i] = q.v[i];
            stc<2>(A_row + c * P2B_HPAD, x);
        }
    } else if (!u.mixed) {
#pragma unroll 1
        for (int c = 0; c < k; ++c) stc<2>(A_row + c * P2B_HPAD, ldc<2>(slot(c, kUpPolicy)));
    }
    if (!u.update) return;
    const FV<2> wgt = ldc<2>(node_rows);
    const bool no_regret = ((u.sn.do_mix >> 1) & 3) == a + 1;  // linear CFR: this player's actions get none
    FV<2> sum;
    sum.v[0] = sum.v[1] = 0.0f;
#pragma unroll 2
    for (int c = 0; c < k; ++c) {
        FV<2> R = ldc<2>(slot(c, kUpRegret)), W;
        const FV<2> Va = ldc<2>(slot(c, kUpValueA));
        W = R;
        if (u.tracked) W = ldc<2>(slot(c, kUpSum));
        DivGuard g = guard_begin(u.d_pos.ok && u.d_neg.ok);
        FV<2> rn, rq, wn, wq, dy;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const bool pos = R.v[i] > 0.0f;
            const float num = pos ? u.sn.num_pos : u.sn.num_neg, dr = pos ? u.d_pos.r : u.d_neg.r;
            dy.v[i] = pos ? u.d_pos.y : u.d_neg.y;
            rn.v[i] = __fmul_rn(R.v[i], num);
            rq.v[i] = div_g<false>(rn.v[i], dy.v[i], dr, g);
            if (u.tracked) {
                wn.v[i] = __fmul_rn(W.v[i], num);
                wq.v[i] = div_g<true>(wn.v[i], dy.v[i], dr, g);
            }
        }
        if (__builtin_expect(guard_bad(g), 0)) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                rq.v[i] = __fdiv_rn(rn.v[i], dy.v[i]);
                if (u.tracked) wq.v[i] = __fdiv_rn(wn.v[i], dy.v[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float reg = no_regret ? 0.0f : __fmul_rn(wgt.v[i], __fsub_rn(Va.v[i], acc_a.v[i]));
            float rr = __fadd_rn(rq.v[i], reg);
            if (p.cfr_plus) rr = fmaxf(rr, 0.0f);
            R.v[i] = rr;
            if (u.tracked) W.v[i] = __fadd_rn(wq.v[i], 1.0f);
        }
        stc<2>(p.regrets + kids + c * P2B_HPAD, R);
        if (u.tracked) stc<2>(p.weight_sums + kids + c * P2B_HPAD, W);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            R.v[i] = fmaxf(R.v[i], 0.0f);
            sum.v[i] = __fadd_rn(sum.v[i], R.v[i]);
        }
        stc<2>(slot(c, kUpRegret), R);
    }
    const float invk = __fdiv_rn(1.0f, (float)k);
    Divisor d[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) d[i] = make_divisor(fmaxf(sum.v[i], 1e-8f));
    float* P_row = w.rec + (long long)(it.node_begin + fc) * kRec + h;
#pragma unroll 2
    for (int c = 0; c < k; ++c) {
        const FV<2> x = ldc<2>(slot(c, kUpRegret));
        DivGuard g = guard_begin(d[0].ok && d[1].ok);
        FV<2> q;
#pragma unroll
        for (int i = 0; i < 2; ++i) q.v[i] = div_g<true>(x.v[i], d[i].y, d[i].r, g);
        if (__builtin_expect(guard_bad(g), 0)) {
#pragma unroll
            for (int i = 0; i < 2; ++i) q.v[i] = __fdiv_rn(x.v[i], d[i].y);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) q.v[i] = sum.v[i] > 1e-8f ? q.v[i] : invk;
        stc<2>(P_row + c * kRec, q);
    }
}

// A block holds `slices` slices of one subgame with `lanes` warps each, which take the nodes of a level in turn.  `ring`: rows of a warp's staging area; two nodes that follow one
// another lie at its two ends if they fit together, else the second is copied once the first is done.
__global__ void __launch_bounds__(kUpThreads) split_up_kernel(const CfrParams p, const SplitWork w, int job, int pass, bool advance,
                                                              bool mixed, int lanes, int slices, int ring) {
    constexpr int kSlices = P2B_HPAD / kUpRow;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint64_t ready[kUpSlices][kSplitMaxDepth + 1];
    if (refused(p)) return;
    const int per_subgame = kSlices / slices;
    const int q = blockIdx.x / per_subgame;
    const int s = p.queue_order ? p.queue_order[q] : q;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, mine = warp / lanes, lane_warp = warp - mine * lanes;
    const int h = ((blockIdx.x - q * per_subgame) * slices + mine) * kUpRow + lane * 2;
    const SubgameRec sg = p.subgames[s];
    float* stage = reinterpret_cast<float*>(smem) + (long long)warp * ring * kUpRow + lane * 2;
    SplitItem* items = reinterpret_cast<SplitItem*>(smem + (size_t)lanes * slices * ring * kUpRow * 4);
    NodeRecPacked* nodes = reinterpret_cast<NodeRecPacked*>(items + sg.n_internal);
    const SplitLevels* lv = w.levels + q;
    {
        const uint4* ns = reinterpret_cast<const uint4*>(p.nodes + sg.node_begin);
        for (int i = tid; i < sg.n_nodes; i += blockDim.x) reinterpret_cast<uint4*>(nodes)[i] = ns[i];
        const uint4* is = reinterpret_cast<const uint4*>(w.items + lv->item_begin);
        for (int i = tid; i < sg.n_internal * 4; i += blockDim.x) reinterpret_cast<uint4*>(items)[i] = is[i];
    }
    UpPass u;
    u.job = job;
    u.sc = p.scalars[job == kUpIter ? pass : 0];
    u.update = job <= kUpStart && pass + 1 < p.iterations;
    u.sn = p.scalars[u.update ? pass + 1 : 0];
    u.tracked = u.update && p.weight_sums != nullptr;
    u.mixed = mixed;
    u.mix = job == kUpIter && !mixed && (u.sc.do_mix & 1) != 0;
    u.keep_values = p.iter_values && p.values_avg != nullptr;
    u.keep_policy = job == kUpIter && p.policy != nullptr && pass == p.iterations - 1;
    u.sample = job == kUpIter && p.policy_sample != nullptr && p.sample_pass[s] == pass;
    u.d_pos = make_divisor(u.sn.den_pos);
    u.d_neg = make_divisor(u.sn.den_neg);
    const int leaf0 = p.leaf_begin ? p.leaf_begin[s] : 0;
    if (tid < slices * (kSplitMaxDepth + 1)) level_init(&ready[0][0] + tid, lanes);
    __syncthreads();
    launch_next();
    previous_done();

    uint64_t* level_ready = ready[mine];
    auto first_of = [&](int d) { return (int)lv->begin[d + 1] - 1 - lane_warp; };
    const int n_levels = lv->n_levels;
    int d = n_levels - 1, waited = n_levels;  // levels from `waited` on are known to be stored
    int x = first_of(d);
    auto skip_empty = [&]() {  // to the warp's next node; it has nothing to store at the levels in between
        while (x < lv->begin[d]) {
            level_arrive(level_ready + d);
            if (d == 0) return false;
            x = first_of(--d);
        }
        return true;
    };
    bool any = skip_empty(), top = false;
    if (any) up_stage(p, w, u, items[x], nodes, h, leaf0, stage);
    while (any) {
        const SplitItem& it = items[x];
        const int rows = up_rows(it.n_children);
        float* at = stage + (top ? (ring - rows) * kUpRow : 0);
        if (d + 1 < waited) {  // its children are one level down
            if (!level_wait(level_ready + d + 1, gave_up(p))) atomicMax(gave_up(p), s + 1);
            waited = d + 1;
        }
        up_stage_values(w, it, h, at);
        asm volatile("cp.async.wait_all;" ::: "memory");
        uint64_t* stored = nullptr;
        x -= lanes;
        if (x < lv->begin[d]) {  // the warp's last node of this level; the empty levels above take its arrival now
            stored = level_ready + d;
            any = d > 0;
            if (any) {
                x = first_of(--d);
                any = skip_empty();
            }
        }
        const int next_rows = any ? up_rows(items[x].n_children) : 0;
        float* next_at = stage + (top ? 0 : (ring - next_rows) * kUpRow);
        const bool ahead = rows + next_rows <= ring;
        if (any && ahead) up_stage(p, w, u, items[x], nodes, h, leaf0, next_at);
        up_node(p, w, u, it, h, at, stored);
        if (any && !ahead) up_stage(p, w, u, items[x], nodes, h, leaf0, next_at);
        top = !top;
    }
    if (advance && lane_warp == 0) advance_root(p, s, h);
}

// ---- rows ---------------------------------------------------------------------------------------
// Beliefs of a node (cfr_evaluator.py:363-380), the other player's view of every action (:1076-1093), the regret
// weights (:1117-1165), showdown values (:484-601) and the beliefs handed to the caller's model.
//
// 448 threads with three hands each, a third of a row apart: consecutive threads touch consecutive hands in global
// and shared memory, and two blocks fit an SM (72 registers a thread).
constexpr int kScanQuarter = 352;  // 32 lanes x 11 sorted positions

struct RowLayout {  // byte offsets into dynamic shared memory
    int tab, rows, pref, pc, tot, scan, cs, S, sums, item, bytes;
    int leaf_row;
};
__host__ __device__ constexpr RowLayout row_layout(int max_children, bool showdown) {
    RowLayout l{};
    int at = 0;
    l.tab = at;
    at += showdown ? kTabBytes : 0;
    l.rows = at;
    l.leaf_row = 2 + max_children;
    at += (2 + max_children + (showdown ? 1 : 0)) * P2B_HPAD * 4;
    l.pref = at;
    at += showdown ? 2 * P2B_HPAD * 4 : 0;
    l.pc = at;
    at += showdown ? 2 * 52 * 52 * 4 : 0;
    l.tot = at;
    at += showdown ? 2 * 64 * 4 : 0;
    l.scan = at;
    at += showdown ? 2 * 4 * 32 * 8 : 0;
    l.cs = at;
    at += (2 + max_children) * 52 * 8;
    l.S = at;
    at += (2 + kCfrMaxChildren) * 8;
    l.sums = at;
    at += 2 * 16 * 4;
    l.item = at;
    at += 64;
    l.bytes = at;
    return l;
}

struct Row3 {
    float v[kHandsPerThread];
};
__device__ __forceinline__ Row3 ld3(const float* row, int tid) {
    Row3 r;
#pragma unroll
    for (int i = 0; i < kHandsPerThread; ++i) r.v[i] = row[tid + i * kRowThreads];
    return r;
}
__device__ __forceinline__ void st3(float* row, int tid, const Row3& r) {
#pragma unroll
    for (int i = 0; i < kHandsPerThread; ++i) row[tid + i * kRowThreads] = r.v[i];
}
__device__ __forceinline__ Row3 mul3(const Row3& x, const Row3& y) {
    Row3 r;
#pragma unroll
    for (int i = 0; i < kHandsPerThread; ++i) r.v[i] = __fmul_rn(x.v[i], y.v[i]);
    return r;
}
__device__ __forceinline__ Row3 path3(const float* base, int stride, const uint16_t* path, int n, Row3 r, int tid) {
#pragma unroll 2
    for (int e = 0; e < n; ++e) r = mul3(r, ld3(base + (unsigned)path[e] * (unsigned)stride, tid));
    return r;
}

struct Hands {
    int c1[kHandsPerThread], c2[kHandsPerThread];
    bool real[kHandsPerThread], allowed[kHandsPerThread];
};

// x / sum, or uniform over the allowed hands when the row is (numerically) empty (cfr_evaluator.py:263-273)
__device__ __forceinline__ Row3 normalised(Row3 x, float sum, float allowed_prob, const Hands& hi) {
    const Divisor d = make_divisor(sum);
    DivGuard g = guard_begin(d.ok);
    Row3 q;
#pragma unroll
    for (int i = 0; i < kHandsPerThread; ++i) q.v[i] = div_g<true>(x.v[i], d.y, d.r, g);
    if (__builtin_expect(guard_bad(g), 0)) {
#pragma unroll
        for (int i = 0; i < kHandsPerThread; ++i) q.v[i] = __fdiv_rn(x.v[i], sum);
    }
#pragma unroll
    for (int i = 0; i < kHandsPerThread; ++i) q.v[i] = sum > 1e-5f ? q.v[i] : (hi.allowed[i] ? allowed_prob : 0.0f);
    return q;
}

// Tables of the showdown formula for two ranges (x: the other player's beliefs x0, y: the leaf row x1), their entries side by
// side, so that one gather of a hand's position serves both.  Of each range, four warps scan a quarter of the strength
// order each (a quarter's offset is the sum of the earlier ones, which they hand one another) and 208 threads take a
// quarter of a card's list each.
__device__ __forceinline__ void showdown_tables(const BoardTabView& tv, const float* x0, const float* x1, float2* pref2, float2* pc2,
                                                float2* tot2, double* scan) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (warp < 8) {
        const uint16_t* __restrict__ sorted = tv.sorted;
        const int slot = warp & 1, qi = 3 - (warp >> 1), k0 = qi * kScanQuarter + 11 * lane;
        const float* __restrict__ x = slot ? x1 : x0;
        float* __restrict__ pref = reinterpret_cast<float*>(pref2) + slot;
        float v[11];
#pragma unroll
        for (int i = 0; i < 11; ++i) v[i] = (k0 + i < P2B_NUM_HANDS) ? x[sorted[k0 + i]] : 0.0f;
        double a0 = 0.0, a1 = 0.0, local = 0.0;
#pragma unroll
        for (int i = 0; i < 11; ++i) {
            local += (double)v[i];
            if (i & 1) a1 += (double)v[i];
            else a0 += (double)v[i];
        }
        double* part = scan + slot * 128 + lane;  // what each lane of each quarter adds up to
        part[qi * 32] = a0 + a1;
        asm volatile("bar.sync %0, 128;" ::"r"(slot + 1) : "memory");
        double before = 0.0;
        for (int r = 0; r < qi; ++r) before += part[r * 32];
        before = warp_sum(before);
        double incl = local;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += up;
        }
        double run = before + (incl - local);
        if (qi == 0 && lane == 0) pref[0] = 0.0f;
#pragma unroll
        for (int i = 0; i < 11; ++i) {
            run += (double)v[i];
            if (k0 + i < P2B_NUM_HANDS) pref[2 * (k0 + i + 1)] = (float)run;
        }
    }
    // the lists: the second range from the last 208 threads of the block down
    const int back = kRowThreads - 1 - tid;
    if (back < 416) {
        const int slot = back < 208 ? 1 : 0, u = 207 - (back - (slot ? 0 : 208)), c = u >> 2, q = u & 3;
        const float* __restrict__ x = slot ? x1 : x0;
        const uint16_t* __restrict__ at = tv.cardlist + 13 * q * 52 + c;
        float v[13];
#pragma unroll
        for (int i = 0; i < 12; ++i) v[i] = x[at[i * 52]];
        v[12] = q < 3 ? x[at[12 * 52]] : 0.0f;
        double t_even = 0.0, t_odd = 0.0;
#pragma unroll
        for (int i = 0; i < 13; ++i) {
            if (i & 1) t_odd += (double)v[i];
            else t_even += (double)v[i];
        }
        const double mine = t_even + t_odd;
        const int g = lane & ~3;
        const double t0 = __shfl_sync(0xffffffffu, mine, g), t1 = __shfl_sync(0xffffffffu, mine, g + 1);
        const double t2 = __shfl_sync(0xffffffffu, mine, g + 2);
        double acc = q == 0 ? 0.0 : (q == 1 ? t0 : (q == 2 ? t0 + t1 : (t0 + t1) + t2));
        float* __restrict__ row = reinterpret_cast<float*>(pc2) + 2 * c * 52 + slot;
        if (q == 0) row[0] = 0.0f;
        float* __restrict__ out = row + 2 * (13 * q + 1);
#pragma unroll
        for (int i = 0; i < 12; ++i) {
            acc += (double)v[i];
            out[2 * i] = (float)acc;
        }
        if (q < 3) out[24] = (float)(acc + (double)v[12]);
        else reinterpret_cast<float*>(tot2)[2 * c + slot] = (float)acc;  // == row[51]
    }
}

// Showdown EV (before the pot scaling) of this thread's hands against the two ranges.
__device__ __forceinline__ void showdown_rows(const BoardTabView& tv, const float* x0, const float* x1, const float2* pref,
                                              const float2* pc, const float2* tot, const Hands& hi, Row3& ev0, Row3& ev1) {
    DivGuard g = guard_begin(true);
#pragma unroll
    for (int i = 0; i < kHandsPerThread; ++i) {
        const int h = threadIdx.x + i * kRowThreads;
        showdown_hand_pair<false>(*reinterpret_cast<const uint2*>(tv.rec + (hi.real[i] ? h : 0)), hi.c1[i], hi.c2[i], x0[h], x1[h],
                                  hi.allowed[i], pref, pc, tot, g, ev0.v[i], ev1.v[i]);
    }
    if (__builtin_expect(guard_bad(g), 0)) {
#pragma unroll
        for (int i = 0; i < kHandsPerThread; ++i) {
            const int h = threadIdx.x + i * kRowThreads;
            showdown_hand_pair<true>(*reinterpret_cast<const uint2*>(tv.rec + (hi.real[i] ? h : 0)), hi.c1[i], hi.c2[i], x0[h], x1[h],
                                     hi.allowed[i], pref, pc, tot, g, ev0.v[i], ev1.v[i]);
        }
    }
}

// The start pass at one node.  Upstream pushes the beliefs down one level at a time and re-normalises EVERY row after each
// level (cfr_evaluator.py:855-875): a node at level L is normalised init_depth - L + 1 times, its children derive from its
// once-normalised row, and the root's row, which its children take as given, is normalised once a level itself.
template <int K>
__device__ __forceinline__ void start_rows(const CfrParams& p, const SubgameRec& sg, const SplitItem& it, float* rows, float* sums,
                                           float* leaf, float* rec, float* cr, int leaf0, const Hands& hi, int tid) {
    const int a = it.to_act, o = 1 - a, j = it.node, fc = it.first_child, lane = tid & 31, warp = tid >> 5;
    const int depth = it.n_path[0] + it.n_path[1];
    const long long nb = (long long)sg.node_begin * P2B_HPAD;
    auto normalise = [&](Row3& u, Row3& v, int times) {
#pragma unroll 1
        for (int t = 0; t < times; ++t) {
            __syncthreads();
            st3(rows, tid, u);
            st3(rows + P2B_HPAD, tid, v);
            __syncthreads();
            if (warp < 2) {
                const float sum = row_sum_reference_order(rows + warp * P2B_HPAD);
                if (lane == 0) sums[warp] = sum;
            }
            __syncthreads();
            u = normalised(u, sums[0], sg.allowed_prob, hi);
            v = normalised(v, sums[1], sg.allowed_prob, hi);
        }
    };
    auto policy = [&](int node) {  // the start policy: the caller's, or uniform over the siblings
        if (p.start_policy) return ld3(p.start_policy + nb + (long long)node * P2B_HPAD, tid);
        const int siblings = load_node(p.nodes + sg.node_begin + load_node(p.nodes + sg.node_begin + node).parent).n_children;
        Row3 r;
        r.v[0] = r.v[1] = r.v[2] = __fdiv_rn(1.0f, (float)siblings);
        return r;
    };
    const float* given = p.root_beliefs + (long long)it.subgame * 2 * P2B_HPAD;
    Row3 r_a = ld3(given + a * P2B_HPAD, tid), r_o = ld3(given + o * P2B_HPAD, tid);
#pragma unroll
    for (int i = 0; i < kHandsPerThread; ++i) {
        r_a.v[i] = hi.allowed[i] ? r_a.v[i] : 0.0f;
        r_o.v[i] = hi.allowed[i] ? r_o.v[i] : 0.0f;
    }
    if (j == 0) {
        st3(cr + a * P2B_HPAD, tid, r_a);
        st3(cr + o * P2B_HPAD, tid, r_o);
    }
#pragma unroll 1
    for (int ia = 0, io = it.n_path[0]; ia + io < it.n_path[0] + depth;) {  // down the path, both players' nodes in order
        const bool acting = io >= depth || (ia < it.n_path[0] && it.path[ia] < it.path[io]);
        const Row3 P = policy(acting ? it.path[ia] : it.path[io]);
        if (acting) {
            r_a = mul3(r_a, P);
            ++ia;
        } else {
            r_o = mul3(r_o, P);
            ++io;
        }
        normalise(r_a, r_o, 1);
    }
    Row3 b_a = r_a, b_o = r_o;
    normalise(b_a, b_o, j == 0 ? max(p.init_depth, 1) : p.init_depth - depth);
    if (j == 0) {
        st3(cr + (2 + a) * P2B_HPAD, tid, b_a);
        st3(cr + (2 + o) * P2B_HPAD, tid, b_o);
    }
#pragma unroll 1
    for (int c = 0; c < K; ++c) {
        const Row3 P = policy(fc + c);
        st3(p.policy_avg + nb + (fc + c) * P2B_HPAD, tid, P);
        st3(rec + (fc + c) * kRec, tid, P);
        if (it.kind[c] == kShowdownLeaf || (it.kind[c] == kModelLeaf && p.leaf_beliefs)) {
            Row3 x_a = mul3(r_a, P), x_o = r_o;
            normalise(x_a, x_o, p.init_depth - depth);
            if (it.kind[c] == kModelLeaf) {
                float* out = p.leaf_beliefs + 2ll * (leaf0 + load_node(p.nodes + sg.node_begin + fc + c).internal_idx) * P2B_HPAD;
                st3(out + a * P2B_HPAD, tid, x_a);
                st3(out + o * P2B_HPAD, tid, x_o);
            } else {
                st3(c == it.first_sd ? leaf : rec + (fc + c) * kRec + kRecValue * P2B_HPAD, tid, x_a);
            }
        }
        st3(rows + (2 + c) * P2B_HPAD, tid, mul3(b_a, P));
    }
    __syncthreads();
    st3(rows, tid, b_a);
    st3(rows + P2B_HPAD, tid, b_o);
}

enum RowKind {
    kRowIter = 0,   // iteration pass, beliefs under the current policy
    kRowAvg = 1,    // iteration pass that also needs the beliefs under the average policy (cfr_avg, kept values)
    kRowStart = 2,  // start pass: the start policy, beliefs re-normalised once per level (:830-886)
    kRowFinal = 3   // final pass: the average policy (`update_average_values_final`, :1276-1292)
};

template <int MAXK, bool SD, int KIND>
__global__ void __launch_bounds__(kRowThreads, 2) split_rows_kernel(const CfrParams p, const SplitWork w, int pass) {
    constexpr bool AVG = KIND == kRowAvg;
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr RowLayout L = row_layout(MAXK, SD);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* rows = reinterpret_cast<float*>(smem + L.rows);
    float* leaf = rows + L.leaf_row * P2B_HPAD;
    float2* pref = reinterpret_cast<float2*>(smem + L.pref);
    float2* pc = reinterpret_cast<float2*>(smem + L.pc);
    float2* tot = reinterpret_cast<float2*>(smem + L.tot);
    double* scan = reinterpret_cast<double*>(smem + L.scan);
    double* cs = reinterpret_cast<double*>(smem + L.cs);
    double* S = reinterpret_cast<double*>(smem + L.S);
    float* sums = reinterpret_cast<float*>(smem + L.sums);
    float* sums_avg = sums + 16;
    const SplitItem& it = *reinterpret_cast<const SplitItem*>(smem + L.item);
    if (refused(p)) return;

    Hands hi;
#pragma unroll
    for (int i = 0; i < kHandsPerThread; ++i) {
        const int h = tid + i * kRowThreads;
        hi.real[i] = h < P2B_NUM_HANDS;
        const int hc = hi.real[i] ? h : P2B_NUM_HANDS - 1;
        hi.c1[i] = p.combos->c1[hc];
        hi.c2[i] = p.combos->c2[hc];
    }
    uint32_t idx[7];
    card_indices(tid, idx);
    const bool mix = KIND == kRowIter && (p.scalars[pass].do_mix & 1) != 0;
    launch_next();
    bool waited = false;
    // a block takes consecutive items: mostly nodes of one subgame, whose board tables stay in shared memory
    const long long total = w.total[0];
    const int first = (int)(blockIdx.x * total / gridDim.x), last = (int)((blockIdx.x + 1) * total / gridDim.x);
    int table = -1;
    for (int x = first; x < last; ++x) {
        __syncthreads();  // every thread is done with the shared memory of the item before
        if (tid < 16) reinterpret_cast<uint32_t*>(smem + L.item)[tid] = reinterpret_cast<const uint32_t*>(w.items + x)[tid];
        __syncthreads();
        const SubgameRec sg = p.subgames[it.subgame];
        const int a = it.to_act, o = 1 - a, j = it.node, k = it.n_children, fc = it.first_child;
        const bool showdown = SD && it.first_sd != kNoChild;
        if (showdown && sg.table_index != table) {
            table = sg.table_index;
            const uint4* t = reinterpret_cast<const uint4*>(p.tables + (long long)table * kTabBytes);
            for (int i = tid; i < kTabBytes / 16; i += kRowThreads) reinterpret_cast<uint4*>(smem + L.tab)[i] = t[i];
        }
        Row3 mask;
#pragma unroll
        for (int i = 0; i < kHandsPerThread; ++i) {
            hi.allowed[i] = hi.real[i] && (((sg.board_mask >> hi.c1[i]) | (sg.board_mask >> hi.c2[i])) & 1ull) == 0;
            mask.v[i] = hi.allowed[i] ? 1.0f : 0.0f;
        }
        if (!waited) {
            previous_done();
            waited = true;
        }
        const long long nb = (long long)sg.node_begin * P2B_HPAD;
        float* rec = w.rec + (long long)sg.node_begin * kRec;
        float* cr = p.carry_roots + (long long)it.subgame * 4 * P2B_HPAD;
        const int leaf0 = p.leaf_begin ? p.leaf_begin[it.subgame] : 0;
        // cfr_avg: showdown values, regret weights and the beliefs of the caller's model under the average policy (:1029, :1133)
        const bool avgb = AVG && p.cfr_avg != 0;
        const bool keep_avg = AVG && p.iter_values != 0 && p.beliefs_avg != nullptr;
        const float* avg_sums = avgb ? sums_avg : sums;

        with_children<MAXK>(k, [&](auto kc) {
            constexpr int K = decltype(kc)::value;
            if constexpr (KIND == kRowStart) {
                start_rows<K>(p, sg, it, rows, sums, leaf, rec, cr, leaf0, hi, tid);
                return;
            }
            Row3 P[K];
            const float* policy = KIND == kRowFinal ? p.policy_avg + nb : rec;
            constexpr int kPolicyStride = KIND == kRowFinal ? P2B_HPAD : kRec;
#pragma unroll
            for (int c = 0; c < K; ++c) {
                P[c] = ld3(policy + (fc + c) * kPolicyStride, tid);
                if (KIND == kRowFinal) st3(rec + (fc + c) * kRec, tid, P[c]);
            }
            const Row3 prior_a = ld3(cr + a * P2B_HPAD, tid), prior_o = ld3(cr + o * P2B_HPAD, tid);
            const Row3 r_a = path3(policy, kPolicyStride, it.path, it.n_path[0], mask, tid);
            const Row3 r_o = path3(policy, kPolicyStride, it.path + it.n_path[0], it.n_path[1], mask, tid);
            const Row3 u_a = mul3(prior_a, r_a), u_o = mul3(prior_o, r_o);
            if (KIND == kRowIter && mix) {  // what the average-policy mix weights by
                st3(rec + j * kRec + kRecReach * P2B_HPAD, tid, r_a);
                st3(rec + j * kRec + kRecOldReach * P2B_HPAD, tid,
                    path3(p.policy_avg + nb, P2B_HPAD, it.path, it.n_path[0], mask, tid));
            }
            Row3 bbar_a, bbar_o;  // beliefs under the average policy
            if (AVG) {
                const Row3 rw_a = path3(p.policy_avg + nb, P2B_HPAD, it.path, it.n_path[0], mask, tid);
                const Row3 rw_o = path3(p.policy_avg + nb, P2B_HPAD, it.path + it.n_path[0], it.n_path[1], mask, tid);
                bbar_a = mul3(prior_a, rw_a);
                bbar_o = mul3(prior_o, rw_o);
                st3(rows, tid, bbar_a);
                st3(rows + P2B_HPAD, tid, bbar_o);
#pragma unroll
                for (int c = 0; c < K; ++c) {
                    if (it.kind[c] != kShowdownLeaf && !(it.kind[c] == kModelLeaf && p.leaf_beliefs)) continue;
                    const Row3 A = ld3(p.policy_avg + nb + (fc + c) * P2B_HPAD, tid);
                    st3(rows + (2 + c) * P2B_HPAD, tid, mul3(prior_a, mul3(rw_a, A)));
                }
                __syncthreads();
                if (warp < 2 + K && (warp < 2 || it.kind[warp - 2] >= kShowdownLeaf)) {
                    const float sum = row_sum_reference_order(rows + warp * P2B_HPAD);
                    if (lane == 0) sums_avg[warp] = sum;
                }
                __syncthreads();
                bbar_a = normalised(bbar_a, sums_avg[0], sg.allowed_prob, hi);
                bbar_o = normalised(bbar_o, sums_avg[1], sg.allowed_prob, hi);
                if (keep_avg) {
                    float* out = p.beliefs_avg + 2 * nb;
                    st3(out + (2 * j + a) * P2B_HPAD, tid, bbar_a);
                    st3(out + (2 * j + o) * P2B_HPAD, tid, bbar_o);
#pragma unroll
                    for (int c = 0; c < K; ++c) {
                        if (it.kind[c] != kModelLeaf) continue;
                        const Row3 bl = p.leaf_beliefs ? normalised(ld3(rows + (2 + c) * P2B_HPAD, tid), sums_avg[2 + c],
                                                                    sg.allowed_prob, hi)
                                                       : Row3{};
                        st3(out + (2 * (fc + c) + a) * P2B_HPAD, tid, bl);
                        st3(out + (2 * (fc + c) + o) * P2B_HPAD, tid, bbar_o);
                    }
                }
            }
            // ---- the rows that are normalised: the node's own and those of the leaves that need beliefs ----
            st3(rows, tid, u_a);
            st3(rows + P2B_HPAD, tid, u_o);
            if (!avgb) {
#pragma unroll
                for (int c = 0; c < K; ++c) {
                    if (it.kind[c] != kShowdownLeaf && !(it.kind[c] == kModelLeaf && p.leaf_beliefs)) continue;
                    st3(rows + (2 + c) * P2B_HPAD, tid, mul3(prior_a, mul3(r_a, P[c])));
                }
            }
            __syncthreads();
            if (warp < 2 + K && (warp < 2 || (!avgb && it.kind[warp - 2] >= kShowdownLeaf))) {
                const float sum = row_sum_reference_order(rows + warp * P2B_HPAD);
                if (lane == 0) sums[warp] = sum;
            }
            __syncthreads();
            const Row3 b_a = normalised(u_a, sums[0], sg.allowed_prob, hi);
            const Row3 b_o = normalised(u_o, sums[1], sg.allowed_prob, hi);
            const Row3 x_o = avgb ? bbar_o : b_o;
            if (KIND != kRowFinal && j == 0) {  // the root's own row, and its sums, for the pass after this one
                st3(cr + (2 + a) * P2B_HPAD, tid, b_a);
                st3(cr + (2 + o) * P2B_HPAD, tid, b_o);
                if (tid == 0) {
                    p.carry_sums[2ll * sg.node_begin + a] = sums[0];
                    p.carry_sums[2ll * sg.node_begin + o] = sums[1];
                }
            }
            if (KIND == kRowFinal) {  // for the value outputs and the best responses
                st3(rec + j * kRec + kRecActing * P2B_HPAD, tid, b_a);
                st3(rec + j * kRec + (kRecBelief + a) * P2B_HPAD, tid, b_a);
                st3(rec + j * kRec + (kRecBelief + o) * P2B_HPAD, tid, b_o);
                if (p.beliefs_avg) {
                    float* out = p.beliefs_avg + 2 * nb;
                    st3(out + (2 * j + a) * P2B_HPAD, tid, b_a);
                    st3(out + (2 * j + o) * P2B_HPAD, tid, b_o);
                }
            }
            if (KIND != kRowFinal && p.beliefs_last && pass == p.iterations - 1) {
                float* out = p.beliefs_last + 2 * nb;
                st3(out + (2 * j + a) * P2B_HPAD, tid, b_a);
                st3(out + (2 * j + o) * P2B_HPAD, tid, b_o);
            }
#pragma unroll
            for (int c = 0; c < K; ++c) {
                float* row = rows + (2 + c) * P2B_HPAD;
                if (SD && it.kind[c] == kShowdownLeaf) {
                    const Row3 x = normalised(ld3(row, tid), avg_sums[2 + c], sg.allowed_prob, hi);
                    st3(c == it.first_sd ? leaf : rec + (fc + c) * kRec + kRecValue * P2B_HPAD, tid, x);
                    if (KIND == kRowFinal && p.beliefs_avg) {
                        float* out = p.beliefs_avg + 2 * nb + 2 * (fc + c) * P2B_HPAD;
                        st3(out + a * P2B_HPAD, tid, x);
                        st3(out + o * P2B_HPAD, tid, b_o);
                    }
                } else if (it.kind[c] == kModelLeaf && p.leaf_beliefs) {
                    const int slot = leaf0 + load_node(p.nodes + sg.node_begin + fc + c).internal_idx;
                    float* out = p.leaf_beliefs + 2ll * slot * P2B_HPAD;
                    st3(out + a * P2B_HPAD, tid, normalised(ld3(row, tid), avg_sums[2 + c], sg.allowed_prob, hi));
                    st3(out + o * P2B_HPAD, tid, x_o);
                }
                st3(row, tid, mul3(b_a, P[c]));
            }
            st3(rows, tid, b_a);
            st3(rows + P2B_HPAD, tid, x_o);
        });
        __syncthreads();
        card_sums(rows, 2 + k, cs, S, idx);
        const BoardTabView tv = view_tables(smem + L.tab);
        if (showdown) showdown_tables(tv, rows + P2B_HPAD, leaf, pref, pc, tot, scan);
        __syncthreads();

        const Row3 b_a = ld3(rows, tid), x_o = ld3(rows + P2B_HPAD, tid);
        {
            Row3 wgt;
            Divisor d[kHandsPerThread];
            bool ok = true;
#pragma unroll
            for (int i = 0; i < kHandsPerThread; ++i) {
                wgt.v[i] = unblocked(cs + 52, S[1], hi.c1[i], hi.c2[i], x_o.v[i]);
                d[i] = make_divisor(unblocked(cs, S[0], hi.c1[i], hi.c2[i], b_a.v[i]));
                ok = ok && d[i].ok;
            }
            if (KIND != kRowFinal) st3(rec + j * kRec + kRecWeight * P2B_HPAD, tid, wgt);
#pragma unroll 1
            for (int c = 0; c < k; ++c) {
                const Row3 m = ld3(rows + (2 + c) * P2B_HPAD, tid);
                Row3 blk, pio;
                DivGuard g = guard_begin(ok);
#pragma unroll
                for (int i = 0; i < kHandsPerThread; ++i) {
                    blk.v[i] = unblocked(cs + (2 + c) * 52, S[2 + c], hi.c1[i], hi.c2[i], m.v[i]);
                    pio.v[i] = div_g<true>(blk.v[i], d[i].y, d[i].r, g);
                }
                if (__builtin_expect(guard_bad(g), 0)) {
#pragma unroll
                    for (int i = 0; i < kHandsPerThread; ++i) pio.v[i] = __fdiv_rn(blk.v[i], d[i].y);
                }
#pragma unroll
                for (int i = 0; i < kHandsPerThread; ++i) pio.v[i] = d[i].y > 1e-5f ? pio.v[i] : 0.0f;
                st3(rec + (fc + c) * kRec + kRecSeen * P2B_HPAD, tid, pio);
            }
        }
        if (!showdown) continue;
        // the acting player's hands against the other player's beliefs, and the reverse at each showdown leaf
        Row3 eva, evo;
        showdown_rows(tv, rows + P2B_HPAD, leaf, pref, pc, tot, hi, eva, evo);
        const Divisor dscale = make_divisor(sg.scale);
#pragma unroll 1
        for (int c = it.first_sd; c < k; ++c) {
            if (it.kind[c] != kShowdownLeaf) continue;
            if (c != it.first_sd) {
                // a further showdown child (a call and an all-in of the same size; rare): its tables in place of the first
                // one's, from its beliefs, which wait in its value row
                const Row3 x = ld3(rec + (fc + c) * kRec + kRecValue * P2B_HPAD, tid);
                __syncthreads();
                st3(leaf, tid, x);
                __syncthreads();
                showdown_tables(tv, rows + P2B_HPAD, leaf, pref, pc, tot, scan);
                __syncthreads();
                showdown_rows(tv, rows + P2B_HPAD, leaf, pref, pc, tot, hi, eva, evo);
            }
            const NodeRec ch = load_node(p.nodes + sg.node_begin + fc + c);
            const float pot_a = a == 0 ? ch.v0 : ch.v1, pot_o = a == 0 ? ch.v1 : ch.v0;
            DivGuard g = guard_begin(dscale.ok);
            Row3 na, no, va, vo;
#pragma unroll
            for (int i = 0; i < kHandsPerThread; ++i) {
                na.v[i] = __fmul_rn(eva.v[i], pot_a);
                no.v[i] = __fmul_rn(evo.v[i], pot_o);
                va.v[i] = div_g<false>(na.v[i], dscale.y, dscale.r, g);
                vo.v[i] = div_g<false>(no.v[i], dscale.y, dscale.r, g);
            }
            if (__builtin_expect(guard_bad(g), 0)) {
#pragma unroll
                for (int i = 0; i < kHandsPerThread; ++i) {
                    va.v[i] = __fdiv_rn(na.v[i], sg.scale);
                    vo.v[i] = __fdiv_rn(no.v[i], sg.scale);
                }
            }
            float* v = rec + (fc + c) * kRec + kRecValue * P2B_HPAD;
            st3(v + a * P2B_HPAD, tid, va);
            st3(v + o * P2B_HPAD, tid, vo);
        }
    }
}

// ---- values and best responses after the final pass -----------------------------------------------
// The outputs of the final pass at a node and at the leaves below it, with the zero-sum shift where asked (:957-980: at every
// node that does not end the hand, the mean over the players of sum_h values * beliefs).
__global__ void __launch_bounds__(kRowThreads) split_values_kernel(const CfrParams p, const SplitWork w) {
    __shared__ __align__(16) float prod[2][P2B_HPAD];
    __shared__ float sums[2];
    if (block_refused(p)) return;
    const int tid = threadIdx.x;
    report_gave_up(p);
    for (int x = blockIdx.x; x < w.total[0]; x += gridDim.x) {
        const SplitItem& it = w.items[x];
        const int leaf0 = p.leaf_begin ? p.leaf_begin[it.subgame] : 0;
        auto shift_of = [&](const Row3& v0, const Row3& b0, const Row3& v1, const Row3& b1) {
            __syncthreads();
            st3(prod[0], tid, mul3(v0, b0));
            st3(prod[1], tid, mul3(v1, b1));
            __syncthreads();
            if (tid < 64) {
                const float sum = row_sum_reference_order(prod[tid >> 5]);
                if ((tid & 31) == 0) sums[tid >> 5] = sum;
            }
            __syncthreads();
            return __fmul_rn(__fadd_rn(sums[0], sums[1]), 0.5f);
        };
        auto minus = [&](Row3 v, float s) {
#pragma unroll
            for (int i = 0; i < kHandsPerThread; ++i) v.v[i] = __fsub_rn(v.v[i], s);
            return v;
        };
        if (!p.values_avg && it.node != 0) continue;
        {
            const float* me = w.rec + (long long)(it.node_begin + it.node) * kRec;
            Row3 v0 = ld3(me + kRecValue * P2B_HPAD, tid), v1 = ld3(me + (kRecValue + 1) * P2B_HPAD, tid);
            if (p.enforce_zero_sum) {
                const float s = shift_of(v0, ld3(me + kRecBelief * P2B_HPAD, tid), v1, ld3(me + (kRecBelief + 1) * P2B_HPAD, tid));
                v0 = minus(v0, s);
                v1 = minus(v1, s);
            }
            if (p.values_avg) {
                float* out = p.values_avg + 2ll * (it.node_begin + it.node) * P2B_HPAD;
                st3(out, tid, v0);
                st3(out + P2B_HPAD, tid, v1);
            }
            if (it.node == 0) {
                float* out = p.root_values + 2ll * it.subgame * P2B_HPAD;
                st3(out, tid, v0);
                st3(out + P2B_HPAD, tid, v1);
            }
        }
        if (!p.values_avg) continue;
        for (int c = 0; c < it.n_children; ++c) {
            const int kind = it.kind[c];
            if (kind == kInternal) continue;
            const long long row = it.node_begin + it.first_child + c;
            const NodeRec nd = load_node(p.nodes + row);
            Row3 v0, v1;
            if (kind == kShowdownLeaf) {
                v0 = ld3(w.rec + row * kRec + kRecValue * P2B_HPAD, tid);
                v1 = ld3(w.rec + row * kRec + (kRecValue + 1) * P2B_HPAD, tid);
            } else {
                const bool model = kind == kModelLeaf && p.leaf_values;
                const float f = kind == kFoldLeaf ? nd.v0 : 0.0f;
                const long long slot = 2ll * (leaf0 + nd.internal_idx) * P2B_HPAD;
#pragma unroll
                for (int i = 0; i < kHandsPerThread; ++i) {
                    v0.v[i] = f;
                    v1.v[i] = -f;
                }
                if (model) {
                    v0 = ld3(p.leaf_values + slot, tid);
                    v1 = ld3(p.leaf_values + slot + P2B_HPAD, tid);
                }
                if (p.enforce_zero_sum && kind == kModelLeaf && p.leaf_beliefs) {
                    const float s = shift_of(v0, ld3(p.leaf_beliefs + slot, tid), v1, ld3(p.leaf_beliefs + slot + P2B_HPAD, tid));
                    v0 = minus(v0, s);
                    v1 = minus(v1, s);
                }
            }
            float* out = p.values_avg + 2 * row * P2B_HPAD;
            st3(out, tid, v0);
            st3(out + P2B_HPAD, tid, v1);
        }
    }
}

// One level of the best-response sweeps (`_best_response_values`, :603-716) of both players: block (subgame, deviator, lane)
// takes every lanes-th node of level d.  Where the deviator acts, its best action per hand decides which beliefs the other
// player meets, whose per-card sums make the node's weights; elsewhere the weights are the final pass's own.  Values of
// sweep 0 lie in the value rows of the final pass, those of sweep 1 in its belief rows, both spent by then.
template <int MAXK>
__global__ void __launch_bounds__(kRowThreads, 2) split_best_response_kernel(const CfrParams p, const SplitWork w, int d, int lanes) {
    extern __shared__ __align__(16) unsigned char smem[];
    float* rows = reinterpret_cast<float*>(smem);  // beliefs of the acting player, then a row a child
    double* cs = reinterpret_cast<double*>(smem + (1 + MAXK) * P2B_HPAD * 4);
    double* S = cs + (1 + MAXK) * 52;
    if (block_refused(p)) return;
    const int tid = threadIdx.x;
    const int q = blockIdx.x / (2 * lanes), rest = blockIdx.x - q * 2 * lanes, deviator = rest / lanes;
    const SplitLevels* lv = w.levels + q;
    if (d >= lv->n_levels) return;
    uint32_t idx[7];
    card_indices(tid, idx);
    const int mine = deviator == 0 ? kRecValue : kRecBelief;
    for (int x = lv->begin[d] + rest - deviator * lanes; x < lv->begin[d + 1]; x += lanes) {
        const SplitItem& it = w.items[lv->item_begin + x];
        const int a = it.to_act, o = 1 - a, k = it.n_children;
        const bool deviates = deviator == a;
        float* me = w.rec + (long long)(it.node_begin + it.node) * kRec;
        const float* kids = w.rec + (long long)(it.node_begin + it.first_child) * kRec;
        auto value = [&](int c, int pl) {
            if (it.kind[c] == kInternal) return ld3(kids + c * kRec + (mine + pl) * P2B_HPAD, tid);
            Row3 v = ld3(p.values_avg + (2ll * (it.node_begin + it.first_child + c) + pl) * P2B_HPAD, tid);
#pragma unroll
            for (int i = 0; i < kHandsPerThread; ++i) v.v[i] = fminf(fmaxf(v.v[i], -1.0f), 1.0f);
            return v;
        };
        Row3 acc_a, acc_o, b_a;
        int best[kHandsPerThread];
#pragma unroll
        for (int i = 0; i < kHandsPerThread; ++i) {
            acc_a.v[i] = acc_o.v[i] = b_a.v[i] = 0.0f;
            best[i] = 0;
        }
        if (deviates) {
            // best action per hand: the first maximum (argmax, :653-660)
            acc_a = value(0, a);
#pragma unroll 1
            for (int c = 1; c < k; ++c) {
                const Row3 v = value(c, a);
#pragma unroll
                for (int i = 0; i < kHandsPerThread; ++i)
                    if (v.v[i] > acc_a.v[i]) {
                        acc_a.v[i] = v.v[i];
                        best[i] = c;
                    }
            }
            b_a = ld3(me + kRecActing * P2B_HPAD, tid);
            __syncthreads();  // the tables of the node before have been read
            st3(rows, tid, b_a);
#pragma unroll 1
            for (int c = 0; c < k; ++c) {
                Row3 m;
#pragma unroll
                for (int i = 0; i < kHandsPerThread; ++i) m.v[i] = best[i] == c ? b_a.v[i] : 0.0f;
                st3(rows + (1 + c) * P2B_HPAD, tid, m);
            }
            __syncthreads();
            card_sums(rows, 1 + k, cs, S, idx);
            __syncthreads();
        }
#pragma unroll 1
        for (int c = 0; c < k; ++c) {
            const Row3 Vo = value(c, o);
            Row3 weight;
            if (deviates) {
#pragma unroll
                for (int i = 0; i < kHandsPerThread; ++i) {
                    const int h = tid + i * kRowThreads, hc = h < P2B_NUM_HANDS ? h : P2B_NUM_HANDS - 1;
                    const int c1 = p.combos->c1[hc], c2 = p.combos->c2[hc];
                    const float blk = unblocked(cs + (1 + c) * 52, S[1 + c], c1, c2, best[i] == c ? b_a.v[i] : 0.0f);
                    const float den = unblocked(cs, S[0], c1, c2, b_a.v[i]);
                    weight.v[i] = den > 1e-5f ? __fdiv_rn(blk, den) : 0.0f;
                }
            } else {
                weight = ld3(kids + c * kRec + kRecSeen * P2B_HPAD, tid);
                const Row3 P = ld3(kids + c * kRec + kRecPolicy * P2B_HPAD, tid), Va = value(c, a);
#pragma unroll
                for (int i = 0; i < kHandsPerThread; ++i) acc_a.v[i] = __fadd_rn(acc_a.v[i], __fmul_rn(Va.v[i], P.v[i]));
            }
#pragma unroll
            for (int i = 0; i < kHandsPerThread; ++i) acc_o.v[i] = __fadd_rn(acc_o.v[i], __fmul_rn(weight.v[i], Vo.v[i]));
        }
        st3(me + (mine + a) * P2B_HPAD, tid, acc_a);
        st3(me + (mine + o) * P2B_HPAD, tid, acc_o);
    }
}

// Local exploitability (:718-764) from the root values of the two sweeps and of the plain expectation, which the up kernel has
// left in the rows of the hand-over area where the root's prior was.
__global__ void __launch_bounds__(kRowThreads) split_exploitability_kernel(const CfrParams p, const SplitWork w) {
    __shared__ __align__(16) float prod[4][P2B_HPAD];
    __shared__ float sums[4];
    if (block_refused(p)) return;
    report_gave_up(p);
    const int s = blockIdx.x, tid = threadIdx.x;
    const float* cr = p.carry_roots + (long long)s * 4 * P2B_HPAD;
    const float* root = w.rec + (long long)p.subgames[s].node_begin * kRec;
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        const Row3 rb = ld3(cr + (2 + d) * P2B_HPAD, tid), base = ld3(cr + d * P2B_HPAD, tid);
        const Row3 best = ld3(root + ((d == 0 ? kRecValue : kRecBelief) + d) * P2B_HPAD, tid);
        Row3 gain, value;
#pragma unroll
        for (int i = 0; i < kHandsPerThread; ++i) {
            gain.v[i] = __fmul_rn(__fsub_rn(best.v[i], base.v[i]), rb.v[i]);
            value.v[i] = __fmul_rn(best.v[i], rb.v[i]);
        }
        st3(prod[d], tid, gain);
        st3(prod[2 + d], tid, value);
    }
    __syncthreads();
    if (tid < 128) {
        const float sum = row_sum_reference_order(prod[tid >> 5]);
        if ((tid & 31) == 0) sums[tid >> 5] = sum;
    }
    __syncthreads();
    if (tid == 0) p.exploitability[s] = __fadd_rn(sums[0], sums[1]);
    if (tid < 2 && p.br_values) p.br_values[(long long)s * 2 + tid] = sums[2 + tid];
}

// `follows`: the launch before it on the stream was one of these kernels (see launch_next).
template <typename... Params, typename... Args>
int launch_pass_kernel(void (*kernel)(Params...), const char* name, unsigned grid, unsigned threads, int bytes, bool follows,
                       cudaStream_t stream, Args... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = (size_t)bytes;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = follows ? 1 : 0;
    return check_cuda(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...), name);
}

template <int MAXK, bool SD, int KIND>
int launch_rows(const CfrParams& p, const SplitWork& w, int pass, bool follows, cudaStream_t stream) {
    constexpr int kBytes = row_layout(MAXK, SD).bytes;
    static_assert(kBytes <= 227 * 1024, "one block must fit an SM");
    static SharedLimit had;
    int rc = allow_shared(had, reinterpret_cast<const void*>(split_rows_kernel<MAXK, SD, KIND>), kBytes);
    if (rc) return rc;
    const long long most = (long long)p.num_subgames * p.max_internal, fit = 2ll * sm_count();
    return launch_pass_kernel(split_rows_kernel<MAXK, SD, KIND>, "split_rows_kernel", (unsigned)(most < fit ? most : fit), kRowThreads,
                              kBytes, follows, stream, p, w, pass);
}

template <int MAXK, int KIND>
int launch_rows(const CfrParams& p, const SplitWork& w, int pass, bool follows, cudaStream_t stream) {
    return p.tables ? launch_rows<MAXK, true, KIND>(p, w, pass, follows, stream)
                    : launch_rows<MAXK, false, KIND>(p, w, pass, follows, stream);
}
template <int KIND>
int launch_rows(const CfrParams& p, const SplitWork& w, int pass, int max_children, bool follows, cudaStream_t stream) {
    return max_children <= kIterMaxChildren ? launch_rows<6, KIND>(p, w, pass, follows, stream)
                                            : launch_rows<8, KIND>(p, w, pass, follows, stream);
}

template <int MODE>
int launch_prep(const CfrParams& p, const SplitWork& w, int pass, int max_children, cudaStream_t stream) {
    const unsigned grid = (unsigned)p.num_subgames * (P2B_HPAD / 64);
    if (max_children <= kIterMaxChildren) split_prep_kernel<6, MODE><<<grid, 32 * kPrepWarps, 0, stream>>>(p, w, pass);
    else split_prep_kernel<8, MODE><<<grid, 32 * kPrepWarps, 0, stream>>>(p, w, pass);
    return check_cuda(cudaGetLastError(), "split_prep_kernel");
}

int launch_up(const CfrParams& p, const SplitWork& w, UpJob job, int pass, bool advance, bool mixed, int max_children, bool follows,
              cudaStream_t stream) {
    int ring = 40;  // two nodes of two or three actions, the usual ones, fit together
    if (ring < up_rows(max_children)) ring = up_rows(max_children);
    // Warps a slice: one warp's walk up a tree is the time of a small batch, so nodes of a level are spread over up to eight;
    // but no more warps than twice what the SMs hold at a time, beyond which they only queue.  Measured (us a pass; 8 / 4 /
    // 2 / 1 warps a slice): 1 subgame 17 / 21 / 29 / 49, 37 of 96 nodes 76 / 79 / 114 / 198, 192 of 77 nodes 318 / 257 /
    // 231 / 264, 4096 of 54 nodes - / - / 2550 / 2730.
    const long long held = (long long)sm_count() * (227 * 1024 / (ring * kUpRow * 4));
    int lanes = 8;
    while (lanes > 2 && (long long)p.num_subgames * (P2B_HPAD / kUpRow) * lanes > 2 * held) lanes /= 2;
    const int slices = lanes == 2 ? kUpSlices : 1;
    long long nodes = (long long)p.max_internal * max_children + 1;
    if (nodes > kCfrMaxNodes) nodes = kCfrMaxNodes;
    const int bytes = lanes * slices * ring * kUpRow * 4 + p.max_internal * (int)sizeof(SplitItem) + (int)nodes * (int)sizeof(NodeRecPacked);
    static SharedLimit had;
    int rc = allow_shared(had, reinterpret_cast<const void*>(split_up_kernel), bytes);
    if (rc) return rc;
    const unsigned grid = (unsigned)p.num_subgames * (P2B_HPAD / kUpRow / slices);
    return launch_pass_kernel(split_up_kernel, "split_up_kernel", grid, 32 * lanes * slices, bytes, follows, stream, p, w, job, pass,
                              advance, mixed, lanes, slices, ring);
}

}  // namespace

long long split_scratch_floats(int num_subgames, long long rows) {
    return 4 + rows * kItemFloats + round4(num_subgames * kLevelFloats) + rows * kRec;
}

bool split_applies(const CfrParams& p, int max_children, long long scratch_floats) {
    return p.rows > 0 && p.init_depth <= kSplitMaxDepth && max_children <= kCfrMaxChildren && p.max_internal <= 255 &&
           scratch_floats >= split_scratch_floats(p.num_subgames, p.rows);
}

// The work lists.  Adding up in every block what lies before it is quadratic in the batch, a launch of its own costs a few us and
// more where a thread's run of subgames gets long: measured, us with the launch / without, 2048 subgames 16 / 14, 4096 28 / 26,
// 8192 50 / 63, 16,384 97 / 182.
constexpr int kBeginFrom = 6144;  // subgames
static int launch_lists(const CfrParams& p, const SplitWork& w, cudaStream_t stream) {
    const bool begun = p.num_subgames >= kBeginFrom;
    if (begun) split_begin_kernel<<<1, kBeginThreads, 0, stream>>>(p, w);
    split_items_kernel<<<p.num_subgames, kCfrMaxNodes, 0, stream>>>(p, w, begun);
    return check_cuda(cudaGetLastError(), "split_items_kernel");
}

int launch_split_passes(const CfrParams& p, int max_children, int pass_begin, int pass_end, bool down, bool up, bool continued,
                        cudaStream_t stream) {
    const SplitWork w = carve(p.scratch, p.num_subgames, p.rows);
    const bool avg = p.cfr_avg != 0 || p.iter_values != 0;
    int rc = P2B_OK;
    bool follows = false;
    if (down && !continued) {
        rc = launch_lists(p, w, stream);
        if (!rc) rc = launch_prep<kPrepPolicy>(p, w, pass_begin, max_children, stream);
    }
    for (int pass = pass_begin; pass <= pass_end && !rc; ++pass) {
        if (pass > pass_begin || down) {
            if (avg) {
                rc = launch_prep<kPrepMix>(p, w, pass, max_children, stream);
                follows = false;
            }
            if (!rc)
                rc = avg ? launch_rows<kRowAvg>(p, w, pass, max_children, follows, stream)
                         : launch_rows<kRowIter>(p, w, pass, max_children, follows, stream);
            follows = true;
        }
        if (!rc && (pass < pass_end || up)) {
            rc = launch_up(p, w, kUpIter, pass, pass < pass_end, avg, max_children, follows, stream);
            follows = true;
        }
    }
    return rc;
}

int launch_split_start(const CfrParams& p, int max_children, bool down, bool up, bool advance, cudaStream_t stream) {
    const SplitWork w = carve(p.scratch, p.num_subgames, p.rows);
    int rc = P2B_OK;
    if (down) {
        rc = launch_lists(p, w, stream);
        if (!rc) rc = launch_rows<kRowStart>(p, w, 0, max_children, false, stream);
    }
    if (!rc && up) rc = launch_up(p, w, kUpStart, -1, advance, true, max_children, down, stream);
    return rc;
}

int launch_split_final(const CfrParams& p, int max_children, bool down, bool up, bool best_responses, cudaStream_t stream) {
    const SplitWork w = carve(p.scratch, p.num_subgames, p.rows);
    const int B = p.num_subgames, sms = sm_count();
    int rc = P2B_OK;
    if (down) rc = launch_rows<kRowFinal>(p, w, p.iterations, max_children, false, stream);
    if (!rc && up) {
        rc = launch_up(p, w, kUpFinal, p.iterations, false, true, max_children, down, stream);
        if (rc) return rc;
        const long long most = (long long)B * p.max_internal, fit = 4ll * sms;
        split_values_kernel<<<(unsigned)(most < fit ? most : fit), kRowThreads, 0, stream>>>(p, w);
        rc = check_cuda(cudaGetLastError(), "split_values_kernel");
    }
    if (rc || !best_responses || !p.exploitability || !p.values_avg) return rc;
    rc = launch_up(p, w, kUpBase, p.iterations, false, true, max_children, false, stream);
    if (rc) return rc;
    // as many blocks a subgame and sweep as it takes to fill the chip, up to a level's worth of nodes
    int lanes = sms / B;
    lanes = lanes < 1 ? 1 : lanes > 16 ? 16 : lanes;
    const bool wide = max_children > kIterMaxChildren;
    const auto kernel = wide ? split_best_response_kernel<kCfrMaxChildren> : split_best_response_kernel<kIterMaxChildren>;
    const int bytes = (1 + (wide ? kCfrMaxChildren : kIterMaxChildren)) * (P2B_HPAD * 4 + 52 * 8 + 8);
    static SharedLimit had[2];
    rc = allow_shared(had[wide], reinterpret_cast<const void*>(kernel), bytes);
    for (int d = p.init_depth; d >= 0 && !rc; --d) {
        kernel<<<(unsigned)(B * 2 * lanes), kRowThreads, bytes, stream>>>(p, w, d, lanes);
        rc = check_cuda(cudaGetLastError(), "split_best_response_kernel");
    }
    if (rc) return rc;
    split_exploitability_kernel<<<(unsigned)B, kRowThreads, 0, stream>>>(p, w);
    return check_cuda(cudaGetLastError(), "split_exploitability_kernel");
}

}  // namespace p2b
