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
// So a pass is split_rows_kernel, one block per internal node of the whole batch, followed by
// split_columns_kernel, where a block owns a slice of hands of one subgame and goes up the tree level by level,
// one warp a node.  A solve whose leaves are valued by the caller's model has the model between the two.
// The reach rows of the other kernels do not exist here: both kernels multiply along the path (3 to 5 rows that
// are in L2), and the old average policy of the ancestors, which the average-policy mix weights by, is still in
// place when a node is visited bottom-up.
//
// Arithmetic and results are those of cfr.cu, bit for bit: same operations in the same order, also in the fp64 sums.
//
// Measured on a B200, a pass in the general kernel / here: one subgame of 57 nodes 0.32 / 0.036 ms, 37 of 96 nodes
// 1.15 / 0.21 ms, 192 flop subgames of 77 nodes (largest 271) 1.4 / 0.48 ms.  The row kernel takes 6.3 us an SM and
// node with two blocks resident; shared-memory wavefronts bound it (0.68 of their peak over the whole kernel, gathers of
// the per-card sums and of the showdown tables), with half of the issue slots used.  The column kernel is bound by the
// latency of its row accesses at small batches and runs at 0.6 of the memory bandwidth at large ones.
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
    kRecRows = 5
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

// ---- work lists -------------------------------------------------------------------------------
// One block per subgame, one thread per node.  The items of a batch follow the queue order, those of a subgame the
// node order, which is breadth-first.
__global__ void __launch_bounds__(kCfrMaxNodes) split_items_kernel(const CfrParams p, const SplitWork w) {
    __shared__ int s_before, s_depth[kSplitMaxDepth + 1], s_bad;
    const int q = blockIdx.x, i = threadIdx.x;
    if (i == 0) s_before = s_bad = 0;
    if (i <= kSplitMaxDepth) s_depth[i] = 0;
    __syncthreads();
    if (p.work_counter[1] != 0) {  // the record check refused the batch
        if (q == 0 && i == 0) w.total[0] = 0;
        return;
    }
    const int s = p.queue_order ? p.queue_order[q] : q;
    int before = 0;
    for (int r = i; r < q; r += kCfrMaxNodes) before += p.subgames[p.queue_order ? p.queue_order[r] : r].n_internal;
    for (int d = 16; d > 0; d >>= 1) before += __shfl_xor_sync(0xffffffffu, before, d);
    if ((i & 31) == 0) atomicAdd(&s_before, before);
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

enum ColumnMode {
    kColInit = 0,  // current policy from the regrets, the root's rows moved on to the coming pass
    kColMix = 1,   // average-policy mix alone: solves whose beliefs are taken under the updated average policy
    kColUp = 2     // values, average-policy mix (unless kColMix has done it), regrets, the next policy
};

// One node for the hands of a warp: VPT consecutive ones a thread.  The stages are ordered so that about three rows a
// child are live at a time: values and backup, average-policy mix, regrets, next policy.
template <int VPT, int K, int MODE>
__device__ __forceinline__ void column_node(const CfrParams& p, const SplitWork& w, const SplitItem& it,
                                            const NodeRecPacked* nodes, const FV<VPT>& mask, int h, int pass, int leaf0,
                                            bool sample, bool mixed) {
    const int a = it.to_act, j = it.node, fc = it.first_child;
    const long long kids = (long long)(it.node_begin + fc) * P2B_HPAD + h;
    float* rec = w.rec + (long long)(it.node_begin + fc) * kRec + h;  // of the first child
    float* R_row = p.regrets + kids;
    FV<VPT> P[K];
    if (MODE == kColInit) {
#pragma unroll
        for (int c = 0; c < K; ++c) P[c] = ldc<VPT>(R_row + c * P2B_HPAD);
        regret_matching<VPT, K>(P);
#pragma unroll
        for (int c = 0; c < K; ++c) stc<VPT>(rec + c * kRec, P[c]);
        return;
    }
    const bool update = MODE == kColUp && pass + 1 < p.iterations;
    const IterScalars sc = p.scalars[pass];
    const bool mix_here = MODE == kColMix || !mixed, mix = mix_here && (sc.do_mix & 1) != 0;
    float* A_row = p.policy_avg + kids;
#pragma unroll
    for (int c = 0; c < K; ++c) P[c] = ldc<VPT>(rec + c * kRec);
    FV<VPT> A[K], ra, rba;
    if (mix) {
#pragma unroll
        for (int c = 0; c < K; ++c) A[c] = ldc<VPT>(A_row + c * P2B_HPAD);
        ra = path_product<VPT>(w.rec + (long long)it.node_begin * kRec + h, kRec, it.path, it.n_path[0], mask);
        rba = path_product<VPT>(p.policy_avg + (long long)it.node_begin * P2B_HPAD + h, P2B_HPAD, it.path, it.n_path[0], mask);
    }
    FV<VPT> Va[K], acc_a, wgt;
    const bool tracked = update && p.weight_sums != nullptr;
    float* W_row = p.weight_sums + kids;
    if (MODE == kColUp) {
        // value backup (:1095-1115)
        FV<VPT> acc_o;
#pragma unroll
        for (int i = 0; i < VPT; ++i) acc_a.v[i] = acc_o.v[i] = 0.0f;
        const int va_off = (kRecValue + a) * P2B_HPAD, vo_off = (kRecValue + 1 - a) * P2B_HPAD;
        float* me = w.rec + (long long)(it.node_begin + j) * kRec + h;
        if (update) wgt = ldc<VPT>(me + kRecWeight * P2B_HPAD);
        FV<VPT> Q[K], Vo[K];
#pragma unroll
        for (int c = 0; c < K; ++c) {
            Q[c] = ldc<VPT>(rec + c * kRec + kRecSeen * P2B_HPAD);
            const int kind = it.kind[c];
            const float *va = rec + c * kRec + va_off, *vo = rec + c * kRec + vo_off;
            if (kind == kModelLeaf && p.leaf_values) {
                const float* v = p.leaf_values + (long long)(leaf0 + nodes[fc + c].internal_idx) * 2 * P2B_HPAD + h;
                va = v + a * P2B_HPAD;
                vo = v + (1 - a) * P2B_HPAD;
            }
            if (kind == kFoldLeaf || (kind == kModelLeaf && !p.leaf_values)) {
                const float v0 = kind == kFoldLeaf ? nodes[fc + c].v0 : 0.0f, f = a == 0 ? v0 : -v0;
#pragma unroll
                for (int i = 0; i < VPT; ++i) {
                    Va[c].v[i] = f;
                    Vo[c].v[i] = -f;
                }
            } else {
                Va[c] = ldc<VPT>(va);
                Vo[c] = ldc<VPT>(vo);
            }
        }
#pragma unroll
        for (int c = 0; c < K; ++c)
#pragma unroll
            for (int i = 0; i < VPT; ++i) {
                acc_a.v[i] = __fadd_rn(acc_a.v[i], __fmul_rn(Va[c].v[i], P[c].v[i]));
                acc_o.v[i] = __fadd_rn(acc_o.v[i], __fmul_rn(Vo[c].v[i], Q[c].v[i]));
            }
        if (j != 0) {
            stc<VPT>(me + va_off, acc_a);
            stc<VPT>(me + vo_off, acc_o);
        }
        if (p.iter_values && p.values_avg) {  // the values of this iteration at the node and at the leaves below it
            float* out = p.values_avg + (long long)it.node_begin * 2 * P2B_HPAD + h;
            stc<VPT>(out + (2 * j + a) * P2B_HPAD, acc_a);
            stc<VPT>(out + (2 * j + 1 - a) * P2B_HPAD, acc_o);
#pragma unroll
            for (int c = 0; c < K; ++c)
                if (it.kind[c] != kInternal) {
                    stc<VPT>(out + (2 * (fc + c) + a) * P2B_HPAD, Va[c]);
                    stc<VPT>(out + (2 * (fc + c) + 1 - a) * P2B_HPAD, Vo[c]);
                }
        }
        if (p.policy && pass == p.iterations - 1) {
#pragma unroll
            for (int c = 0; c < K; ++c) stc<VPT>(p.policy + kids + c * P2B_HPAD, P[c]);
        }
        if (sample) {
#pragma unroll
            for (int c = 0; c < K; ++c) stc<VPT>(p.policy_sample + kids + c * P2B_HPAD, P[c]);
        }
    }
    if (mix_here) {
        if (mix) {
            mix_average<VPT, K>(sc, ra, rba, P, A);
#pragma unroll
            for (int c = 0; c < K; ++c) stc<VPT>(A_row + c * P2B_HPAD, A[c]);
        } else {
#pragma unroll
            for (int c = 0; c < K; ++c) stc<VPT>(A_row + c * P2B_HPAD, P[c]);
        }
    }
    if (update) {
        // instantaneous regrets of this pass folded into the discounted update of the next (:1117-1165, :1346-1368)
        const IterScalars sn = p.scalars[pass + 1];
        const Divisor d_pos = make_divisor(sn.den_pos), d_neg = make_divisor(sn.den_neg);
        const bool no_regret = ((sn.do_mix >> 1) & 3) == a + 1;  // linear CFR: this player's actions get none
        FV<VPT> R[K], W[K];
#pragma unroll
        for (int c = 0; c < K; ++c) R[c] = ldc<VPT>(R_row + c * P2B_HPAD);
        if (tracked) {
#pragma unroll
            for (int c = 0; c < K; ++c) W[c] = ldc<VPT>(W_row + c * P2B_HPAD);
        }
#pragma unroll
        for (int c = 0; c < K; ++c) {
            DivGuard g = guard_begin(d_pos.ok && d_neg.ok);
            FV<VPT> rn, rq, wn, wq, dy;
#pragma unroll
            for (int i = 0; i < VPT; ++i) {
                const bool pos = R[c].v[i] > 0.0f;
                const float num = pos ? sn.num_pos : sn.num_neg, dr = pos ? d_pos.r : d_neg.r;
                dy.v[i] = pos ? d_pos.y : d_neg.y;
                rn.v[i] = __fmul_rn(R[c].v[i], num);
                rq.v[i] = div_g<false>(rn.v[i], dy.v[i], dr, g);
                if (tracked) {
                    wn.v[i] = __fmul_rn(W[c].v[i], num);
                    wq.v[i] = div_g<true>(wn.v[i], dy.v[i], dr, g);
                }
            }
            if (__builtin_expect(guard_bad(g), 0)) {
#pragma unroll
                for (int i = 0; i < VPT; ++i) {
                    rq.v[i] = __fdiv_rn(rn.v[i], dy.v[i]);
                    if (tracked) wq.v[i] = __fdiv_rn(wn.v[i], dy.v[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < VPT; ++i) {
                const float reg = no_regret ? 0.0f : __fmul_rn(wgt.v[i], __fsub_rn(Va[c].v[i], acc_a.v[i]));
                float rr = __fadd_rn(rq.v[i], reg);
                if (p.cfr_plus) rr = fmaxf(rr, 0.0f);
                R[c].v[i] = rr;
                if (tracked) W[c].v[i] = __fadd_rn(wq.v[i], 1.0f);
            }
            stc<VPT>(R_row + c * P2B_HPAD, R[c]);
            if (tracked) stc<VPT>(W_row + c * P2B_HPAD, W[c]);
        }
        regret_matching<VPT, K>(R);
#pragma unroll
        for (int c = 0; c < K; ++c) stc<VPT>(rec + c * kRec, R[c]);
    }
}

// A block holds `slices` slices of 32 VPT hands of one subgame with `lanes` warps each, which take the nodes of a level
// in turn; a level is complete when they meet at the slice's barrier.
template <int VPT, int MAXK, int MODE>
__global__ void __launch_bounds__(256, 3) split_columns_kernel(const CfrParams p, const SplitWork w, int pass, bool advance,
                                                               bool mixed, int lanes, int slices) {
    constexpr int kSlices = P2B_HPAD / (32 * VPT);
    extern __shared__ __align__(16) unsigned char smem[];
    if (p.work_counter[1] != 0) return;
    const int per_subgame = kSlices / slices;
    const int q = blockIdx.x / per_subgame;
    const int s = p.queue_order ? p.queue_order[q] : q;
    const int tid = threadIdx.x, warp = tid >> 5, mine = warp / lanes, lane_warp = warp - mine * lanes;
    const int h = ((blockIdx.x - q * per_subgame) * slices + mine) * 32 * VPT + (tid & 31) * VPT;
    const SubgameRec sg = p.subgames[s];
    SplitItem* items = reinterpret_cast<SplitItem*>(smem);
    NodeRecPacked* nodes = reinterpret_cast<NodeRecPacked*>(smem + sg.n_internal * sizeof(SplitItem));
    const SplitLevels* lv = w.levels + q;
    {
        const uint4* ns = reinterpret_cast<const uint4*>(p.nodes + sg.node_begin);
        for (int i = tid; i < sg.n_nodes; i += blockDim.x) reinterpret_cast<uint4*>(nodes)[i] = ns[i];
        const uint4* is = reinterpret_cast<const uint4*>(w.items + lv->item_begin);
        for (int i = tid; i < sg.n_internal * 4; i += blockDim.x) reinterpret_cast<uint4*>(items)[i] = is[i];
    }
    FV<VPT> mask;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        const bool real = h + i < P2B_NUM_HANDS;
        const int hc = real ? h + i : P2B_NUM_HANDS - 1;
        const bool blocked = (((sg.board_mask >> p.combos->c1[hc]) | (sg.board_mask >> p.combos->c2[hc])) & 1ull) != 0;
        mask.v[i] = real && !blocked ? 1.0f : 0.0f;
    }
    const int leaf0 = p.leaf_begin ? p.leaf_begin[s] : 0;
    const bool sample = p.policy_sample && p.sample_pass[s] == pass;
    __syncthreads();
    // one warp a slice: straight up the tree, no barrier
    const bool alone = lanes == 1;
    for (int d = alone ? 0 : lv->n_levels - 1; d >= 0; --d) {
        const int begin = alone ? 0 : lv->begin[d], end = alone ? sg.n_internal : lv->begin[d + 1];
        for (int x = end - 1 - lane_warp; x >= begin; x -= lanes) {
            const SplitItem& it = items[x];
            with_children<MAXK>(it.n_children, [&](auto kc) {
                column_node<VPT, decltype(kc)::value, MODE>(p, w, it, nodes, mask, h, pass, leaf0, sample, mixed);
            });
        }
        if (!alone) asm volatile("bar.sync %0, %1;" ::"r"(mine + 1), "r"(32 * lanes) : "memory");
    }
    // the root's row of the pass becomes what the node beliefs of the next pass derive from
    if (advance && lane_warp == 0) {
        float* cr = p.carry_roots + (long long)s * 4 * P2B_HPAD + h;
        stc<VPT>(cr, ldc<VPT>(cr + 2 * P2B_HPAD));
        stc<VPT>(cr + P2B_HPAD, ldc<VPT>(cr + 3 * P2B_HPAD));
    }
}

// ---- rows ---------------------------------------------------------------------------------------
// Beliefs of a node (cfr_evaluator.py:363-380), the other player's view of every action (:1076-1093), the regret
// weights (:1117-1165), showdown values (:484-601) and the beliefs handed to the caller's model.
//
// 448 threads with three hands each, a third of a row apart: consecutive threads touch consecutive hands in global
// and shared memory, and two blocks fit an SM (72 registers a thread).
constexpr int kRowThreads = 448, kHandsPerThread = 3;
static_assert(kRowThreads * kHandsPerThread == P2B_HPAD, "rows are covered exactly");
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

// Per-card sums and totals of the rows 0 .. n_cs-1 (cs, S).  Thread t < 416 adds quarter (t / 4 mod 52, t mod 4) of
// the 51 hands that hold a card, for the even or (t >= 208) the odd rows: the indices of its 13 hands belong to the
// thread for the whole kernel and are held in registers as byte offsets, two to a word.
__device__ __forceinline__ void card_sums(const float* rows, int n_cs, double* cs, double* S, const uint32_t (&idx)[7]) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int half = tid >= 208 ? 1 : 0, u = tid - 208 * half, c = u >> 2, q = u & 3;
    if (tid < 416) {
        for (int r0 = 0; r0 < n_cs; r0 += 2) {
            const int r = r0 + half;
            const bool live = r < n_cs;
            const char* __restrict__ x = reinterpret_cast<const char*>(rows + (live ? r : 0) * P2B_HPAD);
            float v[13];
#pragma unroll
            for (int i = 0; i < 12; ++i)
                v[i] = *reinterpret_cast<const float*>(x + (i & 1 ? idx[i >> 1] >> 16 : idx[i >> 1] & 0xffffu));
            v[12] = q < 3 ? *reinterpret_cast<const float*>(x + idx[6]) : 0.0f;
            double t_even = 0.0, t_odd = 0.0;
#pragma unroll
            for (int i = 0; i < 13; ++i) {
                if (i & 1) t_odd += (double)v[i];
                else t_even += (double)v[i];
            }
            const double mine = t_even + t_odd;
            const int g = lane & ~3;
            const double t0 = __shfl_sync(0xffffffffu, mine, g), t1 = __shfl_sync(0xffffffffu, mine, g + 1);
            const double t2 = __shfl_sync(0xffffffffu, mine, g + 2), t3 = __shfl_sync(0xffffffffu, mine, g + 3);
            if (live && q == 0) cs[r * 52 + c] = ((t0 + t1) + t2) + t3;
        }
    }
    // total mass of a row, a warp each (the 18 padding entries are zero)
    for (int r = kRowThreads / 32 - 1 - warp; r < n_cs; r += kRowThreads / 32) {
        const float* __restrict__ x = rows + r * P2B_HPAD;
        double acc[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int b = 0; b < 7; ++b) {
            float v[6];
#pragma unroll
            for (int i = 0; i < 6; ++i) v[i] = x[lane + 32 * (6 * b + i)];
#pragma unroll
            for (int i = 0; i < 6; ++i) acc[i] += (double)v[i];
        }
        const double tot = warp_sum(((acc[0] + acc[1]) + (acc[2] + acc[3])) + (acc[4] + acc[5]));
        if (lane == 0) S[r] = tot;
    }
}

// Tables of the showdown formula for the row x of slot 0 (the other player's beliefs) and of slot 1 (the leaf row);
// `slots` = 3 builds both, 2 only slot 1's.
__device__ __forceinline__ void showdown_tables(const BoardTabView& tv, const float* x0, const float* x1, int slots,
                                                float* pref_out, float* pc_out, float* tot_out, double* scan) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint16_t* __restrict__ sorted = tv.sorted;
    if (warp < 8 && ((slots >> (warp & 1)) & 1)) {
        // quarter scan: prefix of 352 sorted positions; the offset is the sum of the earlier quarters, which the four
        // warps of a slot hand one another
        const int slot = warp & 1, qi = 3 - (warp >> 1);
        const float* __restrict__ x = slot ? x1 : x0;
        float* __restrict__ pref = pref_out + slot * P2B_HPAD;
        const int k0 = qi * kScanQuarter + 11 * lane;
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
            if (k0 + i < P2B_NUM_HANDS) pref[k0 + i + 1] = (float)run;
        }
    }
    // per-card prefix sums: a quarter list a thread, slot 1 from the last 208 threads of the block down
    const int back = kRowThreads - 1 - tid;
    if (back < 416) {
        const int slot = back < 208 ? 1 : 0, u = 207 - (back - (slot ? 0 : 208)), c = u >> 2, q = u & 3;
        const bool live = ((slots >> slot) & 1) != 0;
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
        if (live) {
            double acc = q == 0 ? 0.0 : (q == 1 ? t0 : (q == 2 ? t0 + t1 : (t0 + t1) + t2));
            float* __restrict__ row = pc_out + slot * 52 * 52 + c * 52;
            if (q == 0) row[0] = 0.0f;
            float* __restrict__ out = row + 13 * q + 1;
#pragma unroll
            for (int i = 0; i < 12; ++i) {
                acc += (double)v[i];
                out[i] = (float)acc;
            }
            if (q < 3) out[12] = (float)(acc + (double)v[12]);
            else tot_out[slot * 64 + c] = (float)acc;  // == row[51]
        }
    }
}

// Showdown EV (before the pot scaling) of this thread's hands: ev0 (if BOTH) against the range x0 with the tables of
// slot 0, ev1 against x1 with those of slot 1.  The formula of showdown_hand_ev; a hand's positions in the tables are
// unpacked once for both.
template <bool BOTH>
__device__ __forceinline__ void showdown_rows(const BoardTabView& tv, const float* x0, const float* x1, const float* pref,
                                              const float* pc, const float* tot, const Hands& hi, Row3& ev0, Row3& ev1) {
    const int tid = threadIdx.x;
    DivGuard g = guard_begin(true);
#pragma unroll
    for (int i = 0; i < kHandsPerThread; ++i) {
        const int h = tid + i * kRowThreads, hc = hi.real[i] ? h : 0;
        const uint2 rec = *reinterpret_cast<const uint2*>(tv.rec + hc);
        const int l = rec.x & 0xffffu, r = rec.x >> 16;
        const int a0 = hi.c1[i] * 52 + (rec.y & 0xff), a1 = hi.c1[i] * 52 + ((rec.y >> 8) & 0xff);
        const int b0 = hi.c2[i] * 52 + ((rec.y >> 16) & 0xff), b1 = hi.c2[i] * 52 + (rec.y >> 24);
#pragma unroll
        for (int slot = BOTH ? 0 : 1; slot < 2; ++slot) {
            const float* P = pref + slot * P2B_HPAD;
            const float* C = pc + slot * 52 * 52;
            const float* T = tot + slot * 64;
            const float xh = (slot ? x1 : x0)[h];
            const float PL = P[l], C1 = C[a0], C2 = C[b0];
            const float win = __fsub_rn(__fsub_rn(PL, C1), C2);
            const float tie = __fadd_rn(__fsub_rn(__fsub_rn(__fsub_rn(P[r], PL), __fsub_rn(C[a1], C1)), __fsub_rn(C[b1], C2)), xh);
            const float den = fmaxf(__fadd_rn(__fsub_rn(__fsub_rn(1.0f, T[hi.c1[i]]), T[hi.c2[i]]), xh), 1e-8f);
            const Divisor d = make_divisor(den);
            g.dok = g.dok && d.ok;
            const float wp = div_g<false>(win, d.y, d.r, g), tp = div_g<false>(tie, d.y, d.r, g);
            const float ev = __fsub_rn(wp, __fsub_rn(__fsub_rn(1.0f, wp), tp));
            (slot ? ev1 : ev0).v[i] = (hi.allowed[i] && den > 1e-8f) ? ev : 0.0f;
        }
    }
    if (__builtin_expect(guard_bad(g), 0)) {
#pragma unroll 1
        for (int slot = BOTH ? 0 : 1; slot < 2; ++slot)
#pragma unroll
            for (int i = 0; i < kHandsPerThread; ++i) {
                const int h = tid + i * kRowThreads;
                if (!hi.real[i]) continue;
                const float ev = showdown_hand_ev(tv.rec[h], hi.c1[i], hi.c2[i], (slot ? x1 : x0)[h], hi.allowed[i],
                                                  pref + slot * P2B_HPAD, pc + slot * 52 * 52, tot[slot * 64 + hi.c1[i]],
                                                  tot[slot * 64 + hi.c2[i]]);
                if (slot) ev1.v[i] = ev;
                else ev0.v[i] = ev;
            }
    }
}

template <int MAXK, bool SD, bool AVG>
__global__ void __launch_bounds__(kRowThreads, 2) split_rows_kernel(const CfrParams p, const SplitWork w, int pass) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr RowLayout L = row_layout(MAXK, SD);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* rows = reinterpret_cast<float*>(smem + L.rows);
    float* leaf = rows + L.leaf_row * P2B_HPAD;
    float* pref = reinterpret_cast<float*>(smem + L.pref);
    float* pc = reinterpret_cast<float*>(smem + L.pc);
    float* tot = reinterpret_cast<float*>(smem + L.tot);
    double* scan = reinterpret_cast<double*>(smem + L.scan);
    double* cs = reinterpret_cast<double*>(smem + L.cs);
    double* S = reinterpret_cast<double*>(smem + L.S);
    float* sums = reinterpret_cast<float*>(smem + L.sums);
    float* sums_avg = sums + 16;
    const SplitItem& it = *reinterpret_cast<const SplitItem*>(smem + L.item);
    if (p.work_counter[1] != 0) return;

    Hands hi;
#pragma unroll
    for (int i = 0; i < kHandsPerThread; ++i) {
        const int h = tid + i * kRowThreads;
        hi.real[i] = h < P2B_NUM_HANDS;
        const int hc = hi.real[i] ? h : P2B_NUM_HANDS - 1;
        hi.c1[i] = p.combos->c1[hc];
        hi.c2[i] = p.combos->c2[hc];
    }
    uint32_t idx[7];  // see card_sums
    {
        const int u = tid >= 208 ? tid - 208 : tid, c = (u >> 2) % 52, q = u & 3;
#pragma unroll
        for (int i = 0; i < 7; ++i) {
            uint32_t word = 0;
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const int e = q + 4 * (2 * i + b);
                if (2 * i + b < 13 && e < 51)
                    word |= (uint32_t)(4 * (e < c ? combo_index(e, c) : combo_row_offset(c) - c + e)) << (16 * b);
            }
            idx[i] = word;
        }
    }
    // a block takes consecutive items: mostly nodes of one subgame, whose board tables stay in shared memory
    const int total = w.total[0], each = (total + gridDim.x - 1) / gridDim.x;
    const int first = blockIdx.x * each, last = min(first + each, total);
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
            Row3 P[K];
#pragma unroll
            for (int c = 0; c < K; ++c) P[c] = ld3(rec + (fc + c) * kRec, tid);
            const Row3 prior_a = ld3(cr + a * P2B_HPAD, tid), prior_o = ld3(cr + o * P2B_HPAD, tid);
            const Row3 r_a = path3(rec, kRec, it.path, it.n_path[0], mask, tid);
            const Row3 r_o = path3(rec, kRec, it.path + it.n_path[0], it.n_path[1], mask, tid);
            const Row3 u_a = mul3(prior_a, r_a), u_o = mul3(prior_o, r_o);
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
            if (j == 0) {  // the root's own row, and its sums, for the pass after this one
                st3(cr + (2 + a) * P2B_HPAD, tid, b_a);
                st3(cr + (2 + o) * P2B_HPAD, tid, b_o);
                if (tid == 0) {
                    p.carry_sums[2ll * sg.node_begin + a] = sums[0];
                    p.carry_sums[2ll * sg.node_begin + o] = sums[1];
                }
            }
            if (p.beliefs_last && pass == p.iterations - 1) {
                float* out = p.beliefs_last + 2 * nb;
                st3(out + (2 * j + a) * P2B_HPAD, tid, b_a);
                st3(out + (2 * j + o) * P2B_HPAD, tid, b_o);
            }
#pragma unroll
            for (int c = 0; c < K; ++c) {
                float* row = rows + (2 + c) * P2B_HPAD;
                if (SD && c == it.first_sd) {
                    st3(leaf, tid, normalised(ld3(row, tid), avg_sums[2 + c], sg.allowed_prob, hi));
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
        if (showdown) showdown_tables(tv, rows + P2B_HPAD, leaf, 3, pref, pc, tot, scan);
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
            st3(rec + j * kRec + kRecWeight * P2B_HPAD, tid, wgt);
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
        showdown_rows<true>(tv, rows + P2B_HPAD, leaf, pref, pc, tot, hi, eva, evo);
        const Divisor dscale = make_divisor(sg.scale);
#pragma unroll 1
        for (int c = it.first_sd; c < k; ++c) {
            if (it.kind[c] != kShowdownLeaf) continue;
            if (c != it.first_sd) {
                // a further showdown child (a call and an all-in of the same size; rare): its tables in place of the first one's
                const Row3 r = path3(avgb ? p.policy_avg + nb : rec, avgb ? P2B_HPAD : kRec, it.path, it.n_path[0], mask, tid);
                const Row3 P = avgb ? ld3(p.policy_avg + nb + (fc + c) * P2B_HPAD, tid) : ld3(rec + (fc + c) * kRec, tid);
                const Row3 u = mul3(ld3(cr + a * P2B_HPAD, tid), mul3(r, P));
                __syncthreads();
                st3(leaf, tid, normalised(u, avg_sums[2 + c], sg.allowed_prob, hi));
                __syncthreads();
                showdown_tables(tv, rows + P2B_HPAD, leaf, 2, pref, pc, tot, scan);
                __syncthreads();
                showdown_rows<false>(tv, rows + P2B_HPAD, leaf, pref, pc, tot, hi, eva, evo);
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

template <int MAXK, bool SD, bool AVG>
int launch_rows(const CfrParams& p, const SplitWork& w, int pass, cudaStream_t stream) {
    constexpr int kBytes = row_layout(MAXK, SD).bytes;
    static_assert(kBytes <= 227 * 1024, "one block must fit an SM");
    int rc = check_cuda(cudaFuncSetAttribute(split_rows_kernel<MAXK, SD, AVG>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes),
                        "split_rows_kernel shared-memory attribute");
    if (rc) return rc;
    const long long most = (long long)p.num_subgames * p.max_internal, fit = 2ll * sm_count();
    split_rows_kernel<MAXK, SD, AVG><<<(unsigned)(most < fit ? most : fit), kRowThreads, kBytes, stream>>>(p, w, pass);
    return check_cuda(cudaGetLastError(), "split_rows_kernel");
}

template <int MAXK>
int launch_rows(const CfrParams& p, const SplitWork& w, int pass, bool avg, cudaStream_t stream) {
    if (p.tables)
        return avg ? launch_rows<MAXK, true, true>(p, w, pass, stream) : launch_rows<MAXK, true, false>(p, w, pass, stream);
    return avg ? launch_rows<MAXK, false, true>(p, w, pass, stream) : launch_rows<MAXK, false, false>(p, w, pass, stream);
}

template <int VPT, int MAXK>
int launch_columns(const CfrParams& p, const SplitWork& w, ColumnMode mode, int pass, bool advance, bool mixed, int max_children,
                   cudaStream_t stream) {
    long long nodes = (long long)p.max_internal * max_children + 1;
    if (nodes > kCfrMaxNodes) nodes = kCfrMaxNodes;
    const int bytes = p.max_internal * (int)sizeof(SplitItem) + (int)nodes * (int)sizeof(NodeRecPacked);
    // Warps a slice: as many as it takes to fill the chip with about 16 warps an SM; more of them than that only wait at
    // the levels with few nodes.  Measured (us a pass, 8 / 2 / 1 warps a slice): 37 subgames of 96 nodes 120 / 197 / 350,
    // 192 of 77 nodes 428 / 335 / 506, 4096 of 54 nodes 6680 / 4070 / 3750.
    const int B = p.num_subgames, sms = sm_count();
    int lanes = 8, slices = 1;
    if (B >= 4 * sms) lanes = 1, slices = VPT == 2 ? 7 : 6;
    else if (B >= sms) lanes = 2, slices = 3;
    const unsigned grid = (unsigned)B * (P2B_HPAD / (32 * VPT) / slices), threads = 32 * lanes * slices;
    if (mode == kColInit) split_columns_kernel<VPT, MAXK, kColInit><<<grid, threads, bytes, stream>>>(p, w, pass, advance, mixed, lanes, slices);
    else if (mode == kColMix) split_columns_kernel<VPT, MAXK, kColMix><<<grid, threads, bytes, stream>>>(p, w, pass, advance, mixed, lanes, slices);
    else split_columns_kernel<VPT, MAXK, kColUp><<<grid, threads, bytes, stream>>>(p, w, pass, advance, mixed, lanes, slices);
    return check_cuda(cudaGetLastError(), "split_columns_kernel");
}

int columns(const CfrParams& p, const SplitWork& w, ColumnMode mode, int pass, bool advance, bool mixed, int max_children,
            cudaStream_t stream) {
    // one hand a thread while two would leave SMs without a block: a warp's walk is 25 % shorter then
    const bool one = p.num_subgames * (P2B_HPAD / 64) < sm_count();
    if (max_children <= kIterMaxChildren)
        return one ? launch_columns<1, 6>(p, w, mode, pass, advance, mixed, max_children, stream)
                   : launch_columns<2, 6>(p, w, mode, pass, advance, mixed, max_children, stream);
    return one ? launch_columns<1, 8>(p, w, mode, pass, advance, mixed, max_children, stream)
               : launch_columns<2, 8>(p, w, mode, pass, advance, mixed, max_children, stream);
}

}  // namespace

long long split_scratch_floats(int num_subgames, long long rows) {
    return 4 + rows * kItemFloats + round4(num_subgames * kLevelFloats) + rows * kRec;
}

bool split_applies(const CfrParams& p, int max_children, long long scratch_floats) {
    return p.rows > 0 && p.init_depth <= kSplitMaxDepth && max_children <= kCfrMaxChildren && p.max_internal <= 255 &&
           scratch_floats >= split_scratch_floats(p.num_subgames, p.rows);
}

int launch_split_passes(const CfrParams& p, int max_children, int pass_begin, int pass_end, bool down, bool up, cudaStream_t stream) {
    const SplitWork w = carve(p.scratch, p.num_subgames, p.rows);
    const bool avg = p.cfr_avg != 0 || p.iter_values != 0;
    int rc = P2B_OK;
    if (down) {
        split_items_kernel<<<p.num_subgames, kCfrMaxNodes, 0, stream>>>(p, w);
        rc = check_cuda(cudaGetLastError(), "split_items_kernel");
        if (!rc) rc = columns(p, w, kColInit, pass_begin, true, avg, max_children, stream);
    }
    for (int pass = pass_begin; pass <= pass_end && !rc; ++pass) {
        if (pass > pass_begin || down) {
            if (avg) rc = columns(p, w, kColMix, pass, false, avg, max_children, stream);
            if (!rc)
                rc = max_children <= kIterMaxChildren ? launch_rows<6>(p, w, pass, avg, stream)
                                                      : launch_rows<8>(p, w, pass, avg, stream);
        }
        if (!rc && (pass < pass_end || up)) rc = columns(p, w, kColUp, pass, pass < pass_end, avg, max_children, stream);
    }
    return rc;
}

}  // namespace p2b
