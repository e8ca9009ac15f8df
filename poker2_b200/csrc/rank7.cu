// Hand-ranking kernels: packed score of [N,7] card ids, pairwise comparison of card-id
// and one-hot-plane hands.  A thread owns four consecutive hands (int16: 56 B, seven 8-byte loads;
// int64: 224 B, fourteen 16-byte loads) and fetches its next four while it scores the current ones.
// int64 ids are read as they are: their converted copy cost a pass over memory and a launch (300,000 hands 19 us, now 10).
#include <atomic>

#include "common.cuh"
#include "rank7.cuh"

namespace p2b {

constexpr int kRankThreads = 256;
constexpr int kHandsPerThread = 4;

// The 28 card ids of hands h0 .. h0+3 as 14 words of two 16-bit ids (ids beyond hand n: 0).  T = int16_t or int64_t, of
// which the low 16 bits count; VEC: the base pointer is aligned for the wide loads.
template <typename T, bool VEC>
__device__ __forceinline__ void load_words(const T* __restrict__ cards, int64_t h0, int64_t n, uint32_t (&w)[14]) {
    if (VEC && h0 + kHandsPerThread <= n) {
        if constexpr (sizeof(T) == 2) {
            const uint2* mine = reinterpret_cast<const uint2*>(cards + h0 * 7);
#pragma unroll
            for (int i = 0; i < 7; ++i) {
                const uint2 v = __ldcs(mine + i);
                w[2 * i] = v.x;
                w[2 * i + 1] = v.y;
            }
        } else {
            const uint4* mine = reinterpret_cast<const uint4*>(cards + h0 * 7);
#pragma unroll
            for (int i = 0; i < 14; ++i) {
                const uint4 v = __ldcs(mine + i);
                w[i] = __byte_perm(v.x, v.z, 0x5410);
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 14; ++i) {
            const int64_t e = h0 * 7 + 2 * i;
            const uint32_t a0 = e < n * 7 ? (uint16_t)cards[e] : 0u;
            const uint32_t a1 = e + 1 < n * 7 ? (uint16_t)cards[e + 1] : 0u;
            w[i] = a0 | (a1 << 16);
        }
    }
}

// Scores of the four hands in w; rank(m0, m1, m2, m3) scores a hand of distinct cards from its suit masks.
template <typename Rank>
__device__ __forceinline__ void score_four(const uint32_t (&w)[14], int32_t (&score)[kHandsPerThread], Rank&& rank) {
    // card id -> bit position in the four 16-bit suit lanes (id + 3 * suit), for both 16-bit
    // halves of a word at once: (id * 79) >> 10 is id / 13 for ids below 52 and the product
    // of the low half cannot carry into the high half
    uint32_t bp[14];
#pragma unroll
    for (int k = 0; k < 14; ++k) bp[k] = w[k] + 3u * (((w[k] * 79u) >> 10) & 0x003F003Fu);
#pragma unroll
    for (int j = 0; j < kHandsPerThread; ++j) {
        uint32_t lo = 0, hi = 0;
#pragma unroll
        for (int i = 0; i < 7; ++i) {
            const int e = 7 * j + i;  // 16-bit element of the thread's 28
            const uint32_t bit = (e & 1) ? (bp[e >> 1] >> 16) : (bp[e >> 1] & 0xffffu);
            uint32_t blo, bhi;  // 1 << bit as two words: shl.b32 gives 0 for shift counts above 31
            asm("shl.b32 %0, 1, %1;" : "=r"(blo) : "r"(bit));
            asm("shl.b32 %0, 1, %1;" : "=r"(bhi) : "r"(bit - 32u));
            lo |= blo;
            hi |= bhi;
        }
        const uint32_t m0 = lo & 0x1fffu, m1 = (lo >> 16) & 0x1fffu, m2 = hi & 0x1fffu, m3 = (hi >> 16) & 0x1fffu;
        if (__popc(lo) + __popc(hi) == 7) {
            score[j] = rank(m0, m1, m2, m3);
        } else {  // repeated (or out-of-range) ids: the general scorer on the ids themselves
            int c[7];
#pragma unroll
            for (int i = 0; i < 7; ++i) {
                const int e = 7 * j + i;
                c[i] = (int)(int16_t)((e & 1) ? (w[e >> 1] >> 16) : (w[e >> 1] & 0xffffu));
            }
            score[j] = score_cards<7>(c);
        }
    }
}

__device__ __forceinline__ void store_four(int32_t* __restrict__ out, int64_t h0, int64_t n, const int32_t (&score)[kHandsPerThread]) {
    if (h0 + kHandsPerThread <= n && ((reinterpret_cast<uintptr_t>(out) & 15) == 0)) {
        __stcs(reinterpret_cast<int4*>(out + h0), make_int4(score[0], score[1], score[2], score[3]));
    } else {
#pragma unroll
        for (int j = 0; j < kHandsPerThread; ++j)
            if (h0 + j < n) out[h0 + j] = score[j];
    }
}

// cards: [n,7]; out: [n] int32.  A block's threads take consecutive groups of four hands, one grid's worth at a time.
template <typename T, bool VEC, typename Rank>
__device__ __forceinline__ void rank_all(const T* __restrict__ cards, int32_t* __restrict__ out, int64_t n, Rank&& rank) {
    const int64_t step = (int64_t)gridDim.x * blockDim.x * kHandsPerThread;
    int64_t h0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * kHandsPerThread;
    uint32_t w[14], wn[14];
    load_words<T, VEC>(cards, h0, n, w);
    for (; h0 < n; h0 += step) {
        load_words<T, VEC>(cards, h0 + step, n, wn);
        int32_t score[kHandsPerThread];
        score_four(w, score, rank);
        store_four(out, h0, n, score);
#pragma unroll
        for (int i = 0; i < 14; ++i) w[i] = wn[i];
    }
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(kRankThreads) rank7_cards_kernel(const T* __restrict__ cards, int32_t* __restrict__ out,
                                                                   int64_t n, const RankLut* __restrict__ lut) {
    __shared__ __align__(16) uint32_t table[kRankLutEntries];
    __shared__ uint32_t types[32];
    {
        const uint4* src = reinterpret_cast<const uint4*>(lut->mask_entry);
        for (int i = threadIdx.x; i < kRankLutEntries / 4; i += kRankThreads) reinterpret_cast<uint4*>(table)[i] = __ldg(src + i);
        if (threadIdx.x < 32) types[threadIdx.x] = threadIdx.x < kTypeLutEntries ? lut->type_entry[threadIdx.x] : 0u;
    }
    __syncthreads();
    rank_all<T, VEC>(cards, out, n, [&](uint32_t m0, uint32_t m1, uint32_t m2, uint32_t m3) {
        return score_distinct_lut(m0, m1, m2, m3, table, types);
    });
}

// cards: [n,2,7] -> {1,-1,0}
template <typename T>
__global__ void __launch_bounds__(256) compare7_cards_kernel(const T* __restrict__ cards, int32_t* __restrict__ out, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        int a[7], b[7];
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            a[k] = (int16_t)cards[i * 14 + k];
            b[k] = (int16_t)cards[i * 14 + 7 + k];
        }
        const int32_t sa = score_cards<7>(a), sb = score_cards<7>(b);
        out[i] = (sa > sb) - (sa < sb);
    }
}

// planes: [n,2,4,13] bytes (non-zero = card present) -> {1,-1,0}.  A plane set is a set of
// cards, so a rank's count is the number of suits holding it (p2/env/rules.py:157).
__device__ __forceinline__ int32_t score_planes(const int8_t* __restrict__ p) {
    uint32_t m[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        uint32_t bits = 0;
#pragma unroll
        for (int r = 0; r < 13; ++r) bits |= (p[s * 13 + r] != 0 ? 1u : 0u) << r;
        m[s] = bits;
    }
    return score_from_masks(m[0], m[1], m[2], m[3], classes_from_suits(m[0], m[1], m[2], m[3]));
}

__global__ void __launch_bounds__(256) compare7_planes_kernel(const int8_t* __restrict__ planes,
                                                             int32_t* __restrict__ out, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t sa = score_planes(planes + i * 104), sb = score_planes(planes + i * 104 + 52);
        out[i] = (sa > sb) - (sa < sb);
    }
}

static int grid_for(int64_t work_items, int per_block, int max_blocks) {
    int64_t g = (work_items + per_block - 1) / per_block;
    if (g < 1) g = 1;
    if (g > max_blocks) g = max_blocks;
    return (int)g;
}

int sm_count();

template <typename T, bool VEC>
static int launch_rank(const T* cards, int64_t n, int32_t* out, cudaStream_t stream) {
    // one wave of resident blocks: the tile loop is strided by the grid, so a partial second wave
    // would leave most SMs idle at the end
    static std::atomic<int> resident{0};
    if (resident.load() == 0) {
        int per_sm = 0;
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, rank7_cards_kernel<T, VEC>, kRankThreads, 0);
        if (e != cudaSuccess) return check_cuda(e, "rank7 occupancy query");
        resident.store(per_sm > 0 ? per_sm : 1);
    }
    const int grid = grid_for(n, kRankThreads * kHandsPerThread, sm_count() * resident.load());
    rank7_cards_kernel<T, VEC><<<grid, kRankThreads, 0, stream>>>(cards, out, n, device_rank_lut());
    return check_cuda(cudaGetLastError(), "rank7_cards_kernel");
}

template <typename T>
static int rank_cards(const T* cards, int64_t n, int32_t* out, cudaStream_t stream) {
    if (n == 0) return P2B_OK;
    const int rc = ensure_tables();
    if (rc) return rc;
    const bool vec = (reinterpret_cast<uintptr_t>(cards) & (sizeof(T) == 2 ? 7 : 15)) == 0;
    return vec ? launch_rank<T, true>(cards, n, out, stream) : launch_rank<T, false>(cards, n, out, stream);
}

template <typename T>
static int compare_cards(const T* cards, int64_t n, int32_t* out, cudaStream_t stream) {
    if (n == 0) return P2B_OK;
    compare7_cards_kernel<T><<<grid_for(n, 256, sm_count() * 8), 256, 0, stream>>>(cards, out, n);
    return check_cuda(cudaGetLastError(), "compare7_cards_kernel");
}

int launch_rank7_cards(const int16_t* cards, int64_t n, int32_t* out, cudaStream_t s) { return rank_cards(cards, n, out, s); }
int launch_rank7_cards(const int64_t* cards, int64_t n, int32_t* out, cudaStream_t s) { return rank_cards(cards, n, out, s); }
int launch_compare7_cards(const int16_t* cards, int64_t n, int32_t* out, cudaStream_t s) { return compare_cards(cards, n, out, s); }
int launch_compare7_cards(const int64_t* cards, int64_t n, int32_t* out, cudaStream_t s) { return compare_cards(cards, n, out, s); }

int launch_compare7_planes(const int8_t* planes, int64_t n, int32_t* out, cudaStream_t stream) {
    if (n == 0) return P2B_OK;
    compare7_planes_kernel<<<grid_for(n, 256, sm_count() * 8), 256, 0, stream>>>(planes, out, n);
    return check_cuda(cudaGetLastError(), "compare7_planes_kernel");
}

}  // namespace p2b
