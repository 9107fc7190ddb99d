// Batched solver of general river subgames: per-hand CFR, best response and strategy
// evaluation over many independent subgames in one persistent launch.
//
// A CTA takes subgames from a device work queue (atomicAdd on a head counter) until it is
// empty. For one subgame, the 1081 live hands are held in rank order ("positions"); a
// thread owns K consecutive positions. The bet tree (pre-order nodes) sits in shared
// memory. A pass for player p walks the tree twice per thread, with the per-hand state of
// the open path on depth-indexed stacks (thread-local memory; the innermost open node of the
// bottom-up walk in registers):
//  * top-down: reach of the opponent (times its range) along the path, from the opponent's
//    regret matching (or average strategy); at every leaf the opponent weights x(o) go to
//    shared memory;
//  * leaves: for each leaf a CTA-wide pass turns x into p's counterfactual values:
//      showdown  stake * ([W - B] over all live hands - [W - B] over the hands holding each
//                of p's two cards), W / B = weight of strictly worse / better hands, taken
//                at the bounds of the hand's tie group (card removal by inclusion-exclusion);
//      fold      +-stake * (T - C[c1] - C[c2] + x(h)), T the total and C the per-card sums.
//    Prefix sums use a fixed summation tree (scans of fixed 64-hand chunks, two hands per
//    lane, and of the pairs of the card lists), so results do not depend on the CTA size;
//  * bottom-up: values flow to the root; at p's nodes the CFR pass updates regrets
//    r <- max(r + v(child) - v(node), 0) (the child value is added when the child closes and
//    the node value subtracted when the node closes, so no per-child storage is needed), the
//    best response takes the maximum, the evaluation the strategy-weighted sum.
// Leaves are processed in groups sized to shared memory; both walks advance group by group.
// Average-strategy sums (avg += reach of p x action probability) are added in the bottom-up
// walk of CFR passes, before the edge's regret changes: it reads p's rows for the update
// anyway, and the top-down walk then reads the opponent's rows only. (With the sums added top-down
// both walks read p's rows and formed its strategies: 4,096 mixed subgames 1702 us per iteration,
// now 1600; 100 subgames 251, now 233; 4,096 trees of 14 edges 564 us per pass, now 527.)
#include <cuda_runtime.h>
#include <stdint.h>

#include "batch_solver.h"
#include "device_common.cuh"
#include "hand_eval.cuh"

namespace prb {
namespace {

constexpr int kSetupThreads = 256;
constexpr int DS = 5;  // stack depth: decision nodes of trees of depth <= 5 (max_raises <= 3)

// ---------------------------------------------------------------- setup ----

__global__ void __launch_bounds__(kSetupThreads) batch_setup_kernel(const BSub *__restrict__ subs,
                                                                     BPack *__restrict__ packs,
                                                                     const float *__restrict__ ranges_in,
                                                                     float *__restrict__ ranges_pos,
                                                                     int *__restrict__ err) {
    const int s = blockIdx.x;
    const int tid = threadIdx.x;
    const unsigned long long board = subs[s].board;
    BPack *pk = packs + s;
    __shared__ unsigned long long key[2048];
    __shared__ uint16_t hand_at[kBRow];
    __shared__ uint8_t lo_li[kBRow], hi_li[kBRow], lo_gi[kBRow], hi_gi[kBRow];  // list; group within it
    __shared__ uint16_t gid[kBRow], lrow[48];
    __shared__ uint8_t list_card[48], list_groups[48];

    if (__popcll(board) != 5 || (board >> 52)) {
        if (tid == 0) atomicOr(err, 1);
        return;
    }
    for (int i = tid; i < 2048; i += kSetupThreads) {
        unsigned long long k = ~0ull;
        if (i < 1326) {
            int c1, c2;
            hand_cards(i, &c1, &c2);
            const unsigned long long hm = (1ull << c1) | (1ull << c2);
            if (!(hm & board)) k = ((unsigned long long)(hand_value(hm | board) + 1u) << 11) | (unsigned)i;
        }
        key[i] = k;
    }
    // bitonic sort, ascending: weakest hand first, ties by hand index
    for (int size = 2; size <= 2048; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            __syncthreads();
            for (int t = tid; t < 1024; t += kSetupThreads) {
                const int i = 2 * t - (t & (stride - 1));
                const int j = i + stride;
                const bool up = (i & size) == 0;
                const unsigned long long a = key[i], b = key[j];
                if ((a > b) == up) {
                    key[i] = b;
                    key[j] = a;
                }
            }
        }
    }
    __syncthreads();
    for (int p = tid; p < kBRow; p += kSetupThreads) hand_at[p] = p < kBLive ? (uint16_t)(key[p] & 2047) : 0xFFFF;
    if (tid == 0) {
        int n = 0;
        for (int c = 0; c < 52; c++)
            if (!((board >> c) & 1)) list_card[n++] = (uint8_t)c;
        list_card[47] = 0;
        // tie groups: equal hand values
        int g = -1;
        for (int p = 0; p < kBLive; p++) {
            if (p == 0 || (key[p] >> 11) != (key[p - 1] >> 11)) {
                if (g >= 0 && g < kBMaxGroups) pk->last[g] = (uint16_t)(p - 1);
                g++;
            }
            gid[p] = (uint16_t)g;
        }
        if (g >= kBMaxGroups) atomicOr(err, 4);
        else pk->last[g] = (uint16_t)(kBLive - 1);
        pk->num_groups = (uint16_t)(g + 1);
    }
    __syncthreads();
    if (tid < kBLists) {
        // card list: live hands holding the card, in rank order, and each element's tie group
        // bounds inside the list
        const int li = tid;
        const int card = list_card[li];
        uint16_t pos[kBListLen];
        int k = 0;
        for (int p = 0; p < kBLive && k < kBListLen; p++) {
            int c1, c2;
            hand_cards(hand_at[p], &c1, &c2);
            if (c1 == card || c2 == card) pos[k++] = (uint16_t)p;
        }
        if (k != kBListLen) atomicOr(err, 2);
        for (int j = 0; j < 48; j++) pk->clpos[li][j] = j < k ? pos[j] : (uint16_t)(kBRow - 1);
        int n = 0;
        unsigned long long ends = 0;
        for (int j = 0; j < k; j++) {
            if (j == 0 || gid[pos[j]] != gid[pos[j - 1]]) n++;
            if (j + 1 == k || gid[pos[j]] != gid[pos[j + 1]]) ends |= 1ull << j;
            int c1, c2;
            hand_cards(hand_at[pos[j]], &c1, &c2);
            if (c1 == card) {
                lo_li[pos[j]] = (uint8_t)li;
                lo_gi[pos[j]] = (uint8_t)(n - 1);
            } else {
                hi_li[pos[j]] = (uint8_t)li;
                hi_gi[pos[j]] = (uint8_t)(n - 1);
            }
        }
        list_groups[li] = (uint8_t)n;
        pk->ends[li] = make_uint2((uint32_t)ends, (uint32_t)(ends >> 32));
    }
    __syncthreads();
    if (tid == 0) {
        int r = 0;
        for (int li = 0; li < kBLists; li++) {
            lrow[li] = (uint16_t)r;
            r += list_groups[li];
        }
        lrow[kBLists] = (uint16_t)r;
        if (r > kBMaxRows) atomicOr(err, 8);
        for (int li = 0; li < 48; li++) pk->lrow[li] = lrow[li];
    }
    __syncthreads();
    for (int p = tid; p < kBRow; p += kSetupThreads) {
        const bool live = p < kBLive;
        pk->rows[p] = live ? (uint32_t)(lrow[lo_li[p]] + lo_gi[p]) | ((uint32_t)(lrow[hi_li[p]] + hi_gi[p]) << 16) : 0u;
        pk->grp[p] = live ? (uint32_t)gid[p] | ((uint32_t)lo_li[p] << 16) | ((uint32_t)hi_li[p] << 24) : 0u;
        pk->hand[p] = hand_at[p];
        pk->pgrp[p] = live ? (uint16_t)(gid[p] | (p + 1 == kBLive || gid[p + 1] != gid[p] ? 0x8000 : 0)) : 0;
    }
    for (int h = tid; h < 1328; h += kSetupThreads) pk->pos_of[h] = 0xFFFF;
    __syncthreads();
    for (int p = tid; p < kBLive; p += kSetupThreads) pk->pos_of[hand_at[p]] = (uint16_t)p;
    for (int i = tid; i < 2 * kBRow; i += kSetupThreads) {
        const int pl = i / kBRow, p = i % kBRow;
        ranges_pos[((size_t)s * 2 + pl) * kBRow + p] =
            p < kBLive ? ranges_in[((size_t)s * 2 + pl) * 1326 + hand_at[p]] : 0.0f;
    }
}

// ---------------------------------------------------------------- solver ----

template <int K>
struct Cfg {
    static constexpr int NT = K == 2 ? 544 : (K == 3 ? 384 : 288);
    static constexpr int MINB = K == 2 ? 1 : 2;  // CTAs per SM the register budget is sized for
};

template <typename V>
__device__ __forceinline__ V neg_inf();
template <>
__device__ __forceinline__ float neg_inf<float>() {
    return -__int_as_float(0x7f800000);
}
template <>
__device__ __forceinline__ double neg_inf<double>() {
    return -__longlong_as_double(0x7ff0000000000000ll);
}

// Asks L2 to fetch [p, p + bytes) (16-byte aligned, size a multiple of 16) ahead of use.
__device__ __forceinline__ void prefetch_l2(const void *p, size_t bytes) {
    const char *c = reinterpret_cast<const char *>(p);
    while (bytes > 0) {
        const unsigned n = bytes > 65536 ? 65536u : (unsigned)bytes;
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(c), "r"(n) : "memory");
        c += n;
        bytes -= n;
    }
}

// The regret (and average) rows of subgame s, prefetched into L2.
__device__ __forceinline__ void prefetch_subgame(const BLaunch &a, int s) {
    const BSub sub = a.subs[s];
    const size_t off = (size_t)sub.edge_off * kBRow, bytes = (size_t)sub.num_edges * kBRow * sizeof(float);
    prefetch_l2(a.regrets + off, bytes);
    if (a.avg) prefetch_l2(a.avg + off, bytes);
    prefetch_l2(a.ranges + (size_t)s * 2 * kBRow, 2 * kBRow * sizeof(float));
}

// products rounded on their own (no contraction into a following add)
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }

// Words of the pack that every leaf scan reads, staged once per subgame.
struct PackWords {
    uint32_t clpos[kBLists][24];  // the card lists' positions, two per word
    uint2 ends[kBLists + 1];
    uint16_t lrow[48];
    uint16_t pgrp[kBRow];
    uint16_t last[kBMaxGroups + 4];
    uint16_t num_groups, pad[3];
};
static_assert(sizeof(PackWords) == offsetof(BPack, pos_of) - offsetof(BPack, clpos) && sizeof(PackWords) % 8 == 0,
              "a piece of BPack");

// A leaf, or a fold by the pass's player followed by its sibling call (see leaf_values).
template <typename V>
struct Job {
    int x0;         // the scanned leaf's row in X, in values
    uint16_t show;  // it is a showdown
    uint16_t pair;  // ... and the row before it is a fold of the job
    V stake, fold;  // signed stakes of the scanned leaf and of that fold (either may be zero)
};
constexpr int kMaxGroupLeaves = 32;  // leaves of a group: a warp lays out its jobs

template <typename V>
struct Smem {
    V *X;    // [group][kBRow] opponent weights, then leaf values
    V *CT;   // [jobs][kCtRow] chunk totals of the rank order
    V *PE;   // [jobs][kBMaxGroups] chunk-local prefix at each tie group's end
    V *VG;   // [jobs][kBMaxGroups] W - B of each tie group
    V *VC;   // [jobs][kVcRow] W - B of each row (tie group of a card list)
    V *TL;   // [jobs][48] totals of the card lists
    V *T;    // [jobs] totals
    Job<V> *job;
    BNode *tn;
    uint16_t *leaf_node;
    PackWords *words;
    V *wsum;  // [32] warp partial sums
};
constexpr int kCtRow = 18, kVgRow = kBMaxGroups, kVcRow = 920, kTlRow = 48;
static_assert(kBMaxRows <= kVcRow && kBChunks64 <= kCtRow, "rows");

// Jobs whose scans run together: a thread takes a (job, card list) pair, so that 4 jobs give 188 tasks to
// the 288 and 384 threads of K = 4 and 3 and 8 jobs 376 tasks to the 544 of K = 2.
__host__ __device__ constexpr int jobs_of(int K, size_t value) { return K == 2 && value == 4 ? 8 : 4; }

template <typename V>
__host__ __device__ inline size_t smem_bytes(int group, int jobs) {
    size_t b = 0;
    b += (size_t)group * kBRow * sizeof(V);
    b += (size_t)jobs * (kCtRow + 2 * kVgRow + kVcRow + kTlRow + 2) * sizeof(V);
    b += 32 * sizeof(V);
    b += (size_t)kMaxGroupLeaves * sizeof(Job<V>);
    b += (size_t)kBMaxNodes * sizeof(BNode);
    b += (size_t)kBMaxLeaves * sizeof(uint16_t);
    b += sizeof(PackWords);
    return (b + 15) & ~(size_t)15;
}

template <typename V>
__device__ inline Smem<V> carve(unsigned char *base, int group, int jobs) {
    Smem<V> S;
    V *v = reinterpret_cast<V *>(base);
    S.X = v;
    v += (size_t)group * kBRow;
    S.CT = v;
    v += jobs * kCtRow;
    S.PE = v;
    v += jobs * kVgRow;
    S.VG = v;
    v += jobs * kVgRow;
    S.VC = v;
    v += jobs * kVcRow;
    S.TL = v;
    v += jobs * kTlRow;
    S.T = v;
    v += jobs * 2;
    S.wsum = v;
    v += 32;
    S.job = reinterpret_cast<Job<V> *>(v);
    S.tn = reinterpret_cast<BNode *>(S.job + kMaxGroupLeaves);
    S.leaf_node = reinterpret_cast<uint16_t *>(S.tn + kBMaxNodes);
    S.words = reinterpret_cast<PackWords *>(S.leaf_node + kBMaxLeaves);
    return S;
}

// A thread's K consecutive positions of a row. With K = 2 or 4 (and kBRow a multiple of 4)
// they are all inside the row or all past it, and move as vector accesses of at most 16 bytes
// (rows start on 16-byte boundaries); with K = 3 they move one by one. Positions past the row
// read as zero and are not written.
static_assert(kBRow % 4 == 0, "vector row accesses");
template <int K, typename T>
struct alignas(K == 3 ? sizeof(T) : (K * sizeof(T) > 16 ? 16 : K * sizeof(T))) Lanes {
    T v[K];
};

template <int K, typename T, typename U>
__device__ __forceinline__ void ld_k(const T *row, int pos0, U (&out)[K]) {
    if constexpr (K == 3) {
#pragma unroll
        for (int k = 0; k < K; k++) out[k] = pos0 + k < kBRow ? U(row[pos0 + k]) : U(0);
    } else {
        if (pos0 < kBRow) {
            const Lanes<K, T> t = *reinterpret_cast<const Lanes<K, T> *>(row + pos0);
#pragma unroll
            for (int k = 0; k < K; k++) out[k] = U(t.v[k]);
        } else {
#pragma unroll
            for (int k = 0; k < K; k++) out[k] = U(0);
        }
    }
}

template <int K, typename T, typename U>
__device__ __forceinline__ void st_k(T *row, int pos0, const U (&in)[K]) {
    if constexpr (K == 3) {
#pragma unroll
        for (int k = 0; k < K; k++)
            if (pos0 + k < kBRow) row[pos0 + k] = T(in[k]);
    } else {
        if (pos0 < kBRow) {
            Lanes<K, T> t;
#pragma unroll
            for (int k = 0; k < K; k++) t.v[k] = T(in[k]);
            *reinterpret_cast<Lanes<K, T> *>(row + pos0) = t;
        }
    }
}

// Rows read by the walks come in edge order (edges are numbered in pre-order): a node's
// strategy sums read rows [edge, edge + nchild), and the next nodes read the rows after them.
// This asks L1 for the 128-byte lines that a warp's positions of rows [first, first + n)
// occupy (rows from `rows` on, past the subgame's last edge, are skipped), one line per lane.
constexpr int kPfRows = 4;  // rows of lookahead
template <int K>
__device__ __forceinline__ void prefetch_rows(const float *base, int first, int n, int rows, int warp, int lane) {
    constexpr int kSpan = 32 * K;                  // floats of a row that one warp covers
    constexpr int kLines = (kSpan + 31) / 32 + 1;  // 128-byte lines the span can touch
    static_assert(kPfRows * kLines <= 32, "one prefetch per lane");
    if (lane < n * kLines) {
        const int row = first + lane / kLines;
        const int f = warp * kSpan + (lane % kLines) * 32;
        if (row < rows && f < kBRow) asm volatile("prefetch.global.L1 [%0];" ::"l"(base + (size_t)row * kBRow + f));
    }
}

// Regret matching with one division per node and hand: a node whose out-edges have
// positive-part sum S keeps scale(S) = 1 / S, or -1 / n when S is at most the cutoff (1e-4
// for regrets, 0 for average sums) and the strategy is uniform; an edge's probability is then
// sigma(val, scale) = max(val, 0) x scale, or 1 / n.
__device__ __forceinline__ float recip(float x) { return __frcp_rn(x); }  // = 1.0f / x, correctly rounded
__device__ __forceinline__ double recip(double x) { return __drcp_rn(x); }
template <typename V, bool USEAVG>
__device__ __forceinline__ V strategy_scale(V S, int n) {
    const V cut = USEAVG ? V(0) : V(1e-4f);
    return S <= cut ? -(V(1) / V(n)) : recip(S);
}
template <typename V>
__device__ __forceinline__ V sigma(V val, V scale) {
    return scale < V(0) ? -scale : mul(val > V(0) ? val : V(0), scale);
}

// Lays out the jobs of the leaves [g0, g1) and returns their number; all warps call it, the first writes. A job is a leaf, or a fold
// by p followed by its sibling call (a showdown): p's actions leave the opponent weights unchanged, so one
// scan serves both leaves.
template <typename V>
__device__ __forceinline__ int lay_out_jobs(const Smem<V> &S, int g0, int g1, int p) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, j = g0 + lane;
    BNode ln{};
    if (j < g1) ln = S.tn[S.leaf_node[j]];
    const int next_kind = __shfl_down_sync(FULL, (int)ln.kind, 1), next_parent = __shfl_down_sync(FULL, (int)ln.parent, 1);
    const float next_stake = __shfl_down_sync(FULL, ln.stake, 1);
    const bool pair = j + 1 < g1 && lane < 31 && ln.kind == kBFold && ln.actor == p && next_kind == kBShowdown &&
                      next_parent == (int)ln.parent;
    const unsigned pairs = __ballot_sync(FULL, pair), seconds = pairs << 1;
    const bool start = j < g1 && !(seconds >> lane & 1);
    const unsigned starts = __ballot_sync(FULL, start);
    if (start && threadIdx.x < 32) {
        Job<V> &job = S.job[__popc(starts & ((1u << lane) - 1))];
        job.x0 = (lane + (pair ? 1 : 0)) * kBRow;
        job.show = pair || ln.kind == kBShowdown;
        job.pair = pair;
        job.stake = pair ? V(next_stake) : ln.kind == kBFold && ln.actor == p ? -V(ln.stake) : V(ln.stake);
        job.fold = pair ? -V(ln.stake) : V(0);
    }
    return __popc(starts);
}

// A card list's rows, by one thread: a0 holds the first hand of each of its pairs, v the pairs' sums.
// Writes W - B of every tie group of the list (bit j of `ends`: hand j is a group's last) and returns the
// list's total.
template <typename V>
__device__ __forceinline__ V scan_list(const V (&a0)[kBListLen / 2], V (&v)[kBListLen / 2], uint2 ends, V *to) {
    constexpr int kPairs = kBListLen / 2;
#pragma unroll
    for (int off = 1; off < kPairs; off <<= 1) {
#pragma unroll
        for (int i = kPairs - 1; i >= off; i--) v[i] += v[i - off];
    }
    const V total = v[kPairs - 1];
    V before = V(0);  // prefix at the end of the group before
#pragma unroll
    for (int i = 0; i < kPairs; i++) {
        const V even = (i > 0 ? v[i > 0 ? i - 1 : 0] : V(0)) + a0[i];
        if ((2 * i < 32 ? ends.x >> (2 * i) : ends.y >> (2 * i - 32)) & 1) {
            *to++ = (even + before) - total;
            before = even;
        }
        if ((2 * i + 1 < 32 ? ends.x >> (2 * i + 1) : ends.y >> (2 * i + 1 - 32)) & 1) {
            *to++ = (v[i] + before) - total;
            before = v[i];
        }
    }
    return total;
}

// The values of a group's leaves: opponent weights in X -> p's values, in place, for the jobs of
// lay_out_jobs (n of them); all warps of the CTA call it. JOBS jobs go together:
//   A  card lists, one thread per (job, list): the inclusive scan over the list's 23 pairs of hands in
//      registers, by doubling steps, then W - B of every tie group of the list;
//      rank order, on the warps left over: scans of 64-hand chunks, two hands per lane, of which the
//      prefixes at the tie groups' ends are kept;
//   B  W - B of every tie group of the rank order;
//   C  values: a hand looks up its group and its two rows.
// What bounds the phase is its instructions. A list scanned by a warp (23 of 32 lanes, five shuffles per
// step) took about 110 of them per job, by a thread it takes 600 / 32. W - B formed per tie group (76 and
// 542 on the mean board, for 1081 hands and 2162 list entries) has the operands it had per hand. Both
// leave every bit as it was.
template <int K, typename V, int NW, int JOBS>
__device__ __forceinline__ void leaf_values(const Smem<V> &S, const BPack *__restrict__ pk, int n, int pos0) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kPairs = kBListLen / 2;
    uint32_t rows[K], grp[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int pq = pos0 + k < kBRow ? pos0 + k : kBRow - 1;
        rows[k] = __ldg(&pk->rows[pq]);
        grp[k] = __ldg(&pk->grp[pq]);
    }
    const PackWords &W = *S.words;
#pragma unroll 1
    for (int j0 = 0; j0 < n; j0 += JOBS) {
        const int nj = min(JOBS, n - j0);
        const int list_warps = (nj * kBLists + 31) / 32;  // fewer than NW
        // ---- A ----
        if (warp < list_warps) {
            const int q = (int)threadIdx.x / kBLists, li = (int)threadIdx.x % kBLists;
            if (q < nj) {
                const V *x = S.X + S.job[j0 + q].x0;
                V a0[kPairs], v[kPairs];
#pragma unroll
                for (int i = 0; i < kPairs; i++) {
                    const uint32_t w = W.clpos[li][i];
                    a0[i] = x[w & 0xFFFF];
                    v[i] = a0[i] + x[w >> 16];
                }
                const V total = scan_list(a0, v, W.ends[li], S.VC + q * kVcRow + W.lrow[li]);
                S.TL[q * kTlRow + li] = total;
            }
        } else {
            for (int u = warp - list_warps; u < kBChunks64 * nj; u += NW - list_warps) {
                const int q = u / kBChunks64, c = u - q * kBChunks64;
                const V *x = S.X + S.job[j0 + q].x0 + c * 64 + 2 * lane;
                const V a0 = x[0];
                V v = a0 + x[1];
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const V t = __shfl_up_sync(FULL, v, off);
                    if (lane >= off) v += t;
                }
                V ex = __shfl_up_sync(FULL, v, 1);
                if (lane == 0) ex = V(0);
                const uint32_t g = *reinterpret_cast<const uint32_t *>(W.pgrp + c * 64 + 2 * lane);
                if (g & 0x8000u) S.PE[q * kVgRow + (g & 0x7FFF)] = ex + a0;
                if (g & 0x80000000u) S.PE[q * kVgRow + (g >> 16 & 0x7FFF)] = v;
                if (lane == 31) S.CT[q * kCtRow + c] = v;
            }
        }
        __syncthreads();
        // ---- B: a warp per job ----
        for (int q = warp; q < nj; q += NW) {
            V cofs = lane < kBChunks64 ? S.CT[q * kCtRow + lane] : V(0);  // chunk offsets: lane c holds chunk c's
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const V t = __shfl_up_sync(FULL, cofs, off);
                if (lane >= off) cofs += t;
            }
            const V T = __shfl_sync(FULL, cofs, kBChunks64 - 1);
            cofs = __shfl_up_sync(FULL, cofs, 1);
            if (lane == 0) {
                cofs = V(0);
                S.T[q] = T;
            }
            const int G = W.num_groups;
            for (int g0 = 0; g0 < G; g0 += 32) {
                const int g = min(g0 + lane, G - 1);
                const int ge = W.last[g], gs = g > 0 ? W.last[g > 0 ? g - 1 : 0] : 0;  // ends of this group and the one before
                const V oe = __shfl_sync(FULL, cofs, ge >> 6), os = __shfl_sync(FULL, cofs, gs >> 6);
                const V Pe = oe + S.PE[q * kVgRow + g];
                const V Ps = g > 0 ? os + S.PE[q * kVgRow + (g > 0 ? g - 1 : 0)] : V(0);
                if (g0 + lane < G) S.VG[q * kVgRow + g] = (Pe + Ps) - T;
            }
        }
        __syncthreads();
        // ---- C ----
#pragma unroll 2
        for (int q = 0; q < nj; q++) {
            const Job<V> job = S.job[j0 + q];
            V *x = S.X + job.x0;
            V val[K];
            if (job.show) {
#pragma unroll
                for (int k = 0; k < K; k++) {
                    const V vg = S.VG[q * kVgRow + (grp[k] & 0xFFFF)];
                    const V v1 = S.VC[q * kVcRow + (rows[k] & 0xFFFF)], v2 = S.VC[q * kVcRow + (rows[k] >> 16)];
                    val[k] = pos0 + k < kBLive ? mul(job.stake, (vg - v1) - v2) : V(0);
                }
            }
            if (!job.show || job.pair) {
                V xv[K], fold[K];
                ld_k<K>(x, pos0, xv);
                const V T = S.T[q], m = job.show ? job.fold : job.stake;
#pragma unroll
                for (int k = 0; k < K; k++) {
                    const V t1 = S.TL[q * kTlRow + (grp[k] >> 16 & 255)], t2 = S.TL[q * kTlRow + (grp[k] >> 24)];
                    fold[k] = pos0 + k < kBLive ? mul(m, ((T - t1) - t2) + xv[k]) : V(0);
                }
                st_k<K>(x - (job.show ? kBRow : 0), pos0, fold);
            }
            if (job.show) st_k<K>(x, pos0, val);
        }
        __syncthreads();  // the next jobs rewrite the scans
    }
}

// MINB: CTAs per SM the registers are capped for (Cfg<K>::MINB, or 3 for the dense K = 4
// configuration with 10-leaf groups).
template <int K, typename V, int MODE, bool AVG, bool USEAVG, int MINB>
__global__ void __launch_bounds__(Cfg<K>::NT, MINB) batch_kernel(BLaunch a, int group) {
    constexpr int NT = Cfg<K>::NT;
    constexpr int NW = NT / 32;
    static_assert(MODE == kBModeCFR || !AVG, "average sums accumulate in CFR passes");
    static_assert(MODE != kBModeCFR || (sizeof(V) == 4 && !USEAVG), "CFR runs on regrets in single precision");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int kJobs = jobs_of(K, sizeof(V));
    Smem<V> S = carve<V>(smem_raw, group, kJobs);
    __shared__ int s_next;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const unsigned FULL = 0xffffffffu;
    const int p = a.player, o = 1 - p;
    const float *src_all = USEAVG ? a.avg : a.regrets;
    // weight of this pass's average-sum terms (1 unless the caller weights iterations)
    const float wavg = AVG && a.avg_weight ? *a.avg_weight : 1.0f;

    // The next queue entry is taken (and its rows prefetched into L2) while the current one
    // is solved.
    if (tid == 0) {
        s_next = atomicAdd(a.head, 1);
        if (s_next < a.count) prefetch_subgame(a, a.order[s_next]);
    }
    for (;;) {
        __syncthreads();
        const int qi = s_next;
        __syncthreads();
        if (qi >= a.count) break;
        if (tid == 0) {
            s_next = atomicAdd(a.head, 1);
            if (s_next < a.count) prefetch_subgame(a, a.order[s_next]);
        }
        const int s = a.order[qi];
        const BSub sub = a.subs[s];
        const BPack *__restrict__ pk = a.packs + s;
        const int N = sub.num_nodes, L = sub.num_leaves;
        for (int i = tid; i < N; i += NT) {
            const BNode nd = a.nodes[sub.node_off + i];
            S.tn[i] = nd;
            if (nd.kind != kBDecision) S.leaf_node[nd.edge] = (uint16_t)i;
        }
        {
            const uint2 *src = reinterpret_cast<const uint2 *>(&pk->clpos[0][0]);
            uint2 *dst = reinterpret_cast<uint2 *>(S.words);
            for (int i = tid; i < (int)(sizeof(PackWords) / 8); i += NT) dst[i] = __ldg(src + i);
        }
        __syncthreads();
        float *R = a.regrets + (size_t)sub.edge_off * kBRow;
        float *A = a.avg ? a.avg + (size_t)sub.edge_off * kBRow : nullptr;
        const float *Src = src_all + (size_t)sub.edge_off * kBRow;
        const float *rng = a.ranges + (size_t)s * 2 * kBRow;
        const int pos0 = tid * K;

        // walker state, per owned hand: depth-indexed stacks of the open path (indexed at run
        // time, so they live in local memory, cached in L1). Depth-major with the K hands of a
        // depth adjacent and aligned, so that one depth moves as one vector access.
        alignas(16) V po[DS][K];
        alignas(16) V St[DS][K];   // top-down: opponent weight, strategy scales
        alignas(16) V pp[DS][K];   // bottom-up: own reach
        alignas(16) V acc[DS][K];
        alignas(16) V Sb[DS][K];   // bottom-up: node values, strategy scales
        int open_id[DS];
        int open_top = -1;
        int td = 0, bu = 0;
        V root[K];
#pragma unroll
        for (int k = 0; k < K; k++) root[k] = V(0);

        // adds the values v of the child behind edge ie to its parent par, open at depth dp
        // The innermost open node of the bottom-up walk keeps its value and strategy scale in
        // registers (tacc, tsb); the stacks hold the open nodes outside it. Every child's value
        // goes to its parent, which is always that innermost node.
        V tacc[K], tsb[K];
        // between the bottom-up walks of two groups the registers rest in the stack slot of the
        // innermost open node (slot 0 when none is open: then nothing reads them)
        auto park = [&]() {
            const int t = open_top > 0 ? open_top : 0;
#pragma unroll
            for (int k = 0; k < K; k++) {
                acc[t][k] = tacc[k];
                Sb[t][k] = tsb[k];
            }
        };
        auto unpark = [&]() {
            const int t = open_top > 0 ? open_top : 0;
#pragma unroll
            for (int k = 0; k < K; k++) {
                tacc[k] = acc[t][k];
                tsb[k] = Sb[t][k];
            }
        };
#pragma unroll
        for (int k = 0; k < K; k++) tacc[k] = tsb[k] = V(0);
        park();
        auto deliver = [&](int par, int ie, const V(&v)[K]) {
            const BNode pq = S.tn[par];
            if (a.child_out && par == 0) {
                V *co = reinterpret_cast<V *>(a.child_out) + ((size_t)s * 8 + (ie - pq.edge)) * kBRow;
                st_k<K>(co, pos0, v);
            }
            if (pq.actor != p) {
#pragma unroll
                for (int k = 0; k < K; k++) tacc[k] = tacc[k] + v[k];
            } else if (MODE == kBModeBR) {
#pragma unroll
                for (int k = 0; k < K; k++) tacc[k] = tacc[k] > v[k] ? tacc[k] : v[k];
            } else {
                // the edge's strategy from its regret (or average) row; CFR adds the child's
                // value to the regret, which the parent's close turns into the regret update
                const size_t ro = (size_t)ie * kBRow;
                V sv[K];
                if (MODE == kBModeCFR)
                    ld_k<K>(R + ro, pos0, sv);
                else
                    ld_k<K>(Src + ro, pos0, sv);
#pragma unroll
                for (int k = 0; k < K; k++)
                    tacc[k] = tacc[k] + mul(sigma<V>(sv[k], tsb[k]), v[k]);
                if constexpr (AVG) {
                    float av[K];
                    ld_k<K>(A + ro, pos0, av);
#pragma unroll
                    for (int k = 0; k < K; k++)
                        av[k] = __fmaf_rn(wavg, float(mul(pp[open_top][k], sigma<V>(sv[k], tsb[k]))), av[k]);
                    st_k<K>(A + ro, pos0, av);
                }
                if constexpr (MODE == kBModeCFR) {
                    float r[K];
#pragma unroll
                    for (int k = 0; k < K; k++) r[k] = float(sv[k]) + float(v[k]);
                    st_k<K>(R + ro, pos0, r);
                }
            }
        };
        // closes the open nodes at depth >= d, passing each value to its parent
        auto close_to = [&](int d) {
            while (open_top >= d) {
                const int m = open_id[open_top];
                const BNode nm = S.tn[m];
                V v[K];
#pragma unroll
                for (int k = 0; k < K; k++) v[k] = tacc[k];
                if (MODE == kBModeCFR && nm.actor == p) {
                    for (int e = 0; e < nm.nchild; e++) {
                        float *row = R + (size_t)(nm.edge + e) * kBRow;
                        float r[K];
                        ld_k<K>(row, pos0, r);
#pragma unroll
                        for (int k = 0; k < K; k++) r[k] = fmaxf(r[k] - float(v[k]), 0.0f);
                        st_k<K>(row, pos0, r);
                    }
                }
                open_top--;
                if (m == 0) {
#pragma unroll
                    for (int k = 0; k < K; k++) root[k] = v[k];
                } else {
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        tacc[k] = acc[open_top][k];
                        tsb[k] = Sb[open_top][k];
                    }
                    deliver(nm.parent, nm.in_edge, v);
                }
            }
        };
        // node m's children are one or two leaves, the nodes after it, and belong to this group
        auto leafy = [&](int m, const BNode &nd, int end) {
            return nd.nchild <= 2 && m + nd.nchild < end && S.tn[m + nd.nchild].parent == m &&
                   S.tn[m + 1].kind != kBDecision && S.tn[m + nd.nchild].kind != kBDecision;
        };
        for (int g0 = 0; g0 < L; g0 += group) {
            const int g1 = min(L, g0 + group);
            const int end = g1 == L ? N : S.leaf_node[g1];
            // ---- top-down walk over nodes [td, end) ----
            // Only decision nodes put their opponent weight and strategy scale on the stacks: their
            // children read them, and nothing reads a leaf's entry. p's own nodes pass the weights on as
            // they are and read no row here: p's reach and the average sums go with the bottom-up
            // walk, which reads those rows anyway. A node whose children are all leaves is done together
            // with them, without the stacks and with one read of its rows (see `leafy`).
            for (; td < end; td++) {
                const BNode nd = S.tn[td];
                const int d = nd.depth;
                V npo[K];
                if (td == 0) {
                    if (sizeof(V) == 8 && a.ranges64)
                        ld_k<K>(a.ranges64 + ((size_t)s * 2 + o) * kBRow, pos0, npo);
                    else
                        ld_k<K>(rng + o * kBRow, pos0, npo);
                } else if (S.tn[nd.parent].actor == p) {
#pragma unroll
                    for (int k = 0; k < K; k++) npo[k] = po[d - 1][k];
                } else {
                    V sv[K];
                    ld_k<K>(Src + (size_t)nd.in_edge * kBRow, pos0, sv);
#pragma unroll
                    for (int k = 0; k < K; k++) npo[k] = mul(po[d - 1][k], sigma<V>(sv[k], St[d - 1][k]));
                }
                auto put_leaf = [&](int leaf, const V(&w)[K]) {
                    V xv[K];
#pragma unroll
                    for (int k = 0; k < K; k++) xv[k] = pos0 + k < kBLive ? w[k] : V(0);
                    st_k<K>(S.X + (size_t)(leaf - g0) * kBRow, pos0, xv);
                };
                if (nd.kind != kBDecision) {
                    put_leaf(nd.edge, npo);
                    continue;
                }
                const bool own = nd.actor == p;
                if (leafy(td, nd, end)) {
                    V sv[2][K], sum[K];
#pragma unroll
                    for (int k = 0; k < K; k++) sum[k] = V(0);
                    if (!own) {
#pragma unroll
                        for (int c = 0; c < 2; c++) {
                            if (c >= nd.nchild) continue;
                            ld_k<K>(Src + (size_t)(nd.edge + c) * kBRow, pos0, sv[c]);
#pragma unroll
                            for (int k = 0; k < K; k++) sum[k] += sv[c][k] > V(0) ? sv[c][k] : V(0);
                        }
                        prefetch_rows<K>(Src, nd.edge + nd.nchild, kPfRows, sub.num_edges, warp, lane);
#pragma unroll
                        for (int k = 0; k < K; k++) sum[k] = strategy_scale<V, USEAVG>(sum[k], nd.nchild);
                    }
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        if (c >= nd.nchild) continue;
                        V w[K];
#pragma unroll
                        for (int k = 0; k < K; k++) w[k] = own ? npo[k] : mul(npo[k], sigma<V>(sv[c][k], sum[k]));
                        put_leaf(S.tn[td + 1 + c].edge, w);
                    }
                    td += nd.nchild;
                    continue;
                }
                if (!own) {
                    // strategy sums of the node, for its children
                    V sum[K];
#pragma unroll
                    for (int k = 0; k < K; k++) sum[k] = V(0);
                    for (int e = 0; e < nd.nchild; e++) {
                        V sv[K];
                        ld_k<K>(Src + (size_t)(nd.edge + e) * kBRow, pos0, sv);
#pragma unroll
                        for (int k = 0; k < K; k++) sum[k] += sv[k] > V(0) ? sv[k] : V(0);
                    }
                    prefetch_rows<K>(Src, nd.edge + nd.nchild, kPfRows, sub.num_edges, warp, lane);
#pragma unroll
                    for (int k = 0; k < K; k++) St[d][k] = strategy_scale<V, USEAVG>(sum[k], nd.nchild);
                }
#pragma unroll
                for (int k = 0; k < K; k++) po[d][k] = npo[k];
            }
            // (every warp counts them, the first writes them)
            const int jobs = lay_out_jobs(S, g0, g1, p);
            __syncthreads();

            // ---- leaves of the group: opponent weights -> p's values ----
            leaf_values<K, V, NW, kJobs>(S, pk, jobs, pos0);

            // ---- bottom-up walk over nodes [bu, end) ----
            unpark();
            for (; bu < end; bu++) {
                const BNode nd = S.tn[bu];
                const int d = nd.depth;
                close_to(d);
                if (nd.kind == kBDecision) {
                    if constexpr (AVG) {
                        // p's reach, from the parent's (the innermost open node, scale in tsb)
                        if (bu == 0) {
                            V w[K];
                            if (a.own_reach) ld_k<K>(rng + p * kBRow, pos0, w);
#pragma unroll
                            for (int k = 0; k < K; k++) pp[0][k] = a.own_reach ? w[k] : V(1);
                        } else if (S.tn[nd.parent].actor == p) {
                            V sv[K];
                            ld_k<K>(R + (size_t)nd.in_edge * kBRow, pos0, sv);
#pragma unroll
                            for (int k = 0; k < K; k++) pp[d][k] = mul(pp[d - 1][k], sigma<V>(sv[k], tsb[k]));
                        } else {
#pragma unroll
                            for (int k = 0; k < K; k++) pp[d][k] = pp[d - 1][k];
                        }
                        if (nd.actor == p)
                            prefetch_rows<K>(A, nd.edge, min(nd.nchild, kPfRows), sub.num_edges, warp, lane);
                    }
                    // the parent (open at d - 1, or none at the root) moves to the stack
                    if (open_top >= 0) {
#pragma unroll
                        for (int k = 0; k < K; k++) {
                            acc[open_top][k] = tacc[k];
                            Sb[open_top][k] = tsb[k];
                        }
                    }
                    open_top = d;
                    open_id[d] = bu;
                    const bool own = nd.actor == p;
                    V sum[K];
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        tacc[k] = (own && MODE == kBModeBR) ? neg_inf<V>() : V(0);
                        sum[k] = V(0);
                    }
                    if (own && MODE != kBModeBR) {
                        for (int e = 0; e < nd.nchild; e++) {
                            V sv[K];
                            ld_k<K>(Src + (size_t)(nd.edge + e) * kBRow, pos0, sv);
#pragma unroll
                            for (int k = 0; k < K; k++) sum[k] += sv[k] > V(0) ? sv[k] : V(0);
                        }
                        prefetch_rows<K>(Src, nd.edge + nd.nchild, kPfRows, sub.num_edges, warp, lane);
                    }
#pragma unroll
                    for (int k = 0; k < K; k++)
                        tsb[k] = (own && MODE != kBModeBR) ? strategy_scale<V, USEAVG>(sum[k], nd.nchild) : V(0);
                } else {
                    // a leaf: its value goes straight to the parent (the innermost open node)
                    V xv[K];
                    ld_k<K>(S.X + (size_t)(nd.edge - g0) * kBRow, pos0, xv);
                    deliver(nd.parent, nd.in_edge, xv);
                }
            }
            park();
            __syncthreads();  // X is rewritten by the next group
        }
        unpark();
        close_to(0);

        // ---- outputs: root values and their range-weighted sum ----
        if (a.root_out) {
            st_k<K>(reinterpret_cast<V *>(a.root_out) + (size_t)s * kBRow, pos0, root);
        }
        if (a.sum_out) {
            V part = V(0);
            V rv[K];
            ld_k<K>(rng + p * kBRow, pos0, rv);
#pragma unroll
            for (int k = 0; k < K; k++)
                if (pos0 + k < kBRow) part += mul(rv[k], root[k]);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(FULL, part, off);
            if (lane == 0) S.wsum[warp] = part;
            __syncthreads();
            if (tid == 0) {
                V t = V(0);
                for (int w = 0; w < NW; w++) t += S.wsum[w];
                reinterpret_cast<V *>(a.sum_out)[s] = t;
            }
        }
        __syncthreads();
    }
}

// Subgames without a bet (both players check, then the showdown: all-in river leaves) in CFR passes. Their
// tree is two edges and one leaf, so that batch_kernel spends its time on the staging of tree and pack, the
// walks' stacks and barriers, with at most three CTAs per SM: 1028 us for 18,816 of them. Here a CTA keeps
// no tree, stack or leaf group: 9 KB of shared memory and 3 barriers per subgame, so that 4 share an SM
// while the next subgame's rows are asked from L2. That takes 200 us (592: 32 -> 9 us), 4.2 TB/s of the 44 KB
// that a subgame moves (pack, ranges, two regret rows, one sum row, root values); what is left is the wait
// for those rows. 3 CTAs per SM took 215 us, 5 (40 registers, spills) 238.
// The arithmetic is batch_kernel's, operand for operand. As there, a thread scans a card list: by a warp per
// list the pass had 9,070 instructions per subgame and took 298 us, so it has 5,560.
constexpr int kCheckCtas = 4;
constexpr int kCheckThreads = 288;

template <bool AVG>
__global__ void __launch_bounds__(kCheckThreads, kCheckCtas) check_kernel(BLaunch a) {
    constexpr int K = 4, NW = kCheckThreads / 32, kPairs = kBListLen / 2, kListWarps = (kBLists + 31) / 32;
    __shared__ __align__(16) float X[kBRow];
    __shared__ float CT[kCtRow], PE[kVgRow], VG[kVgRow], VC[kVcRow];
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, pos0 = tid * K;
    const int p = a.player, o = 1 - p;
    const float wavg = AVG && a.avg_weight ? *a.avg_weight : 1.0f;
    int qi = blockIdx.x;
    if (qi >= a.count) return;
    int s = a.order[qi];
    BSub sub = a.subs[s];
    for (;;) {
        const BPack *__restrict__ pk = a.packs + s;
        float *R = a.regrets + (size_t)sub.edge_off * kBRow;  // rows: player 0's check, player 1's check
        const float stake = a.nodes[sub.node_off + 2].stake;
        // ---- opponent weights ----
        float w[K], sv[K];
        ld_k<K>(a.ranges + ((size_t)s * 2 + o) * kBRow, pos0, w);
        ld_k<K>(R + (size_t)o * kBRow, pos0, sv);
#pragma unroll
        for (int k = 0; k < K; k++) {
            w[k] = mul(w[k], sigma<float>(sv[k], strategy_scale<float, false>(sv[k] > 0.0f ? sv[k] : 0.0f, 1)));
            if (pos0 + k >= kBLive) w[k] = 0.0f;
        }
        st_k<K>(X, pos0, w);
        const int next = qi + gridDim.x;
        int s_next = 0;
        if (next < a.count) {
            s_next = a.order[next];
            sub = a.subs[s_next];
            if (tid == 0) {
                const BPack *nx = a.packs + s_next;
                prefetch_l2(nx, offsetof(BPack, hand));
                prefetch_l2(&nx->clpos[0][0], sizeof(PackWords) / 16 * 16);
                prefetch_l2(a.ranges + (size_t)s_next * 2 * kBRow, 2 * kBRow * sizeof(float));
                prefetch_l2(a.regrets + (size_t)sub.edge_off * kBRow, 2 * kBRow * sizeof(float));
                if (AVG) prefetch_l2(a.avg + (size_t)(sub.edge_off + p) * kBRow, kBRow * sizeof(float));
            }
        }
        __syncthreads();
        // ---- scans: card lists on the first two warps, 64-hand chunks of the rank order on the others ----
        if (warp < kListWarps) {
            if (tid < kBLists) {
                const uint4 *at = reinterpret_cast<const uint4 *>(&pk->clpos[tid][0]);
                const uint2 ends = __ldg(&pk->ends[tid]);
                float *to = VC + __ldg(&pk->lrow[tid]);
                float a0[kPairs], v[kPairs];
#pragma unroll
                for (int j = 0; j < (kPairs + 3) / 4; j++) {
                    const uint4 w4 = __ldg(at + j);
                    const uint32_t w1[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        const int i = 4 * j + t;
                        if (i >= kPairs) continue;
                        a0[i] = X[w1[t] & 0xFFFF];
                        v[i] = a0[i] + X[w1[t] >> 16];
                    }
                }
                scan_list(a0, v, ends, to);
            }
        } else {
            for (int c = warp - kListWarps; c < kBChunks64; c += NW - kListWarps) {
                const float2 x2 = *reinterpret_cast<const float2 *>(X + c * 64 + 2 * lane);
                float v = x2.x + x2.y;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const float t = __shfl_up_sync(FULL, v, off);
                    if (lane >= off) v += t;
                }
                float ex = __shfl_up_sync(FULL, v, 1);
                if (lane == 0) ex = 0.0f;
                const uint32_t g = __ldg(reinterpret_cast<const uint32_t *>(pk->pgrp + c * 64) + lane);
                if (g & 0x8000u) PE[g & 0x7FFF] = ex + x2.x;
                if (g & 0x80000000u) PE[g >> 16 & 0x7FFF] = v;
                if (lane == 31) CT[c] = v;
            }
        }
        uint32_t rows[K], grp[K];
        ld_k<K>(pk->rows, pos0, rows);
        ld_k<K>(pk->grp, pos0, grp);
        __syncthreads();
        // ---- W - B of the tie groups of the rank order ----
        const int G = __ldg(&pk->num_groups);
        if (warp * 32 < G) {
            float cofs = lane < kBChunks64 ? CT[lane] : 0.0f;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const float t = __shfl_up_sync(FULL, cofs, off);
                if (lane >= off) cofs += t;
            }
            const float T = __shfl_sync(FULL, cofs, kBChunks64 - 1);
            cofs = __shfl_up_sync(FULL, cofs, 1);
            if (lane == 0) cofs = 0.0f;
            const int g = min(tid, G - 1), gp = max(g - 1, 0);
            const int ge = __ldg(&pk->last[g]), gs = g > 0 ? __ldg(&pk->last[gp]) : 0;
            const float oe = __shfl_sync(FULL, cofs, ge >> 6), os = __shfl_sync(FULL, cofs, gs >> 6);
            const float Pe = oe + PE[g], Ps = g > 0 ? os + PE[gp] : 0.0f;
            if (tid < G) VG[g] = (Pe + Ps) - T;
        }
        // the own row, its sums and its reach while the groups are formed
        float npp[K];
        ld_k<K>(R + (size_t)p * kBRow, pos0, sv);
        float scale[K];
#pragma unroll
        for (int k = 0; k < K; k++) scale[k] = strategy_scale<float, false>(sv[k] > 0.0f ? sv[k] : 0.0f, 1);
        if constexpr (AVG) {
            if (a.own_reach) {
                ld_k<K>(a.ranges + ((size_t)s * 2 + p) * kBRow, pos0, npp);
            } else {
#pragma unroll
                for (int k = 0; k < K; k++) npp[k] = 1.0f;
            }
            float *A = a.avg + (R - a.regrets) + (size_t)p * kBRow;
            float av[K];
            ld_k<K>(A, pos0, av);
#pragma unroll
            for (int k = 0; k < K; k++) av[k] = __fmaf_rn(wavg, mul(npp[k], sigma<float>(sv[k], scale[k])), av[k]);
            st_k<K>(A, pos0, av);
        }
        __syncthreads();
        // ---- values; regrets of the own check; root ----
        float r[K], root[K];
#pragma unroll
        for (int k = 0; k < K; k++) {
            const float vg = VG[grp[k] & 0xFFFF], v1 = VC[rows[k] & 0xFFFF], v2 = VC[rows[k] >> 16];
            float v = pos0 + k < kBLive ? mul(stake, (vg - v1) - v2) : 0.0f;
            if (p == 0) v = 0.0f + v;  // passed through player 1's node
            r[k] = sv[k] + v;
            root[k] = 0.0f + mul(sigma<float>(sv[k], scale[k]), v);
            r[k] = fmaxf(r[k] - root[k], 0.0f);
        }
        st_k<K>(R + (size_t)p * kBRow, pos0, r);
        if (a.root_out) st_k<K>(reinterpret_cast<float *>(a.root_out) + (size_t)s * kBRow, pos0, root);
        if (next >= a.count) break;
        qi = next;
        s = s_next;
    }
}

__global__ void weight_step_kernel(float *w) { *w += 1.0f; }

template <int K, typename V, int MODE, bool AVG, bool USEAVG, int MINB = Cfg<K>::MINB>
cudaError_t launch_one(const BLaunch &a, int ctas, int group, cudaStream_t stream) {
    const size_t smem = smem_bytes<V>(group, jobs_of(K, sizeof(V)));
    cudaError_t e = cudaFuncSetAttribute(batch_kernel<K, V, MODE, AVG, USEAVG, MINB>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    batch_kernel<K, V, MODE, AVG, USEAVG, MINB><<<ctas, Cfg<K>::NT, smem, stream>>>(a, group);
    return cudaGetLastError();
}

template <int K>
cudaError_t launch_k(int mode, int fp64, int avg, const BLaunch &a, int ctas, int group, cudaStream_t st,
                     int dense) {
    if (mode == kBModeCFR) {
        if (fp64) return cudaErrorInvalidValue;
        if constexpr (K == 4) {
            if (dense)
                return avg ? launch_one<4, float, kBModeCFR, true, false, 3>(a, ctas, group, st)
                           : launch_one<4, float, kBModeCFR, false, false, 3>(a, ctas, group, st);
        }
        return avg ? launch_one<K, float, kBModeCFR, true, false>(a, ctas, group, st)
                   : launch_one<K, float, kBModeCFR, false, false>(a, ctas, group, st);
    }
    if (mode == kBModeBR) {
        if (fp64)
            return a.use_average ? launch_one<K, double, kBModeBR, false, true>(a, ctas, group, st)
                                 : launch_one<K, double, kBModeBR, false, false>(a, ctas, group, st);
        return a.use_average ? launch_one<K, float, kBModeBR, false, true>(a, ctas, group, st)
                             : launch_one<K, float, kBModeBR, false, false>(a, ctas, group, st);
    }
    if (fp64)
        return a.use_average ? launch_one<K, double, kBModeEval, false, true>(a, ctas, group, st)
                             : launch_one<K, double, kBModeEval, false, false>(a, ctas, group, st);
    return a.use_average ? launch_one<K, float, kBModeEval, false, true>(a, ctas, group, st)
                         : launch_one<K, float, kBModeEval, false, false>(a, ctas, group, st);
}

}  // namespace

cudaError_t launch_batch_setup(const BSub *subs, int count, BPack *packs, const float *ranges_in,
                               float *ranges_pos, int *err, cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    batch_setup_kernel<<<count, kSetupThreads, 0, stream>>>(subs, packs, ranges_in, ranges_pos, err);
    return cudaGetLastError();
}

int batch_threads(int K) { return K == 2 ? Cfg<2>::NT : (K == 3 ? Cfg<3>::NT : Cfg<4>::NT); }

int batch_group_leaves(int fp64) { return fp64 ? 8 : 16; }

int batch_dense_group() { return 9; }

size_t batch_smem_bytes(int K, int fp64, int group) {
    return fp64 ? smem_bytes<double>(group, jobs_of(K, 8)) : smem_bytes<float>(group, jobs_of(K, 4));
}

cudaError_t launch_weight_step(float *w, cudaStream_t stream) {
    weight_step_kernel<<<1, 1, 0, stream>>>(w);
    return cudaGetLastError();
}

cudaError_t launch_check_pass(int avg, const BLaunch &a, int sms, cudaStream_t stream) {
    if (a.sum_out || a.child_out || (avg && !a.avg)) return cudaErrorInvalidValue;
    if (a.count <= 0) return cudaSuccess;
    const int most = kCheckCtas * sms, ctas = a.count < most ? a.count : most;
    if (avg) check_kernel<true><<<ctas, kCheckThreads, 0, stream>>>(a);
    else check_kernel<false><<<ctas, kCheckThreads, 0, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_batch_pass(int mode, int K, int fp64, int avg, const BLaunch &a, int ctas, int group,
                              cudaStream_t stream, int dense) {
    if (group < 1 || group > kMaxGroupLeaves || ctas < 1) return cudaErrorInvalidValue;
    switch (K) {
        case 2: return launch_k<2>(mode, fp64, avg, a, ctas, group, stream, 0);
        case 3: return launch_k<3>(mode, fp64, avg, a, ctas, group, stream, 0);
        case 4: return launch_k<4>(mode, fp64, avg, a, ctas, group, stream, dense);
        default: return cudaErrorInvalidValue;
    }
}

int batch_dense_ctas_per_sm(int avg) {
    int n = 0;
    const size_t smem = smem_bytes<float>(batch_dense_group(), jobs_of(4, 4));
    cudaError_t e;
    if (avg) {
        cudaFuncSetAttribute(batch_kernel<4, float, kBModeCFR, true, false, 3>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_kernel<4, float, kBModeCFR, true, false, 3>,
                                                          Cfg<4>::NT, smem);
    } else {
        cudaFuncSetAttribute(batch_kernel<4, float, kBModeCFR, false, false, 3>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_kernel<4, float, kBModeCFR, false, false, 3>,
                                                          Cfg<4>::NT, smem);
    }
    return e == cudaSuccess ? n : 0;
}

int batch_ctas_per_sm(int mode, int K, int fp64, int avg) {
    int n = 0;
    const int group = batch_group_leaves(fp64);
    const size_t smem = batch_smem_bytes(K, fp64, group);
    cudaError_t e = cudaSuccess;
#define PRB_OCC(KK, VV, MM, AA, UU)                                                                   \
    do {                                                                                              \
        cudaFuncSetAttribute(batch_kernel<KK, VV, MM, AA, UU, Cfg<KK>::MINB>,                           \
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                 \
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_kernel<KK, VV, MM, AA, UU, Cfg<KK>::MINB>, \
                                                          Cfg<KK>::NT, smem);                         \
    } while (0)
    if (mode == kBModeCFR) {
        if (K == 2) { if (avg) PRB_OCC(2, float, kBModeCFR, true, false); else PRB_OCC(2, float, kBModeCFR, false, false); }
        else if (K == 3) { if (avg) PRB_OCC(3, float, kBModeCFR, true, false); else PRB_OCC(3, float, kBModeCFR, false, false); }
        else { if (avg) PRB_OCC(4, float, kBModeCFR, true, false); else PRB_OCC(4, float, kBModeCFR, false, false); }
    } else if (fp64) {
        if (K == 2) PRB_OCC(2, double, kBModeBR, false, false);
        else if (K == 3) PRB_OCC(3, double, kBModeBR, false, false);
        else PRB_OCC(4, double, kBModeBR, false, false);
    } else {
        if (K == 2) PRB_OCC(2, float, kBModeBR, false, false);
        else if (K == 3) PRB_OCC(3, float, kBModeBR, false, false);
        else PRB_OCC(4, float, kBModeBR, false, false);
    }
#undef PRB_OCC
    return e == cudaSuccess ? n : 0;
}

}  // namespace prb
