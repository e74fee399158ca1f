// pairs.cu — read-pair classification and NAM-pair scoring after the NAM sort.
//
// Restates gpu_pre_cal_type (step2/main.cu:3552-3580) with top_dropoff
// (main.cu:889-898) and is_proper_nam_pair (main.cu:870-887): one thread per pair
// reads the two ends' NAM counts and their first NAMs (the first two for the
// dropoff) and writes one type byte.  The bound mu + 10 sigma is computed as one
// fused multiply-add, as nvcc contracts the reference's expression.
#include <cmath>

#include "prims.cuh"
#include "runtime.h"

namespace gbsa {
namespace {

__device__ __forceinline__ float top_dropoff(const gbsa_nam* nams, uint64_t n) {
    const int h0 = nams[0].n_hits;
    if (h0 <= 2) return 1.0f;
    if (n > 1) return __fdiv_rn((float)nams[1].n_hits, (float)h0);
    return 0.0f;
}

__device__ __forceinline__ bool is_proper_nam_pair(const gbsa_nam& n1, const gbsa_nam& n2, float limit) {
    if (n1.ref_id != n2.ref_id || n1.is_rc == n2.is_rc) return false;
    const int a = max(0, n1.ref_start - n1.query_start);
    const int b = max(0, n2.ref_start - n2.query_start);
    const bool r1_r2 = n2.is_rc && (a <= b) && ((float)(b - a) < limit);
    const bool r2_r1 = n1.is_rc && (b <= a) && ((float)(a - b) < limit);
    return r1_r2 || r2_r1;
}

__global__ void k_classify_pairs(const gbsa_nam* __restrict__ nams, const uint64_t* __restrict__ offs,
                                 uint32_t n_pairs, int layout, float threshold, float limit,
                                 uint8_t* __restrict__ types) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_pairs; i += gridDim.x * blockDim.x) {
        const uint64_t r1 = layout == GBSA_PAIRS_HALVES ? i : 2ull * i;
        const uint64_t r2 = layout == GBSA_PAIRS_HALVES ? (uint64_t)i + n_pairs : 2ull * i + 1;
        const uint64_t o1 = offs[r1], c1 = offs[r1 + 1] - o1;
        const uint64_t o2 = offs[r2], c2 = offs[r2 + 1] - o2;
        uint8_t t;
        if (c1 == 0 && c2 == 0) t = 0;
        else if (c2 == 0) t = 1;
        else if (c1 == 0) t = 2;
        else if (top_dropoff(nams + o1, c1) < threshold && top_dropoff(nams + o2, c2) < threshold &&
                 is_proper_nam_pair(nams[o1], nams[o2], limit))
            t = 3;
        else t = 4;
        types[i] = t;
    }
}

// ---- NAM-pair scoring (get_best_scoring_nam_pairs_sort3, step2/main.cu:1475-1716) ----
//
// A warp per read pair.  Most pairs hold a dozen NAMs per end, but a pair inside a
// tandem repeat holds thousands and pairs every one with every other, and the kernel
// lasts as long as its heaviest pair: a thread per pair took 44.4 ms for 50k pairs of a
// repeat-rich genome, nearly all of it one thread's joint tests (with a warp, scoring,
// planning and running the steps of these pairs takes 3.5 ms together, from 47.4).  The
// kernel is bound by the latency of the heaviest pair's scans.  The lanes therefore
// take 32 mate-2 NAMs of the scan at a time, and blocks of 32 that can change nothing
// (no joint above the heap's root, no NAM left to flag) are stepped over by their
// maxima, 32 blocks at a time.  The pair's NAM fields that the scans read lie compact in
// scratch (CompactNam), its top-40 heap in shared memory, its per-NAM "in a pair" flags,
// candidate list and sort keys in scratch indexed by the pair's NAM offsets.
//
// The reference's steps are kept where their order shows: the heap takes its entries in
// the reference's order (an entry that does not beat a full heap's root changes nothing,
// so only those that may are offered), "best" is the running maximum of the joints, and
// the candidates are ranked by the final sort's comparator when it orders them all
// strictly, else sorted by the reference's quicksort steps.

constexpr int kPairWarps = 4;
constexpr uint32_t kAll = 0xFFFFFFFFu;

struct __align__(16) CompactNam {
    int diag, n_hits, ref_id, is_rc;
};

// Maxima over 32 consecutive mate-2 NAMs (those inside the scanned range): n_hits, n_hits
// of the ones not yet in a pair, diagonal.
struct __align__(16) PairBlock {
    int hits, unflagged, diag, pad;
};

// maintain_top_k (main.cu:1464-1473): a min-heap on score; sift-up stops at a
// parent of score <= the child's, sift-down takes the strictly smaller child (the
// left one on a tie)
struct NamPairHeap {
    gbsa_nam_pair h[GBSA_NAM_PAIRS_TOP_K];
    __device__ void add(int& size, const gbsa_nam_pair& p) {
        if (size < GBSA_NAM_PAIRS_TOP_K) {
            int i = size++;
            h[i] = p;
            while (i > 0) {
                const int up = (i - 1) / 2;
                if (h[up].score <= h[i].score) break;
                const gbsa_nam_pair t = h[up];
                h[up] = h[i];
                h[i] = t;
                i = up;
            }
        } else if (p.score > h[0].score) {
            h[0] = p;
            int i = 0;
            while (2 * i + 1 < size) {
                int sm = i;
                const int l = 2 * i + 1, r = l + 1;
                if (l < size && h[l].score < h[sm].score) sm = l;
                if (r < size && h[r].score < h[sm].score) sm = r;
                if (sm == i) break;
                const gbsa_nam_pair t = h[i];
                h[i] = h[sm];
                h[sm] = t;
                i = sm;
            }
        }
    }
};

// The warp's heap: storage in shared memory, size and root alike in every lane.
struct WarpHeap {
    NamPairHeap* H;
    int size, root;
    __device__ __forceinline__ bool full() const { return size == GBSA_NAM_PAIRS_TOP_K; }
    __device__ __forceinline__ bool takes(int score) const { return !full() || score > root; }
    // Offers the entries of the lanes with `want`, in lane order (calls that would leave a
    // full heap as it is are left out).
    __device__ void offer(bool want, const gbsa_nam_pair& p) {
        uint32_t m = __ballot_sync(kAll, want && takes(p.score));
        while (m) {
            const uint32_t src = __ffs(m) - 1;
            gbsa_nam_pair x;
            x.score = __shfl_sync(kAll, p.score, src);
            x.i1 = __shfl_sync(kAll, p.i1, src);
            x.i2 = __shfl_sync(kAll, p.i2, src);
            int n = size;
            if (lane_id() == 0) H->add(n, x);
            __syncwarp();
            size = __shfl_sync(kAll, n, 0);
            root = H->h[0].score;
            m = __ballot_sync(kAll, want && lane_id() > src && takes(p.score));
        }
    }
};

__device__ __forceinline__ int nam_diagonal(const gbsa_nam& n) { return max(0, n.ref_start - n.query_start); }

// The final sort's comparator (main.cu:1674-1713); an absent end is an all-zero NAM
// with ref_start -1.
__device__ bool nam_pair_before(const gbsa_nam_pair& a, const gbsa_nam_pair& b, const gbsa_nam* n1,
                                const gbsa_nam* n2) {
    gbsa_nam none;
    none.nam_id = none.query_start = none.query_end = none.query_prev_hit_startpos = 0;
    none.ref_end = none.ref_prev_hit_startpos = none.n_hits = none.ref_id = 0;
    none.ref_start = -1;
    none.score = 0.0f;
    none.is_rc = 0;
    const gbsa_nam& a1 = a.i1 < 0 ? none : n1[a.i1];
    const gbsa_nam& a2 = a.i2 < 0 ? none : n2[a.i2];
    const gbsa_nam& b1 = b.i1 < 0 ? none : n1[b.i1];
    const gbsa_nam& b2 = b.i2 < 0 ? none : n2[b.i2];
    if (a.score != b.score) return a.score > b.score;
    if (a1.score != b1.score) return a1.score > b1.score;
    if (a1.is_rc != b1.is_rc) return !a1.is_rc;
    if (a1.query_end != b1.query_end) return a1.query_end < b1.query_end;
    if (a1.query_start != b1.query_start) return a1.query_start < b1.query_start;
    if (a1.ref_end != b1.ref_end) return a1.ref_end < b1.ref_end;
    if (a1.ref_start != b1.ref_start) return a1.ref_start < b1.ref_start;
    if (a2.score != b2.score) return a2.score > b2.score;
    if (a2.is_rc != b2.is_rc) return !a2.is_rc;
    if (a2.query_end != b2.query_end) return a2.query_end < b2.query_end;
    if (a2.query_start != b2.query_start) return a2.query_start < b2.query_start;
    if (a2.ref_end != b2.ref_end) return a2.ref_end < b2.ref_end;
    return a2.ref_start < b2.ref_start;
}

__device__ __forceinline__ int warp_max(int v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(kAll, v, o));
    return v;
}

// First index in [from, to) whose NAM fails `keep`, or to.
template <class Keep>
__device__ __forceinline__ int warp_first_not(const CompactNam* n, int from, int to, Keep&& keep) {
    for (int b = from; b < to; b += 32) {
        const int j = b + (int)lane_id();
        const uint32_t m = __ballot_sync(kAll, j < to && !keep(n[j]));
        if (m) return b + __ffs(m) - 1;
    }
    return to;
}

struct PairState {
    WarpHeap heap;
    uint8_t *add1, *add2;
    PairBlock* blocks;
    int best;
};

// Mate-1 NAM i (n_hits h1, diagonal d1) against 32 mate-2 NAMs, one per lane (valid: in
// the scanned range; d2, h2: its diagonal and n_hits; j: its index).  Returns whether
// the scan ends inside these 32.  flag1: whether i is in a pair.
__device__ __forceinline__ bool pair_block(PairState& S, int i, int h1, int d1, bool fwd1, int span, bool valid, int j,
                                           int d2, int h2, bool& flag1) {
    const bool out = valid && (fwd1 ? d2 >= d1 + span : d2 > d1);
    const uint32_t mo = __ballot_sync(kAll, out);
    const bool in = valid && (mo == 0 || (int)lane_id() < __ffs(mo) - 1);
    const int joint = in ? h1 + h2 : -0x7FFFFFFF;
    int before = S.best;   // the running maximum ahead of this lane's NAM
    if (__any_sync(kAll, in && joint > S.best)) {
        int pm = joint;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kAll, pm, o);
            if ((int)lane_id() >= o) pm = max(pm, v);
        }
        const int ex = __shfl_up_sync(kAll, pm, 1);
        if (lane_id() > 0) before = max(before, ex);
        S.best = max(S.best, __shfl_sync(kAll, pm, 31));
    }
    const bool take = in && joint >= before / 2;
    if (take) S.add2[j] = 1;
    if (__any_sync(kAll, take)) flag1 = true;
    gbsa_nam_pair np;
    np.score = joint;
    np.i1 = i;
    np.i2 = j;
    S.heap.offer(take, np);
    return mo != 0;
}

// One strand combination of the pairing, one reference id at a time (ids below
// 3000, main.cu:1520-1570 and 1573-1623).  fwd1: mate 1 on the forward strand, mate 2's
// diagonal in [d1, d1 + span); else mate 2's diagonal in (d1 - span, d1].
__device__ void pair_pass(const CompactNam* n1, int b1, int e1, const CompactNam* n2, int b2, int e2, bool fwd1,
                          int span, PairState& S) {
    const int lane = (int)lane_id();
    int p1 = b1, p2 = b2;
    for (int ref = 0; ref < 3000; ++ref) {
        p1 = warp_first_not(n1, p1, e1, [&](const CompactNam& x) { return x.ref_id < ref; });
        p2 = warp_first_not(n2, p2, e2, [&](const CompactNam& x) { return x.ref_id < ref; });
        if (p1 == e1 || p2 == e2) break;
        const int r1 = n1[p1].ref_id, r2 = n2[p2].ref_id;
        if (r1 != ref || r2 != ref) {
            ref = max(r1, r2) - 1;   // ids in between pair nothing
            if (r1 != r2) continue;
            if (++ref >= 3000) break;
        }
        const int q1 = warp_first_not(n1, p1, e1, [&](const CompactNam& x) { return x.ref_id == ref; });
        const int q2 = warp_first_not(n2, p2, e2, [&](const CompactNam& x) { return x.ref_id == ref; });
        const int len2 = q2 - p2;
        // the range's first 32 mate-2 NAMs stay in registers; a longer range gets the maxima
        // of its blocks of 32 (block c: [p2 + 32 c, + 32))
        const bool valid0 = lane < len2;
        const CompactNam m0 = valid0 ? n2[p2 + lane] : CompactNam{0, 0, 0, 0};
        int best2 = -1;
        bool sorted = true;   // by diagonal, as the sort order leaves them
        int prev = -0x7FFFFFFF - 1;
        for (int c = 0; 32 * c < len2; ++c) {
            const int j = p2 + 32 * c + lane;
            const bool valid = j < q2;
            const CompactNam m = c == 0 ? m0 : (valid ? n2[j] : CompactNam{0, 0, 0, 0});
            const int up = __shfl_up_sync(kAll, m.diag, 1);
            sorted &= !__any_sync(kAll, valid && m.diag < (lane ? up : prev));
            prev = __shfl_sync(kAll, m.diag, 31);
            const int hits = warp_max(valid ? m.n_hits : -0x7FFFFFFF);
            best2 = max(best2, hits);
            if (len2 > 32) {
                const int unfl = warp_max(valid && !S.add2[j] ? m.n_hits : -0x3FFFFFFF);
                const int dg = warp_max(valid ? m.diag : -0x7FFFFFFF - 1);
                if (lane == 0) S.blocks[c] = PairBlock{hits, unfl, dg, 0};
            }
        }
        __syncwarp();
        const int nblk = (len2 + 31) >> 5;
        bool done = false;
        for (int ib = p1; ib < q1 && !done; ib += 32) {
            const CompactNam mine = ib + lane < q1 ? n1[ib + lane] : CompactNam{0, 0, 0, 0};
            const int ni = min(32, q1 - ib);
            for (int t = 0; t < ni; ++t) {
                const int i = ib + t;
                const int h1 = __shfl_sync(kAll, mine.n_hits, t), d1 = __shfl_sync(kAll, mine.diag, t);
                const int round_best = h1 + best2;
                if (round_best < S.best / 2 || (S.heap.full() && round_best < S.heap.root)) {
                    done = true;
                    break;
                }
                // first mate-2 NAM inside the window
                auto inside = [&](int d) { return fwd1 ? d >= d1 : d > d1 - span; };
                int at = q2;
                if (!sorted) {
                    int lo = p2, hi = q2 - 1;
                    while (lo <= hi) {
                        const int mid = (lo + hi) / 2;
                        if (inside(n2[mid].diag)) {
                            at = mid;
                            hi = mid - 1;
                        } else {
                            lo = mid + 1;
                        }
                    }
                } else if (len2 <= 32) {
                    const uint32_t m = __ballot_sync(kAll, valid0 && inside(m0.diag));
                    if (m) at = p2 + __ffs(m) - 1;
                } else {
                    for (int cb = 0; cb < nblk; cb += 32) {
                        const uint32_t m = __ballot_sync(kAll, cb + lane < nblk && inside(S.blocks[cb + lane].diag));
                        if (!m) continue;
                        const int j = p2 + 32 * (cb + __ffs(m) - 1) + lane;
                        const uint32_t mj = __ballot_sync(kAll, j < q2 && inside(n2[j].diag));
                        at = j - lane + __ffs(mj) - 1;
                        break;
                    }
                }
                if (at == q2) continue;
                bool flag1 = false;
                if (len2 <= 32) {
                    pair_block(S, i, h1, d1, fwd1, span, valid0 && p2 + lane >= at, p2 + lane, m0.diag, m0.n_hits,
                               flag1);
                } else {
                    bool stop = false;
                    for (int cb = (at - p2) >> 5; cb < nblk && !stop; cb += 32) {
                        const bool have = cb + lane < nblk;
                        const PairBlock B = have ? S.blocks[cb + lane] : PairBlock{0, 0, 0, 0};
                        // whether the block can change anything, or end the scan
                        auto needs = [&] {
                            const int top = B.hits + h1, half = S.best / 2;
                            return have && ((fwd1 ? B.diag >= d1 + span : B.diag > d1) || B.unflagged + h1 >= half ||
                                            (top >= half && (!flag1 || S.heap.takes(top))));
                        };
                        uint32_t m = __ballot_sync(kAll, needs());
                        while (m) {
                            const int src = __ffs(m) - 1;
                            const int c = cb + src, j = p2 + 32 * c + lane;
                            const bool valid = j < q2;
                            const CompactNam x = valid ? n2[j] : CompactNam{0, 0, 0, 0};
                            stop = pair_block(S, i, h1, d1, fwd1, span, valid && j >= at, j, x.diag, x.n_hits, flag1);
                            __syncwarp();
                            const int unfl = warp_max(valid && !S.add2[j] ? x.n_hits : -0x3FFFFFFF);
                            if (lane == 0) S.blocks[c].unflagged = unfl;
                            if (stop) break;
                            m = __ballot_sync(kAll, lane > src && needs());
                        }
                        __syncwarp();
                    }
                }
                if (flag1 && lane == 0) S.add1[i] = 1;
            }
        }
        __syncwarp();
    }
}

// Sort key of a list entry: the comparator's first two fields (score and mate 1's NAM
// score, both descending).
__device__ __forceinline__ uint64_t nam_pair_key(const gbsa_nam_pair& p, const gbsa_nam* n1, bool& nan) {
    const float f = (p.i1 < 0 ? 0.0f : n1[p.i1].score) + 0.0f;   // -0 compares as 0
    nan |= f != f;
    uint32_t u = __float_as_uint(f);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    return ((uint64_t)(~((uint32_t)p.score ^ 0x80000000u)) << 32) | (~u);
}

__global__ void __launch_bounds__(32 * kPairWarps)
    k_nam_pairs(const gbsa_nam* __restrict__ nams, const uint64_t* __restrict__ offs, uint32_t n_pairs, int layout,
                int span, uint32_t max_tries, uint8_t* flags, CompactNam* compact, PairBlock* blocks,
                gbsa_nam_pair* lists, int* stacks, gbsa_nam_pair* __restrict__ out, uint32_t* __restrict__ counts) {
    __shared__ NamPairHeap s_heap[kPairWarps];
    const int lane = (int)lane_id();
    const uint32_t w = threadIdx.x >> 5;
    const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t p = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < n_pairs; p += warps) {
        const uint64_t r1 = layout == GBSA_PAIRS_HALVES ? p : 2ull * p;
        const uint64_t r2 = layout == GBSA_PAIRS_HALVES ? p + n_pairs : 2ull * p + 1;
        const uint64_t o1 = offs[r1], o2 = offs[r2];
        const int c1 = (int)(offs[r1 + 1] - o1), c2 = (int)(offs[r2 + 1] - o2);
        if (c1 == 0 || c2 == 0) {
            if (lane == 0) counts[p] = 0;
            continue;
        }
        const gbsa_nam* n1 = nams + o1;
        const gbsa_nam* n2 = nams + o2;
        uint8_t* add1 = flags + o1;
        uint8_t* add2 = flags + o2;
        CompactNam* k1 = compact + o1;
        CompactNam* k2 = compact + o2;
        auto pack = [&](const gbsa_nam* n, int c, CompactNam* k, uint8_t* add) {
            int mid = c;   // first reverse-strand NAM
            for (int b = 0; b < c; b += 32) {
                const int i = b + lane;
                bool rc = false;
                if (i < c) {
                    const gbsa_nam& x = n[i];
                    rc = x.is_rc == 1;
                    k[i] = CompactNam{nam_diagonal(x), x.n_hits, x.ref_id, (int)x.is_rc};
                    add[i] = 0;
                }
                const uint32_t m = __ballot_sync(kAll, rc);
                if (m && mid == c) mid = b + __ffs(m) - 1;
            }
            return mid;
        };
        const int mid1 = pack(n1, c1, k1, add1), mid2 = pack(n2, c2, k2, add2);
        __syncwarp();
        PairState S;
        S.heap.H = &s_heap[w];
        S.heap.size = 0;
        S.heap.root = 0;
        S.add1 = add1;
        S.add2 = add2;
        S.blocks = blocks + (o2 >> 5) + r2;   // room for the list's blocks of 32
        S.best = 0;
        pair_pass(k1, 0, mid1, k2, mid2, c2, true, span, S);
        pair_pass(k1, mid1, c1, k2, 0, mid2, false, span, S);
        // the pair's list: room for its mate-1 NAMs and the heap
        const uint64_t base = o1 + (uint64_t)GBSA_NAM_PAIRS_TOP_K * p;
        gbsa_nam_pair* list = lists + base;
        int len = 0;
        auto most_hits = [&](const CompactNam* k, int c) {
            int v = 0;
            for (int i = lane; i < c; i += 32) v = max(v, k[i].n_hits);
            return warp_max(v);
        };
        const int half1 = (S.best ? S.best : most_hits(k1, c1)) / 2;
        int run_start = 0, prev = k1[0].ref_id + 3000 * k1[0].is_rc;
        for (int b = 0; b < c1; b += 32) {   // mate-1 NAMs in no pair, max_tries per (reference, strand)
            const int i = b + lane;
            const CompactNam x = k1[min(i, c1 - 1)];
            const int key = x.ref_id + 3000 * x.is_rc;
            const int up = __shfl_up_sync(kAll, key, 1);
            const uint32_t heads = __ballot_sync(kAll, i < c1 && key != (lane ? up : prev));
            const uint32_t mine = heads & (0xFFFFFFFFu >> (31 - lane));   // heads at or below this lane
            const int start = mine ? b + 31 - __clz(mine) : run_start;
            const bool take = i < c1 && i - start + 1 <= (int)max_tries && x.n_hits >= half1 && !add1[i];
            const uint32_t m = __ballot_sync(kAll, take);
            if (take) {
                gbsa_nam_pair np;
                np.score = x.n_hits;
                np.i1 = i;
                np.i2 = -1;
                list[len + __popc(m & lanemask_lt())] = np;
            }
            len += __popc(m);
            run_start = __shfl_sync(kAll, start, 31);
            prev = __shfl_sync(kAll, key, 31);
        }
        const int half2 = (S.best ? S.best : most_hits(k2, c2)) / 2;
        for (int b = 0; b < c2; b += 32) {   // mate-2 NAMs in no pair, through the heap
            const int i = b + lane;
            const int h = i < c2 ? k2[i].n_hits : 0;
            gbsa_nam_pair np;
            np.score = h;
            np.i1 = -1;
            np.i2 = i;
            S.heap.offer(i < c2 && h >= half2 && !add2[min(i, c2 - 1)], np);
        }
        for (int i = lane; i < S.heap.size; i += 32) list[len + i] = s_heap[w].h[i];
        len += S.heap.size;
        const uint32_t k = min((uint32_t)len, max_tries);
        gbsa_nam_pair* to = out + p * max_tries;
        __syncwarp();
        // rank of every entry by the comparator; entries it does not order need the
        // reference's steps, so the ranking ends at the first such (the thousands of copies'
        // NAMs of reads in repeats: 2,000 pairs of 764 NAMs an end, nearly all time in those
        // steps, took 1,034 ms with the ranks of all, 929 with a thread a pair, now 697)
        uint64_t* keys = reinterpret_cast<uint64_t*>(stacks + 2 * base);
        bool tie = false;
        for (int i = lane; i < len; i += 32) keys[i] = nam_pair_key(list[i], n1, tie);
        __syncwarp();
        tie = __any_sync(kAll, tie);
        for (int b = 0; b < len && !tie; b += 32) {
            const int e = b + lane;
            const uint64_t ke = e < len ? keys[e] : 0;   // (no key is below 0 or equal to it)
            const gbsa_nam_pair pe = list[min(e, len - 1)];
            uint32_t rank = 0;
            for (int c = 0; c < len && !tie; c += 1024) {
                const int end = min(c + 1024, len);
                for (int f = c; f < end; ++f) {
                    const uint64_t kf = keys[f];
                    if (kf < ke) {
                        ++rank;
                    } else if (kf == ke && f != e) {
                        const gbsa_nam_pair pf = list[f];
                        if (nam_pair_before(pf, pe, n1, n2)) ++rank;
                        else tie |= !nam_pair_before(pe, pf, n1, n2);
                    }
                }
                tie = __any_sync(kAll, tie);
            }
            if (e < len && rank < k) to[rank] = pe;
        }
        __syncwarp();
        if (tie && lane == 0) {
            // quick_sort_iterative (main.cu:317-358): Lomuto partition around the last
            // element, ranges on an explicit stack (left part pushed first)
            int* st = stacks + 2 * base;
            int top = -1;
            st[++top] = 0;
            st[++top] = len - 1;
            while (top >= 0) {
                const int hi = st[top--];
                const int lo = st[top--];
                const gbsa_nam_pair pivot = list[hi];
                int i = lo - 1;
                for (int j = lo; j < hi; ++j)
                    if (nam_pair_before(list[j], pivot, n1, n2)) {
                        ++i;
                        const gbsa_nam_pair t = list[i];
                        list[i] = list[j];
                        list[j] = t;
                    }
                const gbsa_nam_pair t = list[i + 1];
                list[i + 1] = list[hi];
                list[hi] = t;
                const int pv = i + 1;
                if (pv - 1 > lo) {
                    st[++top] = lo;
                    st[++top] = pv - 1;
                }
                if (pv + 1 < hi) {
                    st[++top] = pv + 1;
                    st[++top] = hi;
                }
            }
            for (uint32_t i = 0; i < k; ++i) to[i] = list[i];
        }
        if (lane == 0) counts[p] = k;
        __syncwarp();
    }
}

}  // namespace
}  // namespace gbsa

using namespace gbsa;

extern "C" int gbsa_nam_pairs_device(const gbsa_nam* d_nams, const uint64_t* d_nam_offsets, uint32_t n_pairs,
                                     int layout, float mu, float sigma, uint32_t max_tries, gbsa_nam_pair* d_pairs,
                                     uint32_t* d_counts, void* stream) {
    try {
        if (layout != GBSA_PAIRS_INTERLEAVED && layout != GBSA_PAIRS_HALVES)
            throw Error(GBSA_ERR_PARAM, "layout must be GBSA_PAIRS_INTERLEAVED or GBSA_PAIRS_HALVES");
        if (max_tries == 0) throw Error(GBSA_ERR_PARAM, "max_tries must be at least 1");
        if (n_pairs == 0) return GBSA_OK;
        cudaStream_t st = (cudaStream_t)stream;
        // scratch: a flag and a compact copy per NAM, block maxima per 32 NAMs of a read, and
        // per pair a list and sort keys (or a quicksort stack) with room for its mate-1
        // NAMs plus the heap
        uint64_t total = 0;
        GBSA_CUDA(cudaMemcpyAsync(&total, d_nam_offsets + 2ull * n_pairs, 8, cudaMemcpyDeviceToHost, st));
        GBSA_CUDA(cudaStreamSynchronize(st));
        const uint64_t slots = total + (uint64_t)GBSA_NAM_PAIRS_TOP_K * n_pairs + 1;
        // scratch in stream order (cudaMalloc / cudaFree would wait for the whole device,
        // other callers' work included)
        auto pad = [](size_t b) { return (b + 255) & ~size_t(255); };
        const size_t b_flags = pad(total + 1), b_compact = pad(sizeof(CompactNam) * (total + 1));
        const size_t b_blocks = pad(sizeof(PairBlock) * ((total >> 5) + 2ull * n_pairs + 2));
        const size_t b_lists = pad(sizeof(gbsa_nam_pair) * slots);
        uint8_t* scratch = static_cast<uint8_t*>(scratch_alloc(b_flags + b_compact + b_blocks + b_lists + 8 * slots, st));
        uint8_t* s_compact = scratch + b_flags;
        uint8_t* s_blocks = s_compact + b_compact;
        uint8_t* s_lists = s_blocks + b_blocks;
        const int span = (int)mu + 10 * (int)sigma;
        // a block for every kPairWarps pairs: the block scheduler evens out heavy pairs
        k_nam_pairs<<<grid_for(n_pairs, kPairWarps), 32 * kPairWarps, 0, st>>>(
            d_nams, d_nam_offsets, n_pairs, layout, span, max_tries, scratch,
            reinterpret_cast<CompactNam*>(s_compact), reinterpret_cast<PairBlock*>(s_blocks),
            reinterpret_cast<gbsa_nam_pair*>(s_lists), reinterpret_cast<int*>(s_lists + b_lists), d_pairs, d_counts);
        const cudaError_t launch = cudaGetLastError();
        scratch_free(scratch, st);
        GBSA_CUDA(launch);
        GBSA_LAUNCHED();
        return GBSA_OK;
    } catch (const Error& e) {
        set_last_error(e.what());
        return e.code;
    } catch (const std::exception& e) {
        set_last_error(e.what());
        return GBSA_ERR_CUDA;
    }
}

extern "C" int gbsa_classify_pairs_device(const gbsa_nam* d_nams, const uint64_t* d_nam_offsets, uint32_t n_pairs,
                                          int layout, float dropoff_threshold, float mu, float sigma,
                                          uint8_t* d_types, void* stream) {
    try {
        if (layout != GBSA_PAIRS_INTERLEAVED && layout != GBSA_PAIRS_HALVES)
            throw Error(GBSA_ERR_PARAM, "layout must be GBSA_PAIRS_INTERLEAVED or GBSA_PAIRS_HALVES");
        if (n_pairs == 0) return GBSA_OK;
        const float limit = std::fma(10.0f, sigma, mu);
        k_classify_pairs<<<grid_for(n_pairs, 256, (unsigned)device_sm_count() * 8), 256, 0, (cudaStream_t)stream>>>(
            d_nams, d_nam_offsets, n_pairs, layout, dropoff_threshold, limit, d_types);
        GBSA_LAUNCHED();
        return GBSA_OK;
    } catch (const Error& e) {
        set_last_error(e.what());
        return e.code;
    } catch (const std::exception& e) {
        set_last_error(e.what());
        return GBSA_ERR_CUDA;
    }
}

// ---- alignment orchestration (align_PE_part0..4, step2/main.cu:1857-2165) ---------------
//
// A warp per read pair lists, in the order the reference's align_PE_part<type> runs
// them, the seed extensions (extend_seed_part after reverse_nam_if_needed) and mate
// rescues (rescue_mate_part of a NAM after reverse_nam_if_needed) of the pair, and
// computes the pair's mapq for type 3 (get_mapq, main.cu:900-910).  Two passes: the
// first counts each pair's steps, an exclusive scan places them, the second writes them.

namespace gbsa {
namespace {

__device__ __forceinline__ void plan_push(gbsa_align_step* out, uint32_t& k, bool write, uint32_t pair, uint8_t kind,
                                          bool is_read1, uint64_t read, uint64_t nam_read, uint32_t nam) {
    if (write) {
        gbsa_align_step s;
        s.pair = pair;
        s.read = (uint32_t)read;
        s.nam_read = (uint32_t)nam_read;
        s.nam = nam;
        s.kind = kind;
        s.is_read1 = is_read1 ? 1 : 0;
        s._pad[0] = s._pad[1] = 0;
        out[k] = s;
    }
    ++k;
}

// get_mapq (main.cu:900-910): the reference's float expression — min_matches is a float
// rounded from the double n_hits / 10.0 (capped at 1), the log is logf of the float
// score, the products are float in the reference's order — truncated to int, capped at
// 60 and returned as uint8 (a negative value wraps, as the reference's return type makes
// it).
__device__ __forceinline__ uint8_t pair_mapq(const gbsa_nam* nams, uint64_t n) {
    if (n <= 1) return 60;
    const float s1 = nams[0].score, s2 = nams[1].score;
    const double mm = nams[0].n_hits / 10.0;
    const float min_matches = (float)(mm < 1.0 ? mm : 1.0);
    const float f = __fmul_rn(__fmul_rn(__fmul_rn(40.0f, __fsub_rn(1.0f, __fdiv_rn(s2, s1))), min_matches), logf(s1));
    const int uncapped = (int)f;
    return (uint8_t)(uncapped < 60 ? uncapped : 60);
}

// rescue_read_part (main.cu:795-835): the NAMs of the mapped end in order while fewer than
// max_tries were tried and n_hits / the first NAM's n_hits >= dropoff; each is extended on
// its read, then its mate is rescued from it.  The lanes take 32 NAMs at a time.
__device__ void plan_rescue_read(gbsa_align_step* out, uint32_t& k, bool write, uint32_t p, const gbsa_nam* nams,
                                 uint64_t n, uint64_t mapped, uint64_t mate, bool mapped_is_read1, uint32_t max_tries,
                                 float dropoff) {
    const int top = nams[0].n_hits;
    for (uint64_t b = 0; b < n; b += 32) {
        const uint64_t i = b + lane_id();
        bool stop = true;
        if (i < n) {
            const float d = (float)nams[i].n_hits / (float)top;
            stop = i >= max_tries || d < dropoff;
        }
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, stop);
        const uint32_t tried = m ? __ffs(m) - 1 : 32u;
        if (lane_id() < tried) {
            uint32_t at = k + 2 * lane_id();
            plan_push(out, at, write, p, GBSA_STEP_EXTEND, mapped_is_read1, mapped, mapped, (uint32_t)i);
            plan_push(out, at, write, p, GBSA_STEP_RESCUE, !mapped_is_read1, mate, mapped, (uint32_t)i);
        }
        k += 2 * tried;
        if (m) return;
    }
}

// Index of the first of the largest scores among n > 0 NAMs.
__device__ uint32_t warp_best_score(const gbsa_nam* nams, uint64_t n) {
    float s = nams[0].score;
    uint32_t at = 0;
    for (uint64_t i = lane_id(); i < n; i += 32) {
        const float v = nams[i].score;
        if (v > s) {
            s = v;
            at = (uint32_t)i;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float v = __shfl_xor_sync(0xFFFFFFFFu, s, o);
        const uint32_t a = __shfl_xor_sync(0xFFFFFFFFu, at, o);
        if (v > s || (v == s && a < at)) {
            s = v;
            at = a;
        }
    }
    return at;
}

// A warp per pair (a thread per pair took 1.28 ms for 50k pairs: one thread searching the
// thousands of NAMs of a read in a tandem repeat for its best score).  The joint pairs are
// taken 32 at a time; a NAM is extended at its first appearance, found by comparing the
// pairs' NAM indices with one another instead of through a flag per NAM.
template <bool kWrite>
__global__ void __launch_bounds__(32 * kPairWarps)
    k_plan_pairs(const gbsa_nam* __restrict__ nams, const uint64_t* __restrict__ offs, uint32_t n_pairs, int layout,
                 const uint8_t* __restrict__ types, const gbsa_nam_pair* __restrict__ jp,
                 const uint32_t* __restrict__ jcounts, uint32_t max_tries, float dropoff,
                 uint64_t* __restrict__ counts, gbsa_pair_plan* __restrict__ plans,
                 gbsa_align_step* __restrict__ steps, uint64_t step_cap, unsigned int* bad) {
    const uint32_t lane = lane_id();
    const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t p64 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; p64 < n_pairs; p64 += warps) {
        const uint32_t p = (uint32_t)p64;
        const uint64_t e1 = layout == GBSA_PAIRS_HALVES ? p : 2ull * p;
        const uint64_t e2 = layout == GBSA_PAIRS_HALVES ? (uint64_t)p + n_pairs : 2ull * p + 1;
        const uint64_t o1 = offs[e1], c1 = offs[e1 + 1] - o1;
        const uint64_t o2 = offs[e2], c2 = offs[e2 + 1] - o2;
        const gbsa_nam* n1 = nams + o1;
        const gbsa_nam* n2 = nams + o2;
        const uint8_t type = types[p];
        uint64_t first = 0;
        gbsa_align_step* out = steps;
        bool write = false;
        if (kWrite) {
            first = counts[p];
            write = first + (counts[p + 1] - first) <= step_cap;
            out = steps + first;
        }
        uint32_t k = 0;
        gbsa_pair_plan plan;
        plan.type = type;
        plan.mapq1 = plan.mapq2 = 0;
        plan._pad = 0;
        plan.type4_loop_size = 0;
        if (type == 1 && c1 > 0) {
            plan_rescue_read(out, k, write, p, n1, c1, e1, e2, true, max_tries, dropoff);
        } else if (type == 2 && c2 > 0) {
            plan_rescue_read(out, k, write, p, n2, c2, e2, e1, false, max_tries, dropoff);
        } else if ((type == 3 || type == 4) && c1 > 0 && c2 > 0) {
            // type 3: the ends' first NAMs; type 4: the best-scoring NAM of each end first
            const uint32_t b1 = type == 3 ? 0 : warp_best_score(n1, c1);
            const uint32_t b2 = type == 3 ? 0 : warp_best_score(n2, c2);
            uint32_t at = 0;
            plan_push(out, at, write && lane == 0, p, GBSA_STEP_EXTEND, true, e1, e1, b1);
            plan_push(out, at, write && lane == 0, p, GBSA_STEP_EXTEND, false, e2, e2, b2);
            k = 2;
            if (type == 3) {
                plan.mapq1 = pair_mapq(n1, c1);
                plan.mapq2 = pair_mapq(n2, c2);
            } else {
                const uint32_t nj = jcounts[p];
                const gbsa_nam_pair* J = jp + (uint64_t)p * max_tries;
                const double max_score = nj ? (double)J[0].score : 0.0;
                for (uint32_t b = 0; b < nj; b += 32) {
                    const uint32_t i = b + lane;
                    bool stop = true;
                    gbsa_nam_pair x{0, -1, -1};
                    if (i < nj && i < max_tries) {
                        x = J[i];
                        stop = (float)((double)x.score / max_score) < dropoff;
                    }
                    const uint32_t m = __ballot_sync(0xFFFFFFFFu, stop);
                    const uint32_t taken = m ? __ffs(m) - 1 : 32u;
                    const bool in = lane < taken;
                    const bool have1 = in && x.i1 >= 0 && (uint64_t)x.i1 < c1;
                    const bool have2 = in && x.i2 >= 0 && (uint64_t)x.i2 < c2;
                    // NAMs not aligned yet: neither an end's best nor in an earlier pair
                    const uint32_t same1 = __match_any_sync(0xFFFFFFFFu, have1 ? x.i1 : -1);
                    const uint32_t same2 = __match_any_sync(0xFFFFFFFFu, have2 ? x.i2 : -1);
                    bool new1 = have1 && (uint32_t)x.i1 != b1 && (same1 & lanemask_lt()) == 0;
                    bool new2 = have2 && (uint32_t)x.i2 != b2 && (same2 & lanemask_lt()) == 0;
                    for (uint32_t e = 0; e < b; ++e) {
                        new1 = new1 && J[e].i1 != x.i1;
                        new2 = new2 && J[e].i2 != x.i2;
                    }
                    const bool first_step = have1 ? new1 : have2;    // extend i1, or rescue mate 1 from i2
                    const bool second_step = have2 ? new2 : have1;   // extend i2, or rescue mate 2 from i1
                    const uint32_t f1 = __ballot_sync(0xFFFFFFFFu, first_step);
                    const uint32_t f2 = __ballot_sync(0xFFFFFFFFu, second_step);
                    uint32_t to = k + __popc(f1 & lanemask_lt()) + __popc(f2 & lanemask_lt());
                    if (first_step) {
                        if (have1) plan_push(out, to, write, p, GBSA_STEP_EXTEND, true, e1, e1, (uint32_t)x.i1);
                        else plan_push(out, to, write, p, GBSA_STEP_RESCUE, true, e1, e2, (uint32_t)x.i2);
                    }
                    if (second_step) {
                        if (have2) plan_push(out, to, write, p, GBSA_STEP_EXTEND, false, e2, e2, (uint32_t)x.i2);
                        else plan_push(out, to, write, p, GBSA_STEP_RESCUE, false, e2, e1, (uint32_t)x.i1);
                    }
                    // a pair entry with neither NAM: not produced by the pair scoring
                    if (bad && in && !have1 && !have2) atomicAdd(bad, 1u);
                    k += __popc(f1) + __popc(f2);
                    plan.type4_loop_size += (int)taken;
                    if (m) break;
                }
            }
        }
        if (lane == 0) {
            if (!kWrite) {
                counts[p] = k;
            } else {
                plan.first_step = (uint32_t)first;
                plan.n_steps = k;
                plans[p] = plan;
            }
        }
    }
}

}  // namespace
}  // namespace gbsa

using namespace gbsa;

extern "C" int gbsa_plan_pairs_device(const gbsa_nam* d_nams, const uint64_t* d_nam_offsets, uint32_t n_pairs,
                                      int layout, const uint8_t* d_types, const gbsa_nam_pair* d_pairs,
                                      const uint32_t* d_pair_counts, uint32_t max_tries, float dropoff,
                                      gbsa_pair_plan* d_plans, gbsa_align_step* d_steps, uint64_t step_capacity,
                                      uint64_t* n_steps, void* stream) {
    try {
        if (layout != GBSA_PAIRS_INTERLEAVED && layout != GBSA_PAIRS_HALVES)
            throw Error(GBSA_ERR_PARAM, "layout must be GBSA_PAIRS_INTERLEAVED or GBSA_PAIRS_HALVES");
        if (max_tries == 0) throw Error(GBSA_ERR_PARAM, "max_tries must be at least 1");
        if (n_steps) *n_steps = 0;
        if (n_pairs == 0) return GBSA_OK;
        cudaStream_t st = (cudaStream_t)stream;
        // scratch in stream order: step counts (then offsets) per pair, the status word
        const size_t b_cnt = (8ull * (n_pairs + 1) + 255) & ~size_t(255);
        uint8_t* scratch = static_cast<uint8_t*>(scratch_alloc(b_cnt + 256, st));
        uint64_t* counts = reinterpret_cast<uint64_t*>(scratch);
        unsigned int* bad = reinterpret_cast<unsigned int*>(scratch + b_cnt);
        struct Free {
            uint8_t* p;
            cudaStream_t s;
            ~Free() { scratch_free(p, s); }
        } release{scratch, st};
        GBSA_CUDA(cudaMemsetAsync(bad, 0, 4, st));
        const unsigned grid = grid_for(n_pairs, kPairWarps), block = 32 * kPairWarps;
        k_plan_pairs<false><<<grid, block, 0, st>>>(d_nams, d_nam_offsets, n_pairs, layout, d_types, d_pairs,
                                                    d_pair_counts, max_tries, dropoff, counts, nullptr, nullptr, 0,
                                                    nullptr);
        GBSA_LAUNCHED();
        Workspace ws(st);
        scan_exclusive_u64(counts, counts, n_pairs, counts + n_pairs, ws, st);
        k_plan_pairs<true><<<grid, block, 0, st>>>(d_nams, d_nam_offsets, n_pairs, layout, d_types, d_pairs,
                                                   d_pair_counts, max_tries, dropoff, counts, d_plans, d_steps,
                                                   step_capacity, bad);
        GBSA_LAUNCHED();
        uint64_t total = 0;
        unsigned int h_bad = 0;
        GBSA_CUDA(cudaMemcpyAsync(&total, counts + n_pairs, 8, cudaMemcpyDeviceToHost, st));
        GBSA_CUDA(cudaMemcpyAsync(&h_bad, bad, 4, cudaMemcpyDeviceToHost, st));
        GBSA_CUDA(cudaStreamSynchronize(st));
        if (n_steps) *n_steps = total;
        if (h_bad) throw Error(GBSA_ERR_PARAM, "a NAM pair with neither NAM");
        if (total > step_capacity) throw Error(GBSA_ERR_CAPACITY, "step capacity too small");
        return GBSA_OK;
    } catch (const Error& e) {
        set_last_error(e.what());
        return e.code;
    } catch (const std::exception& e) {
        set_last_error(e.what());
        return GBSA_ERR_CUDA;
    }
}
