// prims.cu — exclusive scan and stable sort of the index's records (see prims.cuh).
#include "prims.cuh"

namespace gbsa {

namespace {

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr size_t kScanTile = (size_t)kScanThreads * kScanItems;

template <int NT>
__device__ uint64_t block_exclusive_sum(uint64_t v, uint64_t* s_warp, uint64_t& total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint64_t inc = warp_inclusive_sum(v);
    if (lane == 31) s_warp[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        uint64_t x = lane < NT / 32 ? s_warp[lane] : 0;
        uint64_t xi = warp_inclusive_sum(x);
        if (lane < NT / 32) s_warp[lane] = xi - x;
        if (lane == NT / 32 - 1) s_warp[32] = xi;
    }
    __syncthreads();
    total = s_warp[32];
    const uint64_t r = s_warp[wid] + inc - v;
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_partials(const uint64_t* in, size_t n, uint64_t* partials) {
    __shared__ uint64_t s_warp[33];
    const size_t base = (size_t)blockIdx.x * kScanTile;
    uint64_t v = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const size_t idx = base + (size_t)i * kScanThreads + threadIdx.x;
        if (idx < n) v += in[idx];
    }
    uint64_t total;
    block_exclusive_sum<kScanThreads>(v, s_warp, total);
    if (threadIdx.x == 0) partials[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_apply(const uint64_t* in, uint64_t* out, size_t n,
                                                             const uint64_t* offsets, uint64_t* d_total) {
    __shared__ uint64_t s_warp[33];
    const size_t base = (size_t)blockIdx.x * kScanTile;
    // each thread owns kScanItems consecutive elements
    uint64_t v[kScanItems];
    uint64_t sum = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const size_t idx = base + (size_t)threadIdx.x * kScanItems + i;
        v[i] = idx < n ? in[idx] : 0;
        sum += v[i];
    }
    uint64_t total;
    uint64_t run = block_exclusive_sum<kScanThreads>(sum, s_warp, total) + (offsets ? offsets[blockIdx.x] : 0);
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const size_t idx = base + (size_t)threadIdx.x * kScanItems + i;
        if (idx < n) out[idx] = run;
        run += v[i];
    }
    if (d_total && blockIdx.x == gridDim.x - 1 && threadIdx.x == kScanThreads - 1) *d_total = run;
}

// ---- radix sort --------------------------------------------------------------
constexpr int kSortThreads = 256;
constexpr int kSortRounds = 16;
constexpr size_t kSortTile = (size_t)kSortThreads * kSortRounds;

__device__ __forceinline__ uint32_t digit_of(const gbsa_ref_randstrobe& r, int pass) {
    // passes 0..3: position bytes (least significant key), 4..11: hash bytes
    if (pass < 4) return (r.position >> (8 * pass)) & 0xFF;
    return (uint32_t)(r.hash >> (8 * (pass - 4))) & 0xFF;
}

__global__ void __launch_bounds__(kSortThreads) k_radix_hist(const gbsa_ref_randstrobe* in, size_t n, int pass,
                                                              uint64_t* block_hist, size_t nblocks) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const size_t base = (size_t)blockIdx.x * kSortTile;
    for (int r = 0; r < kSortRounds; ++r) {
        const size_t idx = base + (size_t)r * kSortThreads + threadIdx.x;
        if (idx < n) atomicAdd(&h[digit_of(in[idx], pass)], 1u);
    }
    __syncthreads();
    block_hist[(size_t)threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

__global__ void __launch_bounds__(kSortThreads) k_radix_scatter(const gbsa_ref_randstrobe* in,
                                                                 gbsa_ref_randstrobe* out, size_t n, int pass,
                                                                 const uint64_t* block_off, size_t nblocks) {
    __shared__ uint64_t s_base[256];
    __shared__ uint32_t s_run[256];
    __shared__ uint32_t s_wcnt[kSortThreads / 32][256];
    __shared__ uint32_t s_woff[kSortThreads / 32][256];
    const uint32_t t = threadIdx.x, lane = t & 31, wid = t >> 5;
    s_base[t] = block_off[(size_t)t * nblocks + blockIdx.x];
    s_run[t] = 0;
    for (int w = 0; w < kSortThreads / 32; ++w) s_wcnt[w][t] = 0;
    __syncthreads();
    const size_t base = (size_t)blockIdx.x * kSortTile;
    for (int r = 0; r < kSortRounds; ++r) {
        const size_t idx = base + (size_t)r * kSortThreads + t;
        const bool valid = idx < n;
        gbsa_ref_randstrobe rec;
        uint32_t d = 256;
        if (valid) {
            rec = in[idx];
            d = digit_of(rec, pass);
        }
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
        const uint32_t rank = __popc(peers & lanemask_lt());
        if (valid && lane == (uint32_t)(__ffs(peers) - 1)) s_wcnt[wid][d] = __popc(peers);
        __syncthreads();
        {
            uint32_t run = s_run[t];
            for (int w = 0; w < kSortThreads / 32; ++w) {
                const uint32_t c = s_wcnt[w][t];
                s_woff[w][t] = run;
                run += c;
                s_wcnt[w][t] = 0;
            }
            s_run[t] = run;
        }
        __syncthreads();
        if (valid) out[s_base[d] + s_woff[wid][d] + rank] = rec;
    }
}

// ---- groups of the top hash bits ------------------------------------------------
constexpr size_t kGroupMean = 160;     // largest mean size of a group
constexpr uint32_t kGroupMax = 256;    // records a warp sorts in shared memory
constexpr int kGroupWarps = 8;
constexpr uint32_t kBlockGroupMax = 2048;   // records a block sorts in shared memory
constexpr uint32_t kBlockGroupThreads = 512;

__global__ void k_group_starts(const gbsa_ref_randstrobe* __restrict__ rs, size_t n, int bits,
                               uint64_t* __restrict__ start) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const uint64_t t = rs[i].hash >> (64 - bits);
        for (uint64_t g = i ? (rs[i - 1].hash >> (64 - bits)) + 1 : 0; g <= t; ++g) start[g] = i;
        if (i == n - 1)
            for (uint64_t g = t + 1; g <= (1ULL << bits); ++g) start[g] = n;
    }
}

// A warp sorts each group of up to kGroupMax records by rank in shared memory: 61 records a
// group at 4M records, 122 comparisons a lane instead of six more passes over memory
// (186 us against 105 a pass).  The
// comparisons are of 32 bits, the first that the group does not share: a record comes after
// those with smaller bits and after those with the same that precede it in place.  That is
// right where those are in order already (copies of one seed, in a contig); a group where
// two neighbours among them are not is ranked by all bits.  Groups of up to kBlockGroupMax go
// to the list for a block each, the size of larger ones (repeats) into `large`.
__global__ void __launch_bounds__(32 * kGroupWarps) k_sort_groups(gbsa_ref_randstrobe* __restrict__ rs,
                                                                  const uint64_t* __restrict__ start, uint64_t n_groups,
                                                                  int bits, uint64_t* __restrict__ large,
                                                                  uint32_t* __restrict__ n_medium,
                                                                  uint32_t* __restrict__ medium) {
    __shared__ uint64_t s_hash[kGroupWarps][kGroupMax];
    __shared__ uint32_t s_pos[kGroupWarps][kGroupMax];
    __shared__ __align__(16) uint32_t s_key[kGroupWarps][kGroupMax];
    constexpr uint32_t kRows = kGroupMax / 32, kNone = 0xFFFFFFFFu;
    const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
    uint64_t* hash = s_hash[wid];
    uint32_t* pos = s_pos[wid];
    uint32_t* key = s_key[wid];
    for (uint64_t g = blockIdx.x * (uint64_t)kGroupWarps + wid; g < n_groups; g += (uint64_t)gridDim.x * kGroupWarps) {
        const uint64_t a = start[g], size = start[g + 1] - a;
        if (lane == 0) {
            large[g] = size > kBlockGroupMax ? size : 0;
            if (size > kGroupMax && size <= kBlockGroupMax) medium[atomicAdd(n_medium, 1u)] = (uint32_t)g;
        }
        if (size < 2 || size > kGroupMax) continue;
        const uint32_t m = (uint32_t)size;
        uint4 v[kRows];
        uint4* rec = reinterpret_cast<uint4*>(rs) + a;
#pragma unroll
        for (uint32_t j = 0; j < kRows; ++j) {
            const uint32_t i = 32 * j + lane;
            if (32 * j < m) {
                v[j] = i < m ? rec[i] : make_uint4(~0u, ~0u, ~0u, ~0u);
                const uint64_t h = ((uint64_t)v[j].y << 32) | v[j].x;
                hash[i] = h;
                pos[i] = v[j].z;
                key[i] = i < m ? (uint32_t)(h >> (32 - bits)) : kNone;
            }
        }
        __syncwarp();
        uint32_t rank[kRows];
        bool wrong = false;
#pragma unroll
        for (uint32_t j = 0; j < kRows; ++j) {
            const uint32_t i = 32 * j + lane;
            rank[j] = 0;
            if (32 * j < m) {
                const uint32_t mine = key[i];
                uint32_t r = 0, prev = kNone;
                auto upto = [&](uint32_t x, uint32_t k) {
                    r += k <= mine;
                    if (k == mine) prev = x;
                };
                uint32_t x = 0;
                for (; x < 32 * j; x += 4) {   // records before the row
                    const uint4 k = *reinterpret_cast<const uint4*>(key + x);
                    upto(x, k.x);
                    upto(x + 1, k.y);
                    upto(x + 2, k.z);
                    upto(x + 3, k.w);
                }
                const uint32_t row = min(m, 32 * j + 32);
                for (; x < row; ++x) {
                    const uint32_t k = key[x];
                    if (x < i) upto(x, k);
                    else r += k < mine;
                }
                for (; x < m; x += 4) {   // behind it (past m all ones: below none)
                    const uint4 k = *reinterpret_cast<const uint4*>(key + x);
                    r += (k.x < mine) + (k.y < mine) + (k.z < mine) + (k.w < mine);
                }
                rank[j] = r;
                if (prev != kNone && i < m)
                    wrong |= hash[prev] > hash[i] || (hash[prev] == hash[i] && pos[prev] > pos[i]);
            }
        }
        if (__any_sync(0xFFFFFFFFu, wrong)) {
#pragma unroll
            for (uint32_t j = 0; j < kRows; ++j) {
                const uint32_t i = 32 * j + lane;
                if (i < m) {
                    const uint64_t h = hash[i];
                    const uint32_t p = pos[i];
                    rank[j] = 0;
                    for (uint32_t x = 0; x < m; ++x) {
                        const uint64_t o = hash[x];
                        rank[j] += o < h || (o == h && (pos[x] < p || (pos[x] == p && x < i)));
                    }
                }
            }
        }
#pragma unroll
        for (uint32_t j = 0; j < kRows; ++j)
            if (32 * j + lane < m) rec[rank[j]] = v[j];
        __syncwarp();
    }
}

// The listed groups, a block each: a bitonic sort by (hash, position, place) in shared memory
// (a group of 2,000 equal hashes took 400 us by rank).
__global__ void __launch_bounds__(kBlockGroupThreads) k_sort_medium(gbsa_ref_randstrobe* __restrict__ rs,
                                                                    const uint64_t* __restrict__ start,
                                                                    const uint32_t* __restrict__ n_medium,
                                                                    const uint32_t* __restrict__ medium) {
    __shared__ uint64_t s_hash[kBlockGroupMax];
    __shared__ uint32_t s_pos[kBlockGroupMax];
    __shared__ uint16_t s_at[kBlockGroupMax];
    constexpr uint32_t kRows = kBlockGroupMax / kBlockGroupThreads;
    for (uint32_t t = blockIdx.x; t < *n_medium; t += gridDim.x) {
        const uint64_t g = medium[t], a = start[g];
        const uint32_t m = (uint32_t)(start[g + 1] - a);
        uint32_t size = 2 * kGroupMax;
        while (size < m) size *= 2;
        uint4* rec = reinterpret_cast<uint4*>(rs) + a;
        for (uint32_t i = threadIdx.x; i < size; i += kBlockGroupThreads) {
            const uint4 v = i < m ? rec[i] : make_uint4(~0u, ~0u, ~0u, ~0u);
            s_hash[i] = ((uint64_t)v.y << 32) | v.x;
            s_pos[i] = v.z;
            s_at[i] = (uint16_t)i;
        }
        __syncthreads();
        for (uint32_t k = 2; k <= size; k *= 2)
            for (uint32_t d = k / 2; d; d /= 2) {
                for (uint32_t x = threadIdx.x; x < size / 2; x += kBlockGroupThreads) {
                    const uint32_t i = 2 * x - (x & (d - 1)), l = i + d;
                    const uint64_t hi = s_hash[i], hl = s_hash[l];
                    const uint32_t pi = s_pos[i], pl = s_pos[l];
                    const uint16_t ai = s_at[i], al = s_at[l];
                    const bool after = hi > hl || (hi == hl && (pi > pl || (pi == pl && ai > al)));
                    if (after == ((i & k) == 0)) {
                        s_hash[i] = hl;
                        s_hash[l] = hi;
                        s_pos[i] = pl;
                        s_pos[l] = pi;
                        s_at[i] = al;
                        s_at[l] = ai;
                    }
                }
                __syncthreads();
            }
        uint4 v[kRows];
#pragma unroll
        for (uint32_t j = 0; j < kRows; ++j) {
            const uint32_t i = kBlockGroupThreads * j + threadIdx.x;
            if (i < m) v[j] = rec[s_at[i]];
        }
        __syncthreads();
#pragma unroll
        for (uint32_t j = 0; j < kRows; ++j) {
            const uint32_t i = kBlockGroupThreads * j + threadIdx.x;
            if (i < m) rec[i] = v[j];
        }
    }
}

// The records of the large groups (those with room of their own in `off`) between their
// places in rs and the packed list, a warp a group.
template <bool kOut>
__global__ void k_move_groups(gbsa_ref_randstrobe* __restrict__ rs, gbsa_ref_randstrobe* __restrict__ list,
                              const uint64_t* __restrict__ start, const uint64_t* __restrict__ off, uint64_t n_groups) {
    const uint32_t lane = lane_id();
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x / 32);
    for (uint64_t g = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32; g < n_groups; g += warps) {
        const uint64_t o = off[g], m = off[g + 1] - o;
        uint4* place = reinterpret_cast<uint4*>(rs) + start[g];
        uint4* packed = reinterpret_cast<uint4*>(list) + o;
        for (uint64_t i = lane; i < m; i += 32) {
            if (kOut) packed[i] = place[i];
            else place[i] = packed[i];
        }
    }
}

}  // namespace

void scan_exclusive_u64(const uint64_t* in, uint64_t* out, size_t n, uint64_t* d_total, Workspace& ws,
                        cudaStream_t st) {
    if (n == 0) {
        if (d_total) GBSA_CUDA(cudaMemsetAsync(d_total, 0, sizeof(uint64_t), st));
        return;
    }
    const size_t nb = (n + kScanTile - 1) / kScanTile;
    if (nb == 1) {
        k_scan_apply<<<1, kScanThreads, 0, st>>>(in, out, n, nullptr, d_total);
        GBSA_LAUNCHED();
        return;
    }
    uint64_t* partials = ws.get<uint64_t>(nb);
    k_scan_partials<<<(unsigned)nb, kScanThreads, 0, st>>>(in, n, partials);
    GBSA_LAUNCHED();
    scan_exclusive_u64(partials, partials, nb, nullptr, ws, st);
    k_scan_apply<<<(unsigned)nb, kScanThreads, 0, st>>>(in, out, n, partials, d_total);
    GBSA_LAUNCHED();
}

// One stable pass over the digit `pass` of n records, src to dst.
static void radix_pass(const gbsa_ref_randstrobe* src, gbsa_ref_randstrobe* dst, size_t n, int pass, uint64_t* bh,
                       Workspace& ws, cudaStream_t st) {
    const size_t nb = (n + kSortTile - 1) / kSortTile;
    k_radix_hist<<<(unsigned)nb, kSortThreads, 0, st>>>(src, n, pass, bh, nb);
    GBSA_LAUNCHED();
    const size_t at = ws.mark();
    scan_exclusive_u64(bh, bh, 256 * nb, nullptr, ws, st);
    ws.rewind(at);   // the next pass follows in the stream
    k_radix_scatter<<<(unsigned)nb, kSortThreads, 0, st>>>(src, dst, n, pass, bh, nb);
    GBSA_LAUNCHED();
}

int sort_passes(size_t n) {
    if (n <= 1) return 0;
    int bytes = 1;
    while (bytes < 3 && (n >> (8 * bytes)) >= kGroupMean) ++bytes;
    return bytes;
}

gbsa_ref_randstrobe* sort_ref_randstrobes(gbsa_ref_randstrobe* a, gbsa_ref_randstrobe* b, size_t n, uint32_t max_position,
                                          Workspace& ws, cudaStream_t st) {
    if (n <= 1) return a;
    uint64_t* bh = ws.get<uint64_t>(256 * ((n + kSortTile - 1) / kSortTile));
    // passes over the position's used bytes, then the hash's
    auto all_passes = [&](gbsa_ref_randstrobe* src, gbsa_ref_randstrobe* dst, size_t m) {
        for (int pass = 0; pass < 12; ++pass) {
            if (pass < 4 && (max_position >> (8 * pass)) == 0) continue;
            radix_pass(src, dst, m, pass, bh, ws, st);
            std::swap(src, dst);
        }
        return src;
    };
    // groups by the hash's top bits: of up to kGroupMean records on average while that saves
    // a pass, else of 24 to 48
    const int bytes = sort_passes(n);
    int bits = 8 * bytes;
    while (bits > 8 && (n >> bits) < 24) --bits;
    gbsa_ref_randstrobe* src = a;
    gbsa_ref_randstrobe* dst = b;
    for (int pass = 12 - bytes; pass < 12; ++pass) {
        radix_pass(src, dst, n, pass, bh, ws, st);
        std::swap(src, dst);
    }
    const uint64_t n_groups = 1ULL << bits;
    uint64_t* start = ws.get<uint64_t>(n_groups + 1);
    k_group_starts<<<grid_for(n, 256, 1u << 16), 256, 0, st>>>(src, n, bits, start);
    GBSA_LAUNCHED();
    uint64_t* large = ws.get<uint64_t>(n_groups + 1);   // a large group's size, then the offsets
    uint32_t* medium = ws.get<uint32_t>(n_groups + 1);  // the groups for a block each, their number last
    uint32_t* n_medium = medium + n_groups;
    GBSA_CUDA(cudaMemsetAsync(n_medium, 0, 4, st));
    k_sort_groups<<<grid_for(n_groups, kGroupWarps, 32 * device_sm_count()), 32 * kGroupWarps, 0, st>>>(
        src, start, n_groups, bits, large, n_medium, medium);
    GBSA_LAUNCHED();
    k_sort_medium<<<4 * device_sm_count(), kBlockGroupThreads, 0, st>>>(src, start, n_medium, medium);
    GBSA_LAUNCHED();
    scan_exclusive_u64(large, large, n_groups, large + n_groups, ws, st);
    uint64_t m = 0;
    GBSA_CUDA(cudaMemcpyAsync(&m, large + n_groups, 8, cudaMemcpyDeviceToHost, st));
    GBSA_CUDA(cudaStreamSynchronize(st));
    if (m == 0) return src;
    if (2 * m > n) return all_passes(src, dst, n);
    // the large groups' records, side by side in the free buffer, sorted among themselves:
    // they keep the groups' order, so each goes back into its group's place
    const unsigned blocks = grid_for(n_groups, 8, 64 * device_sm_count());
    k_move_groups<true><<<blocks, 256, 0, st>>>(src, dst, start, large, n_groups);
    GBSA_LAUNCHED();
    k_move_groups<false><<<blocks, 256, 0, st>>>(src, all_passes(dst, dst + m, m), start, large, n_groups);
    GBSA_LAUNCHED();
    return src;
}

}  // namespace gbsa
