// index_build.cu — StrobemerIndex::populate on the GPU.
//
// Restates step2/index.cu:143-311 (populate, count_randstrobes, assign_randstrobes;
// commented out in the reference) with the RandstrobeGenerator of
// step2/randstrobes.cu:161-190:
//   1. pack the contigs into a 2-bit stream + N bitmask (one pass over the bases);
//   2. canonical syncmers of every contig, a warp per 2048-window segment (a bit a
//      window and a count, exclusive scan, write pass); where the state machine is needed
//      a segment starts at an "anchor" window whose syncmer state does not depend on
//      earlier windows;
//   3. one forward randstrobe per syncmer with at least w_min successors in its
//      contig, packed = (ref_index << 8) + (strobe2 - strobe1); contigs shorter than
//      w_max keep zeroed entries (counted, never assigned, as in the reference);
//   4. stable sort by (hash, position) — ties keep generation order, which is
//      (ref_index, position), i.e. the table ends up sorted by (hash, position, packed);
//   5. bucket tables with the reference's first-bucket rule, and the run-length
//      statistics that give filter_cutoff (float product unique_mers * f), in one pass.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "index.h"
#include "prims.cuh"
#include "seed.cuh"

namespace gbsa {

namespace {

constexpr uint32_t kSegWindows = 2048;
constexpr int kSegWarps = 8;

// one thread per 32 bases; g is padded with 'N' to a multiple of 32 plus 64 bytes
__global__ void k_pack_genome(const uint8_t* __restrict__ g, uint64_t nwords, uint64_t* __restrict__ packed,
                              uint32_t* __restrict__ nmask) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nwords; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint4* src = reinterpret_cast<const uint4*>(g + 32 * i);
        const uint4 a = src[0], b = src[1];
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint64_t word = 0;
        uint32_t nm = 0;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const uint32_t c = nt4((uint8_t)(w[j >> 2] >> (8 * (j & 3))));
            nm |= (c == 4u ? 1u : 0u) << j;
            word = (word << 2) | (c & 3u);
        }
        packed[i] = word;
        nmask[i] = nm;
    }
}

struct SegTables {
    const uint32_t* seg_contig;
    const uint32_t* seg_w0;
    const uint32_t* seg_w1;
    const uint64_t* contig_base;
    const uint32_t* contig_nwin;
};

constexpr uint32_t kSegWords = kSegWindows / 32;

// The syncmers of each segment as a bit a window, and their number.  Bound by integer issue
// (a 64-bit hash a window); segments of A, C, G and T without a tied window take the scan
// that needs no state, the others the state machine from their anchor.
__global__ void __launch_bounds__(32 * kSegWarps) k_mark_syncmers(DevParams P, const uint64_t* __restrict__ packed,
                                                                  const uint32_t* __restrict__ nmask, SegTables T,
                                                                  uint32_t n_seg, uint64_t* __restrict__ seg_count,
                                                                  uint32_t* __restrict__ bits) {
    __shared__ uint64_t s_h[kSegWarps][64];
    __shared__ uint32_t s_bits[kSegWarps][kSegWords];
    const uint32_t wid = threadIdx.x >> 5, lane = lane_id();
    uint64_t* hbuf = s_h[wid];
    uint32_t* own = s_bits[wid];
    for (uint32_t s = blockIdx.x * kSegWarps + wid; s < n_seg; s += gridDim.x * kSegWarps) {
        const uint32_t c = T.seg_contig[s];
        const uint32_t w0 = T.seg_w0[s], w1 = T.seg_w1[s];
        const uint64_t base = T.contig_base[c];
        const uint64_t g = base + w0;   // the segment's first base
        const uint32_t words = ((uint32_t)(g & 31) + (w1 - w0) + (uint32_t)P.k - 1 + 31) / 32;
        uint32_t any_n = P.W > 32 ? 1u : 0u;
        for (uint32_t i = lane; i < words; i += 32) any_n |= nmask[(g >> 5) + i];
        uint32_t n = 0;
        const uint32_t shift = (uint32_t)(P.W - 1);
        auto put = [&](uint32_t at, uint32_t b) {   // bit l: window at + l - shift
            if (lane == 0) {
                if (at && shift) own[(at >> 5) - 1] |= b << (32 - shift);
                if (at < w1 - w0) own[at >> 5] = b >> shift;
            }
            n += __popc(b);
        };
        bool ok = !__any_sync(0xFFFFFFFFu, any_n != 0);
        if (ok) {
            uint32_t* buf = reinterpret_cast<uint32_t*>(hbuf);
            const uint64_t* pk = packed + (g >> 5);
            const uint32_t p0 = (uint32_t)(g & 31);
            ok = clean_scan5(P) ? warp_clean_scan<5>(P, pk, p0, w1 - w0, buf, put)
                                : warp_clean_scan<0>(P, pk, p0, w1 - w0, buf, put);
            __syncwarp();
        }
        if (!ok) {
            for (uint32_t i = lane; i < kSegWords; i += 32) own[i] = 0;
            __syncwarp();
            const uint32_t nwin = T.contig_nwin[c];
            const uint32_t anchor = warp_find_anchor(P, packed, nmask, base, nwin, w0, hbuf);
            n = warp_syncmer_scan(P, packed, nmask, base, nwin, anchor, w1, w0, hbuf,
                                  [&](uint32_t, uint32_t w) { atomicOr(&own[(w - w0) >> 5], 1u << ((w - w0) & 31)); });
        }
        __syncwarp();
        for (uint32_t i = lane; 32 * i < w1 - w0; i += 32) bits[(uint64_t)s * kSegWords + i] = own[i];
        if (lane == 0) seg_count[s] = n;
        __syncwarp();
    }
}

// The marked windows' k-mer hashes and positions, in order.
__global__ void __launch_bounds__(32 * kSegWarps) k_write_syncmers(DevParams P, const uint64_t* __restrict__ packed,
                                                                   SegTables T, uint32_t n_seg,
                                                                   const uint64_t* __restrict__ seg_off,
                                                                   const uint32_t* __restrict__ bits,
                                                                   uint64_t* __restrict__ sh,
                                                                   uint32_t* __restrict__ sp) {
    __shared__ uint16_t s_w[kSegWarps][kSegWindows];
    const uint32_t wid = threadIdx.x >> 5, lane = lane_id();
    for (uint32_t s = blockIdx.x * kSegWarps + wid; s < n_seg; s += gridDim.x * kSegWarps) {
        const uint32_t w0 = T.seg_w0[s], w1 = T.seg_w1[s];
        const uint64_t g = T.contig_base[T.seg_contig[s]] + w0;
        uint32_t n = 0;
        for (uint32_t i = 0; 32 * i < w1 - w0; i += 32) {
            uint32_t b = 32 * (i + lane) < w1 - w0 ? bits[(uint64_t)s * kSegWords + i + lane] : 0u;
            const uint32_t cnt = __popc(b), inc = warp_inclusive_sum(cnt);
            for (uint32_t at = n + inc - cnt; b; b &= b - 1) s_w[wid][at++] = (uint16_t)(32 * (i + lane) + __ffs(b) - 1);
            n += __shfl_sync(0xFFFFFFFFu, inc, 31);
        }
        __syncwarp();
        const uint64_t o = seg_off[s];
        for (uint32_t i = lane; i < n; i += 32) {
            const uint32_t w = s_w[wid][i];
            sp[o + i] = w0 + w;
            sh[o + i] = kmer_hash(P, packed, g + w);
        }
        __syncwarp();
    }
}

// The first syncmer of every contig, and their number at the end.
__global__ void k_contig_starts(const uint64_t* __restrict__ seg_off, const uint64_t* __restrict__ first_seg,
                                uint32_t n_contigs, uint32_t n_seg, const uint64_t* __restrict__ total,
                                uint64_t* __restrict__ out) {
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c <= n_contigs; c += gridDim.x * blockDim.x)
        out[c] = first_seg[c] < n_seg ? seg_off[first_seg[c]] : *total;
}

__global__ void k_ref_randstrobes(DevParams P, const uint64_t* __restrict__ sh, const uint32_t* __restrict__ sp,
                                  uint64_t n_sm, const uint64_t* __restrict__ contig_sm, uint32_t n_contigs,
                                  const uint64_t* __restrict__ contig_ref_off, const uint64_t* __restrict__ contig_len,
                                  gbsa_ref_randstrobe* __restrict__ out) {
    for (uint64_t g = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; g < n_sm; g += (uint64_t)gridDim.x * blockDim.x) {
        // contig of syncmer g: last c with contig_sm[c] <= g
        uint32_t lo = 0, hi = n_contigs;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) / 2;
            if (contig_sm[mid] <= g) lo = mid;
            else hi = mid;
        }
        const uint32_t c = lo;
        if (contig_len[c] < P.w_max) continue;   // step2/index.cu:282-284
        const uint64_t b = contig_sm[c];
        const uint32_t nc = (uint32_t)(contig_sm[c + 1] - b);
        const uint32_t j = (uint32_t)(g - b);
        if (j + P.w_min >= nc) continue;
        uint64_t h;
        uint32_t s1, s2;
        randstrobe_fwd(P, sh + b, sp + b, nc, j, h, s1, s2);
        gbsa_ref_randstrobe r;
        r.hash = h;
        r.position = s1;
        r.packed = (uint32_t)((uint64_t)c << 8) + (s2 - s1);
        out[contig_ref_off[c] + j] = r;
    }
}

// First entry whose hash is not rs[0]'s (n when there is none): doubling steps, then a
// binary search; nearly always entry 1.
__device__ __forceinline__ uint64_t second_run(const gbsa_ref_randstrobe* __restrict__ rs, uint64_t n) {
    const uint64_t h0 = rs[0].hash;
    uint64_t lo = 0, step = 1;   // rs[lo] is of the first run
    while (lo + step < n && rs[lo + step].hash == h0) {
        lo += step;
        step *= 2;
    }
    uint64_t hi = lo + step < n ? lo + step : n;
    while (hi - lo > 1) {
        const uint64_t mid = lo + (hi - lo) / 2;
        if (rs[mid].hash == h0) lo = mid;
        else hi = mid;
    }
    return hi;
}

// Bucket b's form for the lookup, its first entry being `at` of n.  kWhole: all entries from
// `at` on are the bucket's.
template <bool kWhole>
__device__ __forceinline__ Bucket bucket_at(const gbsa_ref_randstrobe* __restrict__ rs, uint64_t n, int bits,
                                            uint64_t b, uint64_t at) {
    uint32_t size = 0;
    uint64_t lo = 0;
    uint32_t hi = 0;   // bytes 0..7 and 8..11
    const uint32_t most = kWhole ? kBucketTags : 255;
    for (; size < most && at + size < n; ++size) {
        const uint64_t h = rs[at + size].hash;
        if (!kWhole && (h >> (64 - bits)) != b) break;
        if (size < 7) lo |= (uint64_t)hash_tag(h) << (8 * (size + 1));
        else if (size < kBucketTags) hi |= hash_tag(h) << (8 * (size - 7));
    }
    if (kWhole) size = (uint32_t)(n - at < 255 ? n - at : 255);
    lo |= size;
    return Bucket{(uint32_t)at, {(uint32_t)lo, (uint32_t)(lo >> 32), hi}};
}

// The bucket table (the reference's first-bucket rule: the buckets up to the first entry's
// start at the second run), where `buckets` is set the lookup's form of it, and the
// histogram of the runs' lengths (bins 1..100 exact, bin 101: longer), in one pass: an entry
// that opens a bucket writes it and the empty ones before it (its warp, where there are more
// than 16: a table of few entries for its buckets, 2,000 for 2^24, took 5.3 ms by the entry
// alone, and 2.5 without the tags; now 1.6), one that opens a run walks it (102
// entries at most).
__global__ void __launch_bounds__(256) k_tables(const gbsa_ref_randstrobe* __restrict__ rs, uint64_t n, int bits,
                                                uint64_t* __restrict__ starts, Bucket* __restrict__ buckets,
                                                unsigned long long* __restrict__ hist) {
    __shared__ unsigned int h[102];
    for (int i = threadIdx.x; i < 102; i += blockDim.x) h[i] = 0;
    __syncthreads();
    constexpr uint32_t kFull = 0xFFFFFFFFu;
    const uint64_t nb = 1ULL << bits;
    auto put = [&](uint64_t b, uint64_t at, bool own) {   // own: bucket b is that of entry `at`
        starts[b] = at;
        if (buckets) buckets[b] = own ? bucket_at<false>(rs, n, bits, b, at) : Bucket{(uint32_t)at, {0, 0, 0}};
    };
    auto empty = [&](uint64_t b0, uint64_t b1, uint64_t at) {   // buckets [b0, b1), the warp's lanes each their own
        uint32_t m = __ballot_sync(kFull, b1 > b0 + 16);
        if (b1 <= b0 + 16)
            for (uint64_t b = b0; b < b1; ++b) put(b, at, false);
        for (; m; m &= m - 1) {
            const int src = __ffs(m) - 1;
            const uint64_t to = __shfl_sync(kFull, b1, src), first = __shfl_sync(kFull, at, src);
            for (uint64_t b = __shfl_sync(kFull, b0, src) + lane_id(); b < to; b += 32) put(b, first, false);
        }
    };
    uint32_t once = 0;
    for (uint64_t base = blockIdx.x * (uint64_t)blockDim.x; base < n; base += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = base + threadIdx.x;
        uint64_t b0 = 0, b1 = 0, at = 0, hash = 0, before = 0;
        if (i < n) {
            hash = rs[i].hash;
            before = i ? rs[i - 1].hash : ~hash;
            b1 = hash >> (64 - bits);
            b0 = i ? (before >> (64 - bits)) + 1 : 0;   // (above b1 within a bucket)
            at = i ? i : second_run(rs, n);
            if (b0 <= b1) put(b1, at, true);
        }
        empty(b0, b1, at);
        if (base + blockDim.x >= n) empty(b1 + 1, i == n - 1 ? nb + 1 : 0, n);
        if (i < n && hash != before) {
            uint32_t len = 1;
            while (len < 101 && i + len < n && rs[i + len].hash == hash) ++len;
            if (len == 1) ++once;
            else atomicAdd(&h[len], 1u);
        }
    }
    once = __reduce_add_sync(0xFFFFFFFFu, once);
    if (lane_id() == 0 && once) atomicAdd(&h[1], once);
    __syncthreads();
    for (int i = threadIdx.x; i < 102; i += blockDim.x)
        if (h[i]) atomicAdd(&hist[i], (unsigned long long)h[i]);
}

}  // namespace

// filter_cutoff and the creation statistics from the run-length histogram, with the
// reference's arithmetic (step2/index.cu:213-243).
static void finish_stats(gbsa_index& ix, const std::vector<unsigned long long>& H, uint64_t unique, float f) {
    uint64_t once = 0, high = 0, mid = 0, size = 0;
    uint32_t fc = 30;
    const uint64_t index_cutoff = (uint64_t)((float)unique * f);
    if (ix.n == 0) {
        mid = 1;   // the reference closes an empty "run" of count 0 (index.cu:214-223)
    } else {
        once = H[1];
        high = H[101];
        for (int v = 2; v <= 100; ++v) mid += H[v];
        size = high + mid;
        if (size > 0) {
            uint32_t value = 0;
            if (index_cutoff < size) {
                uint64_t cum = 0;
                for (int v = 101; v >= 2; --v) {
                    if (index_cutoff < cum + H[v]) {
                        value = (uint32_t)v;   // v == 101 stands for any count > 100
                        break;
                    }
                    cum += H[v];
                }
            } else {
                for (int v = 2; v <= 101; ++v)
                    if (H[v]) {
                        value = (uint32_t)v;
                        break;
                    }
            }
            fc = std::min(100u, std::max(30u, value));
        }
    }
    ix.filter_cutoff = fc;
    ix.info.tot_occur_once = once;
    ix.info.tot_high_ab = high;
    ix.info.tot_mid_ab = mid;
    ix.info.index_cutoff = index_cutoff;
    ix.info.distinct_strobemers = unique;
    ix.info.filter_cutoff = fc;
}

void build_index(gbsa_index& ix, const char* seqs, const uint64_t* offsets, const uint64_t* lengths,
                 uint32_t n_contigs, float f) {
    const DevParams P = ix.dp;
    cudaStream_t st;
    GBSA_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    struct StreamGuard {
        cudaStream_t s;
        ~StreamGuard() { cudaStreamDestroy(s); }
    } guard{st};
    Workspace ws(st);

    // ---- genome upload + packing -------------------------------------------
    std::vector<uint64_t> cbase(n_contigs + 1, 0);
    for (uint32_t c = 0; c < n_contigs; ++c) cbase[c + 1] = cbase[c] + lengths[c];
    const uint64_t total = cbase[n_contigs];
    const uint64_t nwords = (total + 31) / 32 + 4;
    DeviceBuffer d_g(nwords * 32 + 64, st);
    GBSA_CUDA(cudaMemsetAsync(d_g.as<uint8_t>(), 'N', nwords * 32 + 64, st));
    {
        // contiguous input → one copy; otherwise one copy per contig
        bool contiguous = true;
        for (uint32_t c = 0; c < n_contigs; ++c) contiguous &= (offsets[c] == offsets[0] + cbase[c]);
        if (contiguous && total) {
            GBSA_CUDA(cudaMemcpyAsync(d_g.as<uint8_t>(), seqs + offsets[0], total, cudaMemcpyHostToDevice, st));
        } else {
            for (uint32_t c = 0; c < n_contigs; ++c)
                if (lengths[c])
                    GBSA_CUDA(cudaMemcpyAsync(d_g.as<uint8_t>() + cbase[c], seqs + offsets[c], lengths[c],
                                              cudaMemcpyHostToDevice, st));
        }
    }
    DeviceBuffer d_packed(nwords * 8 + 64, st), d_nmask(nwords * 4 + 64, st);
    k_pack_genome<<<grid_for(nwords, 256, 65535), 256, 0, st>>>(d_g.as<uint8_t>(), nwords, d_packed.as<uint64_t>(),
                                                                d_nmask.as<uint32_t>());
    GBSA_LAUNCHED();

    // ---- segments -------------------------------------------------------------
    std::vector<uint32_t> seg_c, seg_w0, seg_w1, cnwin(n_contigs);
    std::vector<uint64_t> cfirst_seg(n_contigs + 1, 0);
    for (uint32_t c = 0; c < n_contigs; ++c) {
        cfirst_seg[c] = seg_c.size();
        const uint64_t L = lengths[c];
        if (L >= 1ULL << 32) throw Error(GBSA_ERR_PARAM, "contig longer than 2^32 - 1 bases");
        const uint32_t nwin = L >= (uint64_t)P.k ? (uint32_t)(L - P.k + 1) : 0;
        cnwin[c] = nwin;
        for (uint32_t w = 0; w < nwin; w += kSegWindows) {
            seg_c.push_back(c);
            seg_w0.push_back(w);
            seg_w1.push_back(std::min(nwin, w + kSegWindows));
        }
    }
    cfirst_seg[n_contigs] = seg_c.size();
    const uint32_t n_seg = (uint32_t)seg_c.size();
    DeviceBuffer d_segc(4 * (n_seg + 1), st), d_segw0(4 * (n_seg + 1), st), d_segw1(4 * (n_seg + 1), st);
    DeviceBuffer d_cbase(8 * (n_contigs + 1), st), d_cnwin(4 * (n_contigs + 1), st);
    if (n_seg) {
        GBSA_CUDA(cudaMemcpyAsync(d_segc.as<void>(), seg_c.data(), 4 * n_seg, cudaMemcpyHostToDevice, st));
        GBSA_CUDA(cudaMemcpyAsync(d_segw0.as<void>(), seg_w0.data(), 4 * n_seg, cudaMemcpyHostToDevice, st));
        GBSA_CUDA(cudaMemcpyAsync(d_segw1.as<void>(), seg_w1.data(), 4 * n_seg, cudaMemcpyHostToDevice, st));
    }
    GBSA_CUDA(cudaMemcpyAsync(d_cbase.as<void>(), cbase.data(), 8 * (n_contigs + 1), cudaMemcpyHostToDevice, st));
    if (n_contigs)
        GBSA_CUDA(cudaMemcpyAsync(d_cnwin.as<void>(), cnwin.data(), 4 * n_contigs, cudaMemcpyHostToDevice, st));
    SegTables T{d_segc.as<uint32_t>(), d_segw0.as<uint32_t>(), d_segw1.as<uint32_t>(), d_cbase.as<uint64_t>(),
                d_cnwin.as<uint32_t>()};

    DeviceBuffer d_segcnt(8 * (n_seg + 1), st), d_segoff(8 * (n_seg + 1), st), d_cseg(8 * (n_contigs + 1), st);
    DeviceBuffer d_bits(4ull * kSegWords * (n_seg + 1), st), d_csm(8 * (n_contigs + 1), st);
    const unsigned seg_blocks = grid_for(n_seg, kSegWarps, 1u << 20);
    std::vector<uint64_t> csm(n_contigs + 1, 0);   // first syncmer of every contig, and their number
    if (n_seg) {
        GBSA_CUDA(cudaMemcpyAsync(d_cseg.as<void>(), cfirst_seg.data(), 8 * (n_contigs + 1), cudaMemcpyHostToDevice, st));
        k_mark_syncmers<<<seg_blocks, 32 * kSegWarps, 0, st>>>(P, d_packed.as<uint64_t>(), d_nmask.as<uint32_t>(), T,
                                                               n_seg, d_segcnt.as<uint64_t>(), d_bits.as<uint32_t>());
        GBSA_LAUNCHED();
        uint64_t* d_tot = ws.get<uint64_t>(1);
        scan_exclusive_u64(d_segcnt.as<uint64_t>(), d_segoff.as<uint64_t>(), n_seg, d_tot, ws, st);
        k_contig_starts<<<grid_for(n_contigs + 1, 256, 4096), 256, 0, st>>>(
            d_segoff.as<uint64_t>(), d_cseg.as<uint64_t>(), n_contigs, n_seg, d_tot, d_csm.as<uint64_t>());
        GBSA_LAUNCHED();
        GBSA_CUDA(cudaMemcpyAsync(csm.data(), d_csm.as<uint64_t>(), 8 * (n_contigs + 1), cudaMemcpyDeviceToHost, st));
        GBSA_CUDA(cudaStreamSynchronize(st));
    }
    const uint64_t n_sm = csm[n_contigs];
    DeviceBuffer d_sh(8 * (n_sm + 1), st), d_sp(4 * (n_sm + 1), st);
    if (n_seg) {
        k_write_syncmers<<<seg_blocks, 32 * kSegWarps, 0, st>>>(P, d_packed.as<uint64_t>(), T, n_seg,
                                                                d_segoff.as<uint64_t>(), d_bits.as<uint32_t>(),
                                                                d_sh.as<uint64_t>(), d_sp.as<uint32_t>());
        GBSA_LAUNCHED();
    }
    d_g.release();

    // ---- per-contig randstrobe offsets (count_randstrobes) ----------------------
    std::vector<uint64_t> cref(n_contigs + 1, 0), clen(n_contigs + 1, 0);
    uint64_t n_rs = 0;
    uint32_t max_position = 0;
    for (uint32_t c = 0; c < n_contigs; ++c) {
        max_position = std::max(max_position, (uint32_t)lengths[c]);
        const uint64_t nc = csm[c + 1] - csm[c];
        cref[c] = n_rs;
        n_rs += nc < P.w_min ? 0 : nc - P.w_min;
        clen[c] = lengths[c];
    }
    cref[n_contigs] = n_rs;
    ix.n = n_rs;
    ix.info.tot_strobemer_count = n_rs;
    DeviceBuffer d_cref(8 * (n_contigs + 1), st), d_clen(8 * (n_contigs + 1), st);
    GBSA_CUDA(cudaMemcpyAsync(d_cref.as<void>(), cref.data(), 8 * (n_contigs + 1), cudaMemcpyHostToDevice, st));
    GBSA_CUDA(cudaMemcpyAsync(d_clen.as<void>(), clen.data(), 8 * (n_contigs + 1), cudaMemcpyHostToDevice, st));

    // the sort's passes go back and forth between the table and scratch; they end in the table
    ix.resize_tables();
    DeviceBuffer d_rs(16 * (n_rs + 1), st);
    gbsa_ref_randstrobe* from = ix.rs();
    gbsa_ref_randstrobe* to = d_rs.as<gbsa_ref_randstrobe>();
    if (sort_passes(n_rs) % 2) std::swap(from, to);
    GBSA_CUDA(cudaMemsetAsync(from, 0, 16 * (n_rs + 1), st));
    if (n_sm) {
        k_ref_randstrobes<<<grid_for(n_sm, 256, 1u << 20), 256, 0, st>>>(
            P, d_sh.as<uint64_t>(), d_sp.as<uint32_t>(), n_sm, d_csm.as<uint64_t>(), n_contigs, d_cref.as<uint64_t>(),
            d_clen.as<uint64_t>(), from);
        GBSA_LAUNCHED();
    }
    d_sh.release();
    d_sp.release();
    d_packed.release();
    d_nmask.release();

    // ---- sort --------------------------------------------------------------------
    const gbsa_ref_randstrobe* sorted = sort_ref_randstrobes(from, to, n_rs, max_position, ws, st);
    const gbsa_ref_randstrobe* rs = ix.rs();
    if (sorted != rs)   // (a table of repeats, sorted by all bytes)
        GBSA_CUDA(cudaMemcpyAsync(ix.rs(), sorted, 16 * n_rs, cudaMemcpyDeviceToDevice, st));
    d_rs.release();

    // ---- bucket tables, run-length statistics → filter_cutoff -----------------------
    std::vector<unsigned long long> H(102, 0);
    if (n_rs == 0) {
        GBSA_CUDA(cudaMemsetAsync(ix.starts(), 0, ix.tables.size() - ix.starts_at(), st));
    } else {
        unsigned long long* d_h = ws.get<unsigned long long>(102);
        GBSA_CUDA(cudaMemsetAsync(d_h, 0, 102 * 8, st));
        k_tables<<<grid_for(n_rs, 256, 16 * device_sm_count()), 256, 0, st>>>(rs, n_rs, ix.bits, ix.starts(),
                                                                              ix.buckets(), d_h);
        GBSA_LAUNCHED();
        GBSA_CUDA(cudaMemcpyAsync(H.data(), d_h, 102 * 8, cudaMemcpyDeviceToHost, st));
    }
    GBSA_CUDA(cudaStreamSynchronize(st));
    uint64_t unique = 0;
    for (const unsigned long long runs : H) unique += runs;
    finish_stats(ix, H, unique, f);
    ix.info.size = ix.n;
    ix.info.bits = ix.bits;
}

// As bucket_at, for a table that was not built here: `odd` is set when the entries are
// not in order, a bucket holds one that belongs elsewhere, or one ends before the last entry
// that belongs to it (start indices that stop short of the table's end), for then a tag or a
// bucket's end could answer differently from the search in order and the walk of a run.
__global__ void k_make_buckets(const uint64_t* __restrict__ starts, const gbsa_ref_randstrobe* __restrict__ rs,
                               uint64_t n, int bits, Bucket* __restrict__ out, uint32_t* __restrict__ odd) {
    const uint64_t nb = 1ULL << bits;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i <= nb; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t a = starts[i], e = i < nb ? starts[i + 1] : a;
        auto top = [&](uint64_t at) { return rs[at].hash >> (64 - bits); };
        const bool good = a <= n && e <= n &&
                          (a >= e || (top(a) == i && top(e - 1) == i && (e == n || top(e) != i)));
        if (!good) *odd = 1;
        out[i] = good && a < e ? bucket_at<true>(rs, e, bits, i, a) : Bucket{(uint32_t)a, {0, 0, 0}};
    }
    for (uint64_t i = 1 + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        if (rs[i - 1].hash > rs[i].hash) *odd = 1;
}

void make_buckets(gbsa_index& ix, cudaStream_t st) {
    if (!ix.tagged) return;
    DeviceBuffer d_odd(4, st);
    uint32_t odd = 0;
    GBSA_CUDA(cudaMemsetAsync(d_odd.as<void>(), 0, 4, st));
    k_make_buckets<<<grid_for(std::max(ix.n_starts(), ix.n), 256, 1u << 20), 256, 0, st>>>(
        ix.starts(), ix.rs(), ix.n, ix.bits, ix.buckets(), d_odd.as<uint32_t>());
    GBSA_LAUNCHED();
    GBSA_CUDA(cudaMemcpyAsync(&odd, d_odd.as<void>(), 4, cudaMemcpyDeviceToHost, st));
    GBSA_CUDA(cudaStreamSynchronize(st));
    if (odd) ix.tagged = false;
}

}  // namespace gbsa
