// map_kernels.cu — kernels of the read → NAM path (intermediates in HBM arenas).
//
//   k_seed_lookup               randstrobes_query (step2/randstrobes.cu:195-241) and the
//                               query loop of find_nams (step2/nam.cu:748-790): find,
//                               is_filtered, add_to_hits_per_ref; the rescue decision of
//                               step2/main.cu:3209-3216
//   k_seed_smem / k_seed_long, k_lookup / k_lookup_long   the same in two kernels, and for
//                               long reads
//   k_nams_group, k_nams        merge_hits_into_nams_forward_and_reverse(sort=true)
//                               (step2/nam.cu:515-539, 347-513) + NAM sort
//   k_rescue                    find_nams_rescue (step2/nam.cu:927-985) + NAM sort
#include <algorithm>
#include <mutex>
#include <utility>
#include <vector>

#include <cooperative_groups.h>

#include "map.cuh"
#include "runtime.h"

namespace gbsa {

namespace {

constexpr int kSeedWarps = 8;
constexpr int kWarpsPerBlock = 8;

__device__ __forceinline__ uint32_t warp_global_id() { return (blockIdx.x * blockDim.x + threadIdx.x) >> 5; }
__device__ __forceinline__ uint32_t warp_count() { return (gridDim.x * blockDim.x) >> 5; }

__device__ __forceinline__ uint64_t warp_bump(unsigned long long* ctr, uint64_t n) {
    uint64_t off = 0;
    if (lane_id() == 0) off = atomicAdd(ctr, (unsigned long long)n);
    return __shfl_sync(0xFFFFFFFFu, off, 0);
}

// The next read for the calling warp from a device work counter: warps pull reads one
// at a time, so reads of uneven cost (lengths, repeats) balance over a grid of resident
// warps instead of each warp owning a fixed stride of them.
__device__ __forceinline__ uint32_t warp_take(unsigned int* head, uint32_t n) {
    uint32_t r = 0;
    if (lane_id() == 0) r = atomicAdd(head, n);
    return __shfl_sync(0xFFFFFFFFu, r, 0);
}
__device__ __forceinline__ uint32_t warp_next(unsigned int* head) { return warp_take(head, 1); }

// Work items a warp takes at a time from a counter that all warps share (each take is a
// round trip, and they queue at one address): four while there are many for each warp.
__device__ __forceinline__ uint32_t items_per_take(uint32_t n) { return n >= 32 * warp_count() ? 4u : 1u; }

// Work items of a kernel whose warps share a counter.  A warp's first items are dealt out
// beforehand (about half of all, at most eight a warp), so that small batches touch the
// counter little, the others taken from it, up to four at a time while there are many: one
// address takes about one atomic a nanosecond (2M reads one at a time 8.81 ms, by four 8.71,
// by four behind eight dealt 8.76; uneven lengths 1.49, 1.50, 1.48; 1,000 reads the same).
struct WarpItems {
    uint32_t n, base, at, left, per;
    __device__ __forceinline__ explicit WarpItems(uint32_t n_items) : n(n_items) {
        const uint32_t warps = warp_count();
        left = min(max(n / (2 * warps), 1u), 8u);
        at = warp_global_id() * left;
        base = min((uint64_t)left * warps, (uint64_t)n);
        per = min(max((n - base) / (16 * warps), 1u), 4u);
    }
    // The next item, or n and above at the end.
    __device__ __forceinline__ uint32_t next(unsigned int* head) {
        if (left == 0) {
            at = base + warp_take(head, per);
            left = per;
        }
        --left;
        return at++;
    }
};

// Room in an arena whose bump counter all warps share, taken ahead in pieces of up to
// `piece` entries: a warp's requests come from its piece while they fit.  A piece is given up
// when no more than an eighth of it is left; a request that does not fit before takes just
// what it needs (given up at any size, requests of a third of a piece and more wasted up to
// half of it: reads with 145 hits each outgrew an arena with room for 166 a read).  What is
// left unused of the pieces is counted (`spare`), so that the counters still tell what was
// used.  most 0: no pieces, each request takes what it needs.
struct WarpRoom {
    uint64_t at = 0;
    uint32_t left = 0, spare = 0, most = 512;
    __device__ __forceinline__ uint64_t take(unsigned long long* used, uint64_t n, uint32_t piece) {
        if (n > left) {
            piece = min(piece, most);
            if (n >= piece || left > piece / 8) return warp_bump(used, n);
            spare += left;
            at = warp_bump(used, piece);
            left = piece;
        }
        left -= (uint32_t)n;
        const uint64_t r = at;
        at += n;
        return r;
    }
    __device__ __forceinline__ void done(unsigned long long* total) const {
        if (lane_id() == 0 && spare + left) atomicAdd(total, (unsigned long long)(spare + left));
    }
};
// The pieces that the warps of the grid hold at a time take at most an eighth of the arena.
__device__ __forceinline__ uint32_t arena_piece(uint64_t cap) {
    const uint64_t p = cap / (8ull * warp_count());
    return p < 512 ? (uint32_t)p : 512u;
}

__device__ __forceinline__ void warp_fail(ReadRec& rec, Counters* ctr, uint32_t bit) {
    if (lane_id() == 0) {
        rec.flags |= kReadFailed;
        atomicOr(&ctr->status, bit);
    }
}

// Writes the query randstrobes of read r from its syncmers.
__device__ __forceinline__ void emit_read_queries(const DevParams& P, const uint64_t* sh, const uint32_t* sp,
                                                  uint32_t ns, uint32_t L, ReadRec& rec, const Arenas& A,
                                                  Counters* ctr, WarpRoom& room) {
    const uint32_t nq = n_query_per_dir(P, ns, L);
    const uint64_t off = room.take(&ctr->q_used, 2 * nq, arena_piece(A.q_cap));
    if (off + 2ull * nq > A.q_cap) {
        warp_fail(rec, ctr, kStatusQueryOverflow);
        if (lane_id() == 0) rec.nq = rec.nq2 = 0;
        return;
    }
    warp_write_queries(P, sh, sp, ns, L, nq, A.q + off);
    if (lane_id() == 0) {
        rec.q_off = off;
        rec.nq = nq;
        rec.nq2 = 2 * nq;
    }
}

__global__ void __launch_bounds__(32 * kSeedWarps, 5) k_seed_smem(DevParams P, const uint8_t* __restrict__ seqs,
                                                                const uint64_t* __restrict__ offs,
                                                                const uint32_t* __restrict__ lens, uint32_t n,
                                                                ReadRec* __restrict__ rec, Arenas A, Counters* ctr) {
    __shared__ uint64_t s_pk[kSeedWarps][kSmemMaxLen / 32 + 4];
    __shared__ uint32_t s_nm[kSeedWarps][kSmemMaxLen / 32 + 4];
    __shared__ uint64_t s_hb[kSeedWarps][64];
    __shared__ uint64_t s_sh[kSeedWarps][kSmemSyncmers];
    __shared__ uint32_t s_sp[kSeedWarps][kSmemSyncmers];
    const uint32_t w = threadIdx.x >> 5;
    WarpItems items(n);
    WarpRoom room;
    for (uint32_t r; (r = items.next(&ctr->queue_head)) < n;) {
        const uint32_t L = lens[r];
        ReadRec& R = rec[r];
        if (L > GBSA_MAX_READ_LEN) {
            warp_fail(R, ctr, kStatusReadTooLong);
            continue;
        }
        uint32_t ns = 0xFFFFFFFFu;
        if (L <= kSmemMaxLen)
            ns = warp_read_syncmers(P, seqs + offs[r], L, s_pk[w], s_nm[w], s_hb[w], s_sh[w], s_sp[w], kSmemSyncmers);
        if (ns == 0xFFFFFFFFu) {
            if (lane_id() == 0) {
                R.flags |= kReadLong;
                A.long_list[atomicAdd(&ctr->n_long, 1u)] = r;
            }
            continue;
        }
        emit_read_queries(P, s_sh[w], s_sp[w], ns, L, R, A, ctr, room);
        __syncwarp();
    }
    room.done(&ctr->q_spare);
}

// Reads that did not fit the shared-memory buffers: same code on a per-warp slot of
// global scratch memory sized for GBSA_MAX_READ_LEN.
__global__ void __launch_bounds__(32 * kWarpsPerBlock) k_seed_long(DevParams P, const uint8_t* __restrict__ seqs,
                                                                    const uint64_t* __restrict__ offs,
                                                                    const uint32_t* __restrict__ lens,
                                                                    ReadRec* __restrict__ rec, Arenas A, Counters* ctr,
                                                                    uint8_t* scratch, const BatchDesc* desc) {
    if (desc) {
        seqs = desc->seqs;
        offs = desc->offs;
        lens = desc->lens;
    }
    const uint32_t n_long = *(volatile unsigned int*)&ctr->n_long;
    uint8_t* slot = scratch + (size_t)warp_global_id() * kLongSlotBytes;
    uint64_t* pk = reinterpret_cast<uint64_t*>(slot);
    uint32_t* nm = reinterpret_cast<uint32_t*>(pk + kLongWords);
    uint64_t* hb = reinterpret_cast<uint64_t*>(nm + kLongWords);
    uint64_t* sh = hb + 64;
    uint32_t* sp = reinterpret_cast<uint32_t*>(sh + GBSA_MAX_READ_LEN);
    WarpRoom room;
    for (uint32_t t = warp_global_id(); t < n_long; t += warp_count()) {
        const uint32_t r = A.long_list[t];
        const uint32_t L = lens[r];
        ReadRec& R = rec[r];
        const uint32_t ns = warp_read_syncmers(P, seqs + offs[r], L, pk, nm, hb, sh, sp, GBSA_MAX_READ_LEN);
        if (ns == 0xFFFFFFFFu) {
            warp_fail(R, ctr, kStatusSyncmerOverflow);
            continue;
        }
        emit_read_queries(P, sh, sp, ns, L, R, A, ctr, room);
        __syncwarp();
    }
    room.done(&ctr->q_spare);
}

// Distinct 32 B sectors of [lo, hi) bytes.
__device__ __forceinline__ uint64_t sector_span(uintptr_t lo, uintptr_t hi) {
    return hi > lo ? ((hi - 1) >> 5) - (lo >> 5) + 1 : 0;
}

// Sector form of one query's gathers as the reference performs them: the bucket
// bound pair, the entries examined in the bucket, and for a found key the filter
// probe and the run walk up to the first entry of another hash (entries the search
// already touched count once).
__device__ __forceinline__ uint64_t lookup_sectors(const IndexView& I, uint64_t key, uint32_t ex, uint64_t pos,
                                                   uint32_t run) {
    const uint64_t top = key >> (64 - I.bits);
    const uintptr_t sb = I.buckets ? reinterpret_cast<uintptr_t>(I.buckets + top)
                                   : reinterpret_cast<uintptr_t>(I.starts + top);
    uint64_t n = sector_span(sb, sb + 16);
    const uint64_t a = bucket_start(I, top);
    uint64_t end = a + ex;   // entries [a, end) touched
    if (pos != kNotFound) {
        const uint64_t walk_end = pos + run + 1 < I.n ? pos + run + 1 : I.n;
        end = walk_end > end ? walk_end : end;
        const uint64_t probe = pos + I.filter_cutoff;
        if (probe < I.n && (probe < a || probe >= end))
            n += sector_span(reinterpret_cast<uintptr_t>(I.rs + probe), reinterpret_cast<uintptr_t>(I.rs + probe + 1));
    }
    n += sector_span(reinterpret_cast<uintptr_t>(I.rs + a), reinterpret_cast<uintptr_t>(I.rs + end));
    return n;
}

constexpr uint32_t kRescueHeavyHits = 2000;   // estimated merge hits of a heavy rescued read

// Puts read r, whose queries' positions are in the arena, on the rescue list.  Reads inside
// short tandem repeats merge thousands of hits: their seeds' runs (up to the count cap)
// estimate the merge's hits; reads above kRescueHeavyHits (C.rescue_block_hits when set) go
// to the heavy end of the list, which the rescue kernel takes first.  filtered: some found
// query is filtered (else none has a long run).
__device__ __forceinline__ void enlist_rescue(const IndexView& I, const MapConfig& C, uint32_t r, ReadRec& R,
                                              const Arenas& A, Counters* ctr, bool filtered) {
    const uint32_t lane = lane_id();
    uint32_t w = 0;
    if (filtered) {
        for (uint32_t i = lane; i < R.nq2; i += 32) {
            const uint64_t pos = A.q_pos[R.q_off + i];
            if (pos == kNotFound) continue;
            const uint32_t c = index_get_count(I, pos);
            w += c <= C.count_cap ? c : 0u;
        }
        w = warp_sum(w);
    }
    const bool heavy = w >= (C.rescue_block_hits ? C.rescue_block_hits : kRescueHeavyHits);
    if (lane == 0) {
        R.flags |= kReadRescue;
        if (heavy) A.rescue_list[A.rescue_cap - 1 - atomicAdd(&ctr->n_rescue_heavy, 1u)] = r;
        else A.rescue_list[atomicAdd(&ctr->n_rescue, 1u)] = r;
        R.n_hits = 0;
    }
}

// kCount: also count the reference's algorithmic bytes and gather sectors (a
// separate instance, so that the counting code costs the mapping kernel nothing).
// find / is_filtered / walk for the queries of read r (warp): per-query index
// positions and hit counts, the nonrepetitive fraction and rescue decision, and for a
// read that is not rescued its hits (query order, then run order) in the hit arena.
// The query loop of find_nams (step2/nam.cu:748-790).
template <bool kCount>
__device__ __forceinline__ void lookup_read(const IndexView& I, const MapConfig& C, uint32_t r, ReadRec* __restrict__ rec,
                                            const Arenas& A, Counters* ctr, WarpRoom& room) {
    const uint32_t lane = lane_id();
    ReadRec& R = rec[r];
    if (R.flags & kReadFailed) return;
    const uint32_t nq = R.nq, nq2 = R.nq2;
    Query* Q = A.q + R.q_off;
    uint32_t* aux = A.q_aux + R.q_off;
    uint32_t tot = 0, good = 0;
    uint64_t bytes = 0, sectors = 0;
    for (uint32_t i = lane; i < nq2; i += 32) {
        const Query q = Q[i];
        if (!kCount && I.buckets) {
            const Probe p = index_probe(I, q.hash, (int)(q.end - q.start));
            if (p.pos != kMissing) {
                ++tot;
                good += p.filtered ? 0u : 1u;
            }
            A.q_pos[R.q_off + i] = p.pos == kMissing ? kNotFound : (uint64_t)p.pos;
            aux[i] = p.n_hits;
            continue;
        }
        uint32_t ex = 0;
        uint64_t bend = 0;
        const uint64_t pos = index_find(I, q.hash, &ex, &bend);
        uint32_t nh = 0, run = 0;
        bytes += 16 + 16ull * ex;
        if (pos != kNotFound) {
            ++tot;
            bytes += 16;   // the reference reads hash[pos + filter_cutoff]
            if (!index_is_filtered_in(I, pos, q.hash, bend)) {
                ++good;
                nh = walk_hit_run(I, (int)q.start, (int)q.end, pos, [&](uint32_t, int, int) {}, &run);
                bytes += 16ull * run;
            }
        }
        if (kCount) sectors += lookup_sectors(I, q.hash, ex, pos, run);
        A.q_pos[R.q_off + i] = pos;
        aux[i] = nh;
    }
    tot = warp_sum(tot);
    good = warp_sum(good);
    if (kCount) {
        bytes = warp_sum(bytes);
        sectors = warp_sum(sectors);
        if (lane == 0) {
            atomicAdd(&ctr->alg_bytes, (unsigned long long)bytes);
            atomicAdd(&ctr->alg_sectors, (unsigned long long)sectors);
        }
    }
    // nonrepetitive_fraction (step2/nam.cu:892) and the rescue trigger: a double
    // comparison of the float ratio with 0.7, or no hits (step2/main.cu:3211)
    const float frac = tot > 0 ? ((float)good) / ((float)tot) : 1.0f;
    const bool rescue = C.force_rescue || (C.rescue_level > 1 && (good == 0 || (double)frac < 0.7));
    if (lane == 0) {
        R.frac = frac;
        R.n_found = tot;
    }
    if (rescue) {
        enlist_rescue(I, C, r, R, A, ctr, good < tot);
        return;
    }
    // hit offsets in generation order (query order, then run order)
    uint64_t running = 0;
    for (uint32_t base = 0; base < nq2; base += 32) {
        const uint32_t i = base + lane;
        const uint32_t v = i < nq2 ? aux[i] : 0;
        const uint32_t inc = warp_inclusive_sum(v);
        if (i < nq2) aux[i] = (uint32_t)running + inc - v;
        running += __shfl_sync(0xFFFFFFFFu, inc, 31);
    }
    __syncwarp();
    const uint64_t H = running;
    const uint64_t hoff = room.take(&ctr->hit_used, H, arena_piece(A.hit_cap));
    if (hoff + H > A.hit_cap) {
        warp_fail(R, ctr, kStatusHitOverflow);
        return;
    }
    const uint64_t* qp = A.q_pos + R.q_off;
    for (uint32_t i = lane; i < nq2; i += 32) {
        // queries that emitted hits in the first pass (found and not filtered)
        const uint32_t next = i + 1 < nq2 ? aux[i + 1] : (uint32_t)H;
        if (next == aux[i]) continue;
        const uint64_t pos = qp[i];
        const uint32_t dir = i >= nq ? 1u : 0u;
        HitPacked* out = A.hits + hoff + aux[i];
        uint32_t k = 0;
        const int qs = (int)Q[i].start, qe = (int)Q[i].end;
        walk_hit_run(I, qs, qe, pos, [&](uint32_t ref, int rs, int re) {
            out[k++] = pack_hit((dir << 31) | ref, qs, qe, rs, re);
        }, nullptr, next - aux[i]);
    }
    if (lane == 0) {
        R.hit_off = hoff;
        R.n_hits = (uint32_t)H;
    }
}

template <bool kCount>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) k_lookup(IndexView I, MapConfig C, uint32_t n,
                                                                 ReadRec* __restrict__ rec, Arenas A, Counters* ctr,
                                                                 const BatchDesc* desc) {
    if (desc) n = min(n, desc->n_reads);   // batched form: n is the work areas' capacity
    WarpItems items(n);
    WarpRoom room;
    for (uint32_t r; (r = items.next(&ctr->queue_head2)) < n;) {
        lookup_read<kCount>(I, C, r, rec, A, ctr, room);
    }
    room.done(&ctr->hit_spare);
}

// The lookup of the reads seeded by k_seed_long (the long list).
template <bool kCount>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) k_lookup_long(IndexView I, MapConfig C,
                                                                      ReadRec* __restrict__ rec, Arenas A,
                                                                      Counters* ctr) {
    const uint32_t n_long = *(volatile unsigned int*)&ctr->n_long;
    WarpRoom room;
    for (uint32_t t = warp_global_id(); t < n_long; t += warp_count())
        lookup_read<kCount>(I, C, A.long_list[t], rec, A, ctr, room);
    room.done(&ctr->hit_spare);
}

// Seeding and lookup of a read in one go, for reads of at most kFastQueries queries and `cap`
// syncmers with parameters and an index for which fast_seed() holds (all profiles of read
// lengths).  Returns false, with nothing written, for any other read (the caller then takes
// the steps one by one).  Reads of only A, C, G and T without a tied syncmer window, nearly
// all, take the scan without state in line; the syncmers of one with an N, other letters or a
// tied window come from odd_syncmers, and it goes on here: left to the steps, 500k reads of
// 150 bp that all hold an N, or U for T, spent 2.7 and 3.0 ms in this kernel (1.7 and 1.6
// before there was a fast path), now 1.3 and 1.5.
//
// Both orientations' randstrobes run through one loop (the reverse ones walk the syncmers
// downwards; the distance between two syncmers is the same either way), a query goes from
// the lane that selects it straight into the index, and what is left of it for the hits (its
// interval, the run's place and first entry) lies in the warp's scratch slot, which stays in
// L2, instead of passing query, position and count through the arena.  A third of the
// queries have a candidate in their bucket: those are collected and looked at 32 at a time,
// so that the entries' part runs about once a read and not with a few lanes in each round.
// 1,880 warp instructions a read of 150 bp (2,710 by the steps), both bound by integer
// issue: packing 190, syncmers 650, their k-mer hashes 190, selection 440, buckets 110,
// entries 290, hits 150.  With the tags and with few atomics (WarpRoom, WarpItems) 2M reads
// 6.05 -> 4.3 ms, 100k pairs of 300 bp 1.12 -> 0.86 ms, of 400 bp 1.36 -> 0.99 ms.
constexpr uint32_t kFastQueries = 256;
// Queries of a warp's read that wait for a look at the entries.
struct FastQueue {
    uint64_t key[64];
    uint32_t start[64], what[64], se[64];   // the bucket's start; match | size << 16; the query
    uint8_t hits[32];
};
constexpr uint32_t kFastPad = 24;      // words before and behind the list: the most strobes ahead
constexpr uint32_t kFastShift = 256;   // added to positions: more than any max_dist

__host__ __device__ __forceinline__ bool fast_seed(const DevParams& P, const IndexView& I, const MapConfig& C) {
    return P.q <= 0xFF && P.W <= 32 && P.w_max <= kFastPad && I.buckets != nullptr && I.filter_cutoff <= 255 && !C.force_rescue && !C.count_bytes;
}

// Syncmers of a read with other letters than A, C, G and T (packed again, with its N bits) or
// (acgt, packed) with a tied window, which takes the scan with state.  Out of line.
__device__ __noinline__ uint32_t odd_syncmers(const DevParams& P, const uint8_t* seq, uint32_t L, bool acgt,
                                              uint64_t* pk, uint32_t* nm, uint64_t* hb, uint32_t* sp, uint32_t cap) {
    const uint32_t nwin = L - (uint32_t)P.k + 1;
    const bool has_n = !acgt && warp_pack_read(seq, L, pk, nm);
    uint32_t n = 0xFFFFFFFFu;
    if (!acgt) n = warp_clean_syncmers(P, pk, nwin, reinterpret_cast<uint32_t*>(hb), sp, cap, has_n ? nm : nullptr);
    return n != 0xFFFFFFFFu ? n : warp_state_syncmers(P, pk, nm, has_n, nwin, hb, sp, cap);
}

__device__ __forceinline__ bool fast_read(const DevParams& P, const IndexView& I, const MapConfig& C,
                                          const uint8_t* __restrict__ seq, uint32_t L, uint32_t r,
                                          ReadRec* __restrict__ rec, const Arenas& A, Counters* ctr, uint64_t* pk,
                                          uint32_t* nm, uint64_t* hb, uint64_t* sh, uint32_t* sp, uint32_t cap,
                                          FastQueue& Q, WarpRoom& room, uint32_t& direct) {
    constexpr uint32_t kFull = 0xFFFFFFFFu;
    const uint32_t lane = lane_id();
    if (L < (uint32_t)P.k) return false;
    const bool acgt = warp_pack_clean(seq, L, pk);
    uint32_t n = 0xFFFFFFFFu;
    if (acgt) n = warp_clean_syncmers(P, pk, L - (uint32_t)P.k + 1, reinterpret_cast<uint32_t*>(hb), sp, cap);
    if (n == 0xFFFFFFFFu) n = odd_syncmers(P, seq, L, acgt, pk, nm, hb, sp, cap);
    const uint32_t nq = n_query_per_dir(P, n, L), nq2 = 2 * nq;
    if (n > cap || nq2 > kFastQueries) return false;
    // the syncmers' hashes; their positions and the hash bits that the selection compares
    for (uint32_t i = lane; i < n; i += 32) {
        const uint32_t w = sp[i];
        const uint64_t h = kmer_hash(P, pk, w);
        sh[i] = h;
        sp[i] = ((w + kFastShift) << 8) | ((uint32_t)h & (uint32_t)P.q);
    }
    // beside the list positions that are too far from any: the selection needs no bounds
    if (lane < kFastPad) {
        sp[(int)lane - (int)kFastPad] = 0;
        sp[n + lane] = 0xFFFFFFFFu;
    }
    __syncwarp();
    const uint32_t k = (uint32_t)P.k;
    // per found query, in order: start | end << 10 | query << 20, the run's place, the run's
    // first entry
    uint4* found = reinterpret_cast<uint4*>(A.slots + (uint64_t)warp_global_id() * A.slot_bytes);
    uint64_t hits = 0;   // a byte for each 32 found queries: the hits of the one that is this lane's
    uint32_t tot = 0, good = 0, sum = 0, pending = 0;
    // query i's strobes: its key, and its interval and number
    auto select = [&](uint32_t i, uint64_t& key, uint32_t& se) {
        const bool rev = i >= nq;
        const uint32_t j = rev ? i - nq : i;
        const int i1 = (int)(rev ? n - 1 - j : j), dir = rev ? -1 : 1;
        // a strobe at most max_dist away: no larger than `limit`, bits inverted for the
        // reverse strand, whose strobes lie at smaller positions
        const uint32_t v1 = sp[i1], flip = rev ? 0xFFFFFFFFu : 0u;
        const uint32_t limit = ((v1 ^ flip) | 0xFFu) + (P.max_dist << 8);
        const uint32_t* strobe = sp + i1 + dir * (int)P.w_min;
        uint32_t best = 0xFFFFFFFFu;
#pragma unroll 4
        for (uint32_t x = P.w_min; x <= P.w_max; ++x, strobe += dir) {
            const uint32_t v = *strobe;
            const uint32_t of = ((uint32_t)__popc((v ^ v1) & 0xFFu) << 16) | x;   // the first of the least
            if ((v ^ flip) <= limit) best = min(best, of);
        }
        const int i2 = best == 0xFFFFFFFFu ? i1 : i1 + dir * (int)(best & 0xFFFFu);
        const uint32_t p1 = (v1 >> 8) - kFastShift, p2 = (sp[i2] >> 8) - kFastShift;
        const uint32_t s1 = rev ? L - p1 - k : p1, e2 = rev ? L - p2 : p2 + k;
        se = s1 | (e2 << 10) | (i << 20);
        key = sh[i1] + sh[i2];
    };
    for (uint32_t round = 0; 32 * round < nq2; ++round) {
        const uint32_t i = 32 * round + lane;
        Candidates c;
        c.match = 0;
        uint64_t key = 0;
        uint32_t se = 0;
        if (i < nq2) {
            select(i, key, se);
            c = bucket_candidates(load_bucket(I, key), key);
        }
        // queries with candidates wait until there are 32 of them (or no more to come)
        const uint32_t some = __ballot_sync(kFull, c.match != 0);
        if (c.match) {
            const uint32_t at = pending + __popc(some & lanemask_lt());
            Q.key[at] = key;
            Q.start[at] = c.start;
            Q.what[at] = c.match | (c.size << 16);
            Q.se[at] = se;
        }
        pending += __popc(some);
        __syncwarp();
        while (pending >= 32 || (pending && 32 * (round + 1) >= nq2)) {
            const uint32_t m = min(pending, 32u);
            Probe p;
            p.pos = kMissing;
            p.filtered = false;
            uint32_t x = 0;
            if (lane < m) {
                Candidates d;
                d.start = Q.start[lane];
                d.match = Q.what[lane] & 0xFFFFu;
                d.size = Q.what[lane] >> 16;
                x = Q.se[lane];
                p = probe_candidates(I, Q.key[lane], (int)((x >> 10) & 0x3FFu) - (int)(x & 0x3FFu), d);
            }
            const uint32_t is = __ballot_sync(kFull, p.pos != kMissing);
            good += __popc(__ballot_sync(kFull, p.pos != kMissing && !p.filtered));
            // the found ones to their places, their hits' number to the lane that writes them
            if (p.pos != kMissing) {
                const uint32_t at = tot + __popc(is & lanemask_lt());
                found[at] = make_uint4(x, p.pos, p.position, p.packed);
                Q.hits[at & 31] = (uint8_t)p.n_hits;
            }
            __syncwarp();
            const uint32_t mine = tot + ((lane - tot) & 31u);
            if (mine < tot + __popc(is)) {
                const uint32_t nh = Q.hits[lane];
                hits |= (uint64_t)nh << (8 * (mine >> 5));
                sum += nh;
            }
            tot += __popc(is);
            pending -= m;
            // what is left moves to the front (fewer than 32)
            uint64_t rk = 0;
            uint32_t r0 = 0, r1 = 0, r2 = 0;
            if (lane < pending) {
                rk = Q.key[32 + lane];
                r0 = Q.start[32 + lane];
                r1 = Q.what[32 + lane];
                r2 = Q.se[32 + lane];
            }
            __syncwarp();
            if (lane < pending) {
                Q.key[lane] = rk;
                Q.start[lane] = r0;
                Q.what[lane] = r1;
                Q.se[lane] = r2;
            }
            __syncwarp();
        }
    }
    ReadRec& R = rec[r];
    // nonrepetitive_fraction (step2/nam.cu:892) and the rescue trigger, as in lookup_read
    const float frac = tot > 0 ? ((float)good) / ((float)tot) : 1.0f;
    const bool rescue = C.rescue_level > 1 && (good == 0 || (double)frac < 0.7);
    if (lane == 0) {
        R.frac = frac;
        R.n_found = tot;
    }
    if (rescue) {
        // the rescue kernel reads the found queries from the arena
        const uint64_t off = warp_bump(&ctr->q_used, nq2);
        if (off + nq2 > A.q_cap) {
            warp_fail(R, ctr, kStatusQueryOverflow);
            if (lane == 0) R.nq = R.nq2 = 0;
            return true;
        }
        if (lane == 0) {
            R.q_off = off;
            R.nq = nq;
            R.nq2 = nq2;
        }
        for (uint32_t i = lane; i < nq2; i += 32) A.q_pos[off + i] = kNotFound;
        __syncwarp();
        for (uint32_t f = lane; f < tot; f += 32) {
            const uint4 v = found[f];
            const uint32_t i = v.x >> 20;
            A.q[off + i] = Query{0, v.x & 0x3FFu, (v.x >> 10) & 0x3FFu};
            A.q_pos[off + i] = v.y;
        }
        __syncwarp();
        enlist_rescue(I, C, r, R, A, ctr, good < tot);
        __syncwarp();
        return true;
    }
    const uint32_t H = __reduce_add_sync(kFull, sum);
    direct += nq2;
    const uint64_t hoff = room.take(&ctr->hit_used, H, arena_piece(A.hit_cap));
    if (hoff + H > A.hit_cap) {
        warp_fail(R, ctr, kStatusHitOverflow);
        return true;
    }
    // the hits in generation order (query order, then run order)
    HitPacked* out = A.hits + hoff;
    uint32_t at = 0;
    for (uint32_t round = 0; 32 * round < tot; ++round) {
        const uint32_t nh = (uint32_t)(hits >> (8 * round)) & 0xFFu;
        const uint32_t any = __ballot_sync(kFull, nh != 0);
        if (!any) continue;
        uint32_t to = at + __popc(any & lanemask_lt());
        if (__any_sync(kFull, nh > 1)) {
            const uint32_t inc = warp_inclusive_sum(nh);
            to = at + inc - nh;
            at += __shfl_sync(kFull, inc, 31);
        } else {
            at += __popc(any);
        }
        if (nh) {
            const uint4 f = found[32 * round + lane];
            const uint32_t rc = (f.x >> 20) >= nq ? 0x80000000u : 0u;
            const int qs = (int)(f.x & 0x3FFu), qe = (int)((f.x >> 10) & 0x3FFu);
            if (nh == 1) {
                out[to] = pack_hit(rc | (f.w >> 8), qs, qe, (int)f.z, (int)(f.z + (f.w & 0xFFu) + k));
            } else {
                walk_hit_run(I, qs, qe, f.y, [&](uint32_t ref, int rs, int re) {
                    out[to++] = pack_hit(rc | ref, qs, qe, rs, re);
                }, nullptr, nh);
            }
        }
    }
    if (lane == 0) {
        R.hit_off = hoff;
        R.n_hits = H;
    }
    __syncwarp();
    return true;
}

// The same read by the steps: seeding into the query arena, then lookup_read.  Reads that do
// not fit the shared-memory buffers go to the long list.
template <bool kCount, bool kLookup>
__device__ __forceinline__ void step_read(const DevParams& P, const IndexView& I, const MapConfig& C,
                                          const uint8_t* seq, uint32_t L, uint32_t r, ReadRec* rec, const Arenas& A,
                                          Counters* ctr, uint64_t* pk, uint32_t* nm, uint64_t* hb, uint64_t* sh,
                                          uint32_t* sp, uint32_t max_len, uint32_t cap, WarpRoom& queries,
                                          WarpRoom& hits) {
    ReadRec& R = rec[r];
    uint32_t ns = 0xFFFFFFFFu;
    if (L <= max_len) ns = warp_read_syncmers(P, seq, L, pk, nm, hb, sh, sp, cap);
    if (ns == 0xFFFFFFFFu) {
        if (lane_id() == 0) {
            R.flags |= kReadLong;
            A.long_list[atomicAdd(&ctr->n_long, 1u)] = r;
        }
        return;
    }
    emit_read_queries(P, sh, sp, ns, L, R, A, ctr, queries);
    __syncwarp();
    if (kLookup) {
        lookup_read<kCount>(I, C, r, rec, A, ctr, hits);
        __syncwarp();
    }
}

// step_read beside the fast path: out of line, for the few reads that need it, which take just
// the arena room that they use (a piece each, of which a read leaves nine tenths, made batches
// of many such reads outgrow the arenas).
__device__ __noinline__ void slow_read(const DevParams& P, const IndexView& I, const MapConfig& C, const uint8_t* seq,
                                       uint32_t L, uint32_t r, ReadRec* rec, const Arenas& A, Counters* ctr,
                                       uint64_t* pk, uint32_t* nm, uint64_t* hb, uint64_t* sh, uint32_t* sp,
                                       uint32_t max_len, uint32_t cap) {
    WarpRoom queries, hits;
    queries.most = hits.most = 0;
    step_read<false, true>(P, I, C, seq, L, r, rec, A, ctr, pk, nm, hb, sh, sp, max_len, cap, queries, hits);
}

// A read of the fast kernels: in one go, else by the steps.
template <uint32_t kMaxLen, uint32_t kSyncmers>
__device__ __forceinline__ void fast_or_slow_read(const DevParams& P, const IndexView& I, const MapConfig& C,
                                                  const uint8_t* seq, uint32_t L, uint32_t r, ReadRec* rec,
                                                  const Arenas& A, Counters* ctr, uint64_t* pk, uint32_t* nm,
                                                  uint64_t* hb, uint64_t* sh, uint32_t* sp, FastQueue& Q,
                                                  WarpRoom& room, uint32_t& direct) {
    if (L > kMaxLen ||
        !fast_read(P, I, C, seq, L, r, rec, A, ctr, pk, nm, hb, sh, sp + kFastPad, kSyncmers, Q, room, direct))
        slow_read(P, I, C, seq, L, r, rec, A, ctr, pk, nm, hb, sh, sp, kMaxLen, kSyncmers);
}

// Seeding and lookup of a read by one warp (the main path): randstrobes_query, then
// the query loop of find_nams on the queries just written.  Seeding is bound by
// integer issue and the lookup by the latency of random index reads, so the warps of
// an SM interleave the two: while some wait on gathers, others hash.  Reads that do
// not fit the shared-memory buffers go to the long list (k_seed_long, then
// k_lookup_long).
// 4 blocks of 8 warps per SM: 64 registers, with which nothing spills (6 blocks, 40
// registers: 10% more instructions; 2M reads 9.03 ms a batch, 5 blocks 8.78, 4 blocks 8.83,
// uneven lengths 1.44 / 1.45 / 1.43), and per-warp buffers for reads up to 512 bases and 160
// syncmers (33 KB per block, leaving the rest of the SM's unified L1 to cache index
// entries); longer reads take the long path.
constexpr int kFusedBlocksPerSm = 4;
constexpr uint32_t kFusedMaxLen = 512;
constexpr uint32_t kFusedSyncmers = 160;

template <bool kCount, bool kFast>
__global__ void __launch_bounds__(32 * kSeedWarps, kFusedBlocksPerSm)
    k_seed_lookup(DevParams P, IndexView I, MapConfig C, const uint8_t* __restrict__ seqs,
                  const uint64_t* __restrict__ offs, const uint32_t* __restrict__ lens, uint32_t n,
                  ReadRec* __restrict__ rec, Arenas A, Counters* ctr) {
    __shared__ uint64_t s_pk[kSeedWarps][kFusedMaxLen / 32 + 4];
    __shared__ uint32_t s_nm[kSeedWarps][kFusedMaxLen / 32 + 4];
    __shared__ uint64_t s_hb[kSeedWarps][64];
    __shared__ uint64_t s_sh[kSeedWarps][kFusedSyncmers];
    __shared__ uint32_t s_sp[kSeedWarps][kFusedSyncmers + 2 * kFastPad];
    __shared__ FastQueue s_q[kFast ? kSeedWarps : 1];
    const uint32_t w = threadIdx.x >> 5;
    WarpItems items(n);
    WarpRoom room, queries;
    uint32_t direct = 0;
    for (uint32_t r; (r = items.next(&ctr->queue_head)) < n;) {
        const uint32_t L = lens[r];
        if (L > GBSA_MAX_READ_LEN) {
            warp_fail(rec[r], ctr, kStatusReadTooLong);
            continue;
        }
        if (kFast)
            fast_or_slow_read<kFusedMaxLen, kFusedSyncmers>(P, I, C, seqs + offs[r], L, r, rec, A, ctr, s_pk[w],
                                                            s_nm[w], s_hb[w], s_sh[w], s_sp[w], s_q[kFast ? w : 0],
                                                            room, direct);
        else
            step_read<kCount, true>(P, I, C, seqs + offs[r], L, r, rec, A, ctr, s_pk[w], s_nm[w], s_hb[w], s_sh[w],
                                    s_sp[w], kFusedMaxLen, kFusedSyncmers, queries, room);
    }
    room.done(&ctr->hit_spare);
    if (!kFast) queries.done(&ctr->q_spare);
    if (direct && lane_id() == 0) atomicAdd(&ctr->q_direct, (unsigned long long)direct);
}

// The batched form's seeding + lookup: the body of k_seed_lookup, but each warp pulls
// work items from a device queue (an atomic counter) until the batch's items run out,
// so reads of uneven lengths and the two mates of a pair (one item) balance over the
// persistent grid; the batch (reads, count, items) is read from desc in device memory.
// The shape (warps per block, resident blocks per SM, shared-memory read window) is a
// template of its own per variant, picked at run time.
// kLookup false: seeding alone (indexes whose entries exceed the fuse limit are looked
// up by k_lookup afterwards, as in the plain form).
template <bool kCount, bool kLookup, bool kFast, int kWarps, int kBlocks, uint32_t kMaxLen, uint32_t kSyncmers>
__global__ void __launch_bounds__(32 * kWarps, kBlocks)
    k_seed_lookup_q(DevParams P, IndexView I, MapConfig C, const BatchDesc* __restrict__ desc,
                    ReadRec* __restrict__ rec, Arenas A, Counters* ctr) {
    __shared__ uint64_t s_pk[kWarps][kMaxLen / 32 + 4];
    __shared__ uint32_t s_nm[kWarps][kMaxLen / 32 + 4];
    __shared__ uint64_t s_hb[kWarps][64];
    __shared__ uint64_t s_sh[kWarps][kSyncmers];
    __shared__ uint32_t s_sp[kWarps][kSyncmers + 2 * kFastPad];
    __shared__ FastQueue s_q[kFast ? kWarps : 1];
    const uint32_t w = threadIdx.x >> 5;
    const uint8_t* __restrict__ seqs = desc->seqs;
    const uint64_t* __restrict__ offs = desc->offs;
    const uint32_t* __restrict__ lens = desc->lens;
    const uint32_t* __restrict__ items = desc->items;
    const uint32_t n_items = items ? desc->n_items : desc->n_reads;
    WarpItems queue(n_items);
    WarpRoom room, queries;
    uint32_t direct = 0;
    for (uint32_t it; (it = queue.next(&ctr->queue_head)) < n_items;) {
        // item bounds outside [0, n_reads] are clamped (reads no item covers stay empty)
        const uint32_t n_reads = desc->n_reads;
        const uint32_t r0 = min(items ? items[it] : it, n_reads);
        const uint32_t r1 = min(items ? items[it + 1] : it + 1, n_reads);
        for (uint32_t r = r0; r < r1; ++r) {
            const uint32_t L = lens[r];
            if (L > GBSA_MAX_READ_LEN) {
                warp_fail(rec[r], ctr, kStatusReadTooLong);
                continue;
            }
            if (kFast)
                fast_or_slow_read<kMaxLen, kSyncmers>(P, I, C, seqs + offs[r], L, r, rec, A, ctr, s_pk[w], s_nm[w],
                                                      s_hb[w], s_sh[w], s_sp[w], s_q[kFast ? w : 0], room, direct);
            else
                step_read<kCount, kLookup>(P, I, C, seqs + offs[r], L, r, rec, A, ctr, s_pk[w], s_nm[w], s_hb[w],
                                           s_sh[w], s_sp[w], kMaxLen, kSyncmers, queries, room);
        }
    }
    room.done(&ctr->hit_spare);
    if (!kFast) queries.done(&ctr->q_spare);
    if (direct && lane_id() == 0) atomicAdd(&ctr->q_direct, (unsigned long long)direct);
}

// Scratch of `bytes` for the calling warp: its own slot from byte `slot_off` on when
// the request fits, else a bump allocation in the shared overflow arena (nullptr
// when that is full too).
__device__ __forceinline__ uint8_t* warp_scratch(const Arenas& A, Counters* ctr, uint64_t slot_off, uint64_t bytes) {
    bytes = (bytes + 255) & ~255ull;   // keep every region 256-byte aligned
    const uint32_t slot = warp_global_id();
    if (slot < A.n_slots && slot_off + bytes <= A.slot_bytes) return A.slots + (uint64_t)slot * A.slot_bytes + slot_off;
    const uint64_t o = warp_bump(&ctr->scratch_used, bytes);
    if (o + bytes > A.ovf_cap) return nullptr;
    return A.ovf + o;
}


// Scores, sorts and writes the closed NAMs of a read to the NAM arena.  keys needs
// room for next_pow2(n_closed) entries.
// Warp bitonic sort of P (a power of two) entries that moves only the first key word
// (k1) and the NAM index (ix); the second and third words stay by NAM index and are
// read when the first words tie.
__device__ void warp_sort_idx(uint64_t* k1, uint32_t* ix, const uint64_t* k2, const uint64_t* k3, uint32_t P) {
    const uint32_t lane = lane_id();
    for (uint32_t k = 2; k <= P; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t q = lane; q < P / 2; q += 32) {
                const uint32_t i = ((q & ~(j - 1)) << 1) | (q & (j - 1));
                const uint32_t ixj = i | j;
                const uint64_t xb = k1[ixj], xa = k1[i];
                bool less;
                if (xb != xa) {
                    less = xb < xa;
                } else {
                    const uint32_t ib = ix[ixj], ia = ix[i];
                    const uint64_t b2 = k2[ib], a2 = k2[ia], b3 = k3[ib], a3 = k3[ia];
                    less = b2 != a2 ? b2 < a2 : (b3 != a3 ? b3 < a3 : ib < ia);
                }
                if (less == ((i & k) == 0)) {
                    k1[i] = xb;
                    k1[ixj] = xa;
                    const uint32_t t = ix[i];
                    ix[i] = ix[ixj];
                    ix[ixj] = t;
                }
            }
            __syncwarp();
        }
    }
}

// Sorts a rescued read's NN <= kWarpSortMax NAMs with the warp in its shared buffer (7 KB,
// free after the merge) and writes them to the NAM arena.
__device__ void warp_finish_nams(const MapConfig& C, const NamState* closed, uint32_t NN, uint32_t* buf, ReadRec& R,
                                 const Arenas& A, Counters* ctr) {
    const uint32_t lane = lane_id();
    const uint32_t P = next_pow2(NN);
    uint64_t* k1 = reinterpret_cast<uint64_t*>(buf);      // P <= 256: 2 KB
    uint64_t* k2 = k1 + 256;                              // 2 KB
    uint64_t* k3 = k2 + 256;                              // 2 KB
    uint32_t* ix = reinterpret_cast<uint32_t*>(k3 + 256); // 1 KB
    for (uint32_t t = lane; t < P; t += 32) {
        NamKey k;
        if (t < NN) {
            k = nam_key(closed[t], t, C.sort_mode);
        } else {   // padding sorts last (a NAM's first key word is never all ones)
            k.k1 = k.k2 = k.k3 = ~0ULL;
        }
        k1[t] = k.k1;
        ix[t] = t;
        k2[t] = k.k2;
        k3[t] = k.k3;
    }
    __syncwarp();
    warp_sort_idx(k1, ix, k2, k3, P);
    const uint64_t noff = warp_bump(&ctr->nam_used, NN);
    if (noff + NN > A.nam_cap) {
        warp_fail(R, ctr, kStatusNamOverflow);
        return;
    }
    for (uint32_t t = lane; t < NN; t += 32) A.nams[noff + t] = closed[ix[t]];
    if (lane == 0) {
        R.nam_off = noff;
        R.n_nams = NN;
    }
    __syncwarp();
}

// ---- the NAM merge in registers --------------------------------------------------------
//
// find_nams merge with the read's NAMs in registers: a group of G lanes (4 to 32 by hit
// count) takes a read, 32 / G reads a warp, with R slots a lane: NAM i is slot (row) i / G
// of lane i % G.  Slots are never given back (a read has at most as many NAMs as hits;
// the few reads with more NAMs than slots go to a list in memory), so slot order is
// creation order.  The hit-major rule of merge_hits_into_nams (step2/nam.cu:347-513): hits
// in (orientation, query_start, position) order, each joins the first NAM in creation order
// that accepts it, found with one ballot a row; a NAM that the query start has passed, or of the other
// orientation, accepts nothing, so it needs no closing (rows with no other NAM are
// skipped).  The NAMs are then ranked by their keys through shared memory and written
// once, in order.
//
// A lane a read (open NAMs in shared memory) ran 7.9 of 32 lanes an instruction at 15%
// occupancy, waiting on shared memory, and its sort of many NAMs went through HBM: one
// read of 128 hits took as long as a thousand reads.
constexpr int kGroupWarps = 4;
constexpr int kGroupBlocksPerSm = 8;     // 64 registers a thread
// The rescue chain runs beside the NAM kernels on another stream; the persistent grids are
// sized so that its blocks (RescueShared, 97 KB each) keep room beside them.
constexpr int kRescueBlocksPerSm = 2;

__device__ __forceinline__ HitRec load_hit(const HitPacked* __restrict__ hits, uint32_t i, uint32_t H) {
    HitRec h;
    if (i < H) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(hits + i));
        h.ref_rc = v.x;
        h.qs = (int32_t)(v.y & 0xFFFFu);
        h.qe = (int32_t)(v.y >> 16);
        h.rs = (int32_t)v.z;
        h.re = (int32_t)v.w;
    } else {
        h.ref_rc = 0;
        h.qs = h.qe = h.rs = h.re = -1;
    }
    return h;
}

// Hit-count bucket of a read for the register merge: 8 wide up to 64 hits, 32 wide up to
// 128, 64 wide up to 256, then one for all above.
__device__ __forceinline__ uint32_t lane_bucket(uint32_t H) {
    if (H <= 64) return (H - 1) >> 3;
    if (H <= 128) return 8 + ((H - 65) >> 5);
    return H <= 256 ? 10 + ((H - 129) >> 6) : kLaneBuckets - 1;
}

// Sorts the reads with hits into lists by hit count for the register merge, so that the
// groups of a warp merge reads of similar size (a warp runs as long as its longest read).
// Appends are aggregated per warp and bucket.
__global__ void k_bucket_reads(uint32_t n, const ReadRec* __restrict__ rec, Arenas A, Counters* ctr,
                               const BatchDesc* desc) {
    if (desc) n = min(n, desc->n_reads);
    const uint32_t lane = lane_id();
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
        const uint32_t r = base + threadIdx.x;
        uint32_t key = 0xFFFFFFFFu;   // no list
        if (r < n) {
            const uint32_t flags = rec[r].flags;
            const uint32_t H = rec[r].n_hits;
            if (!(flags & (kReadFailed | kReadRescue)) && H > 0) key = lane_bucket(H);
        }
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, key);
        const uint32_t leader = __ffs(peers) - 1;
        uint32_t at = 0;
        if (key != 0xFFFFFFFFu && lane == leader)
            at = atomicAdd(&ctr->lane_cnt[key], (unsigned)__popc(peers));
        at = __shfl_sync(0xFFFFFFFFu, at, leader) + __popc(peers & lanemask_lt());
        if (key != 0xFFFFFFFFu) A.lane_lists[(size_t)key * A.lane_cap + at] = r;
    }
}

// Shared memory of a warp's register merge: the hits in flight, and the NAMs' sort keys by
// slot (row * 32 + lane).
template <int R>
struct GroupShared {
    uint4 hits[2][32];
    uint64_t k1[32 * R], k2[32 * R], k3[32 * R];
    uint8_t at[32 * R];   // slot that took a rank
};

// f(r) for every row, r a compile-time constant (the rows' state must stay in registers).
template <class F, int... I>
__device__ __forceinline__ void each_row_of(std::integer_sequence<int, I...>, F&& f) {
    (f(std::integral_constant<int, I>{}), ...);
}
template <int R, class F>
__device__ __forceinline__ void each_row(F&& f) {
    each_row_of(std::make_integer_sequence<int, R>{}, f);
}

// Merges the reads list[first ..] (one a group of G lanes, those below cnt) and writes
// their sorted NAMs; S: the warp's shared memory.  Returns a group's read with more than
// G * R NAMs in its lanes (its NAMs are not written), else kNoRead.
// kLong (G 32): NAMs that can take no more hits leave full lanes for `closed` (room for the
// read's hits), which holds all of them in creation order at the end, `n_closed`; a read with
// more than kFewOpen NAMs left in full lanes is returned.
constexpr uint32_t kNoRead = 0xFFFFFFFFu;
constexpr uint32_t kFewOpen = 96;
template <int G, int R, bool kLong = false>
__device__ uint32_t group_merge(const MapConfig& C, ReadRec* __restrict__ rec, const Arenas& A, Counters* ctr,
                                const uint32_t* __restrict__ list, uint32_t first, uint32_t cnt, GroupShared<R>& S,
                                WarpRoom& room, NamState* closed = nullptr, uint32_t* n_closed = nullptr) {
    constexpr uint32_t kFull = 0xFFFFFFFFu;
    constexpr uint32_t kNoRef = 0xFFFFFFFFu;   // a hit's reference id has 24 bits
    const uint32_t lane = lane_id();
    const uint32_t sub = lane & (G - 1), base = lane & ~(uint32_t)(G - 1);
    const uint32_t gmask = (G == 32 ? kFull : (1u << (G & 31)) - 1) << base;
    const uint32_t at = first + lane / G;
    const bool have = at < cnt;
    const uint32_t rd = have ? list[at] : 0;
    const uint32_t H = have ? rec[rd].n_hits : 0;
    const uint4* hits = reinterpret_cast<const uint4*>(A.hits + (have ? rec[rd].hit_off : 0));
    const uint32_t Hm = __reduce_max_sync(kFull, H);
    int32_t rs[R], re[R], rp[R];
    uint32_t ref[R], qep[R], qn[R];   // qep: query end << 16 | previous hit's start; qn: n_hits << 16 | query start
    each_row<R>([&](auto row_c) {
        constexpr int r = decltype(row_c)::value;
        ref[r] = kNoRef;
        qep[r] = qn[r] = 0;
        rs[r] = re[r] = rp[r] = 0;
    });
    uint32_t n = 0;              // the group's NAMs
    uint32_t rows = 0, live = 0; // rows in use by any group, and those that may still accept a hit (bits)
    // the group's hits, G at a time through shared memory, the next G in flight
    const uint4 none = make_uint4(kNoRef - 1, 0, 0, 0);
    uint4 nx = sub < H ? __ldg(hits + sub) : none;
    bool over = false;
    auto nam = [&](int r) {
        NamState m;
        m.qs = (int32_t)(qn[r] & 0xFFFFu);
        m.qe = (int32_t)(qep[r] >> 16);
        m.qprev = (int32_t)(qep[r] & 0xFFFFu);
        m.rs = rs[r];
        m.re = re[r];
        m.rprev = rp[r];
        m.n_hits = (int32_t)(qn[r] >> 16);
        m.ref_rc = ref[r];
        return m;
    };
    uint32_t* number = reinterpret_cast<uint32_t*>(S.k3);   // kLong: of each slot's NAM
    uint32_t created = 0;
    for (uint32_t c = 0; c < Hm; c += G) {
        uint4* buf = S.hits[(c / G) & 1];
        buf[lane] = nx;
        nx = c + G + sub < H ? __ldg(hits + c + G + sub) : none;
        __syncwarp();
        const uint32_t steps = min((uint32_t)G, Hm - c);
        if (R <= 4 && rows > 1) {   // rows the query start has passed in every group
            const uint4 v = buf[base];
            const uint32_t xqs = v.y & 0xFFFFu;
            live = 0;
            each_row<R>([&](auto row_c) {
                constexpr int r = decltype(row_c)::value;
                if ((uint32_t)r < rows &&
                    __any_sync(kFull, ref[r] != kNoRef && (int32_t)(ref[r] ^ v.x) >= 0 && (qep[r] >> 16) >= xqs))
                    live |= 1u << r;
            });
        }
        for (uint32_t j = 0; j < steps; ++j) {
            const uint4 v = buf[base + j];
            const uint32_t xqs = v.y & 0xFFFFu, xqe = v.y >> 16;
            const int32_t xrs = (int32_t)v.z, xre = (int32_t)v.w;
            bool done = c + j >= H;
            // rows where some NAM could take the hit by its reference interval: most fail this
            // (with 8 slots a lane the rows are tested without branches, so that their
            // latencies overlap: that merge is a few long reads, each on one warp)
            uint32_t may = 0;
            auto in_ref = [&](int r) { return ref[r] == v.x && rp[r] < xrs && xrs <= re[r]; };
            if (R > 4)
                each_row<R>([&](auto row_c) {
                    constexpr int r = decltype(row_c)::value;
                    may |= __any_sync(kFull, in_ref(r)) ? 1u << r : 0u;
                });
            each_row<R>([&](auto row_c) {
                constexpr int r = decltype(row_c)::value;
                if (R > 4 ? !((may >> r) & 1u) : (!((live >> r) & 1u) || !__any_sync(kFull, in_ref(r)))) return;
                const uint32_t qe = qep[r] >> 16;
                const bool ok = !done && in_ref(r) && (qep[r] & 0xFFFFu) < xqs && xqs <= qe &&
                                (xqe > qe) == (xre > re[r]);
                const uint32_t b = __ballot_sync(kFull, ok) & gmask;
                if (ok && (b & lanemask_lt()) == 0) {   // the first accepting NAM takes the hit
                    qep[r] = (max(qe, xqe) << 16) | xqs;   // both ends grow or neither
                    re[r] = max(re[r], xre);
                    rp[r] = xrs;
                    qn[r] += 1u << 16;
                }
                done = done || b != 0;
            });
            // a hit that no NAM took opens one in the group's next slot
            if (__any_sync(kFull, !done)) {
                if (n == G * R) {   // (never for reads of up to G * R hits)
                    if constexpr (kLong) {   // the NAMs that may take another hit move to the front
                        uint32_t open = 0, to[R];
                        each_row<R>([&](auto row_c) {
                            constexpr int r = decltype(row_c)::value;
                            const bool stay = (int32_t)(ref[r] ^ v.x) >= 0 && (qep[r] >> 16) >= xqs;
                            const uint32_t b = __ballot_sync(kFull, stay);
                            to[r] = stay ? open + __popc(b & lanemask_lt()) : kNoRef;
                            open += __popc(b);
                        });
                        if (open > kFewOpen) return rd;
                        uint32_t* word = reinterpret_cast<uint32_t*>(S.k1);
                        auto move = [&](auto& x) {
                            each_row<R>([&](auto row_c) {
                                constexpr int r = decltype(row_c)::value;
                                if (to[r] != kNoRef) word[to[r]] = (uint32_t)x[r];
                            });
                            __syncwarp();
                            each_row<R>([&](auto row_c) {
                                constexpr int r = decltype(row_c)::value;
                                if (r * G + lane < open) x[r] = word[r * G + lane];
                            });
                            __syncwarp();
                        };
                        uint32_t at[R];
                        each_row<R>([&](auto row_c) {
                            constexpr int r = decltype(row_c)::value;
                            at[r] = number[r * G + lane];
                            if (to[r] == kNoRef) closed[at[r]] = nam(r);
                        });
                        move(ref);
                        move(qep);
                        move(qn);
                        move(rs);
                        move(re);
                        move(rp);
                        move(at);
                        each_row<R>([&](auto row_c) {
                            constexpr int r = decltype(row_c)::value;
                            number[r * G + lane] = at[r];
                            if (r * G + lane >= open) ref[r] = kNoRef;
                        });
                        n = open;
                        rows = (n + G - 1) / G;
                        live = (1u << rows) - 1;
                    } else {
                        over = true;
                        done = true;
                    }
                }
                const bool mine = !done && sub == (n & (G - 1));
                each_row<R>([&](auto row_c) {
                    constexpr int r = decltype(row_c)::value;
                    if (mine && n / G == (uint32_t)r) {
                        ref[r] = v.x;
                        qep[r] = (xqe << 16) | xqs;
                        rs[r] = xrs;
                        re[r] = xre;
                        rp[r] = xrs;
                        qn[r] = (1u << 16) | xqs;
                        if (kLong) number[r * G + lane] = created;
                    }
                });
                if (kLong) ++created;
                const uint32_t row = done ? 0u : 1u << (n / G);
                const uint32_t opened = G == 32 ? row : __reduce_or_sync(kFull, row);
                if (!done) ++n;
                live |= opened;
                rows = max(rows, 32u - (uint32_t)__clz(opened));
            }
        }
        if (G == 32 && over) return rd;
    }
    if constexpr (kLong) {
        __syncwarp();
        each_row<R>([&](auto row_c) {
            constexpr int r = decltype(row_c)::value;
            if (r * G + lane < n) closed[number[r * G + lane]] = nam(r);
        });
        __syncwarp();
        *n_closed = created;
        return kNoRead;
    }
    // ranks by the first key word (a NAM's is never all ones), one byte a row
    uint64_t ranks = 0;
    each_row<R>([&](auto row_c) {
        constexpr int r = decltype(row_c)::value;
        if ((uint32_t)r < rows) S.k1[32 * r + lane] = r * G + sub < n ? nam_key(nam(r), 0, C.sort_mode).k1 : ~0ULL;
    });
    __syncwarp();
    const uint32_t nm = __reduce_max_sync(kFull, n);
    for (uint32_t r = 0; r < rows; ++r) {   // (the keys are read by slot: no register array is indexed)
        const uint64_t mine = S.k1[32 * r + lane];
        uint32_t rank = 0;
        for (uint32_t row = 0; row * G < nm; ++row) {
            const uint64_t* k = S.k1 + 32 * row + base;
            const uint32_t in_row = min((uint32_t)G, nm - row * G);
#pragma unroll 4
            for (uint32_t j = 0; j < in_row; ++j) rank += k[j] < mine ? 1u : 0u;
        }
        if (r * G + sub < n) S.at[R * base + rank] = (uint8_t)(r * G + sub);
        ranks |= (uint64_t)(rank & 0xFFu) << (8 * r);
    }
    __syncwarp();
    // NAMs whose first words tie took the same rank: then all three words and the
    // creation order decide
    bool tie = false;
    each_row<R>([&](auto row_c) {
        constexpr int r = decltype(row_c)::value;
        if (r * G + sub < n) tie |= S.at[R * base + ((ranks >> (8 * r)) & 0xFFu)] != (uint8_t)(r * G + sub);
    });
    if (__any_sync(kFull, tie)) {
        each_row<R>([&](auto row_c) {
            constexpr int r = decltype(row_c)::value;
            if (r * G + sub < n) {
                const NamKey k = nam_key(nam(r), 0, C.sort_mode);
                S.k2[32 * r + lane] = k.k2;
                S.k3[32 * r + lane] = k.k3;
            }
        });
        __syncwarp();
        for (uint32_t f = lane; f < 32 * rows; f += 32) {   // the lane's slots again, by row
            const uint32_t own = (f >> 5) * G + sub;
            uint32_t more = 0;
            for (uint32_t o = 0; own < n && o < n; ++o) {
                const uint32_t e = 32 * (o / G) + base + (o & (G - 1));
                if (S.k1[e] != S.k1[f] || o == own) continue;
                const uint64_t a2 = S.k2[e], b2 = S.k2[f], a3 = S.k3[e], b3 = S.k3[f];
                if (a2 != b2 ? a2 < b2 : (a3 != b3 ? a3 < b3 : o < own)) ++more;
            }
            ranks += (uint64_t)more << (8 * (f >> 5));
        }
    }
    // NAM arena
    const uint32_t count = sub == 0 ? n : 0;
    const uint32_t inc = warp_inclusive_sum(count);
    const uint32_t total = __shfl_sync(kFull, inc, 31);
    const uint64_t off0 = room.take(&ctr->nam_used, total, arena_piece(A.nam_cap));
    const uint64_t off = off0 + __shfl_sync(kFull, inc - count, base);
    if (off0 + total > A.nam_cap) {
        if (have && sub == 0) {
            rec[rd].flags |= kReadFailed;
            atomicOr(&ctr->status, kStatusNamOverflow);
        }
        __syncwarp();
        return kNoRead;
    }
    each_row<R>([&](auto row_c) {
        constexpr int r = decltype(row_c)::value;
        if (r * G + sub < n) {
            // the fields of NamState in order
            uint4* to = reinterpret_cast<uint4*>(A.nams + off + ((ranks >> (8 * r)) & 0xFFu));
            to[0] = make_uint4(qn[r] & 0xFFFFu, qep[r] >> 16, qep[r] & 0xFFFFu, (uint32_t)rs[r]);
            to[1] = make_uint4((uint32_t)re[r], (uint32_t)rp[r], qn[r] >> 16, ref[r]);
        }
    });
    if (have && sub == 0) {
        rec[rd].nam_off = off;
        rec[rd].n_nams = n;
    }
    __syncwarp();
    return kNoRead;
}

// Lists a read with more NAMs than a warp's slots for k_nams: from the front, or, where its
// first queries have kFewHits hits or fewer each, from the back.  A query costs a block 3,500
// cycles whatever it brings, a hit a warp some 200, and the block sorts faster: reads of a few
// dozen queries with many hits each were slower by the warp (100k pairs 0.77 -> 0.86 ms, 100k
// reads of 250 bp 1.74 -> 2.15), reads of 4,000 bp by the block (see long_merge).
constexpr uint32_t kFewHits = 4;
__device__ __forceinline__ void list_big_read(const Arenas& A, Counters* ctr, uint32_t r, const ReadRec& R) {
    const uint32_t lane = lane_id();
    const uint4* hits = reinterpret_cast<const uint4*>(A.hits + R.hit_off);
    const uint32_t m = min(R.n_hits, 160u);   // (more than 128)
    uint32_t q = 0;
    for (uint32_t h = lane; h < m; h += 32) q += h == 0 || __ldg(&hits[h].y) != __ldg(&hits[h - 1].y) ? 1u : 0u;
    q = __reduce_add_sync(0xFFFFFFFFu, q);
    if (lane == 0) {
        if (m <= kFewHits * q) A.big_list[A.rescue_cap - 1 - atomicAdd(&ctr->n_few, 1u)] = r;
        else A.big_list[atomicAdd(&ctr->n_big, 1u)] = r;
    }
}

// The register merge: persistent warps take the reads by bucket from a work counter, the
// most hits first.  Groups of 4 lanes take reads of up to 16 hits, of 8 up to 32, of 16 up
// to 64, a warp all others; a read with more than 128 NAMs (one in a thousand) goes to
// k_nams.  4 slots a lane fit 64 registers, 32 warps an SM; with 8 slots (twice the reads
// a warp for the same hits) they took 128 registers and three times as long a hit.
__global__ void __launch_bounds__(32 * kGroupWarps, kGroupBlocksPerSm)
    k_nams_group(MapConfig C, ReadRec* __restrict__ rec, Arenas A, Counters* ctr) {
    __shared__ GroupShared<4> s_group[kGroupWarps];
    __shared__ uint32_t s_cnt[kLaneBuckets];
    if (threadIdx.x < kLaneBuckets) s_cnt[threadIdx.x] = *(volatile unsigned int*)&ctr->lane_cnt[threadIdx.x];
    __syncthreads();
    GroupShared<4>& S = s_group[threadIdx.x >> 5];
    uint32_t all = 0;
    for (uint32_t b = 0; b < kLaneBuckets; ++b) all += s_cnt[b];
    const uint32_t per = items_per_take(all / 4);
    WarpRoom room;
    uint32_t next = 0, left = 0;
    for (;; ++next, --left) {
        if (left == 0) {
            next = warp_take(&ctr->group_next, per);
            left = per;
        }
        uint32_t t = next;
        int b = (int)kLaneBuckets - 1;
        for (; b >= 0; --b) {
            const uint32_t shift = b < 2 ? 3u : (b < 4 ? 2u : (b < 8 ? 1u : 0u));   // log2 of the reads a warp
            const uint32_t items = (s_cnt[b] + (1u << shift) - 1) >> shift;
            if (t < items) {
                t <<= shift;
                break;
            }
            t -= items;
        }
        if (b < 0) break;
        const uint32_t* list = A.lane_lists + (size_t)b * A.lane_cap;
        if (b < 2) {
            group_merge<4, 4>(C, rec, A, ctr, list, t, s_cnt[b], S, room);
        } else if (b < 4) {
            group_merge<8, 4>(C, rec, A, ctr, list, t, s_cnt[b], S, room);
        } else if (b < 8) {
            group_merge<16, 4>(C, rec, A, ctr, list, t, s_cnt[b], S, room);
        } else {
            const uint32_t r = group_merge<32, 4>(C, rec, A, ctr, list, t, s_cnt[b], S, room);
            if (r != kNoRead) list_big_read(A, ctr, r, rec[r]);
            __syncwarp();
        }
    }
    room.done(&ctr->nam_spare);
}

// A NAM list in struct-of-arrays form (field f of NAM o at b[f * stride + o]), so that 32
// lanes reading one field of 32 NAMs touch 32 consecutive words.
struct OpenSoA {
    int32_t* b;
    uint32_t stride;
    __device__ int32_t* f(int k) const { return b + (size_t)k * stride; }
    __device__ NamState get(uint32_t o) const {
        NamState n;
        n.qs = b[o];
        n.qe = b[stride + o];
        n.qprev = b[2 * stride + o];
        n.rs = b[3 * stride + o];
        n.re = b[4 * stride + o];
        n.rprev = b[5 * stride + o];
        n.n_hits = b[6 * stride + o];
        n.ref_rc = (uint32_t)b[7 * stride + o];
        return n;
    }
    __device__ void put(uint32_t o, const NamState& n) const {
        b[o] = n.qs;
        b[stride + o] = n.qe;
        b[2 * stride + o] = n.qprev;
        b[3 * stride + o] = n.rs;
        b[4 * stride + o] = n.re;
        b[5 * stride + o] = n.rprev;
        b[6 * stride + o] = n.n_hits;
        b[7 * stride + o] = (int32_t)n.ref_rc;
    }
};

// Phase 1 of find_nams_rescue for one read (warp): RescueHit{position, count, qs,
// qe} of every found query of each orientation, sorted by (count, query_start) —
// query_start is unique per orientation, so this is the reference's
// (count, query_start, query_end) order (cmp1, step2/nam.cu:909-912); the prefix
// taken until (count > rescue_cutoff && taken >= 5) || count > cap
// (step2/nam.cu:960-969); re-sorted by query_start (cmp2).  rk/tk: 2 x Pq u64 each.
// Returns the sum and the maximum of the run lengths of the taken ones.
struct RescuePlan {
    uint32_t m[2];
    uint64_t bound;
    uint32_t maxrun;
};

// One orientation d: adds its taken prefix to plan.
__device__ void rescue_prepare_dir(const IndexView& I, const MapConfig& C, const Query* const* Qd,
                                   const uint64_t* const* Pd, const uint32_t* nqd, uint32_t Pq, uint64_t* buf, int d,
                                   RescuePlan& plan) {
    const uint32_t lane = lane_id();
    uint64_t* rk[2] = {buf, buf + Pq};
    uint64_t* tk[2] = {buf + 2 * Pq, buf + 3 * Pq};
    {
        uint32_t nd = 0;
        const uint32_t nq = nqd[d];
        for (uint32_t base = 0; base < nq; base += 32) {
            const uint32_t qi = base + lane;
            bool f = false;
            uint64_t key = 0;
            if (qi < nq) {
                const uint64_t pos = Pd[d][qi];
                if (pos != kNotFound) {
                    f = true;
                    const uint32_t cnt = index_get_count(I, pos);
                    key = ((uint64_t)cnt << 32) | ((uint64_t)Qd[d][qi].start << 16) | qi;
                }
            }
            const uint32_t bm = __ballot_sync(0xFFFFFFFFu, f);
            if (f) rk[d][nd + __popc(bm & lanemask_lt())] = key;
            nd += __popc(bm);
        }
        __syncwarp();
        warp_sort_u64(rk[d], nd);
        uint32_t stop = nd;
        for (uint32_t base = 0; base < nd; base += 32) {
            const uint32_t j = base + lane;
            bool brk = false;
            if (j < nd) {
                const uint32_t cnt = (uint32_t)(rk[d][j] >> 32);
                brk = (cnt > C.rescue_cutoff && j >= 5) || cnt > C.count_cap;
            }
            const uint32_t bm = __ballot_sync(0xFFFFFFFFu, brk);
            if (bm) {
                stop = base + (__ffs(bm) - 1);
                break;
            }
        }
        plan.m[d] = stop;
        uint64_t bsum = 0;
        uint32_t bmax = 0;
        for (uint32_t j = lane; j < stop; j += 32) {
            const uint32_t cnt = (uint32_t)(rk[d][j] >> 32);
            bsum += cnt;
            bmax = cnt > bmax ? cnt : bmax;
            tk[d][j] = ((rk[d][j] & 0xFFFFFFFFull) << 32) | cnt;   // (start, index) order, run length
        }
        plan.bound += warp_sum(bsum);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const uint32_t v = __shfl_xor_sync(0xFFFFFFFFu, bmax, o);
            bmax = v > bmax ? v : bmax;
        }
        plan.maxrun = bmax > plan.maxrun ? bmax : plan.maxrun;
        __syncwarp();
        warp_sort_u64(tk[d], stop);
    }
}

constexpr uint32_t kWarpSortMax = 256;   // rescued reads with more NAMs are sorted by k_sort_jobs
constexpr uint32_t kSortTile = 2048;      // keys per shared-memory tile of the small block sort (56 KB)
constexpr int kClusterCtas = 8;           // CTAs of a cluster sort
constexpr uint32_t kRescueSmemHits = 1024;// per-warp shared buffer for one query's hits

// Words a merge needs for queries of up to n hits: their positions, packed words and the
// NAM that claims each, and a bit each for the ones claimed by earlier NAMs.
__host__ __device__ constexpr uint32_t rescue_hit_words(uint32_t n) { return 3 * n + (n + 31) / 32; }

// Shared memory of the rescue kernel: a buffer a warp (a block's merge uses all warps'
// buffers as one).
struct RescueShared {
    uint32_t buf[kWarpsPerBlock][rescue_hit_words(kRescueSmemHits)];
    uint32_t cnt[kWarpsPerBlock];   // block merge: kept or untaken hits per warp
    int least[kWarpsPerBlock];      // block walk: least length difference per warp
    uint32_t item;
    uint8_t* scratch;
    RescuePlan plan[2];
};

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// warp_walk_run_n by the block: 128 entries a warp at a time (a run of up to 1024 in one
// pass); the running minimum and the kept hits' places cross the warps through S.
__device__ __forceinline__ uint32_t block_walk_run(const IndexView& I, int qs, int qe, uint64_t pos, uint32_t cnt,
                                                   uint32_t* rs_out, uint32_t* pk_out, RescueShared& S,
                                                   uint32_t& min_span, uint32_t& max_span) {
    constexpr uint32_t kFull = 0xFFFFFFFFu;
    const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
    const uint2* ent = reinterpret_cast<const uint2*>(I.rs + pos);   // (position, packed) at offset 8
    int carry = 0x7FFFFFFF;   // least difference of the passes before
    uint32_t n = 0, mn = 0xFFu, mx = 0;
    for (uint32_t pass = 0; pass < cnt; pass += 128 * kWarpsPerBlock) {
        const uint32_t base = pass + 128 * w;
        uint2 e[4];
        int before[4];   // least difference ahead of the entry, within the warp's 128
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t j = base + 32 * u + lane;
            e[u] = j < cnt ? __ldg(&ent[2 * (size_t)j + 1]) : make_uint2(0, 0);
        }
        int least = 0x7FFFFFFF;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int x = (qe - qs) - ((int)(e[u].y & 0xFF) + I.k);
            const int diff = base + 32 * u + lane < cnt ? (x < 0 ? -x : x) : 0x7FFFFFFF;
            int pm = diff;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(kFull, pm, o);
                if (lane >= (uint32_t)o) pm = min(pm, v);
            }
            const int ex = __shfl_up_sync(kFull, pm, 1);
            before[u] = lane ? min(ex, least) : least;
            least = min(least, __shfl_sync(kFull, pm, 31));
        }
        if (lane == 0) S.least[w] = least;
        __syncthreads();
        int ahead = carry;
        for (uint32_t v = 0; v < kWarpsPerBlock; ++v) {
            if (v < w) ahead = min(ahead, S.least[v]);
            carry = min(carry, S.least[v]);
        }
        uint32_t keep = 0, kept = 0;
        uint32_t km[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t j = base + 32 * u + lane;
            const int x = (qe - qs) - ((int)(e[u].y & 0xFF) + I.k);
            const bool take = j < cnt && (x < 0 ? -x : x) <= min(before[u], ahead);
            keep |= take ? 1u << u : 0u;
            km[u] = __ballot_sync(kFull, take);
            kept += __popc(km[u]);
        }
        if (lane == 0) S.cnt[w] = kept;
        __syncthreads();
        uint32_t to = n;
        for (uint32_t v = 0; v < kWarpsPerBlock; ++v) {
            if (v < w) to += S.cnt[v];
            n += S.cnt[v];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if ((keep >> u) & 1u) {
                const uint32_t k = to + __popc(km[u] & lanemask_lt());
                rs_out[k] = e[u].x;
                pk_out[k] = e[u].y;
                mn = min(mn, e[u].y & 0xFFu);
                mx = max(mx, e[u].y & 0xFFu);
            }
            to += __popc(km[u]);
        }
        __syncthreads();
    }
    mn = __reduce_min_sync(kFull, mn);
    mx = __reduce_max_sync(kFull, mx);
    if (lane == 0) {
        S.least[w] = (int)mn;
        S.cnt[w] = mx;
    }
    __syncthreads();
    for (uint32_t v = 0; v < kWarpsPerBlock; ++v) {
        mn = min(mn, (uint32_t)S.least[v]);
        mx = max(mx, S.cnt[v]);
    }
    min_span = mn + (uint32_t)I.k;
    max_span = mx + (uint32_t)I.k;
    return n;   // (the caller synchronises before the hits are read or S is written again)
}

// Merges one query's hits into the NAMs [lo, n) of its orientation d in O (struct of
// arrays, in creation order) and returns the new number of NAMs: hits h of nh (positions
// hrs, packed words hpk as in the index, sorted by position, all from query_start qs to
// query_end qe, of spans min_span to max_span).  claim: kFree for every hit, gone: their bits
// 0; the team (kBlock: the block, else the warp) has synchronised since they were written,
// and has again on return.  cnt: a word a warp (kBlock).
//
// Which hit joins which NAM.  NAM-major (merge_hits_into_nams_fast, step2/nam.cu:94-343):
// for each open NAM in creation order, the first hit that it accepts and that no NAM before
// it took.  Hit-major (merge_hits_into_nams, step2/nam.cu:347-513): for each hit in order,
// the first NAM in creation order that accepts it (a NAM takes one hit of a query, as the
// next must start behind it).  Both give the one pairing that no NAM and hit would leave
// for each other, NAMs preferring earlier hits and hits earlier NAMs, and that is what all
// proposing at once comes to, each NAM to its first acceptable hit, a hit keeping the NAM
// created first and a NAM that loses its hit going on to its next one, in whatever order
// the proposals come.  The threads take a round of NAMs (one each) at a time: hits are
// claimed with an atomic minimum of the NAM's number, and the thread that displaces a NAM
// goes on with that one.  Hits claimed in earlier rounds are gone for good: a bit each lets
// a NAM step over any number of them at once.  A hit lies where a NAM can accept it only
// near the NAM's end, as its length is known to within the query's shortest and longest
// hit.  A NAM that the query has passed (query_end < query_start) accepts nothing and stays
// where it is, so nothing is moved between lists; then a thread a hit updates the NAM that
// holds it, and unclaimed hits open NAMs in ref_start order.  (A warp resolving 32 NAMs
// after the other, testing every hit between a NAM's last hit and its end and moving every
// NAM of the list for every query, took 2.7M cycles for a read of 8550 hits, 1.5 ms of a
// batch.)
//
// kPrev: queries may share their start, and a NAM takes one hit of all of them.
constexpr uint32_t kFree = 0xFFFFFFFFu;

template <bool kBlock, bool kPrev>
__device__ __forceinline__ uint32_t merge_query(const OpenSoA& O, uint32_t lo, uint32_t n, int qs, int qe, uint32_t d,
                                                int k, uint32_t nh, uint32_t min_span, uint32_t max_span,
                                                const uint32_t* hrs, const uint32_t* hpk, uint32_t* claim,
                                                uint32_t* gone, uint32_t* cnt) {
    const uint32_t lane = lane_id(), w = kBlock ? threadIdx.x >> 5 : 0;
    const uint32_t tid = kBlock ? threadIdx.x : lane, nt = kBlock ? blockDim.x : 32u;
    const uint32_t nw = kBlock ? blockDim.x >> 5 : 1u;
    auto sync = [] {
        if (kBlock) __syncthreads();
        else __syncwarp();
    };
    int32_t *fqe = O.f(1), *fqprev = O.f(2), *fre = O.f(4), *frprev = O.f(5), *fnh = O.f(6);
    const uint32_t* fref = reinterpret_cast<const uint32_t*>(O.f(7));
    const volatile uint32_t* held = claim;
    // proposals, a round of nt NAMs at a time (the next round's fields on their way)
    auto fields = [&](uint32_t i) {   // (a NAM the query has passed, or that took one of its hits: none)
        if (i >= n || (kPrev && fqprev[i] >= qs)) return make_int4(-1, 0, 0, 0);
        return make_int4(fqe[i], fre[i], frprev[i], (int)fref[i]);
    };
    int4 nx = fields(lo + tid);
    for (uint32_t r0 = lo; r0 < n; r0 += nt) {
        const int4 f = nx;
        nx = fields(r0 + nt + tid);
        uint32_t i = r0 + tid, fresh = kFree;
        if (f.x >= qs) {
            int nqe = f.x, nre = f.y, from = f.z + 1, last = nre;
            uint32_t want = (uint32_t)f.w & 0x7FFFFFFFu;
            // a hit is accepted when both its ends lie beyond the NAM's or neither does
            if (qe > nqe) from = max(from, nre - (int)max_span + 1);
            else last = nre - (int)min_span;
            uint32_t at = 0, hi = nh;
            while (at < hi) {   // hits are sorted by ref_start
                const uint32_t mid = (at + hi) >> 1;
                if ((int)hrs[mid] < from) at = mid + 1;
                else hi = mid;
            }
            for (; at < nh; ++at) {
                // the next hit that no NAM of an earlier round took
                uint32_t free = ~gone[at >> 5] & (0xFFFFFFFFu << (at & 31));
                if (!free) {
                    at |= 31u;
                    if (at + 1 >= nh || (int)hrs[at + 1] > last) break;
                    continue;
                }
                at = (at & ~31u) + (uint32_t)__ffs(free) - 1;
                if (at >= nh) break;
                const int rs = (int)hrs[at];
                if (rs > last) break;
                const uint32_t pk = hpk[at];
                const int re = rs + (int)(pk & 0xFF) + k;
                if ((pk >> 8) != want || held[at] < i || (qe > nqe) != (re > nre)) continue;
                const uint32_t old = atomicMin(&claim[at], i);
                if (old < i) continue;
                if (old == kFree) {
                    fresh = at;
                    break;
                }
                i = old;   // displaced: on with its next hit
                nqe = fqe[i];
                nre = fre[i];
                last = qe > nqe ? nre : nre - (int)min_span;
                want = fref[i] & 0x7FFFFFFFu;
            }
        }
        if (r0 + nt >= n) break;   // the last round: its claims need no bits
        sync();
        if (fresh != kFree) atomicOr(&gone[fresh >> 5], 1u << (fresh & 31));
        sync();
    }
    sync();
    // hits to their NAMs; the others open NAMs in order
    const uint32_t per = ((nh + nw - 1) / nw + 31) & ~31u;
    const uint32_t h0 = min(w * per, nh), h1 = min(h0 + per, nh);
    uint32_t mine = 0;
    for (uint32_t b = h0; b < h1; b += 32)
        mine += __popc(__ballot_sync(0xFFFFFFFFu, b + lane < h1 && held[b + lane] == kFree));
    uint32_t to = n, opened = mine;
    if constexpr (kBlock) {
        if (lane == 0) cnt[w] = mine;
        __syncthreads();
        opened = 0;
        for (uint32_t v = 0; v < nw; ++v) {
            if (v < w) to += cnt[v];
            opened += cnt[v];
        }
    }
    for (uint32_t b = h0; b < h1; b += 32) {
        const uint32_t h = b + lane;
        const bool in = h < h1;
        const uint32_t i = in ? held[h] : 0u;
        const bool open = in && i == kFree;
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, open);
        if (in) {
            const int rs = (int)hrs[h];
            const uint32_t pk = hpk[h];
            const int re = rs + (int)(pk & 0xFF) + k;
            if (open) {
                HitRec x;
                x.ref_rc = (d << 31) | (pk >> 8);
                x.qs = qs;
                x.qe = qe;
                x.rs = rs;
                x.re = re;
                O.put(to + __popc(m & lanemask_lt()), nam_from_hit(x));
            } else {
                if (qe > fqe[i] && re > fre[i]) {
                    fqe[i] = qe;
                    fre[i] = re;
                }
                fqprev[i] = qs;
                frprev[i] = rs;
                fnh[i] += 1;
            }
        }
        to += __popc(m);
    }
    sync();
    return n + opened;
}

// Phase 2 of find_nams_rescue: walks the runs of the taken rescue hits in (orientation,
// query_start) order and merges them into O (merge_query); returns the number of NAMs.
// kBlock: by the block, else by the warp alone.
// buf: rescue_hit_words(cap) words, plan.maxrun <= cap.
template <bool kBlock>
__device__ __forceinline__ uint32_t rescue_merge(const IndexView& I, const Query* const* Qd, const uint64_t* const* Pd,
                                                 const RescuePlan& plan, const uint64_t* tkbuf, uint32_t Pq,
                                                 const OpenSoA& O, uint32_t* buf, uint32_t cap, RescueShared& S,
                                                 uint64_t& walk_cycles) {
    const uint32_t tid = kBlock ? threadIdx.x : lane_id(), nt = kBlock ? blockDim.x : 32u;
    uint32_t *hrs = buf, *hpk = buf + cap, *claim = buf + 2 * (size_t)cap, *gone = buf + 3 * (size_t)cap;
    uint32_t n = 0;
    for (int d = 0; d < 2; ++d) {
        const uint64_t* tk = tkbuf + (2 + d) * Pq;
        const uint32_t lo = n;   // the other orientation's NAMs can take no hit
        for (uint32_t j = 0; j < plan.m[d]; ++j) {
            const uint32_t qi = (uint32_t)(tk[j] >> 32) & 0xFFFF;
            const uint32_t cnt = (uint32_t)tk[j];
            const int qs = (int)Qd[d][qi].start, qe = (int)Qd[d][qi].end;
            uint32_t nh = 0, min_span = 0, max_span = 0;
            const long long tw = clock64();
            if constexpr (kBlock) nh = block_walk_run(I, qs, qe, Pd[d][qi], cnt, hrs, hpk, S, min_span, max_span);
            else nh = warp_walk_run_n(I, qs, qe, Pd[d][qi], cnt, hrs, hpk, cap, min_span, max_span);
            walk_cycles += (uint64_t)(clock64() - tw);
            for (uint32_t t = tid; t < cnt; t += nt) claim[t] = kFree;
            for (uint32_t t = tid; 32 * t < cnt; t += nt) gone[t] = 0;
            // the next query's run (its first entries), on its way while this one merges
            if (!kBlock && j + 1 < plan.m[d] && 8 * tid < (uint32_t)tk[j + 1])
                prefetch_l2(I.rs + Pd[d][(uint32_t)(tk[j + 1] >> 32) & 0xFFFF] + 8 * tid);
            if (kBlock) __syncthreads();
            else __syncwarp();
            n = merge_query<kBlock, false>(O, lo, n, qs, qe, (uint32_t)d, I.k, nh, min_span, max_span, hrs, hpk, claim,
                                           gone, S.cnt);
        }
    }
    return n;
}

// Hands a rescued read's NAMs to the block sort when they are more than kWarpSortMax and
// returns true, else false (the caller's warp sorts them).
__device__ __forceinline__ bool rescue_sort_job(const Arenas& A, Counters* ctr, ReadRec& R, NamState* closed,
                                                uint32_t n, NamKey* keys, uint32_t r, uint32_t t) {
    if (n <= kWarpSortMax) return false;
    // many NAMs: the block-per-read sort kernel orders them.  The count is known now
    // (the sort only orders them), so the NAM offsets of the batch can be computed
    // while the sorts run; the sort sets nam_off.
    if (lane_id() == 0) {
        R.n_nams = n;
        const uint32_t j = n > kSortTile ? A.jobs_cap - 1 - atomicAdd(&ctr->n_huge, 1u)
                                         : atomicAdd(&ctr->n_heavy, 1u);
        SortJob job;
        job.closed = closed;
        job.keys = keys;
        job.n = n;
        job.read = r;
        job.note = t;
        job.pad = 0;
        A.sort_jobs[j] = job;
    }
    return true;
}

// find_nams_rescue for the rescued read r (entry t of the rescue list) by the calling warp
// or, kBlock, by the block (a heavy read: the two orientations' plans on two warps, each
// query's run walked by one).
template <bool kBlock>
__device__ __forceinline__ void rescue_read(const IndexView& I, const MapConfig& C, ReadRec* __restrict__ rec,
                                            const Arenas& A, Counters* ctr, uint32_t t, uint32_t r, RescueShared& S) {
    const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
    const bool first = !kBlock || w == 0;   // the warp that takes scratch and writes the result
    const uint32_t tid = kBlock ? threadIdx.x : lane, nt = kBlock ? blockDim.x : 32u;
    const long long t0 = clock64();
    ReadRec& R = rec[r];
    uint64_t* note = A.rescue_cycles && first && lane == 0 ? A.rescue_cycles + 8ull * t : nullptr;
    // scratch for the team (nullptr, with the read marked failed, when there is none)
    auto scratch = [&](uint64_t slot_off, uint64_t bytes) {
        uint8_t* p = nullptr;
        if (first) {
            p = warp_scratch(A, ctr, slot_off, bytes);
            if (!p) warp_fail(R, ctr, kStatusScratchOverflow);
        }
        if (kBlock) {
            if (threadIdx.x == 0) S.scratch = p;
            __syncthreads();
            p = S.scratch;
            __syncthreads();
        }
        return p;
    };
    const uint32_t nqd[2] = {R.nq, R.nq2 - R.nq};
    const Query* Qd[2] = {A.q + R.q_off, A.q + R.q_off + R.nq};
    const uint64_t* Pd[2] = {A.q_pos + R.q_off, A.q_pos + R.q_off + R.nq};
    const uint32_t Pq = next_pow2(max(max(nqd[0], nqd[1]), 1u));
    const uint64_t b1 = 4ull * 8 * Pq + 64;
    uint64_t* buf = reinterpret_cast<uint64_t*>(scratch(0, b1));
    if (!buf) return;
    RescuePlan plan{};
    if (kBlock) {
        if (w < 2) {
            RescuePlan p{};
            rescue_prepare_dir(I, C, Qd, Pd, nqd, Pq, buf, (int)w, p);
            if (lane == 0) S.plan[w] = p;
        }
        __syncthreads();
        plan.m[0] = S.plan[0].m[0];
        plan.m[1] = S.plan[1].m[1];
        plan.bound = S.plan[0].bound + S.plan[1].bound;
        plan.maxrun = max(S.plan[0].maxrun, S.plan[1].maxrun);
    } else {
        rescue_prepare_dir(I, C, Qd, Pd, nqd, Pq, buf, 0, plan);
        rescue_prepare_dir(I, C, Qd, Pd, nqd, Pq, buf, 1, plan);
    }
    if (note) {
        note[0] = note[1] = (uint64_t)(clock64() - t0);
        note[4] = plan.bound;
        note[7] = plan.maxrun;
    }
    if (plan.bound == 0) {
        if (first && lane == 0) R.n_nams = 0;
        if (kBlock) __syncthreads();
        return;
    }
    // the NAMs (as many as hits), sort keys only for more than the cluster sort's tiles
    // hold, and a long run's hits
    const uint32_t H = (uint32_t)plan.bound;
    const uint32_t smem_hits = kBlock ? kWarpsPerBlock * kRescueSmemHits : kRescueSmemHits;
    const bool big_run = plan.maxrun > smem_hits;
    const uint64_t key_bytes = H > kClusterCtas * kSortTile ? 32ull * next_pow2(H) : 0;
    const uint64_t off2 = (b1 + 255) & ~255ull;
    const uint64_t b2 = 32ull * H + key_bytes + (big_run ? 4ull * rescue_hit_words(plan.maxrun) : 0) + 64;
    uint8_t* sc2 = scratch(off2, b2);
    if (!sc2) return;
    NamKey* keys = reinterpret_cast<NamKey*>(sc2);
    const OpenSoA O{reinterpret_cast<int32_t*>(sc2 + key_bytes), H};
    uint32_t* hits = big_run ? reinterpret_cast<uint32_t*>(sc2 + key_bytes + 32ull * H)
                             : (kBlock ? &S.buf[0][0] : S.buf[w]);
    const long long t_merge = clock64();
    uint64_t walk_cycles = 0;
    const uint32_t n = rescue_merge<kBlock>(I, Qd, Pd, plan, buf, Pq, O, hits, big_run ? plan.maxrun : smem_hits, S,
                                            walk_cycles);
    if (note) {
        note[2] = (uint64_t)(clock64() - t_merge);
        note[5] = n;
        note[6] = walk_cycles;
    }
    // the NAMs as records; those of a sort job outlive this read, so not in the warp's slot
    NamState* closed = reinterpret_cast<NamState*>(
        scratch(n > kWarpSortMax ? A.slot_bytes : off2 + ((b2 + 255) & ~255ull), 32ull * n + 32));
    if (!closed) return;
    for (uint32_t i = tid; i < n; i += nt) closed[i] = O.get(i);
    if (kBlock) __syncthreads();
    else __syncwarp();
    if (first && !rescue_sort_job(A, ctr, R, closed, n, key_bytes ? keys : nullptr, r, t)) {
        const long long t_fin = clock64();
        warp_finish_nams(C, closed, n, S.buf[w], R, A, ctr);
        if (note) note[3] = (uint64_t)(clock64() - t_fin);
    }
    if (note) note[0] = (uint64_t)(clock64() - t0);
    if (kBlock) __syncthreads();
    else __syncwarp();
}

// find_nams_rescue for the reads on the rescue list, heavy ones (at the list's heavy end)
// first, a warp a read; with C.rescue_block_hits set, and few heavy reads for the grid or
// few rescued reads for its warps, the heavy ones a block each, which ends a read in a third
// of a warp's time but takes eight warps for it: 22900 rescued reads of 2M, 1742 of them
// heavy, took 1.95 ms with blocks and 1.05 with warps (1.54 before this merge); the 10 of
// 1000 reads 0.09 ms with blocks (0.23 before).
__global__ void __launch_bounds__(32 * kWarpsPerBlock, 3)
    k_rescue(IndexView I, MapConfig C, ReadRec* __restrict__ rec, Arenas A, Counters* ctr) {
    extern __shared__ __align__(16) uint8_t s_dyn[];
    RescueShared& S = *reinterpret_cast<RescueShared*>(s_dyn);
    static_assert(sizeof(S.buf[0]) >= 7168 && kWarpSortMax <= 256, "the sort entries fit a warp's buffer");
    const uint32_t n_heavy = *(volatile unsigned int*)&ctr->n_rescue_heavy;
    const uint32_t n_rescue = n_heavy + *(volatile unsigned int*)&ctr->n_rescue;
    uint32_t first = 0;
    if (C.rescue_block_hits && (n_rescue <= warp_count() || n_heavy <= 3 * gridDim.x)) {
        for (;;) {
            if (threadIdx.x == 0) S.item = atomicAdd(&ctr->rescue_block_next, 1u);
            __syncthreads();
            const uint32_t t = S.item;
            __syncthreads();
            if (t >= n_heavy) break;
            rescue_read<true>(I, C, rec, A, ctr, t, A.rescue_list[A.rescue_cap - 1 - t], S);
        }
        first = n_heavy;
    }
    // resident warps take reads in list order, heavy ones first
    for (;;) {
        const uint32_t t = warp_next(&ctr->rescue_next) + first;
        if (t >= n_rescue) break;
        rescue_read<false>(I, C, rec, A, ctr, t,
                           t < n_heavy ? A.rescue_list[A.rescue_cap - 1 - t] : A.rescue_list[t - n_heavy], S);
    }
}

// ---- sort of rescued reads with packed keys --------------------------------------------
//
// In the score order (score descending, orientation, reference id, query start, query end,
// reference start, ...) the NAMs of one read need few bits a field, and they are created in
// (orientation, query start, reference start) order, so their number stands for what comes
// after the query end: score | orientation | reference | query start | query end | number
// makes one 64-bit word without ties: no two NAMs agree in orientation, reference, query
// start and reference start (queries with the same start and hash can open such NAMs, and
// these go to the sorts below).  Up to 8192 such words sort in a block's registers
// (bitonic; partners in other lanes by shuffles, in other warps through shared memory),
// with nothing but the word to move; a read whose fields do not fit, or whose NAMs are not
// in that order, goes to the sorts below.  Those move a key word and an index through
// shared memory at every stage and read two more words on ties: 0.96 + 1.29 ms for the
// 5629 reads of a batch of 2M, against 0.47.
constexpr int kPackThreads = 512;
constexpr uint32_t kPackMax = 16 * kPackThreads;   // NAMs

// Bitonic stages (k, j), j = j0, j0 / 2, .., 1, of the words x of a block, word
// t * kKeys + r at x[r] of thread t.
template <int kKeys>
__device__ __forceinline__ void pack_merge(uint64_t (&x)[kKeys], uint32_t k, uint32_t j0, uint64_t* sm) {
    const uint32_t t = threadIdx.x;
    const bool asc = ((t * kKeys) & k) == 0;   // (k >= kKeys: alike for the thread's words)
    for (uint32_t j = j0; j >= kKeys; j >>= 1) {
        const uint32_t m = j / kKeys;   // partner thread t ^ m
        const bool keep_min = ((t & m) == 0) == asc;
        if (m < 32) {
#pragma unroll
            for (int r = 0; r < kKeys; ++r) {
                const uint64_t y = __shfl_xor_sync(0xFFFFFFFFu, x[r], m);
                if ((x[r] > y) == keep_min) x[r] = y;
            }
        } else {
            __syncthreads();
#pragma unroll
            for (int r = 0; r < kKeys; ++r) sm[r * kPackThreads + t] = x[r];
            __syncthreads();
#pragma unroll
            for (int r = 0; r < kKeys; ++r) {
                const uint64_t y = sm[r * kPackThreads + (t ^ m)];
                if ((x[r] > y) == keep_min) x[r] = y;
            }
        }
    }
    if (j0 >= kKeys) j0 = kKeys / 2;
#pragma unroll
    for (int j = kKeys / 2; j > 0; j >>= 1) {
        if ((uint32_t)j > j0) continue;
#pragma unroll
        for (int r = 0; r < kKeys; ++r) {
            if (r & j) continue;
            const bool up = ((t * kKeys + r) & k) == 0;
            const uint64_t u = x[r], v = x[r | j];
            if ((u > v) == up) {
                x[r] = v;
                x[r | j] = u;
            }
        }
    }
}

// Sorts one job of at most kKeys * kPackThreads NAMs; false when its keys cannot be packed.
template <int kKeys>
__device__ __noinline__ bool pack_sort(const SortJob& job, ReadRec& R, const Arenas& A, Counters* ctr, uint64_t* sm) {
    __shared__ uint32_t s_max[3];   // score, reference id, query end
    __shared__ uint64_t s_noff;
    const uint32_t t = threadIdx.x, n = job.n;
    const NamState* closed = job.closed;
    if (t < 3) s_max[t] = 0;
    __syncthreads();
    uint32_t ms = 0, mr = 0, mq = 0;
    bool ok = true;
    for (uint32_t i = t; i < n; i += kPackThreads) {
        const NamState a = closed[i];
        ms = max(ms, (uint32_t)nam_score_int(a));
        mr = max(mr, a.ref_rc & 0x7FFFFFFFu);
        mq = max(mq, (uint32_t)a.qe);
        if (i + 1 < n) {   // created in (orientation, query start, reference start, reference) order
            const NamState b = closed[i + 1];
            const uint32_t oa = a.ref_rc >> 31, ob = b.ref_rc >> 31;
            ok &= oa != ob ? oa < ob
                           : (a.qs != b.qs ? a.qs < b.qs : (a.rs != b.rs ? a.rs < b.rs : a.ref_rc < b.ref_rc));
        }
    }
    ms = __reduce_max_sync(0xFFFFFFFFu, ms);
    mr = __reduce_max_sync(0xFFFFFFFFu, mr);
    mq = __reduce_max_sync(0xFFFFFFFFu, mq);
    if (lane_id() == 0) {
        atomicMax(&s_max[0], ms);
        atomicMax(&s_max[1], mr);
        atomicMax(&s_max[2], mq);
    }
    if (!__syncthreads_and(ok)) return false;
    ms = s_max[0];
    mr = s_max[1];
    mq = s_max[2];
    const uint32_t br = 32 - __clz(mr), bq = 32 - __clz(mq), bn = 32 - __clz(n - 1);
    if (32 - __clz(ms) + 1 + br + 2 * bq + bn > 63) return false;   // (padding is all ones)
    uint64_t x[kKeys];
#pragma unroll
    for (int r = 0; r < kKeys; ++r) {
        const uint32_t i = r * kPackThreads + t;
        x[r] = ~0ULL;
        if (i < n) {
            const NamState a = closed[i];
            uint64_t v = ((uint64_t)(ms - (uint32_t)nam_score_int(a)) << 1) | (a.ref_rc >> 31);
            v = (v << br) | (a.ref_rc & 0x7FFFFFFFu);
            v = (v << bq) | (uint32_t)a.qs;
            v = (v << bq) | (uint32_t)a.qe;
            x[r] = (v << bn) | i;
        }
    }
    for (uint32_t k = 2; k <= kKeys * kPackThreads; k <<= 1) pack_merge<kKeys>(x, k, k >> 1, sm);
    if (t == 0) {
        const uint64_t noff = atomicAdd(&ctr->nam_used, (unsigned long long)n);
        if (noff + n > A.nam_cap) {
            R.flags |= kReadFailed;
            R.n_nams = 0;   // the rescue kernel set the count ahead of the sort
            atomicOr(&ctr->status, kStatusNamOverflow);
            s_noff = ~0ULL;
        } else {
            R.nam_off = noff;
            s_noff = noff;
        }
    }
    // the order to shared memory, so that consecutive threads write consecutive NAMs
    __syncthreads();
    uint32_t* order = reinterpret_cast<uint32_t*>(sm);
#pragma unroll
    for (int r = 0; r < kKeys; ++r) order[t * kKeys + r] = (uint32_t)x[r] & ((1u << bn) - 1);
    __syncthreads();
    const uint64_t noff = s_noff;
    if (noff != ~0ULL)
        for (uint32_t i = t; i < n; i += kPackThreads) A.nams[noff + i] = closed[order[i]];
    return true;
}

// The packed sort of the rescued reads with more than kWarpSortMax NAMs, the ones with more
// than kSortTile first; jobs that it passes on go to the slow list (those above kSortTile
// from its back).
__global__ void __launch_bounds__(kPackThreads, 2)
    k_sort_packed(MapConfig C, ReadRec* __restrict__ rec, Arenas A, Counters* ctr) {
    extern __shared__ __align__(16) uint8_t s_dyn[];   // kPackMax words
    uint64_t* sm = reinterpret_cast<uint64_t*>(s_dyn);
    __shared__ uint32_t s_next;
    const uint32_t n_huge = *(volatile unsigned int*)&ctr->n_huge;
    const uint32_t n_jobs = n_huge + *(volatile unsigned int*)&ctr->n_heavy;
    for (;;) {
        if (threadIdx.x == 0) s_next = atomicAdd(&ctr->sort_next, 1u);
        __syncthreads();
        const uint32_t h = s_next;
        if (h >= n_jobs) break;
        const long long t0 = clock64();
        const uint32_t at = h < n_huge ? A.jobs_cap - 1 - h : h - n_huge;
        const SortJob job = A.sort_jobs[at];
        ReadRec& R = rec[job.read];
        bool done = false;
        if (C.sort_mode == GBSA_SORT_SCORE && job.n <= kPackMax) {
            if (job.n <= kPackThreads) done = pack_sort<1>(job, R, A, ctr, sm);
            else if (job.n <= 2 * kPackThreads) done = pack_sort<2>(job, R, A, ctr, sm);
            else if (job.n <= 4 * kPackThreads) done = pack_sort<4>(job, R, A, ctr, sm);
            else if (job.n <= 8 * kPackThreads) done = pack_sort<8>(job, R, A, ctr, sm);
            else done = pack_sort<16>(job, R, A, ctr, sm);
        }
        if (threadIdx.x == 0) {
            if (!done) {
                if (h < n_huge) A.slow_list[A.rescue_cap - 1 - atomicAdd(&ctr->n_slow_huge, 1u)] = at;
                else A.slow_list[atomicAdd(&ctr->n_slow, 1u)] = at;
            } else if (A.rescue_cycles) {
                A.rescue_cycles[8ull * job.note + 3] = (uint64_t)(clock64() - t0);
            }
        }
        __syncthreads();
    }
}

// A read with more than 128 NAMs of which few are open at a time (one of a thousand bases and
// more, whose queries have a hit or two each), by the warp: the slots are given back as the
// queries pass their NAMs, and the NAMs are sorted through scratch.  False: too many are open.
// 10,000 reads of 4,000 bp, two thirds of them such: this stage 22.7 ms with a block a read, 2.6
// so (3.9 with a warp and the open NAMs in memory), the call 28.4 -> 8.1 ms (10.3).
__device__ __noinline__ bool long_merge(const MapConfig& C, ReadRec* __restrict__ rec, const Arenas& A, Counters* ctr,
                                        uint32_t rd, GroupShared<4>& S) {
    const uint32_t lane = lane_id();
    ReadRec& R = rec[rd];
    const uint32_t H = R.n_hits;
    const uint64_t b_list = (32ull * H + 255) & ~255ull;
    NamState* list = reinterpret_cast<NamState*>(warp_scratch(A, ctr, 0, b_list));
    if (!list) {
        warp_fail(R, ctr, kStatusScratchOverflow);
        return true;
    }
    WarpRoom room;
    uint32_t n = 0;
    if (group_merge<32, 4, true>(C, rec, A, ctr, &rd, 0, 1, S, room, list, &n) != kNoRead) return false;
    const uint32_t P = next_pow2(n);
    uint8_t* sc = warp_scratch(A, ctr, b_list <= A.slot_bytes ? b_list : 0, 28ull * P);
    if (!sc) {
        warp_fail(R, ctr, kStatusScratchOverflow);
        return true;
    }
    uint64_t* k2 = reinterpret_cast<uint64_t*>(sc);
    uint64_t* k3 = k2 + P;
    // what moves lies in shared memory where it fits
    static_assert(sizeof(S.k1) + sizeof(S.k2) + sizeof(S.k3) >= 256 * 12, "256 keys with their numbers");
    uint64_t* k1 = P <= 256 ? S.k1 : k3 + P;
    uint32_t* ix = reinterpret_cast<uint32_t*>(k1 + P);
    for (uint32_t t = lane; t < P; t += 32) {
        NamKey k;
        k.k1 = k.k2 = k.k3 = ~0ULL;   // padding sorts last (a NAM's first key word is never all ones)
        if (t < n) k = nam_key(list[t], t, C.sort_mode);
        k1[t] = k.k1;
        ix[t] = t;
        k2[t] = k.k2;
        k3[t] = k.k3;
    }
    __syncwarp();
    warp_sort_idx(k1, ix, k2, k3, P);
    const uint64_t noff = warp_bump(&ctr->nam_used, n);
    if (noff + n > A.nam_cap) {
        warp_fail(R, ctr, kStatusNamOverflow);
        return true;
    }
    for (uint32_t t = lane; t < n; t += 32) A.nams[noff + t] = list[ix[t]];
    if (lane == 0) {
        R.nam_off = noff;
        R.n_nams = n;
    }
    __syncwarp();
    return true;
}

// find_nams for the reads with more NAMs than k_nams_group's slots (reads in repeats, with
// queries of dozens of hits): a block a read, a query's hits merged at once (merge_query).
// A warp a read, hit by hit with 8 slots a lane, took 0.36 ms for the longest of 81 such
// reads of 100k, 0.95 ms where some of 250 bp had more than 256 NAMs; here 0.12 and 0.17.
// Before them the reads with few hits a query, a warp each (long_merge).
constexpr int kBigThreads = kPackThreads;
constexpr int kBigWarps = kBigThreads / 32;
constexpr uint32_t kBigHits = 512;   // hits of one query in shared memory
union BigShared {
    uint32_t hits[rescue_hit_words(kBigHits)];
    uint64_t sort[4 * kPackThreads];   // also the warp sort's buffer
    GroupShared<4> merge[kBigWarps];
};

__global__ void __launch_bounds__(kBigThreads, 2)
    k_nams(const __grid_constant__ MapConfig C, int k, ReadRec* __restrict__ rec, const __grid_constant__ Arenas A,
           Counters* ctr) {
    extern __shared__ __align__(16) uint8_t s_dyn[];
    BigShared& s = *reinterpret_cast<BigShared*>(s_dyn);
    __shared__ uint32_t s_left[2 * kBigWarps], s_n_left;   // reads that long_merge left
    __shared__ uint32_t s_cnt[kBigThreads / 32];
    __shared__ uint32_t s_item, s_run, s_min, s_max;
    __shared__ uint8_t* s_scratch;
    static_assert(sizeof(s) >= 7168 && kWarpSortMax <= 256, "a warp's sort entries fit");
    const uint32_t tid = threadIdx.x, lane = lane_id(), w = tid >> 5;
    const uint32_t n_big = *(volatile unsigned int*)&ctr->n_big, n_few = *(volatile unsigned int*)&ctr->n_few;
    uint32_t left = 0, left_at = 0;
    for (bool few = n_few != 0;;) {
        if (few && left_at == left) {   // until the list ends, or there are reads for the block
            if (tid == 0) s_n_left = 0;
            __syncthreads();
            while (__shfl_sync(0xFFFFFFFFu, *(volatile uint32_t*)&s_n_left, 0) < kBigWarps) {
                const uint32_t t = warp_next(&ctr->few_next);
                if (t >= n_few) break;
                const uint32_t r = A.big_list[A.rescue_cap - 1 - t];
                if (!long_merge(C, rec, A, ctr, r, s.merge[w]) && lane == 0) s_left[atomicAdd(&s_n_left, 1u)] = r;
                __syncwarp();
            }
            __syncthreads();
            left = s_n_left;
            left_at = 0;
            few = left >= kBigWarps;
        }
        uint32_t r, b = 0xFFFFFFFFu;
        if (left_at < left) {
            r = s_left[left_at++];
        } else {
            if (tid == 0) s_item = atomicAdd(&ctr->big_next, 1u);
            __syncthreads();
            b = s_item;
            if (b >= n_big) break;
            r = A.big_list[b];
        }
        const long long t0 = clock64();
        ReadRec& R = rec[r];
        const uint32_t H = R.n_hits;
        const HitPacked* hits = A.hits + R.hit_off;
        // the NAMs (at most H), their records, sort keys, and the hits of a query with more
        // than kBigHits
        const uint32_t P2 = next_pow2(H);
        const uint64_t b_soa = 32ull * H, b_keys = 32ull * P2;
        if (w == 0) {
            uint8_t* p = warp_scratch(A, ctr, 0, b_soa + 32ull * H + b_keys + 4ull * rescue_hit_words(H) + 64);
            if (!p) warp_fail(R, ctr, kStatusScratchOverflow);
            if (lane == 0) s_scratch = p;
        }
        __syncthreads();
        uint8_t* sc = s_scratch;
        if (!sc) continue;
        const OpenSoA O{reinterpret_cast<int32_t*>(sc), H};
        NamState* closed = reinterpret_cast<NamState*>(sc + b_soa);
        NamKey* keys = reinterpret_cast<NamKey*>(closed + H);
        uint32_t* big_buf = reinterpret_cast<uint32_t*>(sc + b_soa + 32ull * H + b_keys);
        uint32_t n = 0, lo = 0, cur_dir = 0;
        for (uint32_t i = 0; i < H;) {
            // hits [i, i + nh) of one query
            const HitRec x = load_hit(hits, i, H);
            const uint32_t dir = x.ref_rc >> 31;
            if (tid == 0) {
                s_run = 0xFFFFFFFFu;
                s_min = 0xFFFFFFFFu;
                s_max = 0;
            }
            if (dir != cur_dir) {   // the other orientation's NAMs can take no more hits
                lo = n;
                cur_dir = dir;
            }
            __syncthreads();
            uint32_t nh = 0;
            for (uint32_t c = 0;; c += kBigThreads) {
                const HitRec y = load_hit(hits, i + c + tid, H);
                const bool same = i + c + tid < H && (y.ref_rc >> 31) == dir && y.qs == x.qs && y.qe == x.qe;
                if (!same) atomicMin(&s_run, c + tid);
                if (__syncthreads_and(same)) continue;
                nh = s_run;
                break;
            }
            const uint32_t cap = nh <= kBigHits ? kBigHits : H;
            uint32_t* buf = nh <= kBigHits ? s.hits : big_buf;
            uint32_t *hrs = buf, *hpk = buf + cap, *claim = buf + 2 * (size_t)cap, *gone = buf + 3 * (size_t)cap;
            bool bad = false;
            for (uint32_t t = tid; t < nh; t += kBigThreads) {
                const HitRec y = load_hit(hits, i + t, H);
                const uint32_t span = (uint32_t)(y.re - y.rs);
                bad |= t > 0 && load_hit(hits, i + t - 1, H).rs > y.rs;
                hrs[t] = (uint32_t)y.rs;
                hpk[t] = (y.ref_rc << 8) | (span - (uint32_t)k);   // as in the index
                claim[t] = kFree;
                atomicMin(&s_min, span);
                atomicMax(&s_max, span);
            }
            for (uint32_t t = tid; 32 * t < nh; t += kBigThreads) gone[t] = 0;
            // (an index whose runs are not in position order: hit by hit)
            if (__syncthreads_or(bad)) nh = 1;
            n = merge_query<true, true>(O, lo, n, x.qs, x.qe, dir, k, nh, s_min, s_max, hrs, hpk, claim, gone, s_cnt);
            i += nh;
        }
        for (uint32_t i = tid; i < n; i += kBigThreads) closed[i] = O.get(i);
        if (tid == 0) R.n_nams = n;
        __syncthreads();
        const long long t_merge = clock64();
        SortJob job;
        job.closed = closed;
        job.n = n;
        bool done = false;
        if (C.sort_mode == GBSA_SORT_SCORE && n <= 4 * kPackThreads) {
            if (n <= kPackThreads) done = pack_sort<1>(job, R, A, ctr, s.sort);
            else if (n <= 2 * kPackThreads) done = pack_sort<2>(job, R, A, ctr, s.sort);
            else done = pack_sort<4>(job, R, A, ctr, s.sort);
        }
        __syncthreads();
        if (!done && w == 0) {
            if (n <= kWarpSortMax) {
                warp_finish_nams(C, closed, n, reinterpret_cast<uint32_t*>(s_dyn), R, A, ctr);
            } else {
                for (uint32_t t = lane; t < n; t += 32) keys[t] = nam_key(closed[t], t, C.sort_mode);
                __syncwarp();
                warp_sort_keys(keys, n);
                const uint64_t noff = warp_bump(&ctr->nam_used, n);
                if (noff + n > A.nam_cap) {
                    warp_fail(R, ctr, kStatusNamOverflow);
                    if (lane == 0) R.n_nams = 0;
                } else {
                    for (uint32_t t = lane; t < n; t += 32) A.nams[noff + t] = closed[keys[t].idx];
                    if (lane == 0) R.nam_off = noff;
                }
            }
        }
        if (A.nam_cycles && tid == 0 && b < n_big) {
            uint64_t* note = A.nam_cycles + 4ull * b;   // cycles, hits, NAMs, merge cycles
            note[0] = (uint64_t)(clock64() - t0);
            note[1] = H;
            note[2] = n;
            note[3] = (uint64_t)(t_merge - t0);
        }
        __syncthreads();
    }
}

// Shared-memory tile of the block sort, one array per key field so that a warp's
// accesses are conflict-free and a compare usually reads only k1.
struct SortTile {
    uint64_t* k1;
    uint64_t* k2;
    uint64_t* k3;
    uint32_t* idx;
    __device__ NamKey get(uint32_t i) const {
        NamKey k;
        k.k1 = k1[i];
        k.k2 = k2[i];
        k.k3 = k3[i];
        k.idx = idx[i];
        k.pad = 0;
        return k;
    }
    __device__ void put(uint32_t i, const NamKey& k) {
        k1[i] = k.k1;
        k2[i] = k.k2;
        k3[i] = k.k3;
        idx[i] = k.idx;
    }
    // b < a, reading the secondary fields only when the first ones tie
    __device__ bool less_at(uint32_t b, uint32_t a) const {
        const uint64_t x = k1[b], y = k1[a];
        if (x != y) return x < y;
        const uint64_t x2 = k2[b], y2 = k2[a];
        if (x2 != y2) return x2 < y2;
        const uint64_t x3 = k3[b], y3 = k3[a];
        if (x3 != y3) return x3 < y3;
        return idx[b] < idx[a];
    }
    __device__ void swap(uint32_t i, uint32_t j) {
        const NamKey a = get(i), b = get(j);
        put(i, b);
        put(j, a);
    }
};


__device__ __forceinline__ void cmp_swap(NamKey* keys, uint32_t i, uint32_t j, uint32_t k) {
    const uint32_t ixj = i ^ j;
    if (ixj > i) {
        const NamKey a = keys[i], b = keys[ixj];
        const bool up = (i & k) == 0;
        if (key_less(b, a) == up) {
            keys[i] = b;
            keys[ixj] = a;
        }
    }
}

// Block bitonic sort of n keys (room for next_pow2(n) in global memory) by all
// threads of the block.  Every stage whose partner distance is below tcap runs on a
// shared-memory tile of tcap keys; only the stages with larger distances touch
// global memory.
__device__ void block_sort_keys(NamKey* keys, uint32_t n, SortTile tile, uint32_t tcap) {
    const uint32_t P = next_pow2(n);
    for (uint32_t i = n + threadIdx.x; i < P; i += blockDim.x) {
        NamKey k;
        k.k1 = k.k2 = k.k3 = ~0ULL;
        k.idx = 0xFFFFFFFFu;
        k.pad = 0;
        keys[i] = k;
    }
    __syncthreads();
    const uint32_t T = P < tcap ? P : tcap;
    // Runs all stages (k, j) with j < T inside each tile; k is the current merge size
    // (k <= T: the tile-local sort from scratch; k > T: finish merge level k).
    auto tile_pass = [&](uint32_t k_from, uint32_t k_to, uint32_t j_from) {
        for (uint32_t t0 = 0; t0 < P; t0 += T) {
            for (uint32_t i = threadIdx.x; i < T; i += blockDim.x) tile.put(i, keys[t0 + i]);
            __syncthreads();
            for (uint32_t k = k_from; k <= k_to; k <<= 1) {
                for (uint32_t j = (k == k_from ? j_from : k >> 1); j > 0; j >>= 1) {
                    // one compare per thread and pair: i is the lower index of the pair
                    for (uint32_t q = threadIdx.x; q < T / 2; q += blockDim.x) {
                        const uint32_t i = ((q & ~(j - 1)) << 1) | (q & (j - 1));
                        const uint32_t ixj = i | j;
                        const bool up = ((t0 + i) & k) == 0;   // direction uses the global index
                        if (tile.less_at(ixj, i) == up) tile.swap(i, ixj);
                    }
                    __syncthreads();
                }
            }
            for (uint32_t i = threadIdx.x; i < T; i += blockDim.x) keys[t0 + i] = tile.get(i);
            __syncthreads();
        }
    };
    tile_pass(2, T, 1);
    for (uint32_t k = 2 * T; k <= P; k <<= 1) {
        for (uint32_t j = k >> 1; j >= T; j >>= 1) {
            for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) cmp_swap(keys, i, j, k);
            __syncthreads();
        }
        tile_pass(k, k, T >> 1);
    }
}

// Shared-memory tile of the block sort that moves only the first key word and the
// NAM index: the other key words stay where they were loaded (indexed by NAM) and
// are read only when the first words tie.  A compare-exchange then moves 12 bytes
// instead of 28.
struct IdxSortTile {
    uint64_t* k1;    // first key word, moves with ix
    uint32_t* ix;    // NAM index, moves
    uint64_t* k2;    // second and third key words by NAM index (fixed)
    uint64_t* k3;
    __device__ bool less_at(uint32_t b, uint32_t a) const {
        const uint64_t x = k1[b], y = k1[a];
        if (x != y) return x < y;
        const uint32_t ib = ix[b], ia = ix[a];
        const uint64_t x2 = k2[ib], y2 = k2[ia];
        if (x2 != y2) return x2 < y2;
        const uint64_t x3 = k3[ib], y3 = k3[ia];
        if (x3 != y3) return x3 < y3;
        return ib < ia;
    }
    __device__ void swap(uint32_t i, uint32_t j) {
        const uint64_t a = k1[i];
        k1[i] = k1[j];
        k1[j] = a;
        const uint32_t b = ix[i];
        ix[i] = ix[j];
        ix[j] = b;
    }
};

// Bitonic sort of the P (a power of two) keys held in the tile.
__device__ void idx_tile_sort(IdxSortTile tile, uint32_t P) {
    for (uint32_t k = 2; k <= P; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t q = threadIdx.x; q < P / 2; q += blockDim.x) {
                const uint32_t i = ((q & ~(j - 1)) << 1) | (q & (j - 1));
                const uint32_t ixj = i | j;
                if (tile.less_at(ixj, i) == ((i & k) == 0)) tile.swap(i, ixj);
            }
            __syncthreads();
        }
    }
}

// Sorts the NAMs of the rescued reads with kWarpSortMax < NAMs <= kSortTile that the packed
// sort passed on: one block per read, bitonic sort in a shared-memory tile, then the
// read's NAMs are written to the NAM arena in order.
template <int kThreads, uint32_t kTile>
__global__ void __launch_bounds__(kThreads) k_sort_jobs(MapConfig C, ReadRec* __restrict__ rec, Arenas A,
                                                         Counters* ctr) {
    extern __shared__ __align__(16) uint8_t s_dyn[];   // kTile sort keys, one array per field
    __shared__ uint64_t s_noff;
    SortTile tile;
    tile.k1 = reinterpret_cast<uint64_t*>(s_dyn);
    tile.k2 = tile.k1 + kTile;
    tile.k3 = tile.k2 + kTile;
    tile.idx = reinterpret_cast<uint32_t*>(tile.k3 + kTile);
    IdxSortTile itile;   // the same shared memory, for jobs that fit it
    itile.k1 = tile.k1;
    itile.k2 = tile.k2;
    itile.k3 = tile.k3;
    itile.ix = tile.idx;
    const uint32_t n_jobs = *(volatile unsigned int*)&ctr->n_slow;
    for (uint32_t h = blockIdx.x; h < n_jobs; h += gridDim.x) {
        const long long t0 = clock64();
        const SortJob job = A.sort_jobs[A.slow_list[h]];
        ReadRec& R = rec[job.read];
        const NamState* closed = job.closed;
        const uint32_t NN = job.n;
        const uint32_t P = next_pow2(NN);
        const bool in_tile = P <= kTile;
        if (in_tile) {
            for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
                NamKey k;
                if (i < NN) {
                    k = nam_key(closed[i], i, C.sort_mode);
                } else {   // padding sorts last (a NAM's first key word is never all ones)
                    k.k1 = k.k2 = k.k3 = ~0ULL;
                }
                itile.k1[i] = k.k1;
                itile.ix[i] = i;
                itile.k2[i] = k.k2;
                itile.k3[i] = k.k3;
            }
            __syncthreads();
            idx_tile_sort(itile, P);
        } else {
            for (uint32_t i = threadIdx.x; i < NN; i += blockDim.x) job.keys[i] = nam_key(closed[i], i, C.sort_mode);
            __syncthreads();
            block_sort_keys(job.keys, NN, tile, kTile);
        }
        if (threadIdx.x == 0) {
            const uint64_t noff = atomicAdd(&ctr->nam_used, (unsigned long long)NN);
            if (noff + NN > A.nam_cap) {
                R.flags |= kReadFailed;
                R.n_nams = 0;   // the rescue kernel set the count ahead of the sort
                atomicOr(&ctr->status, kStatusNamOverflow);
                s_noff = ~0ULL;
            } else {
                R.nam_off = noff;
                R.n_nams = NN;
                s_noff = noff;
            }
        }
        __syncthreads();
        const uint64_t noff = s_noff;
        if (noff != ~0ULL)
            for (uint32_t i = threadIdx.x; i < NN; i += blockDim.x)
                A.nams[noff + i] = closed[in_tile ? tile.idx[i] : job.keys[i].idx];
        __syncthreads();
        if (A.rescue_cycles && threadIdx.x == 0) A.rescue_cycles[8ull * job.note + 3] = (uint64_t)(clock64() - t0);
    }
}

// ---- cluster sort of the other rescued reads with more than kSortTile NAMs -------------
//
// A cluster of kClusterCtas CTAs sorts one read's keys: each CTA holds T = P /
// kClusterCtas of the P (next power of two) keys in its shared-memory tile, so up to
// kClusterCtas * kSortTile keys are sorted without touching global memory.  Bitonic
// stages whose partner distance is below T stay within a CTA (block barrier); the
// few with larger distances compare and swap across the CTAs' tiles through
// distributed shared memory (cluster barrier).  Each CTA needs only kSortTile keys of
// shared memory, so the clusters run beside the NAM kernels of the other stream.
// Tie break of the index-moving cluster sort: NAM indices ib and ia whose first key
// words are equal, by their second and third words (fixed, NAM e in CTA e / T at e % T)
// and then the index.
__device__ __forceinline__ bool cluster_tie_less(uint32_t ib, uint32_t ia, uint64_t* k2, uint64_t* k3, uint32_t T) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const uint64_t b2 = *cl.map_shared_rank(k2 + ib % T, ib / T), a2 = *cl.map_shared_rank(k2 + ia % T, ia / T);
    if (b2 != a2) return b2 < a2;
    const uint64_t b3 = *cl.map_shared_rank(k3 + ib % T, ib / T), a3 = *cl.map_shared_rank(k3 + ia % T, ia / T);
    if (b3 != a3) return b3 < a3;
    return ib < ia;
}

__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(256)
    k_sort_jobs_cluster(MapConfig C, ReadRec* __restrict__ rec, Arenas A, Counters* ctr) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) uint8_t s_dyn[];   // kSortTile keys, one array per field
    __shared__ uint64_t s_noff;
    cg::cluster_group cl = cg::this_cluster();
    const uint32_t rank = cl.block_rank();
    SortTile tile;
    tile.k1 = reinterpret_cast<uint64_t*>(s_dyn);
    tile.k2 = tile.k1 + kSortTile;
    tile.k3 = tile.k2 + kSortTile;
    tile.idx = reinterpret_cast<uint32_t*>(tile.k3 + kSortTile);
    const uint32_t n_jobs = *(volatile unsigned int*)&ctr->n_slow_huge;
    const uint32_t n_clusters = gridDim.x / kClusterCtas;
    for (uint32_t h = blockIdx.x / kClusterCtas; h < n_jobs; h += n_clusters) {
        const long long t0 = clock64();
        const SortJob job = A.sort_jobs[A.slow_list[A.rescue_cap - 1 - h]];
        const NamState* closed = job.closed;
        const uint32_t NN = job.n;
        const uint32_t P = next_pow2(NN);
        const bool in_tiles = P <= kClusterCtas * kSortTile;
        if (in_tiles) {
            // Each CTA's tile moves only the first key word (k1) and the NAM index (idx) of
            // its T positions; the second and third words stay where they were loaded,
            // by NAM index, and are read (possibly from another CTA) only on ties.
            const uint32_t T = P / kClusterCtas;   // NN > kSortTile: T >= kSortTile / 4
            const uint32_t e0 = rank * T;
            for (uint32_t i = threadIdx.x; i < T; i += blockDim.x) {
                const uint32_t e = e0 + i;
                NamKey k;
                if (e < NN) {
                    k = nam_key(closed[e], e, C.sort_mode);
                } else {   // padding sorts last (a NAM's first key word is never all ones)
                    k.k1 = k.k2 = k.k3 = ~0ULL;
                }
                tile.k1[i] = k.k1;
                tile.idx[i] = e;
                tile.k2[i] = k.k2;
                tile.k3[i] = k.k3;
            }
            cl.sync();
            for (uint32_t k = 2; k <= P; k <<= 1) {
                for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                    if (j < T) {
                        for (uint32_t q = threadIdx.x; q < T / 2; q += blockDim.x) {
                            const uint32_t i = ((q & ~(j - 1)) << 1) | (q & (j - 1));
                            const uint32_t ixj = i | j;
                            const uint64_t xb = tile.k1[ixj], xa = tile.k1[i];
                            const bool less =
                                xb != xa ? xb < xa : cluster_tie_less(tile.idx[ixj], tile.idx[i], tile.k2, tile.k3, T);
                            if (less == (((e0 + i) & k) == 0)) {
                                tile.k1[i] = xb;
                                tile.k1[ixj] = xa;
                                const uint32_t t = tile.idx[i];
                                tile.idx[i] = tile.idx[ixj];
                                tile.idx[ixj] = t;
                            }
                        }
                        if (j > 1) __syncthreads();
                        else cl.sync();   // the next stage may cross CTAs
                    } else {
                        // pairs (i, i | j) across CTAs; this CTA takes an equal share
                        for (uint32_t q = rank * (T / 2) + threadIdx.x; q < (rank + 1) * (T / 2); q += blockDim.x) {
                            const uint32_t i = ((q & ~(j - 1)) << 1) | (q & (j - 1));
                            const uint32_t ixj = i | j;
                            uint64_t* pa = cl.map_shared_rank(tile.k1 + i % T, i / T);
                            uint64_t* pb = cl.map_shared_rank(tile.k1 + ixj % T, ixj / T);
                            uint32_t* qa = cl.map_shared_rank(tile.idx + i % T, i / T);
                            uint32_t* qb = cl.map_shared_rank(tile.idx + ixj % T, ixj / T);
                            const uint64_t xa = *pa, xb = *pb;
                            const bool less = xb != xa ? xb < xa : cluster_tie_less(*qb, *qa, tile.k2, tile.k3, T);
                            if (less == ((i & k) == 0)) {
                                *pa = xb;
                                *pb = xa;
                                const uint32_t t = *qa;
                                *qa = *qb;
                                *qb = t;
                            }
                        }
                        cl.sync();
                    }
                }
            }
        }
        if (rank == 0) {
            if (!in_tiles) {
                // beyond the cluster's tiles (rare): the first CTA sorts through global memory
                for (uint32_t i = threadIdx.x; i < NN; i += blockDim.x)
                    job.keys[i] = nam_key(closed[i], i, C.sort_mode);
                __syncthreads();
                block_sort_keys(job.keys, NN, tile, kSortTile);
            }
            if (threadIdx.x == 0) {
                ReadRec& R = rec[job.read];
                const uint64_t noff = atomicAdd(&ctr->nam_used, (unsigned long long)NN);
                if (noff + NN > A.nam_cap) {
                    R.flags |= kReadFailed;
                    R.n_nams = 0;   // the rescue kernel set the count ahead of the sort
                    atomicOr(&ctr->status, kStatusNamOverflow);
                    s_noff = ~0ULL;
                } else {
                    R.nam_off = noff;
                    R.n_nams = NN;
                    s_noff = noff;
                }
            }
        }
        cl.sync();
        const uint64_t noff = *cl.map_shared_rank(&s_noff, 0u);
        if (noff != ~0ULL) {
            if (in_tiles) {
                const uint32_t T = P / kClusterCtas, e0 = rank * T;
                for (uint32_t i = threadIdx.x; i < T && e0 + i < NN; i += blockDim.x)
                    A.nams[noff + e0 + i] = closed[tile.idx[i]];
            } else if (rank == 0) {
                for (uint32_t i = threadIdx.x; i < NN; i += blockDim.x) A.nams[noff + i] = closed[job.keys[i].idx];
            }
        }
        if (A.rescue_cycles && rank == 0 && threadIdx.x == 0)
            A.rescue_cycles[8ull * job.note + 3] = (uint64_t)(clock64() - t0);
        cl.sync();   // tiles and s_noff are reused by the next job
    }
}

// Writes the records x of the first m lanes to out[0 .. m).  A record has 11 words: written
// by each lane for itself, a store touches up to 44 sectors for 4 bytes of each; through
// `words` (32 records of shared memory) they leave in whole sectors (the two gathers of
// 100,000 reads 93 -> 60 us, of 2M reads 0.90 -> 0.60 ms with the first of them alone).
static_assert(sizeof(gbsa_nam) == 44, "a record is 11 words");
__device__ __forceinline__ void write_records(uint32_t* words, const gbsa_nam& x, uint32_t m, gbsa_nam* out) {
    const uint32_t lane = lane_id();
    if (lane < m) {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(&x);
#pragma unroll
        for (uint32_t i = 0; i < 11; ++i) words[11 * lane + i] = w[i];
    }
    __syncwarp();
    uint32_t* to = reinterpret_cast<uint32_t*>(out);
#pragma unroll
    for (uint32_t i = 0; i < 11; ++i)
        if (32 * i + lane < 11 * m) to[32 * i + lane] = words[32 * i + lane];
    __syncwarp();
}

// Records at or beyond out_cap are not written (the caller sized out from an estimate
// and gathers again when the total turns out larger).
// mode 0: every read; 1: the reads that were not rescued (fractions and rescue flags
// of every read), while the rescued reads' sorts may still run; 2: the rescued reads
// (through the rescue list), after their sorts.
__global__ void k_gather_nams(uint32_t n, const ReadRec* __restrict__ rec, const NamState* __restrict__ arena,
                              const uint64_t* __restrict__ out_off, gbsa_nam* __restrict__ out, uint64_t out_cap,
                              float* frac, uint8_t* rescued, int mode, Arenas A, const Counters* ctr,
                              const BatchDesc* desc) {
    __shared__ uint32_t s_words[kWarpsPerBlock][32 * 11];
    __shared__ uint32_t s_many[kWarpsPerBlock];   // mode 2: reads for the block
    __shared__ uint64_t s_from[kWarpsPerBlock], s_to[kWarpsPerBlock];
    uint32_t* words = s_words[threadIdx.x >> 5];
    const uint32_t lane = lane_id();
    uint64_t* copy_off = nullptr;
    if (desc) {
        const uint32_t cap = n;
        n = min(n, desc->n_reads);
        out = desc->out;
        out_cap = desc->out_cap;
        frac = mode == 2 ? nullptr : desc->frac;
        rescued = mode == 2 ? nullptr : desc->rescued;
        if (mode != 2) {
            copy_off = desc->out_off;
            // slots past the batch hold no NAMs: out_off[cap] is the batch's total
            if (blockIdx.x == 0 && threadIdx.x == 0) copy_off[n] = out_off[cap];
        }
    }
    // a rescued read with up to 64 NAMs by a warp, one with more by the block (it may hold
    // thousands: by a warp, the longest took 30 us of a batch of 1000 reads; but 100,000 reads
    // that are not in the index, a block each, 55 us); a block's reads lie apart on the list,
    // whose heavy ones are side by side
    if (mode == 2) {
        const uint32_t w = threadIdx.x >> 5, n_light = ctr->n_rescue, total = n_light + ctr->n_rescue_heavy;
        auto copy = [&](uint64_t from, uint64_t o, uint32_t m, uint32_t first, uint32_t step) {
            for (uint32_t j = first; j < m; j += step) {
                gbsa_nam x;
                if (j + lane < m) to_gbsa_nam(arena[from + j + lane], (int)(j + lane), x);
                write_records(words, x, min(m - j, 32u), out + o + j);
            }
        };
        for (uint32_t t0 = blockIdx.x; t0 < total; t0 += gridDim.x * kWarpsPerBlock) {
            const uint32_t t = t0 + w * gridDim.x;
            uint64_t from = 0, o = 0;
            uint32_t m = 0;
            if (t < total) {
                const uint32_t r = t < n_light ? A.rescue_list[t] : A.rescue_list[A.rescue_cap - 1 - (t - n_light)];
                from = rec[r].nam_off;
                o = out_off[r];
                m = o >= out_cap ? 0u : (uint32_t)min((uint64_t)rec[r].n_nams, out_cap - o);
            }
            if (m <= 64) {
                copy(from, o, m, 0, 32);
                m = 0;
            }
            if (lane == 0) {
                s_many[w] = m;
                s_from[w] = from;
                s_to[w] = o;
            }
            if (!__syncthreads_or(m != 0)) continue;
            for (uint32_t v = 0; v < kWarpsPerBlock; ++v) copy(s_from[v], s_to[v], s_many[v], 32 * w, blockDim.x);
            __syncthreads();
        }
        return;
    }
    // up to 32 reads in turn a warp, their NAMs side by side over the lanes
    const uint32_t group = min(max(n / warp_count(), 1u), 32u);
    for (uint32_t r0 = warp_global_id() * group; r0 < n; r0 += warp_count() * group) {
        const uint32_t r = r0 + lane;
        uint32_t count = 0;
        uint64_t from = 0, o = 0;   // the read's first NAM, its first record
        if (lane < group && r < n) {
            const ReadRec& R = rec[r];
            const bool resc = (R.flags & kReadRescue) != 0;
            count = mode == 1 && resc ? 0u : R.n_nams;
            from = R.nam_off;
            o = out_off[r];
            if (frac) frac[r] = R.frac;
            if (rescued) rescued[r] = resc ? 1 : 0;
            if (copy_off) copy_off[r] = o;
        }
        const uint32_t upto = warp_inclusive_sum(count);
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, upto, 31);
        from -= upto - count;
        o -= upto - count;
        const uint32_t before = upto - count;
        for (uint32_t c = 0; c < total; c += 32) {
            const uint32_t t = c + lane;
            // the read of NAM t: the first whose NAMs end behind it
            uint32_t at = 0;
#pragma unroll
            for (uint32_t step = 16; step; step /= 2)
                if (__shfl_sync(0xFFFFFFFFu, upto, at + step - 1) <= t) at += step;
            const uint64_t src = __shfl_sync(0xFFFFFFFFu, from, at) + t;
            const uint64_t dst = __shfl_sync(0xFFFFFFFFu, o, at) + t;
            const uint32_t id = t - __shfl_sync(0xFFFFFFFFu, before, at);
            const bool in = t < total && dst < out_cap;
            const uint64_t first = __shfl_sync(0xFFFFFFFFu, dst, 0);
            const uint32_t m = __popc(__ballot_sync(0xFFFFFFFFu, in));
            gbsa_nam x;
            if (in) to_gbsa_nam(arena[src], (int)id, x);
            if (__all_sync(0xFFFFFFFFu, !in || dst == first + lane)) write_records(words, x, m, out + first);
            else if (in) out[dst] = x;
        }
    }
}

__global__ void k_gather_queries(uint32_t n, const ReadRec* __restrict__ rec, const Query* __restrict__ arena,
                                 const uint64_t* __restrict__ out_off, gbsa_query_randstrobe* __restrict__ out) {
    const uint32_t lane = lane_id();
    for (uint32_t r = warp_global_id(); r < n; r += warp_count()) {
        const ReadRec R = rec[r];
        const uint64_t o = out_off[r];
        for (uint32_t j = lane; j < R.nq2; j += 32) {
            const Query q = arena[R.q_off + j];
            gbsa_query_randstrobe x;
            x.hash = q.hash;
            x.start = q.start;
            x.end = q.end;
            x.is_reverse = j >= R.nq ? 1 : 0;
            for (int b = 0; b < 7; ++b) x._pad[b] = 0;
            out[o + j] = x;
        }
    }
}

__global__ void k_read_counts(uint32_t n, const ReadRec* __restrict__ rec, int what, uint64_t* __restrict__ out,
                              const BatchDesc* desc) {
    const uint32_t live = desc ? min(n, desc->n_reads) : n;
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
        out[r] = r >= live ? 0 : (what == 0 ? rec[r].n_nams : (uint64_t)rec[r].nq2);
}

__global__ void k_clear_recs(uint32_t cap, ReadRec* __restrict__ rec, const BatchDesc* desc) {
    const uint32_t n = min(cap, desc->n_reads);
    unsigned long long* w = reinterpret_cast<unsigned long long*>(rec);
    static_assert(sizeof(ReadRec) % 8 == 0, "ReadRec is a whole number of 8-byte words");
    const uint64_t words = (uint64_t)n * (sizeof(ReadRec) / 8);
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < words; i += (uint64_t)gridDim.x * blockDim.x)
        w[i] = 0ull;
}

__global__ void k_reset_recs(uint32_t n, ReadRec* __restrict__ rec) {
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        ReadRec& R = rec[r];
        R.flags = 0;
        R.hit_off = 0;
        R.n_hits = 0;
        R.frac = 0.0f;
        R.nam_off = 0;
        R.n_nams = 0;
        R.n_found = 0;
    }
}

__global__ void k_find(IndexView I, const uint64_t* __restrict__ h, uint64_t n, uint64_t* __restrict__ pos) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        pos[i] = index_find(I, h[i]);
}

__global__ void k_get_count(IndexView I, const uint64_t* __restrict__ p, uint64_t n, uint32_t* __restrict__ c) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        c[i] = p[i] < I.n ? index_get_count(I, p[i]) : 0;
}

unsigned warp_grid(uint64_t items, int warps_per_block) {
    const int sms = device_sm_count();
    const uint64_t want = (items + warps_per_block - 1) / warps_per_block;
    const uint64_t cap = (uint64_t)sms * 16;
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(want, cap));
}

}  // namespace

uint32_t nam_kernel_warps(uint32_t n_reads) { return warp_grid(n_reads, kWarpsPerBlock) * kWarpsPerBlock; }

// Launches a kernel that probes the index, with the mapper's L2 access-policy window
// (the bucket table held persisting in L2) as a launch attribute, so that only these
// launches carry it and the caller's stream keeps its own attributes.
template <class... Exp, class... Act>
static void launch_probe(void (*kernel)(Exp...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                         const MapConfig& C, Act&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    if (C.l2_bytes) {
        attr[0].id = cudaLaunchAttributeAccessPolicyWindow;
        attr[0].val.accessPolicyWindow.base_ptr = const_cast<void*>(C.l2_base);
        attr[0].val.accessPolicyWindow.num_bytes = C.l2_bytes;
        attr[0].val.accessPolicyWindow.hitRatio = C.l2_hit_ratio;
        attr[0].val.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
        attr[0].val.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    GBSA_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<Act>(args)...));
}

void launch_seed(const DevParams& P, const uint8_t* seqs, const uint64_t* offs, const uint32_t* lens, uint32_t n,
                 ReadRec* rec, Arenas A, Counters* ctr, cudaStream_t st) {
    if (!n) return;
    k_seed_smem<<<warp_grid(n, kSeedWarps), 32 * kSeedWarps, 0, st>>>(P, seqs, offs, lens, n, rec, A, ctr);
    GBSA_LAUNCHED();
}

void launch_seed_long(const DevParams& P, const uint8_t* seqs, const uint64_t* offs, const uint32_t* lens,
                      ReadRec* rec, Arenas A, Counters* ctr, uint8_t* long_scratch, uint32_t long_warps,
                      cudaStream_t st, const BatchDesc* desc) {
    const unsigned blocks = std::max(1u, long_warps / kWarpsPerBlock);
    k_seed_long<<<blocks, 32 * kWarpsPerBlock, 0, st>>>(P, seqs, offs, lens, rec, A, ctr, long_scratch, desc);
    GBSA_LAUNCHED();
}

// Shapes of the batched form's seeding + lookup kernel (the autotuner's choices).
// Variant 0 is the plain form's fused kernel shape.
SeedVariant seed_variant(int v) {
    static const SeedVariant table[kSeedVariants] = {
        {8, 4, 512, 160}, {8, 5, 512, 160}, {4, 12, 512, 160}, {8, 7, 256, 96}, {16, 2, 512, 160}, {8, 6, 256, 96},
    };
    return table[v < 0 || v >= kSeedVariants ? 0 : v];
}

template <bool kCount, bool kLookup, bool kFast, int kWarps, int kBlocks, uint32_t kMaxLen, uint32_t kSyncmers>
static void launch_q(const DevParams& P, const IndexView& I, const MapConfig& C, const BatchDesc* desc, ReadRec* rec,
                     Arenas A, Counters* ctr, uint32_t cap, cudaStream_t st) {
    // resident blocks, and a scratch slot a warp (the work areas hold nam_kernel_warps(cap))
    const unsigned grid = std::min<unsigned>((unsigned)device_sm_count() * kBlocks,
                                             std::max(1u, nam_kernel_warps(cap) / kWarps));
    launch_probe(k_seed_lookup_q<kCount, kLookup, kFast, kWarps, kBlocks, kMaxLen, kSyncmers>, grid, 32 * kWarps, 0, st, C,
                 P, I, C, desc, rec, A, ctr);
}

template <bool kCount, bool kLookup, bool kFast>
static void launch_q_variant(int v, const DevParams& P, const IndexView& I, const MapConfig& C, const BatchDesc* desc,
                             ReadRec* rec, Arenas A, Counters* ctr, uint32_t cap, cudaStream_t st) {
    switch (v) {
        case 1: launch_q<kCount, kLookup, kFast, 8, 5, 512, 160>(P, I, C, desc, rec, A, ctr, cap, st); break;
        case 2: launch_q<kCount, kLookup, kFast, 4, 12, 512, 160>(P, I, C, desc, rec, A, ctr, cap, st); break;
        case 3: launch_q<kCount, kLookup, kFast, 8, 7, 256, 96>(P, I, C, desc, rec, A, ctr, cap, st); break;
        case 4: launch_q<kCount, kLookup, kFast, 16, 2, 512, 160>(P, I, C, desc, rec, A, ctr, cap, st); break;
        case 5: launch_q<kCount, kLookup, kFast, 8, 6, 256, 96>(P, I, C, desc, rec, A, ctr, cap, st); break;
        default: launch_q<kCount, kLookup, kFast, 8, 4, 512, 160>(P, I, C, desc, rec, A, ctr, cap, st); break;
    }
}

bool seeds_fast(const DevParams& P, const IndexView& I, const MapConfig& C) { return fast_seed(P, I, C); }

void launch_seed_lookup_queue(const DevParams& P, const IndexView& I, const MapConfig& C, const BatchDesc* desc,
                              ReadRec* rec, Arenas A, Counters* ctr, int variant, bool lookup, uint32_t cap,
                              cudaStream_t st) {
    if (!lookup) launch_q_variant<false, false, false>(variant, P, I, C, desc, rec, A, ctr, cap, st);
    else if (C.count_bytes) launch_q_variant<true, true, false>(variant, P, I, C, desc, rec, A, ctr, cap, st);
    else if (fast_seed(P, I, C)) launch_q_variant<false, true, true>(variant, P, I, C, desc, rec, A, ctr, cap, st);
    else launch_q_variant<false, true, false>(variant, P, I, C, desc, rec, A, ctr, cap, st);
    GBSA_LAUNCHED();
}

void launch_seed_lookup(const DevParams& P, const IndexView& I, const MapConfig& C, const uint8_t* seqs,
                        const uint64_t* offs, const uint32_t* lens, uint32_t n, ReadRec* rec, Arenas A, Counters* ctr,
                        cudaStream_t st) {
    if (!n) return;
    // resident blocks only: the warps pull reads from the work counter until none is left
    const unsigned grid = std::min<unsigned>(warp_grid(n, kSeedWarps), (unsigned)device_sm_count() * kFusedBlocksPerSm);
    launch_probe(C.count_bytes ? k_seed_lookup<true, false>
                               : (fast_seed(P, I, C) ? k_seed_lookup<false, true> : k_seed_lookup<false, false>), grid, 32 * kSeedWarps, 0, st, C, P, I, C,
                 seqs, offs, lens, n, rec, A, ctr);
    GBSA_LAUNCHED();
}

void launch_lookup_long(const IndexView& I, const MapConfig& C, uint32_t n, ReadRec* rec, Arenas A, Counters* ctr,
                        cudaStream_t st) {
    if (!n) return;
    // sized for n long reads (every read, for long-read parameter sets); warps beyond
    // the long-list count exit at once
    const unsigned blocks = warp_grid(n, kWarpsPerBlock);
    launch_probe(C.count_bytes ? k_lookup_long<true> : k_lookup_long<false>, blocks, 32 * kWarpsPerBlock, 0, st, C, I,
                 C, rec, A, ctr);
    GBSA_LAUNCHED();
}

void launch_lookup(const IndexView& I, const MapConfig& C, uint32_t n, ReadRec* rec, Arenas A, Counters* ctr,
                   cudaStream_t st, const BatchDesc* desc) {
    if (!n) return;
    launch_probe(C.count_bytes ? k_lookup<true> : k_lookup<false>, warp_grid(n, kWarpsPerBlock), 32 * kWarpsPerBlock, 0,
                 st, C, I, C, n, rec, A, ctr, desc);
    GBSA_LAUNCHED();
}

// The NAM phase's kernels (group and block merges, rescue, NAM gather) run beside each
// other and need most of an SM's shared memory together (rescue 2 x 97 KB, group merge
// 17 KB a block): they ask for the largest shared-memory carveout, so that the SM keeps
// that configuration through the phase instead of switching it as each kernel's blocks
// arrive (left to CUDA, an earlier merge took 5.0 instead of 3.3 ms on the C2 batch
// inside the batch graph).  The seeding + lookup kernels keep the default: they use the
// rest of the unified L1 to cache index entries.  Set once per device.
void nam_phase_carveout() {
    static std::mutex mu;
    static std::vector<char> done;
    int dev = 0;
    GBSA_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> g(mu);
    if ((int)done.size() <= dev) done.resize(dev + 1, 0);
    if (done[dev]) return;
    const void* fs[] = {(const void*)k_nams_group, (const void*)k_nams, (const void*)k_rescue, (const void*)k_gather_nams};
    for (const void* f : fs)
        GBSA_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout,
                                       (int)cudaSharedmemCarveoutMaxShared));
    GBSA_CUDA(cudaFuncSetAttribute(k_rescue, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RescueShared)));
    GBSA_CUDA(cudaFuncSetAttribute(k_nams, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BigShared)));
    done[dev] = 1;
}

void launch_nams(const MapConfig& C, uint32_t n, ReadRec* rec, Arenas A, Counters* ctr, cudaStream_t st) {
    if (!n) return;
    nam_phase_carveout();
    const unsigned blocks = grid_for(n, kGroupWarps, (unsigned)device_sm_count() * kGroupBlocksPerSm);
    k_nams_group<<<blocks, 32 * kGroupWarps, 0, st>>>(C, rec, A, ctr);
    GBSA_LAUNCHED();
}

void launch_bucket_reads(uint32_t n, ReadRec* rec, Arenas A, Counters* ctr, cudaStream_t st, const BatchDesc* desc) {
    if (!n) return;
    k_bucket_reads<<<grid_for(n, 256, (unsigned)device_sm_count() * 8), 256, 0, st>>>(n, rec, A, ctr, desc);
    GBSA_LAUNCHED();
}

void launch_nams_warp(const MapConfig& C, int k, uint32_t n, ReadRec* rec, Arenas A, Counters* ctr, cudaStream_t st) {
    if (!n) return;
    nam_phase_carveout();
    // a block for 16 reads, 64 at least (a hundred reads of 4,000 bp went through 7 blocks); a
    // warp without a scratch slot takes the overflow arena's room
    const unsigned blocks =
        std::min<unsigned>((unsigned)device_sm_count() * 2, std::min(n, std::max(64u, (n + 15) / 16)));
    k_nams<<<blocks, kBigThreads, sizeof(BigShared), st>>>(C, k, rec, A, ctr);
    GBSA_LAUNCHED();
}

void launch_rescue(const IndexView& I, const MapConfig& C, uint32_t n_reads, ReadRec* rec, Arenas A, Counters* ctr,
                   cudaStream_t st) {
    if (!n_reads) return;
    nam_phase_carveout();
    // persistent, kRescueBlocksPerSm per SM (at most one scratch slot per warp)
    const unsigned blocks =
        std::min<unsigned>(warp_grid(n_reads, kWarpsPerBlock), (unsigned)device_sm_count() * kRescueBlocksPerSm);
    launch_probe(k_rescue, blocks, 32 * kWarpsPerBlock, sizeof(RescueShared), st, C, I, C, rec, A, ctr);
    GBSA_LAUNCHED();
}

// The sorts' dynamic shared memory: a tile of kSortTile keys; their limit is set once per
// device (mappers may launch from several threads at once).
constexpr int kSortThreads = 256;
constexpr size_t kSortSmem = kSortTile * 28;

static void sort_smem_limit() {
    static std::mutex mu;
    static std::vector<char> done;
    int dev = 0;
    GBSA_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> g(mu);
    if ((int)done.size() <= dev) done.resize(dev + 1, 0);
    if (done[dev]) return;
    for (const void* f : {(const void*)k_sort_jobs<kSortThreads, kSortTile>,
                          (const void*)k_sort_jobs<2 * kSortThreads, kSortTile>, (const void*)k_sort_jobs_cluster})
        GBSA_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSortSmem));
    GBSA_CUDA(cudaFuncSetAttribute(k_sort_packed, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(8 * kPackMax)));
    done[dev] = 1;
}

// The sorts' grids: resident blocks, no more than there can be jobs.
void launch_sort_packed(const MapConfig& C, uint32_t n, ReadRec* rec, Arenas A, Counters* ctr, cudaStream_t st) {
    sort_smem_limit();
    k_sort_packed<<<std::min(n, (unsigned)device_sm_count() * 2), kPackThreads, 8 * kPackMax, st>>>(C, rec, A, ctr);
    GBSA_LAUNCHED();
}

void launch_sort_jobs(const MapConfig& C, uint32_t n, ReadRec* rec, Arenas A, Counters* ctr, cudaStream_t st) {
    sort_smem_limit();
    const unsigned sms = (unsigned)device_sm_count();
    if (C.sort_variant == 1)
        k_sort_jobs<2 * kSortThreads, kSortTile><<<std::min(n, sms * 3), 2 * kSortThreads, kSortSmem, st>>>(C, rec, A, ctr);
    else
        k_sort_jobs<kSortThreads, kSortTile><<<std::min(n, sms * 4), kSortThreads, kSortSmem, st>>>(C, rec, A, ctr);
    GBSA_LAUNCHED();
}

void launch_sort_jobs_cluster(const MapConfig& C, uint32_t n, ReadRec* rec, Arenas A, Counters* ctr, cudaStream_t st) {
    sort_smem_limit();
    // SMs / 2 clusters of kClusterCtas CTAs
    const unsigned clusters = std::min(n, std::max(1u, (unsigned)device_sm_count() / 2));
    k_sort_jobs_cluster<<<clusters * kClusterCtas, 256, kSortSmem, st>>>(C, rec, A, ctr);
    GBSA_LAUNCHED();
}

void launch_gather_nams(uint32_t n, const ReadRec* rec, const NamState* arena, const uint64_t* out_off,
                        gbsa_nam* out, float* frac, uint8_t* rescued, cudaStream_t st, uint64_t out_cap, int mode,
                        const Arenas* A, const Counters* ctr, const BatchDesc* desc) {
    if (!n) return;
    const Arenas none{};
    k_gather_nams<<<warp_grid(n, kWarpsPerBlock), 32 * kWarpsPerBlock, 0, st>>>(
        n, rec, arena, out_off, out, out_cap, frac, rescued, mode, A ? *A : none, ctr, desc);
    GBSA_LAUNCHED();
}

// The queries of each read forward-first, each orientation ordered by start (stable), and the
// read's record, a warp a read.  Queries in that order already (as randstrobes_query gives
// them) are copied; others are placed by rank, or when a read has more than kRankQueries of
// them `left` is set and the caller lays the batch out itself.  Bound by the upload.  (On the
// host, a sort a read: 5,000 reads of 150 bp 1.67 ms a call, now 0.31.)
__global__ void k_layout_queries(uint32_t n, const gbsa_query_randstrobe* __restrict__ in,
                                 const uint64_t* __restrict__ offs, Query* __restrict__ out, ReadRec* __restrict__ rec,
                                 uint32_t* __restrict__ left) {
    const uint32_t lane = lane_id();
    const uint64_t first = offs[0];
    // orientation above the start
    auto key = [](const gbsa_query_randstrobe& q) { return ((uint64_t)(q.is_reverse != 0) << 32) | q.start; };
    for (uint32_t r = warp_global_id(); r < n; r += warp_count()) {
        const uint64_t a = offs[r] - first, m = offs[r + 1] - offs[r];
        uint32_t nf = 0;
        bool late = false;
        for (uint64_t i = lane; i < m; i += 32) {
            const gbsa_query_randstrobe q = in[a + i];
            nf += q.is_reverse ? 0 : 1;
            if (i) late |= key(in[a + i - 1]) > key(q);
            out[a + i] = Query{q.hash, q.start, q.end};
        }
        nf = __reduce_add_sync(0xFFFFFFFFu, nf);
        if (__any_sync(0xFFFFFFFFu, late)) {
            if (m > kRankQueries) {
                if (lane == 0) *left = 1;
                continue;
            }
            __syncwarp();
            for (uint64_t i = lane; i < m; i += 32) {
                const gbsa_query_randstrobe q = in[a + i];
                uint32_t rank = 0;
                for (uint64_t j = 0; j < m; ++j) {
                    const uint64_t o = key(in[a + j]);
                    rank += o < key(q) || (o == key(q) && j < i);
                }
                out[a + rank] = Query{q.hash, q.start, q.end};
            }
        }
        if (lane == 0) {
            ReadRec R{};
            R.q_off = a;
            R.nq = nf;
            R.nq2 = (uint32_t)m;
            rec[r] = R;
        }
    }
}

void launch_layout_queries(uint32_t n, const gbsa_query_randstrobe* in, const uint64_t* offs, Query* out, ReadRec* rec,
                           uint32_t* left, cudaStream_t st) {
    if (!n) return;
    k_layout_queries<<<warp_grid(n, kWarpsPerBlock), 32 * kWarpsPerBlock, 0, st>>>(n, in, offs, out, rec, left);
    GBSA_LAUNCHED();
}

void launch_gather_queries(uint32_t n, const ReadRec* rec, const Query* arena, const uint64_t* out_off,
                           gbsa_query_randstrobe* out, cudaStream_t st) {
    if (!n) return;
    k_gather_queries<<<warp_grid(n, kWarpsPerBlock), 32 * kWarpsPerBlock, 0, st>>>(n, rec, arena, out_off, out);
    GBSA_LAUNCHED();
}

void launch_find(const IndexView& I, const uint64_t* hashes, uint64_t n, uint64_t* pos, cudaStream_t st) {
    if (!n) return;
    k_find<<<grid_for(n, 256, 1u << 20), 256, 0, st>>>(I, hashes, n, pos);
    GBSA_LAUNCHED();
}

void launch_get_count(const IndexView& I, const uint64_t* pos, uint64_t n, uint32_t* counts, cudaStream_t st) {
    if (!n) return;
    k_get_count<<<grid_for(n, 256, 1u << 20), 256, 0, st>>>(I, pos, n, counts);
    GBSA_LAUNCHED();
}

void launch_reset_recs(uint32_t n, ReadRec* rec, cudaStream_t st) {
    if (!n) return;
    k_reset_recs<<<grid_for(n, 256, 1u << 16), 256, 0, st>>>(n, rec);
    GBSA_LAUNCHED();
}

void launch_clear_recs(uint32_t cap, ReadRec* rec, const BatchDesc* desc, cudaStream_t st) {
    if (!cap) return;
    k_clear_recs<<<(unsigned)device_sm_count() * 4, 256, 0, st>>>(cap, rec, desc);
    GBSA_LAUNCHED();
}

__global__ void k_offsets_add(const uint64_t* __restrict__ in, uint64_t* __restrict__ out, uint64_t n, uint64_t base) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = in[i] + base;
}

void launch_offsets_add(const uint64_t* in, uint64_t* out, uint64_t n, uint64_t base, cudaStream_t st) {
    if (!n) return;
    k_offsets_add<<<grid_for(n, 256, 4096), 256, 0, st>>>(in, out, n, base);
    GBSA_LAUNCHED();
}

void launch_read_counts(uint32_t n, const ReadRec* rec, int what, uint64_t* out, cudaStream_t st,
                        const BatchDesc* desc) {
    if (!n) return;
    k_read_counts<<<grid_for(n, 256, 1u << 16), 256, 0, st>>>(n, rec, what, out, desc);
    GBSA_LAUNCHED();
}

}  // namespace gbsa
