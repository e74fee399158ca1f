// nam.cuh — hit → NAM merging and NAM ordering, warp-cooperative.
//
// The reference keeps one hit list per (orientation, reference id) in robin_hood
// maps (step2/nam.cu:45-62) and merges each list on its own:
//   merge_hits_into_nams      (hit-major, step2/nam.cu:347-513; find_nams)
//   merge_hits_into_nams_fast (NAM-major, step2/nam.cu:94-343; find_nams_rescue)
// over hits sorted by (query_start, ref_start).  Lists never interact, so the warp
// processes all of them at once, one query randstrobe at a time: the hits of one
// query randstrobe share query_start, arrive sorted by ref_start (a hash run is
// sorted by position) and only meet NAMs of their own (orientation, reference id).
//
// NAMs are kept in creation order (the reference's open list order).  A NAM whose
// query_end is behind the current query_start can take no later hit (the reference
// removes such NAMs at its flush points; which NAMs are removed when only changes
// iteration, not results).
//
//   hit-major: for each hit (ref_start order), the first open NAM in creation order
//     that accepts it takes it — found with a warp ballot over 32 NAMs at a time.
//   NAM-major: for each open NAM (creation order), the first untaken hit of the
//     query with ref_start in (ref_prev, ref_end] that extends it or lies inside it —
//     all NAMs propose at once and a hit keeps the NAM created first.
#pragma once

#include "lookup.cuh"

namespace gbsa {

// Working state of one NAM (step2/my_struct.hpp:48-62 fields used by the merge).
struct NamState {
    int32_t qs, qe, qprev, rs, re, rprev, n_hits;
    uint32_t ref_rc;
};

__device__ __forceinline__ NamState nam_from_hit(const HitRec& h) {
    NamState n;
    n.qs = h.qs;
    n.qe = h.qe;
    n.qprev = h.qs;
    n.rs = h.rs;
    n.re = h.re;
    n.rprev = h.rs;
    n.n_hits = 1;
    n.ref_rc = h.ref_rc;
    return n;
}

// Warp-cooperative add_to_hits_per_ref (step2/nam.cu:45-62) for one query whose
// equal-hash run [pos, pos + cnt) is known: an entry is kept when its length
// difference is <= every earlier difference of the run (the reference's running
// minimum), found with a warp prefix minimum.  Writes the kept hits in compact form
// (rs[] = position, pk[] = packed, in run order) and returns their count (at most
// cap are written) and the spans of the shortest and the longest kept hit.  The entries are loaded 128 at a time, four per lane, so a run
// of up to 128 costs one memory round trip.
__device__ __forceinline__ uint32_t warp_walk_run_n(const IndexView& I, int qs, int qe, uint64_t pos, uint32_t cnt,
                                                    uint32_t* rs_out, uint32_t* pk_out, uint32_t cap,
                                                    uint32_t& min_span, uint32_t& max_span) {
    const uint32_t lane = lane_id();
    uint32_t mn = 0xFFu, mx = 0;   // of the packed words' low bytes (span - k)
    int carry = 0x7FFFFFFF;
    uint32_t n = 0;
    const uint2* ent = reinterpret_cast<const uint2*>(I.rs + pos);   // (position, packed) at offset 8
    for (uint32_t base = 0; base < cnt; base += 128) {
        uint2 e[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t j = base + 32 * u + lane;
            e[u] = j < cnt ? __ldg(&ent[2 * (size_t)j + 1]) : make_uint2(0, 0);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t j = base + 32 * u + lane;
            const bool mine = j < cnt;
            int diff = 0x7FFFFFFF;
            if (mine) {
                const int d = (qe - qs) - ((int)(e[u].y & 0xFF) + I.k);
                diff = d < 0 ? -d : d;
            }
            int pm = diff;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xFFFFFFFFu, pm, o);
                if (lane >= (uint32_t)o) pm = v < pm ? v : pm;
            }
            int excl = __shfl_up_sync(0xFFFFFFFFu, pm, 1);
            if (lane == 0) excl = 0x7FFFFFFF;
            excl = excl < carry ? excl : carry;
            const bool keep = mine && diff <= excl;
            const uint32_t km = __ballot_sync(0xFFFFFFFFu, keep);
            if (keep) {
                mn = min(mn, e[u].y & 0xFFu);
                mx = max(mx, e[u].y & 0xFFu);
                const uint32_t k = n + __popc(km & lanemask_lt());
                if (k < cap) {
                    rs_out[k] = e[u].x;
                    pk_out[k] = e[u].y;
                }
            }
            n += __popc(km);
            const int tot = __shfl_sync(0xFFFFFFFFu, pm, 31);
            carry = tot < carry ? tot : carry;
        }
    }
    min_span = __reduce_min_sync(0xFFFFFFFFu, mn) + (uint32_t)I.k;
    max_span = __reduce_max_sync(0xFFFFFFFFu, mx) + (uint32_t)I.k;
    __syncwarp();
    return n;
}

// Score (step2/nam.cu:454-463): n_hits * (2*min_span - max_span) if positive, else 1.
__device__ __forceinline__ int nam_score_int(const NamState& n) {
    const int qspan = n.qe - n.qs, rspan = n.re - n.rs;
    const int mx = qspan > rspan ? qspan : rspan;
    const int mn = qspan < rspan ? qspan : rspan;
    const int v = 2 * mn - mx;
    return v > 0 ? n.n_hits * v : 1;
}

__device__ __forceinline__ void to_gbsa_nam(const NamState& n, int id, gbsa_nam& o) {
    o.nam_id = id;
    o.query_start = n.qs;
    o.query_end = n.qe;
    o.query_prev_hit_startpos = n.qprev;
    o.ref_start = n.rs;
    o.ref_end = n.re;
    o.ref_prev_hit_startpos = n.rprev;
    o.n_hits = n.n_hits;
    o.ref_id = (int32_t)(n.ref_rc & 0x7FFFFFFFu);
    o.score = (float)nam_score_int(n);
    o.is_rc = (n.ref_rc >> 31) ? 1 : 0;
    o._pad[0] = o._pad[1] = o._pad[2] = 0;
}

// Sort key of a NAM: three u64 compared in order, then the index (stable).
//   GBSA_SORT_SCORE:     score desc, is_rc, ref_id, qs | qe, rs, re | n_hits desc
//   GBSA_SORT_REF_MATE2: is_rc, ref_id, max(0, rs-qs) | n_hits desc, qe, qs | re, rs
//                        (Nam::operator<, step2/my_struct.hpp:78-92)
//   GBSA_SORT_REF_MATE1: is_rc, ref_id | n_hits desc, qe, qs | re, rs
//                        (sort_nams_single2, step2/main.cu:2271-2289)
// All compared fields enter a key, so the order is total over the compared fields
// (the score is a function of n_hits and the coordinates).  Field widths: ref_id <
// 2^24 (RefRandstrobe packs it in 24 bits), query coordinates <= GBSA_MAX_READ_LEN,
// score < 2^24, NAM ref spans < 2^19.
struct NamKey {
    uint64_t k1, k2, k3;
    uint32_t idx;
    uint32_t pad;
};

__device__ __forceinline__ NamKey nam_key(const NamState& n, uint32_t idx, int mode) {
    const uint64_t rc = n.ref_rc >> 31, ref = n.ref_rc & 0xFFFFFFu;
    NamKey k;
    k.idx = idx;
    k.pad = 0;
    if (mode == GBSA_SORT_SCORE) {
        const uint64_t sc = (uint64_t)nam_score_int(n);
        k.k1 = ((0xFFFFFFull - sc) << 40) | (rc << 39) | (ref << 15) | ((uint64_t)n.qs & 0x7FFF);
        k.k2 = ((uint64_t)n.qe << 51) | ((uint64_t)(uint32_t)n.rs << 19) | ((uint64_t)(n.re - n.rs) & 0x7FFFF);
        k.k3 = 0xFFFFFFFFull - (uint32_t)n.n_hits;
    } else {
        const int d = n.rs - n.qs;
        const uint64_t diag = mode == GBSA_SORT_REF_MATE2 ? (uint64_t)(uint32_t)(d > 0 ? d : 0) : 0;
        k.k1 = (rc << 56) | (ref << 32) | diag;
        k.k2 = ((0xFFFFull - (uint32_t)n.n_hits) << 48) | ((uint64_t)n.qe << 24) | (uint64_t)n.qs;
        k.k3 = ((uint64_t)(uint32_t)n.re << 32) | (uint32_t)n.rs;
    }
    return k;
}

__device__ __forceinline__ bool key_less(const NamKey& a, const NamKey& b) {
    if (a.k1 != b.k1) return a.k1 < b.k1;
    if (a.k2 != b.k2) return a.k2 < b.k2;
    if (a.k3 != b.k3) return a.k3 < b.k3;
    return a.idx < b.idx;
}

__device__ __forceinline__ uint32_t next_pow2(uint32_t n) {
    return n <= 1 ? 1 : 1u << (32 - __clz(n - 1));
}

// Warp bitonic sort of n keys; keys must have room for next_pow2(n) entries.
__device__ inline void warp_sort_keys(NamKey* keys, uint32_t n) {
    const uint32_t lane = lane_id();
    const uint32_t P = next_pow2(n);
    for (uint32_t i = n + lane; i < P; i += 32) {
        NamKey k;
        k.k1 = k.k2 = k.k3 = ~0ULL;
        k.idx = 0xFFFFFFFFu;
        k.pad = 0;
        keys[i] = k;
    }
    __syncwarp();
    for (uint32_t k = 2; k <= P; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t i = lane; i < P; i += 32) {
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
            __syncwarp();
        }
    }
}

// Warp bitonic sort of u64 keys; keys must have room for next_pow2(n) entries.
__device__ inline void warp_sort_u64(uint64_t* keys, uint32_t n) {
    const uint32_t lane = lane_id();
    if (n <= 32) {   // in registers
        uint64_t x = lane < n ? keys[lane] : ~0ULL;
#pragma unroll
        for (uint32_t k = 2; k <= 32; k <<= 1)
#pragma unroll
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                const uint64_t y = __shfl_xor_sync(0xFFFFFFFFu, x, j);
                // the lower lane of a pair keeps the smaller key where the run ascends
                if ((x > y) == (((lane & j) == 0) == ((lane & k) == 0))) x = y;
            }
        if (lane < n) keys[lane] = x;
        __syncwarp();
        return;
    }
    const uint32_t P = next_pow2(n);
    for (uint32_t i = n + lane; i < P; i += 32) keys[i] = ~0ULL;
    __syncwarp();
    for (uint32_t k = 2; k <= P; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t i = lane; i < P; i += 32) {
                const uint32_t ixj = i ^ j;
                if (ixj > i) {
                    const uint64_t a = keys[i], b = keys[ixj];
                    const bool up = (i & k) == 0;
                    if ((a > b) == up) {
                        keys[i] = b;
                        keys[ixj] = a;
                    }
                }
            }
            __syncwarp();
        }
    }
}

}  // namespace gbsa
