// lookup.cuh — index probes: StrobemerIndex::find / is_filtered / get_count and the
// hit-run walk of add_to_hits_per_ref, as device functions.
#pragma once

#include "index.h"

namespace gbsa {

// Hit record of the NAM stage (step2/my_struct.hpp:95-110 plus its map key):
// ref_rc = is_rc << 31 | ref_id.
struct HitRec {
    uint32_t ref_rc;
    int32_t qs, qe, rs, re;
};

// A hit as stored in the hit arena: 16 bytes, one vector load.  Query coordinates are
// below GBSA_MAX_READ_LEN, so query start and end share a word.
struct __align__(16) HitPacked {
    uint32_t ref_rc;
    uint32_t qse;    // query start | query end << 16
    int32_t rs, re;
};
static_assert(GBSA_MAX_READ_LEN < 65536, "query coordinates fit 16 bits");

__device__ __forceinline__ HitPacked pack_hit(uint32_t ref_rc, int qs, int qe, int rs, int re) {
    HitPacked p;
    p.ref_rc = ref_rc;
    p.qse = (uint32_t)qs | ((uint32_t)qe << 16);
    p.rs = rs;
    p.re = re;
    return p;
}

__device__ __forceinline__ uint64_t get_hash(const IndexView& I, uint64_t pos) {   // index.hpp:83-89
    return pos < I.n ? __ldg(&I.rs[pos].hash) : ~0ULL;
}

// Start of bucket i.
__device__ __forceinline__ uint64_t bucket_start(const IndexView& I, uint64_t i) {
    return I.buckets ? (uint64_t)__ldg(&I.buckets[i].start) : __ldg(&I.starts[i]);
}

// First entry of [a, b), sorted by hash, whose hash equals the key, or kNotFound: entries in
// order until one is >= key (buckets hold ~2 entries on average), or a binary search for a
// long range; both give the reference's answer.  ex receives the number of entries
// examined by the linear rule (for the byte count).
__device__ __forceinline__ uint64_t find_in(const IndexView& I, uint64_t key, uint64_t a, uint64_t b,
                                            uint32_t* ex = nullptr) {
    if (b - a <= 16) {
        for (uint64_t x = a; x < b; ++x) {
            const uint64_t h = __ldg(&I.rs[x].hash);
            if (h >= key) {
                if (ex) *ex = (uint32_t)(x - a + 1);
                return h == key ? x : kNotFound;
            }
        }
        if (ex) *ex = (uint32_t)(b - a);
        return kNotFound;
    }
    uint64_t lo = a, hi = b;
    while (lo < hi) {
        const uint64_t mid = lo + (hi - lo) / 2;
        if (__ldg(&I.rs[mid].hash) < key) lo = mid + 1;
        else hi = mid;
    }
    if (ex) *ex = (uint32_t)(lo - a + 1 < b - a ? lo - a + 1 : b - a);
    return (lo < b && __ldg(&I.rs[lo].hash) == key) ? lo : kNotFound;
}

// StrobemerIndex::find (step2/index.hpp:57-81): first entry of the key's bucket
// whose hash equals the key, or kNotFound.
__device__ __forceinline__ uint64_t index_find(const IndexView& I, uint64_t key, uint32_t* ex = nullptr,
                                               uint64_t* bucket_end = nullptr) {
    const uint64_t top = key >> (64 - I.bits);
    const uint64_t a = bucket_start(I, top);
    const uint64_t b = bucket_start(I, top + 1);
    if (bucket_end) *bucket_end = b;
    if (a >= b) {
        if (ex) *ex = 0;
        return kNotFound;
    }
    return find_in(I, key, a, b, ex);
}

// An index entry as one 16-byte load.
struct Entry {
    uint64_t hash;
    uint32_t position, packed;
};
__device__ __forceinline__ Entry load_entry(const IndexView& I, uint32_t pos) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(I.rs) + pos);
    return Entry{((uint64_t)v.y << 32) | v.x, v.z, v.w};
}

// A query's answer from the tagged buckets (I.buckets set): the position of its hash
// (kMissing: not in the index), whether it is filtered, and for one that is not the hits
// that add_to_hits_per_ref keeps and the first of them (the run's first entry, which is
// always kept).
constexpr uint32_t kMissing = 0xFFFFFFFFu;   // fewer than 2^32 entries: no entry's position
struct Probe {
    uint32_t pos;
    bool filtered;
    uint32_t n_hits;
    uint32_t position, packed;
};

// What the bucket alone says of a key: the entries that may equal it.  None (`match` 0): the
// key is not in the index.
struct Candidates {
    uint32_t start;
    uint32_t size;    // 255: or more
    uint32_t match;   // bit i: entry i's tag agrees (kBucketTags or fewer entries), else bit 0
};
__device__ __forceinline__ uint4 load_bucket(const IndexView& I, uint64_t key) {
    return __ldg(reinterpret_cast<const uint4*>(I.buckets) + (uint32_t)(key >> (64 - I.bits)));
}
__device__ __forceinline__ Candidates bucket_candidates(const uint4& b, uint64_t key) {
    const uint32_t tag = hash_tag(key) * 0x01010101u;
    // a bit for each byte that agrees, gathered in bits 24..27
    auto bits = [&](uint32_t w, uint32_t bytes) { return (__vcmpeq4(w, tag) & bytes) * 0x01020408u; };
    Candidates c;
    c.start = b.x;
    c.size = b.y & 0xFFu;
    c.match = (bits(b.y, 0x01010100u) >> 25) & 0x7u;
    c.match |= (bits(b.z, 0x01010101u) >> 21) & 0x78u;
    c.match |= (bits(b.w, 0x01010101u) >> 17) & 0x780u;
    c.match &= (1u << min(c.size, kBucketTags)) - 1;
    if (c.size > kBucketTags) c.match = 1;
    return c;
}

// The answer for a key with candidates: those entries in order, or a bucket of more than
// kBucketTags searched as a whole.  `len` is the query's length.
__device__ __forceinline__ Probe probe_candidates(const IndexView& I, uint64_t key, int len, const Candidates& c) {
    Probe p;
    p.pos = kMissing;
    p.filtered = false;
    p.n_hits = 0;
    p.position = p.packed = 0;
    const uint32_t a = c.start;
    uint32_t end = a + c.size;
    Entry e;
    if (c.size <= kBucketTags) {
        for (uint32_t m = c.match;; m &= m - 1) {
            if (!m) return p;
            const uint32_t i = (uint32_t)__ffs(m) - 1;
            e = load_entry(I, a + i);
            if (e.hash == key) {
                p.pos = a + i;
                break;
            }
        }
    } else {
        if (c.size == 255) end = __ldg(&I.buckets[(uint32_t)(key >> (64 - I.bits)) + 1].start);
        const uint64_t x = find_in(I, key, a, end);
        if (x == kNotFound) return p;
        p.pos = (uint32_t)x;
        e = load_entry(I, p.pos);
    }
    // an entry at or past the bucket's end has other top bits, so it cannot equal key; past
    // the table's end the reference reads all ones
    const uint64_t far = (uint64_t)p.pos + I.filter_cutoff;
    p.filtered = far >= end ? far >= I.n && key == ~0ULL : __ldg(&I.rs[far].hash) == key;
    if (p.filtered) return p;
    p.position = e.position;
    p.packed = e.packed;
    p.n_hits = 1;
    int least = len - ((int)(e.packed & 0xFF) + I.k);
    least = least < 0 ? -least : least;
    for (uint32_t x = p.pos + 1; x < end; ++x) {
        if (c.size <= kBucketTags && !((c.match >> (x - a)) & 1u)) break;
        const Entry f = load_entry(I, x);
        if (f.hash != key) break;
        int diff = len - ((int)(f.packed & 0xFF) + I.k);
        diff = diff < 0 ? -diff : diff;
        if (diff <= least) {
            least = diff;
            ++p.n_hits;
        }
    }
    return p;
}

__device__ __forceinline__ Probe index_probe(const IndexView& I, uint64_t key, int len) {
    const Candidates c = bucket_candidates(load_bucket(I, key), key);
    if (c.match) return probe_candidates(I, key, len, c);
    Probe p;
    p.pos = kMissing;
    p.filtered = false;
    p.n_hits = 0;
    p.position = p.packed = 0;
    return p;
}

__device__ __forceinline__ bool index_is_filtered(const IndexView& I, uint64_t pos) {   // index.hpp:91-93
    return get_hash(I, pos) == get_hash(I, pos + I.filter_cutoff);
}

// index_is_filtered for a position returned by index_find(key) whose bucket ends at
// bucket_end: an entry at or past the bucket's end has other top bits, so it cannot
// equal key, and the second load is needed only when pos + filter_cutoff is still
// inside the bucket (past the table's end get_hash reads all ones).
__device__ __forceinline__ bool index_is_filtered_in(const IndexView& I, uint64_t pos, uint64_t key,
                                                     uint64_t bucket_end) {
    const uint64_t p2 = pos + I.filter_cutoff;
    if (p2 >= bucket_end) return p2 >= I.n && key == ~0ULL;
    return __ldg(&I.rs[p2].hash) == key;
}

// StrobemerIndex::get_count (step2/index.hpp:115-147): length of the equal-hash run
// starting at pos, within the bucket.
__device__ __forceinline__ uint32_t index_get_count(const IndexView& I, uint64_t pos) {
    const uint64_t key = __ldg(&I.rs[pos].hash);
    const uint64_t end = bucket_start(I, (key >> (64 - I.bits)) + 1);
    if (end - pos < 8) {
        uint32_t c = 1;
        for (uint64_t x = pos + 1; x < end && __ldg(&I.rs[x].hash) == key; ++x) ++c;
        return c;
    }
    // upper bound of key in [pos, end)
    uint64_t lo = pos, hi = end;
    while (lo < hi) {
        const uint64_t mid = lo + (hi - lo) / 2;
        if (__ldg(&I.rs[mid].hash) <= key) lo = mid + 1;
        else hi = mid;
    }
    return (uint32_t)(lo - pos);
}

// add_to_hits_per_ref (step2/nam.cu:45-62): walks the run of entries equal to the
// hash at pos and calls emit(ref_id, rs, re) for each entry whose length difference
// to the query is <= the running minimum.  Stops at the end of the table.
template <class Emit>
__device__ __forceinline__ uint32_t walk_hit_run(const IndexView& I, int qs, int qe, uint64_t pos, Emit&& emit,
                                                 uint32_t* run_len = nullptr, uint32_t most = 0xFFFFFFFFu) {
    int min_diff = 0x7FFFFFFF;
    const uint64_t key = get_hash(I, pos);
    const uint64_t p0 = pos;
    uint32_t n = 0;
    for (; pos < I.n && n < most; ++pos) {
        const gbsa_ref_randstrobe e = I.rs[pos];
        if (e.hash != key) break;
        const int rs = (int)e.position;
        const int re = rs + (int)(e.packed & 0xFF) + I.k;
        const int d = (qe - qs) - (re - rs);
        const int diff = d < 0 ? -d : d;
        if (diff <= min_diff) {
            emit(e.packed >> 8, rs, re);
            min_diff = diff;
            ++n;
        }
    }
    if (run_len) *run_len = (uint32_t)(pos - p0);
    return n;
}

}  // namespace gbsa
