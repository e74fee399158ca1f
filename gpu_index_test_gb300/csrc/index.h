// index.h — the device-resident StrobemerIndex behind the opaque gbsa_index handle.
//
// Layout in HBM (step2/index.hpp:180-182 kept as is, so export is a plain copy):
//   rs      RefRandstrobe[n], 16 B each, sorted by (hash, position, packed)
//   starts  u64[2^bits + 1]  bucket start table; starts[top bits of hash] .. starts[+1]
//           bounds the bucket, with the reference's first-bucket rule
//           (step2/index.cu:207-210: buckets up to the first hash's own start at the
//           second distinct hash)
//   buckets Bucket[2^bits + 1], the lookup's form of the table
#pragma once

#include <cstdint>

#include "common.cuh"
#include "runtime.h"

namespace gbsa {
struct Bucket;
}

struct gbsa_index {
    gbsa_params params{};
    gbsa::DevParams dp{};
    int bits = 0;
    uint32_t filter_cutoff = 0;
    uint64_t n = 0;
    gbsa_index_info info{};
    int device = 0;
    gbsa::ScratchLease lease;
    // One allocation: gbsa_ref_randstrobe[n], uint64_t[2^bits + 1], and when n < 2^32 and the
    // table is in order (`tagged`) Bucket[2^bits + 1], which the kernels read.  (Three of them
    // took 95 us more to load an index of 1 Mbp.)
    gbsa::DeviceBuffer tables;
    bool tagged = false;

    void resize_tables() {
        tagged = n < (1ull << 32);
        tables.resize(buckets_at() + (tagged ? 16 * n_starts() : 0));
    }
    uint64_t n_starts() const { return (1ull << bits) + 1; }
    uint64_t starts_at() const { return (16 * (n + 1) + 255) & ~255ull; }
    uint64_t buckets_at() const { return (starts_at() + 8 * n_starts() + 255) & ~255ull; }
    gbsa_ref_randstrobe* rs() const { return tables.as<gbsa_ref_randstrobe>(); }
    uint64_t* starts() const { return reinterpret_cast<uint64_t*>(tables.as<uint8_t>() + starts_at()); }
    gbsa::Bucket* buckets() const;   // null when not `tagged`
};

namespace gbsa {

// A bucket as the lookup reads it, in one 16-byte load: its start, its size (255: or more,
// see the next bucket's start), and a tag (8 bits of the hash, hash_tag) of each of its first
// kBucketTags entries.  Two thirds of a read's queries are not in the index (its other
// strand, and seeds with a sequencing error): the tags answer nearly all of those without
// the dependent fetch of an entry.  Buckets hold up to 5 entries on average (3.8 at 20 Mbp);
// with 4 tags a third of them had to be searched (551 of 2,150 warp instructions a read).
constexpr uint32_t kBucketTags = 11;
struct __align__(16) Bucket {
    uint32_t start;
    uint32_t w[3];   // the size in byte 0, entry i's tag in byte i + 1 (0 past the bucket's end)
};

}  // namespace gbsa

inline gbsa::Bucket* gbsa_index::buckets() const {
    return tagged ? reinterpret_cast<gbsa::Bucket*>(tables.as<uint8_t>() + buckets_at()) : nullptr;
}

namespace gbsa {

// Read-only view of the index used by device code.
struct IndexView {
    const gbsa_ref_randstrobe* rs;
    const uint64_t* starts;
    const Bucket* buckets;      // or null (2^32 entries or more, or a loaded table out of order)
    uint64_t n;
    int bits;
    uint32_t filter_cutoff;
    int k;
};

inline IndexView view_of(const gbsa_index& ix) {
    return IndexView{ix.rs(), ix.starts(), ix.buckets(), ix.n, ix.bits, ix.filter_cutoff, ix.params.k};
}

// Builds the lookup's bucket table of a loaded index, when every start fits 32 bits
// (n < 2^32) and the entries lie in their buckets in order.
void make_buckets(gbsa_index& ix, cudaStream_t st);

// Validates parameters like the reference constructors (step2/indexparameters.hpp:24-68).
bool params_valid(const gbsa_params& p);
int pick_bits_host(const gbsa_params& p, uint64_t total_length);

}  // namespace gbsa
