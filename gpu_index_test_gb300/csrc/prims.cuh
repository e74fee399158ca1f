// prims.cuh — device-wide primitives: exclusive scan and a stable sort of
// 16-byte RefRandstrobe records.  Hand-written; no library sort or scan is used.
#pragma once

#include <cstddef>
#include <cstdint>
#include <vector>

#include "common.cuh"
#include "runtime.h"

namespace gbsa {

// Exclusive prefix sum of n u64 values (in may equal out).  If total is non-null it
// receives the sum (device pointer).  Uses ws for block partials.
void scan_exclusive_u64(const uint64_t* in, uint64_t* out, size_t n, uint64_t* d_total, Workspace& ws,
                        cudaStream_t st);

// Sorts n RefRandstrobe records by (hash, position), stably: records that tie on both
// keep their input order.  a and b are two device buffers of n records; returns the
// one holding the result.  No position exceeds max_position.
//
// A radix sort over all of the key's bytes is bound by its passes over memory (each reads
// the records twice and writes them once).  Hashes are spread evenly, so passes over their
// first two bytes (one below 40 k records, three above 10 M) leave groups of few records,
// which a warp finishes in shared memory (a block above 256).  Groups of more than 2048
// (the copies of repeats) are put side by side and sorted by all bytes among themselves.
// 4M records 1.30 -> 0.49 ms (12 passes before, with a look at each histogram on the host).
gbsa_ref_randstrobe* sort_ref_randstrobes(gbsa_ref_randstrobe* a, gbsa_ref_randstrobe* b, size_t n, uint32_t max_position,
                                          Workspace& ws, cudaStream_t st);
// Its passes over all records: a holds the result after an even number of them, b after an
// odd one (either when large groups are more than half of the records).
int sort_passes(size_t n);

}  // namespace gbsa
