// extend.cu — seed extension of NAMs, the first step of the reference's alignment
// kernels (align_PE_part1..4, step2/main.cu:1876-2165): reverse_nam_if_needed
// (main.cu:759-793), then extend_seed_part (main.cu:582-643) with my_hamming_align
// (main.cu:506-580).
//
// Both are comparisons of a stretch of the read with a stretch of the contig, so the
// warp compares for its 32 NAMs in turn, 8 lanes a NAM and 8 bases a lane (aligned 32-bit
// loads), into a mismatch bit per base; a lane then reads its own NAM's bits.  The
// reference runs the best-segment scan only when the Hamming distance admits the ungapped
// path, which leaves a handful of mismatches: the scan steps over the runs between them.
// A thread per NAM walking bytes waited on its loads (0.70 ms for 1M NAMs of 150 bp reads
// against 0.23 here; 0.06 ms is what the bytes take).
#include "common.cuh"
#include "runtime.h"

namespace gbsa {
namespace {

// revcomp_table (step2/main.cu:1832-1849): A/C/G/T/U in either case to the upper-case
// complement, every other byte to 'N'.  c & 0xDF equals one of these letters only for
// that letter in either case.  (The reference indexes its table with a signed char, so
// bytes of 128 and above read outside it; here they give 'N'.)
__device__ __forceinline__ uint8_t revcomp_base(uint8_t c) {
    switch (c & 0xDF) {
        case 'A': return 'T';
        case 'C': return 'G';
        case 'G': return 'C';
        case 'T':
        case 'U': return 'A';
        default: return 'N';
    }
}

// The read in one orientation: the reverse complement is read backwards through the
// table, as the reference's rc copy (main.cu:1893-1900).
struct ReadView {
    const uint8_t* fwd;
    int L;
    bool rc;
    __device__ __forceinline__ uint8_t at(int j) const {
        return rc ? revcomp_base(__ldg(fwd + (L - 1 - j))) : __ldg(fwd + j);
    }
};

// No early exit, so that the k loads are independent and in flight together.
__device__ __forceinline__ bool kmer_equal(const uint8_t* ref, const ReadView& q, int qpos, int k) {
    bool eq = true;
#pragma unroll 8
    for (int t = 0; t < k; ++t) eq &= __ldg(ref + t) == q.at(qpos + t);
    return eq;
}

// 2-bit codes of 4 bases (A, C, G, T in either case: 0..3), a byte each, and whether all
// four are such letters.
__device__ __forceinline__ uint32_t codes4(uint32_t w, uint32_t& sel, bool& acgt) {
    const uint32_t c4 = ((w >> 1) ^ (w >> 2)) & 0x03030303u;
    const uint32_t t = (c4 | (c4 >> 4)) & 0x00FF00FFu;
    sel = (t | (t >> 8)) & 0xFFFFu;   // the codes as byte-permute selectors
    acgt = ((w & 0xDFDFDFDFu) == __byte_perm(0x54474341u, 0u, sel));
    return c4;
}

// The complements of 4 bases (revcomp_base of each byte).
__device__ __forceinline__ uint32_t complement4(uint32_t w) {
    uint32_t sel;
    bool acgt;
    codes4(w, sel, acgt);
    if (acgt) return __byte_perm(0x41434754u, 0u, sel);   // A, C, G, T: T, G, C, A
    uint32_t r = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) r |= (uint32_t)revcomp_base((uint8_t)(w >> (8 * u))) << (8 * u);
    return r;
}

// 8 bytes from p on, as two words in memory order; only aligned words that hold a byte of
// the sequence are read (the others' bytes are 0): `off` bytes of it lie before p (negative:
// it starts behind p), `rem` bytes from p on.
__device__ __forceinline__ uint2 load8(const uint8_t* p, int off, int rem) {
    const int mis = (int)(reinterpret_cast<uintptr_t>(p) & 3);
    const uint32_t* w = reinterpret_cast<const uint32_t*>(p - mis);
    const uint32_t w0 = off + 4 - mis > 0 ? __ldg(w) : 0u;
    const uint32_t w1 = off + 8 - mis > 0 && 4 - mis < rem ? __ldg(w + 1) : 0u;
    const uint32_t w2 = mis != 0 && 8 - mis < rem ? __ldg(w + 2) : 0u;
    return make_uint2(__funnelshift_r(w0, w1, 8 * mis), __funnelshift_r(w1, w2, 8 * mis));
}

constexpr int kExtendWarps = 4;
constexpr int kMaskBases = 512;                  // longest comparison of the warp
constexpr int kMaskWords = kMaskBases / 32 + 1;  // (odd: the lanes' words lie in different banks)
constexpr int kMaxKmer = 32;                     // longest k-mer of the warp's checks

// What a lane has the warp compare: n bases of the contig with the read's in the orientation
// rc, from (ref, q) on; and for the k-mer checks a second pair of the same length.
struct Compare {
    const uint8_t* ref;
    const uint8_t* fwd;   // the read as given, L bases
    int L, n;
    int q, q2, ref2;      // ref2: the second stretch's place after ref
    uint32_t rc;
};

struct ExtendShared {
    Compare task[32];
    uint32_t mask[32][kMaskWords];   // mismatch bits of each lane's comparison
    uint8_t list[32];
};

// Mismatch bits of the n (1 to 8 counted, more allowed) bases from ref + j and q + j on.
__device__ __forceinline__ uint32_t compare8(const Compare& t, const uint8_t* ref, int q, int j) {
    const int n = t.n - j;
    const uint2 r = load8(ref + j, 0, n);
    // the read's bases q + j on, or L - 1 - q - j downwards and complemented
    const int at = t.rc ? t.L - 8 - q - j : q + j;
    uint2 x = load8(t.fwd + at, at, t.L - at);
    if (t.rc)
        x = make_uint2(complement4(__byte_perm(x.y, 0u, 0x0123)), complement4(__byte_perm(x.x, 0u, 0x0123)));
    // a one in each differing byte, then side by side
    const uint32_t d0 = __vcmpne4(r.x, x.x) & 0x01010101u, d1 = __vcmpne4(r.y, x.y) & 0x01010101u;
    const uint32_t bits = ((d0 * 0x01020408u) >> 24) | (((d1 * 0x01020408u) >> 24) << 4);
    return n < 8 ? bits & ((1u << n) - 1) : bits;
}

// Runs the comparisons of the lanes with `want` (n <= kMaskBases): afterwards bit j of
// S.mask[lane] says that base j differs (bits from n on are 0); kKmers: both stretches
// (n <= kMaxKmer), the first's bits in word 0 and the second's in word 1.
template <bool kKmers>
__device__ __noinline__ void warp_compare(ExtendShared& S, bool want, const Compare& c) {
    const uint32_t lane = lane_id();
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, want);
    if (want) {
        S.task[lane] = c;
        S.list[__popc(m & lanemask_lt())] = (uint8_t)lane;
    }
    __syncwarp();
    const uint32_t cnt = __popc(m), sub = lane & 7u;
    for (uint32_t g = lane >> 3; g < cnt; g += 4) {   // (no warp operation inside: groups run apart)
        const uint32_t owner = S.list[g];
        const Compare t = S.task[owner];
        uint8_t* out = reinterpret_cast<uint8_t*>(S.mask[owner]);
        if (kKmers) {
            const int j = 8 * (int)(sub & 3u);
            const bool second = sub >= 4;
            out[sub] = j < t.n ? (uint8_t)compare8(t, second ? t.ref + t.ref2 : t.ref, second ? t.q2 : t.q, j) : 0;
        } else {
            for (int j = 8 * (int)sub; j < ((t.n + 31) & ~31); j += 64)
                out[j >> 3] = j < t.n ? (uint8_t)compare8(t, t.ref, t.q, j) : 0;
        }
    }
    __syncwarp();
}

// Whether bits [from, from + n) of a lane's mask are all 0.
__device__ __forceinline__ bool mask_clear(const uint32_t* m, int from, int n) {
    bool clear = true;
    for (int w = from >> 5; w <= (from + n - 1) >> 5; ++w) {
        uint32_t x = m[w];
        if (w == from >> 5) x &= 0xFFFFFFFFu << (from & 31);
        const int end = from + n - 32 * w;
        if (end < 32) x &= (1u << end) - 1;
        clear = clear && x == 0;
    }
    return clear;
}

// my_hamming_align (main.cu:506-580): its scan's state, fed base by base or run by run.
struct SegmentScan {
    gbsa_align_params ap;
    int start = 0, score, best_start = 0, best_end = 0, best_score = 0;
    // mismatches so far, at the current segment's start and at the best segment's ends
    int mm = 0, cm_start = 0, best_cm_start = 0, best_cm_end = 0;
    __device__ explicit SegmentScan(const gbsa_align_params& p) : ap(p), score(p.end_bonus) {}
    __device__ __forceinline__ void best_at(int end) {
        if (score > best_score) {
            best_start = start;
            best_score = score;
            best_end = end;
            best_cm_start = cm_start;
            best_cm_end = mm;
        }
    }
    __device__ __forceinline__ void step(int j, bool differs) {
        mm += differs ? 1 : 0;
        score += differs ? -ap.mismatch : ap.match;
        if (score < 0) {
            start = j + 1;
            score = 0;
            cm_start = mm;
        }
        best_at(j + 1);
    }
    // n > 0 matches from base j on, with match > 0 and score >= 0: the score only grows, so
    // the best segment's end is the run's
    __device__ __forceinline__ void run(int j, int n) {
        score += n * ap.match;
        best_at(j + n);
    }
    __device__ __forceinline__ void finish(int L) {
        if (score + ap.end_bonus > best_score) {
            best_score = score + ap.end_bonus;
            best_end = L;
            best_start = start;
            best_cm_start = cm_start;
            best_cm_end = mm;
        }
    }
    __device__ __forceinline__ void record(gbsa_seed_alignment& o, int pstart, int L) const {
        o.done = 1;
        o.edit_distance = best_cm_end - best_cm_start;
        o.global_ed = o.edit_distance + best_start + (L - best_end);
        o.score = best_score;
        o.ref_start = pstart + best_start;
        o.length = best_end - best_start;
    }
};

// extend_seed_part's test of the Hamming distance (an int limit, a float ratio compared in
// double); the reference's count stops once it exceeds the limit.
__device__ __forceinline__ bool hamming_admits(int mismatches, int L) {
    const int hamming_dist = min(mismatches, (int)(L * 0.05) + 1);
    return hamming_dist >= 0 && ((float)hamming_dist / L) < 0.05;
}

// The whole step for one NAM by one thread, base by base: reads longer than kMaskBases, k
// above kMaxKmer.
__device__ __noinline__ void extend_long(gbsa_nam nam, const uint8_t* fwd, const uint8_t* ref, int L, int rlen, int k,
                                         const gbsa_align_params& ap, gbsa_seed_alignment& o) {
    bool consistent = kmer_equal(ref + nam.ref_start, ReadView{fwd, L, nam.is_rc != 0}, nam.query_start, k) &&
                      kmer_equal(ref + nam.ref_end - k, ReadView{fwd, L, nam.is_rc != 0}, nam.query_end - k, k);
    if (!consistent) {
        const int qs2 = L - nam.query_end, qe2 = L - nam.query_start;
        const ReadView other{fwd, L, nam.is_rc == 0};
        if (kmer_equal(ref + nam.ref_start, other, qs2, k) && kmer_equal(ref + nam.ref_end - k, other, qe2 - k, k)) {
            nam.is_rc = nam.is_rc ? 0 : 1;
            nam.query_start = qs2;
            nam.query_end = qe2;
            consistent = true;
        }
    }
    o.query_start = nam.query_start;
    o.query_end = nam.query_end;
    o.is_rc = nam.is_rc;
    o.consistent = consistent ? 1 : 0;
    const int pstart = max(0, nam.ref_start - nam.query_start);
    const int pend = min(nam.ref_end + L - nam.query_end, rlen);
    if (pend - pstart != L || !consistent) return;
    const ReadView q{fwd, L, nam.is_rc != 0};
    SegmentScan scan(ap);
    for (int j = 0; j < L; ++j) scan.step(j, q.at(j) != __ldg(ref + pstart + j));
    scan.finish(L);
    if (hamming_admits(scan.mm, L)) scan.record(o, pstart, L);
}

__global__ void __launch_bounds__(32 * kExtendWarps)
    k_extend_seeds(const uint8_t* __restrict__ ref_seqs, const uint64_t* __restrict__ ref_offs,
                   const uint64_t* __restrict__ ref_lens, uint32_t n_refs, const uint8_t* __restrict__ read_seqs,
                   const uint64_t* __restrict__ read_offs, const uint32_t* __restrict__ read_lens, uint32_t n_reads,
                   const gbsa_nam* __restrict__ nams, const uint32_t* __restrict__ nam_reads, uint64_t n, int k,
                   gbsa_align_params ap, gbsa_seed_alignment* __restrict__ out, unsigned int* bad) {
    __shared__ ExtendShared s_ext[kExtendWarps];
    ExtendShared& S = s_ext[threadIdx.x >> 5];
    const uint32_t lane = lane_id();
    uint32_t* mask = S.mask[lane];
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t first = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x - lane;
    for (uint64_t i0 = first; i0 < n; i0 += stride) {   // the warp's 32 NAMs
        const uint64_t i = i0 + lane;
        const bool valid = i < n;
        gbsa_nam nam = nams[valid ? i : n - 1];
        gbsa_seed_alignment o;
        o.ref_id = o.ref_start = o.edit_distance = o.global_ed = o.score = o.length = 0;
        o.query_start = o.query_end = 0;
        o.is_rc = o.done = o.consistent = o._pad = 0;
        const uint32_t r = nam_reads[valid ? i : n - 1];
        bool ok = valid && r < n_reads && nam.ref_id >= 0 && (uint32_t)nam.ref_id < n_refs;
        int L = 0, rlen = 0;
        if (ok) {
            L = (int)read_lens[r];
            rlen = (int)ref_lens[nam.ref_id];
            // every k-mer the checks compare then lies inside its sequence
            ok = nam.query_start >= 0 && nam.query_end <= L && nam.query_end - nam.query_start >= k &&
                 nam.ref_start >= 0 && nam.ref_end <= rlen && nam.ref_end - nam.ref_start >= k;
        }
        if (valid && !ok) atomicAdd(bad, 1u);
        const uint8_t* fwd = ok ? read_seqs + read_offs[r] : nullptr;
        const uint8_t* ref = ok ? ref_seqs + ref_offs[nam.ref_id] : nullptr;
        if (ok) o.ref_id = nam.ref_id;
        if (ok && (L > kMaskBases || k > kMaxKmer)) {
            gbsa_seed_alignment x = o;   // (o itself stays in registers)
            extend_long(nam, fwd, ref, L, rlen, k, ap, x);
            o = x;
            ok = false;
        }
        // reverse_nam_if_needed (step2/main.cu:759-793).  When the NAM's k-mers lie on the
        // diagonal of its projected window, the window's comparison answers them too.
        auto window = [&](int& pstart) {
            pstart = max(0, nam.ref_start - nam.query_start);
            return min(nam.ref_end + L - nam.query_end, rlen) - pstart == L;
        };
        int pstart = 0;
        const bool diag = ok && nam.ref_start >= nam.query_start &&
                          nam.ref_end - nam.ref_start == nam.query_end - nam.query_start && window(pstart);
        Compare c;
        c.fwd = fwd;
        c.L = L;
        bool consistent = false, compared = false;   // compared: the mask is the window's, in the NAM's orientation
        for (int pass = 0; pass < 2; ++pass) {
            // extend_seed_part's window (step2/main.cu:582-643); in the second pass of the
            // NAMs whose k-mers were checked apart
            const bool want = pass == 0 ? diag : ok && consistent && !compared && window(pstart);
            c.ref = ref + pstart;
            c.q = 0;
            c.n = L;
            c.rc = nam.is_rc != 0;
            warp_compare<false>(S, want, c);
            if (pass == 0 && diag)
                consistent = mask_clear(mask, nam.query_start, k) && mask_clear(mask, nam.query_end - k, k);
            compared = compared || (want && consistent);
            if (pass == 1 || !__any_sync(0xFFFFFFFFu, ok && !consistent)) break;
            // off the diagonal: the k-mers themselves; then the other orientation
            const int qs2 = L - nam.query_end, qe2 = L - nam.query_start;
            c.ref = ref + nam.ref_start;
            c.ref2 = nam.ref_end - k - nam.ref_start;
            c.n = k;
            for (int flip = 0; flip < 2; ++flip) {
                const bool check = ok && !consistent && (flip || !diag);
                c.rc = (nam.is_rc != 0) != (flip != 0);
                c.q = flip ? qs2 : nam.query_start;
                c.q2 = (flip ? qe2 : nam.query_end) - k;
                warp_compare<true>(S, check, c);
                if (check && mask[0] == 0 && mask[1] == 0) {
                    consistent = true;
                    if (flip) {
                        nam.is_rc = nam.is_rc ? 0 : 1;
                        nam.query_start = qs2;
                        nam.query_end = qe2;
                    }
                }
            }
        }
        if (ok) {
            o.query_start = nam.query_start;
            o.query_end = nam.query_end;
            o.is_rc = nam.is_rc;
            o.consistent = consistent ? 1 : 0;
            if (compared) {
                int mm = 0;
                for (int w = 0; 32 * w < L; ++w) mm += __popc(mask[w]);
                if (hamming_admits(mm, L)) {
                    SegmentScan scan(ap);
                    if (ap.match > 0 && ap.end_bonus >= 0) {
                        int j = 0;
                        for (int w = 0; 32 * w < L; ++w)
                            for (uint32_t x = mask[w]; x; x &= x - 1) {
                                const int at = 32 * w + __ffs(x) - 1;
                                if (at > j) scan.run(j, at - j);
                                scan.step(at, true);
                                j = at + 1;
                            }
                        if (j < L) scan.run(j, L - j);
                    } else {
                        for (int j = 0; j < L; ++j) scan.step(j, (mask[j >> 5] >> (j & 31)) & 1u);
                    }
                    scan.finish(L);
                    scan.record(o, pstart, L);
                }
            }
        }
        if (valid) out[i] = o;
        __syncwarp();   // the masks are rewritten
    }
}

// ---- mate rescue (rescue_mate_part with has_shared_substring) --------------------------
constexpr int kMaxMateSubstrings = 64;   // sampled substrings of a mate (the reference keeps 50)
constexpr int kRescueWarps = 8;
// Longest mate with that many substrings: k = 32 takes substrings of 21 bases, 10 apart.
constexpr int kMateWords = (21 + 10 * kMaxMateSubstrings) / 16 + 4;

// nt2int_mod8 (step2/main.cu:645-654) of 4 bases: the codes 0, 0, 0, 1, 3, 0, 0, 2 by byte
// value mod 8, a byte each.
__device__ __forceinline__ uint32_t codes4_mod8(uint32_t w) {
    const uint32_t x = w & 0x07070707u;
    const uint32_t t = (x | (x >> 4)) & 0x00FF00FFu;
    return __byte_perm(0x01000000u, 0x02000003u, (t | (t >> 8)) & 0xFFFFu);
}

// nt2int_mod8 of the complements of 4 bases, a byte each.
__device__ __forceinline__ uint32_t codes4_complement(uint32_t w) {
    uint32_t sel;
    bool acgt;
    const uint32_t c = codes4(w, sel, acgt);
    return acgt ? 0x03030303u - c : codes4_mod8(complement4(w));
}

// Four codes (a byte each, the first base lowest) packed into 8 bits, the first base highest.
__device__ __forceinline__ uint32_t pack4(uint32_t c) { return (c * 0x40100401u) >> 24; }

// A warp per NAM: the window where the mate lies (float arithmetic as the reference's:
// the int offset converted to float, mu + 5 sigma as one fused multiply-add, truncation
// back to int), then has_shared_substring (step2/main.cu:657-693): whether any of the
// mate's 2k/3-base substrings at multiples of k/3 equals a substring of the window.  Both
// position sets stop one substring short of the end, as the reference's loops.
//
// The bases are packed 2 bits each four at a time; a lane then holds the 32 bases from its
// own 4 window positions on (three exchanges with its neighbours) and cuts each position's
// substring out with a shift.  The mate's substrings sit in the lanes' registers, and a
// 1024-bit filter over them, a word a lane, passes the few positions that are compared
// with all of them.  Any match answers the question, so the window's 128-position blocks
// are taken from where the insert size puts the mate outwards: most mates are found in the
// first.  Scanned from the window's start, with 13 byte loads and 23 compares a position,
// 1M NAMs of 150 bp pairs took 4.16 ms against 0.68 here (bound by integer issue).
__global__ void __launch_bounds__(32 * kRescueWarps)
    k_rescue_mates(const uint8_t* __restrict__ ref_seqs, const uint64_t* __restrict__ ref_offs,
                   const uint64_t* __restrict__ ref_lens, uint32_t n_refs, const uint8_t* __restrict__ read_seqs,
                   const uint64_t* __restrict__ read_offs, const uint32_t* __restrict__ read_lens, uint32_t n_reads,
                   const gbsa_nam* __restrict__ nams, const uint32_t* __restrict__ mate_reads, uint64_t n, int k,
                   float mu, float sigma, gbsa_mate_rescue* __restrict__ out, unsigned int* bad) {
    __shared__ uint32_t s_mate[kRescueWarps][kMateWords];   // the mate, 16 bases a word, the first highest
    __shared__ uint32_t s_filter[kRescueWarps][32];
    constexpr uint32_t kFull = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    uint32_t* mate = s_mate[w];
    const int sub = 2 * k / 3, step = k / 3;
    const uint32_t hmask = sub >= 16 ? kFull : (1u << (2 * sub)) - 1;   // a longer substring keeps its last 16 bases
    const float spread = __fmaf_rn(5.0f, sigma, mu);
    const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    // filter word and two bits of a substring
    auto filter_word = [](uint32_t h) { return (h * 0x9E3779B1u) >> 27; };
    auto filter_bits = [](uint32_t h) {
        const uint32_t z = h * 0x9E3779B1u;
        return (1u << ((z >> 22) & 31u)) | (1u << ((z >> 17) & 31u));
    };
    for (uint64_t i = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
        const gbsa_nam nam = nams[i];
        const uint32_t r = mate_reads[i];
        gbsa_mate_rescue o;
        o.ref_id = o.window_start = o.window_end = o.edit_distance = 0;
        o.is_rc = o.done = o.is_unaligned = o._pad = 0;
        bool ok = r < n_reads && nam.ref_id >= 0 && (uint32_t)nam.ref_id < n_refs;
        const int L = ok ? (int)read_lens[r] : 0;
        const int n_sub = L > sub ? (L - sub + step - 1) / step : 0;   // p = 0, step, ... with p + sub < L
        if (n_sub > kMaxMateSubstrings) ok = false;
        if (!ok) {
            if (lane == 0) {
                atomicAdd(bad, 1u);
                out[i] = o;
            }
            continue;
        }
        const uint8_t* fwd = read_seqs + read_offs[r];
        // rescue_mate_part (step2/main.cu:695-757)
        const bool mate_fwd = nam.is_rc != 0;   // the mate in the orientation opposite to the NAM
        int a, b;
        if (mate_fwd) {
            a = __float2int_rz(__fsub_rn(__int2float_rn(nam.ref_start - nam.query_start), spread));
            b = nam.ref_start - nam.query_start + L / 2;
        } else {
            a = nam.ref_end + (L - nam.query_end) - L / 2;
            b = __float2int_rz(__fadd_rn(__int2float_rn(nam.ref_end + (L - nam.query_end)), spread));
        }
        const int ref_len = (int)ref_lens[nam.ref_id];
        const int ws = max(0, min(a, ref_len));
        const int we = min(ref_len, max(0, b));
        bool shared = false;
        if (we >= ws + k && n_sub > 0) {
            // the mate's codes (of its complement when it is taken reversed)
            s_filter[w][lane] = 0;
            for (int p = 4 * (int)lane; p < L; p += 128) {
                const uintptr_t at = reinterpret_cast<uintptr_t>(fwd + p);
                const uint32_t* src = reinterpret_cast<const uint32_t*>(at & ~uintptr_t(3));
                const uint32_t mis = (uint32_t)(at & 3);
                const uint32_t hi = mis != 0 && 4 - (int)mis < L - p ? __ldg(src + 1) : 0u;
                const uint32_t x = __funnelshift_r(__ldg(src), hi, 8 * mis);
                // byte p / 4 of the words' stream
                reinterpret_cast<uint8_t*>(mate)[(p >> 2) ^ 3] =
                    (uint8_t)pack4(mate_fwd ? codes4_mod8(x) : codes4_complement(x));
            }
            __syncwarp();
            // substrings lane and lane + 32
            uint32_t e[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int t = (int)lane + 32 * u;
                e[u] = 0;
                if (t >= n_sub) continue;
                const int q = mate_fwd ? t * step : L - t * step - sub;   // where it starts in the read as given
                const uint32_t sh = 2 * (q & 15);
                const uint32_t w0 = mate[q >> 4], w1 = mate[(q >> 4) + 1], w2 = mate[(q >> 4) + 2];
                uint64_t h = ((uint64_t)__funnelshift_l(w1, w0, sh) << 32) | __funnelshift_l(w2, w1, sh);
                h >>= 64 - 2 * sub;
                if (!mate_fwd) h = revcomp_bits(~h, sub);   // (complemented already: only reversed)
                e[u] = (uint32_t)h & hmask;
                atomicOr(&s_filter[w][filter_word(e[u])], filter_bits(e[u]));
            }
            __syncwarp();
            const uint32_t filter = s_filter[w][lane];
            const uint8_t* win = ref_seqs + ref_offs[nam.ref_id] + ws;
            const int len = we - ws, n_pos = len - sub;   // positions p with p + sub < window length
            const int mis = (int)(reinterpret_cast<uintptr_t>(win) & 3);
            const int n_blk = n_pos > 0 ? (n_pos + mis + 127) / 128 : 0;   // block c: positions 128 c - mis on
            // the block in the middle of where the mate is expected (it starts mu - L before
            // the NAM's read ends, or ends mu after it starts)
            const float start = mate_fwd ? (float)(nam.ref_start - nam.query_start + L - ws) - mu
                                         : (float)(nam.ref_end - nam.query_end - L - ws) + mu;
            const int mid = (int)fminf(fmaxf(start + 0.5f * (float)L, 0.0f), (float)max(n_pos - 1, 0));
            const int c0 = n_blk ? (mid + mis) / 128 : 0;
            for (int t = 0; t < 2 * n_blk && !shared; ++t) {   // c0, c0 + 1, c0 - 1, c0 + 2, ...
                const int c = c0 + ((t & 1) ? (t + 1) / 2 : -(t / 2));
                if (c < 0 || c >= n_blk) continue;
                const int p0 = 128 * c - mis + 4 * (int)lane;   // the lane's first position (a word boundary)
                const uint32_t x = p0 + 4 > 0 && p0 < len ? __ldg(reinterpret_cast<const uint32_t*>(win + p0)) : 0u;
                const uint32_t y = lane < 8 && p0 + 132 > 0 && p0 + 128 < len
                                       ? __ldg(reinterpret_cast<const uint32_t*>(win + p0 + 128))
                                       : 0u;
                // cur: the lane's bases, nxt: the first lanes' of the block after; 4, 8, 16, 32 bases
                const uint32_t cur4 = pack4(codes4_mod8(x)), nxt4 = pack4(codes4_mod8(y));
                const uint32_t cur8 = (cur4 << 8) | __shfl_sync(kFull, lane < 1 ? nxt4 : cur4, (lane + 1) & 31);
                const uint32_t nxt8 = (nxt4 << 8) | __shfl_down_sync(kFull, nxt4, 1);
                const uint32_t cur16 = (cur8 << 16) | __shfl_sync(kFull, lane < 2 ? nxt8 : cur8, (lane + 2) & 31);
                const uint32_t nxt16 = (nxt8 << 16) | __shfl_down_sync(kFull, nxt8, 2);
                const uint32_t low16 = __shfl_sync(kFull, lane < 4 ? nxt16 : cur16, (lane + 4) & 31);
                const uint64_t bases = ((uint64_t)cur16 << 32) | low16;
                uint32_t h[4];
                uint32_t pass = 0;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    h[u] = (uint32_t)(bases >> (64 - 2 * (u + sub))) & hmask;
                    const uint32_t bits = filter_bits(h[u]);
                    const uint32_t word = __shfl_sync(kFull, filter, filter_word(h[u]));
                    const bool in = p0 + u >= 0 && p0 + u < n_pos;
                    pass |= in && (word & bits) == bits ? 1u << u : 0u;
                }
                if (!__any_sync(kFull, pass != 0)) continue;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    uint32_t m = __ballot_sync(kFull, (pass >> u) & 1u);
                    while (m && !shared) {
                        const uint32_t x1 = __shfl_sync(kFull, h[u], __ffs(m) - 1);
                        m &= m - 1;
                        shared = __any_sync(kFull, ((int)lane < n_sub && e[0] == x1) ||
                                                       ((int)lane + 32 < n_sub && e[1] == x1));
                    }
                }
            }
            __syncwarp();   // the next NAM rewrites the mate and the filter
        }
        if (lane == 0) {
            o.ref_id = nam.ref_id;
            o.window_start = ws;
            o.window_end = we;
            o.is_rc = nam.is_rc;
            if (!shared) {
                o.done = 1;
                o.is_unaligned = 1;
                o.edit_distance = L;
            }
            out[i] = o;
        }
    }
}

}  // namespace
}  // namespace gbsa

using namespace gbsa;

extern "C" int gbsa_extend_seeds_device(const uint8_t* d_ref_seqs, const uint64_t* d_ref_offsets,
                                        const uint64_t* d_ref_lengths, uint32_t n_refs, const uint8_t* d_read_seqs,
                                        const uint64_t* d_read_offsets, const uint32_t* d_read_lengths,
                                        uint32_t n_reads, const gbsa_nam* d_nams, const uint32_t* d_nam_reads,
                                        uint64_t n_nams, int k, const gbsa_align_params* params,
                                        gbsa_seed_alignment* d_out, void* stream) {
    try {
        if (!params) throw Error(GBSA_ERR_PARAM, "params must not be null");
        if (k < 1) throw Error(GBSA_ERR_PARAM, "k must be at least 1");
        if (n_nams == 0) return GBSA_OK;
        cudaStream_t st = (cudaStream_t)stream;
        // the status word is allocated in stream order: a cudaFree would wait for the
        // whole device
        unsigned int* bad = static_cast<unsigned int*>(scratch_alloc(sizeof(unsigned int), st));
        unsigned int h_bad = 0;
        const cudaError_t e = [&] {
            // one wave of resident blocks (the loop strides over the NAMs)
            int per_sm = 0;
            cudaError_t r =
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_extend_seeds, 32 * kExtendWarps, 0);
            if (r != cudaSuccess) return r;
            const unsigned max_blocks = (unsigned)device_sm_count() * (unsigned)(per_sm > 0 ? per_sm : 1);
            r = cudaMemsetAsync(bad, 0, sizeof(unsigned int), st);
            if (r != cudaSuccess) return r;
            k_extend_seeds<<<grid_for(n_nams, 32 * kExtendWarps, max_blocks), 32 * kExtendWarps, 0, st>>>(
                d_ref_seqs, d_ref_offsets, d_ref_lengths, n_refs, d_read_seqs, d_read_offsets, d_read_lengths,
                n_reads, d_nams, d_nam_reads, n_nams, k, *params, d_out, bad);
            g_launches.fetch_add(1, std::memory_order_relaxed);   // counted as GBSA_LAUNCHED, without a throw
            r = cudaGetLastError();
            if (r != cudaSuccess) return r;
            return cudaMemcpyAsync(&h_bad, bad, sizeof h_bad, cudaMemcpyDeviceToHost, st);
        }();
        scratch_free(bad, st);
        GBSA_CUDA(e);
        GBSA_CUDA(cudaStreamSynchronize(st));
        if (h_bad)
            throw Error(GBSA_ERR_PARAM, std::to_string(h_bad) +
                                            " NAM(s) name a read or contig out of range or leave their read or contig");
        return GBSA_OK;
    } catch (const Error& e) {
        set_last_error(e.what());
        return e.code;
    } catch (const std::exception& e) {
        set_last_error(e.what());
        return GBSA_ERR_CUDA;
    }
}

extern "C" int gbsa_rescue_mates_device(const uint8_t* d_ref_seqs, const uint64_t* d_ref_offsets,
                                        const uint64_t* d_ref_lengths, uint32_t n_refs, const uint8_t* d_read_seqs,
                                        const uint64_t* d_read_offsets, const uint32_t* d_read_lengths,
                                        uint32_t n_reads, const gbsa_nam* d_nams, const uint32_t* d_mate_reads,
                                        uint64_t n_nams, int k, float mu, float sigma, gbsa_mate_rescue* d_out,
                                        void* stream) {
    try {
        if (k < 3 || k > 32) throw Error(GBSA_ERR_PARAM, "k must be in [3, 32]");
        if (n_nams == 0) return GBSA_OK;
        cudaStream_t st = (cudaStream_t)stream;
        unsigned int* bad = static_cast<unsigned int*>(scratch_alloc(sizeof(unsigned int), st));
        unsigned int h_bad = 0;
        const cudaError_t e = [&] {
            int per_sm = 0;
            cudaError_t r =
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_rescue_mates, 32 * kRescueWarps, 0);
            if (r != cudaSuccess) return r;
            const uint64_t want = (n_nams + kRescueWarps - 1) / kRescueWarps;   // a warp per NAM
            const unsigned blocks = (unsigned)std::min<uint64_t>(
                want, (uint64_t)device_sm_count() * (uint64_t)(per_sm > 0 ? per_sm : 1));
            r = cudaMemsetAsync(bad, 0, sizeof(unsigned int), st);
            if (r != cudaSuccess) return r;
            k_rescue_mates<<<blocks, 32 * kRescueWarps, 0, st>>>(
                d_ref_seqs, d_ref_offsets, d_ref_lengths, n_refs, d_read_seqs, d_read_offsets, d_read_lengths,
                n_reads, d_nams, d_mate_reads, n_nams, k, mu, sigma, d_out, bad);
            g_launches.fetch_add(1, std::memory_order_relaxed);   // counted as GBSA_LAUNCHED, without a throw
            r = cudaGetLastError();
            if (r != cudaSuccess) return r;
            return cudaMemcpyAsync(&h_bad, bad, sizeof h_bad, cudaMemcpyDeviceToHost, st);
        }();
        scratch_free(bad, st);
        GBSA_CUDA(e);
        GBSA_CUDA(cudaStreamSynchronize(st));
        if (h_bad)
            throw Error(GBSA_ERR_PARAM, std::to_string(h_bad) +
                                            " NAM(s) name a contig or mate out of range or a mate with more than 64 "
                                            "sampled substrings");
        return GBSA_OK;
    } catch (const Error& e) {
        set_last_error(e.what());
        return e.code;
    } catch (const std::exception& e) {
        set_last_error(e.what());
        return GBSA_ERR_CUDA;
    }
}

// ---- the steps of the alignment orchestration ------------------------------------------
//
// Runs the step lists of gbsa_plan_pairs_device: every step's NAM goes through the seed
// extension kernel on its own read (an extension step keeps the record; a rescue step
// keeps only reverse_nam_if_needed's answer — orientation, query interval, consistency —
// since the reference runs only that check before rescue_mate_part), then the rescue
// steps' NAMs, in the orientation that check left them, through the mate rescue kernel.

namespace gbsa {
namespace {

__global__ void k_gather_step_nams(const gbsa_nam* __restrict__ nams, const uint64_t* __restrict__ offs,
                                   const gbsa_align_step* __restrict__ steps, uint64_t n, gbsa_nam* __restrict__ out,
                                   uint32_t* __restrict__ out_reads) {
    for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < n; s += (uint64_t)gridDim.x * blockDim.x) {
        const gbsa_align_step st = steps[s];
        out[s] = nams[offs[st.nam_read] + st.nam];
        out_reads[s] = st.nam_read;
    }
}

__global__ void k_rescue_list(const gbsa_align_step* __restrict__ steps, uint64_t n, const gbsa_nam* __restrict__ step_nams,
                              gbsa_seed_alignment* __restrict__ ext, gbsa_nam* __restrict__ rnams,
                              uint32_t* __restrict__ rmates, uint64_t* __restrict__ ridx, unsigned long long* count,
                              gbsa_mate_rescue* __restrict__ resc) {
    for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < n; s += (uint64_t)gridDim.x * blockDim.x) {
        gbsa_mate_rescue none;
        none.ref_id = none.window_start = none.window_end = none.edit_distance = 0;
        none.is_rc = none.done = none.is_unaligned = none._pad = 0;
        resc[s] = none;
        const gbsa_align_step st = steps[s];
        if (st.kind != GBSA_STEP_RESCUE) continue;
        gbsa_seed_alignment e = ext[s];
        gbsa_nam nm = step_nams[s];
        nm.is_rc = e.is_rc;
        nm.query_start = e.query_start;
        nm.query_end = e.query_end;
        // the reference only checks the orientation before the rescue: no alignment record
        e.ref_start = e.edit_distance = e.global_ed = e.score = e.length = 0;
        e.done = 0;
        ext[s] = e;
        const unsigned long long j = atomicAdd(count, 1ull);
        rnams[j] = nm;
        rmates[j] = st.read;
        ridx[j] = s;
    }
}

__global__ void k_scatter_rescues(const gbsa_mate_rescue* __restrict__ in, const uint64_t* __restrict__ idx, uint64_t n,
                                  gbsa_mate_rescue* __restrict__ out) {
    for (uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; j < n; j += (uint64_t)gridDim.x * blockDim.x)
        out[idx[j]] = in[j];
}

}  // namespace
}  // namespace gbsa

extern "C" int gbsa_run_align_steps_device(const uint8_t* d_ref_seqs, const uint64_t* d_ref_offsets,
                                           const uint64_t* d_ref_lengths, uint32_t n_refs, const uint8_t* d_read_seqs,
                                           const uint64_t* d_read_offsets, const uint32_t* d_read_lengths,
                                           uint32_t n_reads, const gbsa_nam* d_nams, const uint64_t* d_nam_offsets,
                                           const gbsa_align_step* d_steps, uint64_t n_steps, int k,
                                           const gbsa_align_params* params, float mu, float sigma,
                                           gbsa_seed_alignment* d_ext, gbsa_mate_rescue* d_resc, void* stream) {
    try {
        if (n_steps == 0) return GBSA_OK;
        cudaStream_t st = (cudaStream_t)stream;
        // scratch in stream order: the steps' NAMs and reads, the rescue list (NAMs, mates,
        // step indices), its count and the rescue records
        const size_t b_nams = (sizeof(gbsa_nam) * n_steps + 255) & ~size_t(255);
        const size_t b_u32 = (4ull * n_steps + 255) & ~size_t(255);
        const size_t b_u64 = (8ull * n_steps + 255) & ~size_t(255);
        const size_t b_res = (sizeof(gbsa_mate_rescue) * n_steps + 255) & ~size_t(255);
        uint8_t* sc = static_cast<uint8_t*>(scratch_alloc(2 * b_nams + 2 * b_u32 + b_u64 + b_res + 256, st));
        struct Free {
            uint8_t* p;
            cudaStream_t s;
            ~Free() { scratch_free(p, s); }
        } release{sc, st};
        gbsa_nam* step_nams = reinterpret_cast<gbsa_nam*>(sc);
        uint32_t* step_reads = reinterpret_cast<uint32_t*>(sc + b_nams);
        gbsa_nam* rnams = reinterpret_cast<gbsa_nam*>(sc + b_nams + b_u32);
        uint32_t* rmates = reinterpret_cast<uint32_t*>(sc + 2 * b_nams + b_u32);
        uint64_t* ridx = reinterpret_cast<uint64_t*>(sc + 2 * b_nams + 2 * b_u32);
        gbsa_mate_rescue* rout = reinterpret_cast<gbsa_mate_rescue*>(sc + 2 * b_nams + 2 * b_u32 + b_u64);
        unsigned long long* count = reinterpret_cast<unsigned long long*>(sc + 2 * b_nams + 2 * b_u32 + b_u64 + b_res);
        GBSA_CUDA(cudaMemsetAsync(count, 0, 8, st));
        const unsigned grid = grid_for(n_steps, 256, (unsigned)device_sm_count() * 8);
        k_gather_step_nams<<<grid, 256, 0, st>>>(d_nams, d_nam_offsets, d_steps, n_steps, step_nams, step_reads);
        GBSA_LAUNCHED();
        int rc = gbsa_extend_seeds_device(d_ref_seqs, d_ref_offsets, d_ref_lengths, n_refs, d_read_seqs, d_read_offsets,
                                          d_read_lengths, n_reads, step_nams, step_reads, n_steps, k, params, d_ext,
                                          stream);
        if (rc != GBSA_OK) throw Error(rc, gbsa_last_error());
        k_rescue_list<<<grid, 256, 0, st>>>(d_steps, n_steps, step_nams, d_ext, rnams, rmates, ridx, count, d_resc);
        GBSA_LAUNCHED();
        unsigned long long n_resc = 0;
        GBSA_CUDA(cudaMemcpyAsync(&n_resc, count, 8, cudaMemcpyDeviceToHost, st));
        GBSA_CUDA(cudaStreamSynchronize(st));
        if (n_resc) {
            rc = gbsa_rescue_mates_device(d_ref_seqs, d_ref_offsets, d_ref_lengths, n_refs, d_read_seqs, d_read_offsets,
                                          d_read_lengths, n_reads, rnams, rmates, n_resc, k, mu, sigma, rout, stream);
            if (rc != GBSA_OK) throw Error(rc, gbsa_last_error());
            k_scatter_rescues<<<grid_for(n_resc, 256, (unsigned)device_sm_count() * 8), 256, 0, st>>>(rout, ridx, n_resc,
                                                                                                    d_resc);
            GBSA_LAUNCHED();
        }
        GBSA_CUDA(cudaStreamSynchronize(st));
        return GBSA_OK;
    } catch (const Error& e) {
        set_last_error(e.what());
        return e.code;
    } catch (const std::exception& e) {
        set_last_error(e.what());
        return GBSA_ERR_CUDA;
    }
}
