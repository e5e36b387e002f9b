// kernels.cuh -- the three device stages of one correction batch.
//
//   k_candidates : minhash signature + table lookup + de-duplication
//                  (one CTA per anchor)
//   k_align      : shifted Hamming distance, both strands, orientation,
//                  pair flag (one thread per (anchor, candidate) pair); most
//                  calls take k_align_tc (align_tc.cuh) in its place
//   k_msa        : alignment filters, MSA build/refine, consensus
//                  correction of anchor and candidates (one CTA per anchor)
#pragma once
#include <type_traits>
#include "device.cuh"

namespace careb200 {

__constant__ float c_qweight[256];    // QualityScoreConversion table (qualityscoreweights.hpp:16-31)

// ---------------------------------------------------------------------------
// Stage 1: candidate read ids per anchor.
//   CPUSequenceHasher::hashInto       include/cpusequencehasher.hpp:88-125
//   forEachEncodedCanonicalKmer...    include/sequencehelpers.hpp:844-926
//   OrdinaryCpuMinhasher::determineNumValues/retrieveValues/queryMap
//                                     include/ordinaryminhasher.hpp:135-221,437-449
//   determineCandidateReadIds         include/corrector.hpp:571-650
// The table-major concatenation is followed by sort+unique in the reference;
// here a shared-memory hash set removes duplicates, and the unique ids are
// placed by counting the smaller ones (up to an id per thread) or by a bitonic
// sort: same set, same ascending order.
// ---------------------------------------------------------------------------
constexpr uint32_t kEmpty = 0xFFFFFFFFu;

// Shared memory that a launch of k_candidates or k_candidates_spill may take.
// The limit is set to this at every launch: it belongs to the function on the
// device, and a limit of each call's own size could fall below another
// thread's between that thread's setting and its launch.
constexpr size_t kCandSmemLimit = 227 * 1024 - 256;

struct CandSmem {
    // dynamic shared memory layout, all offsets in bytes
    static __host__ __device__ size_t canon(int) { return 0; }
    static __host__ __device__ size_t partial(int maxlen) { return (size_t)(maxlen + 8) * 8; }
    static __host__ __device__ size_t seq(int maxlen, int groups, int maps) {
        return partial(maxlen) + (size_t)groups * maps * 8;
    }
    static __host__ __device__ size_t qinfo(int maxlen, int groups, int maps, int pitch) {
        return seq(maxlen, groups, maps) + (size_t)(pitch + 4) * 4;
    }
    static __host__ __device__ size_t set(int maxlen, int groups, int maps, int pitch) {
        return (qinfo(maxlen, groups, maps, pitch) + (size_t)(3 * kMaxMaps + 8) * 4 + 15) & ~(size_t)15;
    }
    static __host__ __device__ size_t total(int maxlen, int groups, int maps, int pitch, int setcap) {
        return set(maxlen, groups, maps, pitch) + (size_t)setcap * 4 * 2;
    }
};

// The candidate list of anchor ai, by one CTA. The de-duplication set has
// 2^sl2 entries, sl2 the smallest with 2^sl2 >= 2T (T ids retrieved), at most
// 2^set_log2. With a spill list the capacity is small (most anchors hold a few
// dozen unique ids among hundreds retrieved) and an anchor with more than
// half as many unique ids is appended to the list instead: its segment is
// then written by k_candidates_spill with a set large enough for every id.
template <int BLOCK>
__device__ __forceinline__ void candidates_of(
    const DevOptions& o, const DevReads& r, const TableDesc* __restrict__ td, const Slot* __restrict__ slots,
    const uint32_t* __restrict__ values, const unsigned long long* __restrict__ sig, uint32_t first, uint32_t ai,
    int set_log2, uint32_t* __restrict__ spill_list, unsigned int* __restrict__ spill_n,
    uint32_t* __restrict__ cand_ids, uint32_t* __restrict__ cand_anchor, uint32_t* __restrict__ seg_off,
    uint32_t* __restrict__ seg_cnt, unsigned long long* __restrict__ arena_count, unsigned long long arena_cap,
    int* __restrict__ status, unsigned char* smem, uint32_t& s_unique, uint32_t& s_ins, uint32_t& s_full,
    unsigned long long& s_base) {
    const int tid = threadIdx.x;
    const uint32_t a = first + ai;
    const int h = o.num_maps;
    const int groups = BLOCK / h;
    const int setcap = 1 << set_log2;
    unsigned long long* canon = (unsigned long long*)(smem + CandSmem::canon(r.max_len));
    unsigned long long* partial = (unsigned long long*)(smem + CandSmem::partial(r.max_len));
    uint32_t* sseq = (uint32_t*)(smem + CandSmem::seq(r.max_len, groups, h));
    uint32_t* qoff = (uint32_t*)(smem + CandSmem::qinfo(r.max_len, groups, h, r.seq_pitch));
    uint32_t* qcnt = qoff + kMaxMaps;
    uint32_t* qpre = qcnt + kMaxMaps;              // kMaxMaps + 1 entries
    uint32_t* set = (uint32_t*)(smem + CandSmem::set(r.max_len, groups, h, r.seq_pitch));
    uint32_t* list = set + setcap;

    const int L = r.len[a];
    const bool skip = (o.exclude_ambiguous && r.ambig[a]) || L < o.k;
    if (skip) {
        if (tid == 0) { seg_off[ai] = 0; seg_cnt[ai] = 0; }
        return;
    }
    // the anchor's signature: resident (computed once per read storage by
    // k_signatures), or hashed here
    if (!sig) {
        // anchor row into shared memory, two zero words of padding for kmer_at
        const uint32_t* arow = r.seq + (size_t)a * r.seq_pitch;
        for (int i = tid; i < r.seq_pitch + 2; i += BLOCK) sseq[i] = i < r.seq_pitch ? __ldg(arow + i) : 0u;
        __syncthreads();

        // canonical k-mers
        const int npos = L - o.k + 1;
        const int rcshift = 64 - 2 * o.k;
        for (int p = tid; p < npos; p += BLOCK) {
            const unsigned long long fw = kmer_at(sseq, o.k, p);
            const unsigned long long rv = revcomp64(fw) >> rcshift;
            canon[p] = fw < rv ? fw : rv;
        }
        __syncthreads();

        // per map: min over k-mers of murmur64(kmer + map)
        {
            const int m = tid % h, g = tid / h;
            if (g < groups) {
                unsigned long long mn = ~0ull;
                for (int p = g; p < npos; p += groups) {
                    const unsigned long long v = murmur64(canon[p] + (unsigned long long)m);
                    mn = v < mn ? v : mn;
                }
                partial[g * h + m] = mn;
            }
        }
        __syncthreads();
    }

    // table lookup (linear probing from murmur64(key))
    if (tid < h) {
        unsigned long long key = ~0ull;
        if (sig) {
            key = __ldg(sig + (size_t)a * h + tid);
        } else {
            for (int g = 0; g < groups; ++g) { const unsigned long long v = partial[g * h + tid]; key = v < key ? v : key; }
            key &= o.kmer_mask;
        }
        const TableDesc d = td[tid];
        uint32_t pos = (uint32_t)murmur64(key) & d.mask;
        uint32_t off = 0, cnt = 0;
        for (uint32_t probe = 0; probe <= d.mask; ++probe) {
            const Slot sl = slots[d.slot_base + pos];
            if (sl.count == 0) break;
            if (sl.key == key) { off = sl.offset; cnt = sl.count; break; }
            pos = (pos + 1) & d.mask;
        }
        if ((int)cnt > o.threshold) cnt = 0;      // queryMap :443-446
        qoff[tid] = (uint32_t)d.value_base + off;
        qcnt[tid] = cnt;
    }
    if (tid == 0) { s_unique = 0; s_ins = 0; s_full = 0; }
    __syncthreads();
    if (tid < 32) {                                  // offsets of the maps' runs: warp scan, two maps per lane
        const uint32_t c0 = tid < h ? qcnt[tid] : 0u, c1 = tid + 32 < h ? qcnt[tid + 32] : 0u;
        uint32_t s0 = c0, s1 = c1;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t t0 = __shfl_up_sync(0xffffffffu, s0, d), t1 = __shfl_up_sync(0xffffffffu, s1, d);
            if (tid >= d) { s0 += t0; s1 += t1; }
        }
        const uint32_t tot0 = __shfl_sync(0xffffffffu, s0, 31);
        if (tid < h) qpre[tid] = s0 - c0;
        if (tid + 32 < h) qpre[tid + 32] = tot0 + s1 - c1;
        if (tid == 31) qpre[h] = tot0 + s1;
    }
    __syncthreads();

    // the hash set is sized for the ids actually retrieved: a power of two
    // >= 2 * T (at least 64), within the allocated capacity
    const uint32_t T = qpre[h];
    int sl2 = 6;
    while (sl2 < set_log2 && (1u << sl2) < 2 * T) ++sl2;
    const int scap = 1 << sl2;
    // without a spill list the set always has room (2^set_log2 > h * threshold >= T)
    const uint32_t limit = spill_list ? (uint32_t)scap / 2 : 0xffffffffu;
    for (int i = tid; i < scap; i += BLOCK) set[i] = kEmpty;
    __syncthreads();

    // insert all retrieved ids into the shared hash set, eight loads in
    // flight per thread ahead of their inserts
    constexpr int kInFlight = 8;
    for (uint32_t e0 = 0; e0 < T; e0 += BLOCK * kInFlight) {
        uint32_t ids[kInFlight];
#pragma unroll
        for (int k = 0; k < kInFlight; ++k) {
            const uint32_t e = e0 + (uint32_t)(k * BLOCK + tid);
            ids[k] = kEmpty;
            if (e < T) {
                int lo = 0, hi = h - 1;             // map of element e
                while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (qpre[mid] <= e) lo = mid; else hi = mid - 1; }
                ids[k] = __ldg(values + qoff[lo] + (e - qpre[lo]));
            }
        }
#pragma unroll
        for (int k = 0; k < kInFlight; ++k) {
            const uint32_t id = ids[k];                // read ids are < 2^32 - 1: kEmpty marks none
            if (id == kEmpty || *(volatile uint32_t*)&s_full) continue;
            uint32_t pos = (id * 2654435761u) >> (32 - sl2);
            bool placed = false;
            for (int probe = 0; probe < scap; ++probe) {
                const uint32_t prev = atomicCAS(&set[pos], kEmpty, id);
                if (prev == kEmpty) {
                    placed = true;
                    if (atomicAdd(&s_ins, 1u) >= limit) s_full = 1;
                    break;
                }
                if (prev == id) { placed = true; break; }
                pos = (pos + 1) & (scap - 1);
            }
            if (!placed) s_full = 1;
        }
    }
    __syncthreads();
    if (s_full) {                                   // block-uniform: the second pass takes the anchor
        if (tid == 0) spill_list[atomicAdd(spill_n, 1u)] = ai;
        return;
    }

    // unique ids minus the anchor itself and (optionally) ambiguous reads
    for (int i = tid; i < scap; i += BLOCK) {
        const uint32_t v = set[i];
        if (v != kEmpty && v != a && !(o.exclude_ambiguous && r.ambig[v])) list[atomicAdd(&s_unique, 1u)] = v;
    }
    __syncthreads();
    const uint32_t U = s_unique;
    if (U <= BLOCK) {
        // an id per thread (nearly every anchor): its place is the number of
        // smaller ids, counted four at a time. No barriers between steps as
        // the sort below has, and a quarter of its instructions at 48 ids:
        // 4.7 -> 4.0 ms per 1M anchors.
        if (tid < 4) list[U + tid] = kEmpty;
        if (tid == 0) s_base = atomicAdd(arena_count, (unsigned long long)U);
        __syncthreads();
        const unsigned long long at = s_base;
        if (tid == 0) { seg_off[ai] = (uint32_t)at; seg_cnt[ai] = U; }
        if (at + U > arena_cap) {
            if (tid == 0) atomicOr(status, kStatusCandOverflow | kStatusIncomplete);
            return;
        }
        if ((uint32_t)tid < U) {
            const uint32_t id = list[tid];
            uint32_t rank = 0;
            for (uint32_t i = 0; i < U; i += 4) {
                const uint4 v = *reinterpret_cast<const uint4*>(list + i);
                rank += (v.x < id ? 1u : 0u) + (v.y < id ? 1u : 0u) + (v.z < id ? 1u : 0u) + (v.w < id ? 1u : 0u);
            }
            cand_ids[at + rank] = id;
            cand_anchor[at + tid] = ai;
        }
        return;
    }
    uint32_t P = 32;
    while (P < U) P <<= 1;
    for (uint32_t i = U + tid; i < P; i += BLOCK) list[i] = kEmpty;
    __syncthreads();
    // bitonic sort of list[0..P): exchanges across warps (partner distance
    // >= 32) through shared memory, one barrier each; the exchanges within a
    // warp (distance < 32) of a merge level in registers with shuffles
    const int wid = tid >> 5, ln = tid & 31;
    for (uint32_t kk = 2; kk <= P; kk <<= 1) {
        for (uint32_t j = kk >> 1; j >= 32; j >>= 1) {
            for (uint32_t i = tid; i < P; i += BLOCK) {
                const uint32_t ixj = i ^ j;
                if (ixj > i) {
                    const uint32_t x = list[i], y = list[ixj];
                    const bool up = (i & kk) == 0;
                    if ((x > y) == up) { list[i] = y; list[ixj] = x; }
                }
            }
            __syncthreads();
        }
        for (uint32_t i0 = 32u * wid; i0 < P; i0 += BLOCK) {      // warp-uniform
            const uint32_t i = i0 + ln;
            uint32_t x = list[i];
            const bool up = (i & kk) == 0;
            for (uint32_t j = min(kk >> 1, 16u); j > 0; j >>= 1) {
                const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
                x = (up == ((i & j) == 0)) ? min(x, y) : max(x, y);
            }
            list[i] = x;
        }
        __syncthreads();
    }
    if (tid == 0) s_base = atomicAdd(arena_count, (unsigned long long)U);
    __syncthreads();
    const unsigned long long base = s_base;
    if (tid == 0) { seg_off[ai] = (uint32_t)base; seg_cnt[ai] = U; }
    if (base + U > arena_cap) {
        if (tid == 0) atomicOr(status, kStatusCandOverflow | kStatusIncomplete);
        return;
    }
    for (uint32_t i = tid; i < U; i += BLOCK) { cand_ids[base + i] = list[i]; cand_anchor[base + i] = ai; }
}

// One anchor per CTA, the set capacity 2^set_log2 (small when spill_list is
// given: the anchors that overflow it are listed for k_candidates_spill).
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK)
k_candidates(DevOptions o, DevReads r, const TableDesc* __restrict__ td, const Slot* __restrict__ slots,
             const uint32_t* __restrict__ values, const unsigned long long* __restrict__ sig,
             uint32_t first, uint32_t count, int set_log2, uint32_t* __restrict__ spill_list,
             unsigned int* __restrict__ spill_n, uint32_t* __restrict__ cand_ids, uint32_t* __restrict__ cand_anchor,
             uint32_t* __restrict__ seg_off, uint32_t* __restrict__ seg_cnt,
             unsigned long long* __restrict__ arena_count, unsigned long long arena_cap,
             int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t s_unique, s_ins, s_full;
    __shared__ unsigned long long s_base;
    if (blockIdx.x >= count) return;
    candidates_of<BLOCK>(o, r, td, slots, values, sig, first, blockIdx.x, set_log2, spill_list, spill_n, cand_ids,
                         cand_anchor, seg_off, seg_cnt, arena_count, arena_cap, status, smem, s_unique, s_ins,
                         s_full, s_base);
}

// The listed anchors with a set for every retrieved id (persistent CTAs).
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK)
k_candidates_spill(DevOptions o, DevReads r, const TableDesc* __restrict__ td, const Slot* __restrict__ slots,
                   const uint32_t* __restrict__ values, const unsigned long long* __restrict__ sig, uint32_t first,
                   int set_log2, const uint32_t* __restrict__ spill_list, const unsigned int* __restrict__ spill_n,
                   uint32_t* __restrict__ cand_ids, uint32_t* __restrict__ cand_anchor,
                   uint32_t* __restrict__ seg_off, uint32_t* __restrict__ seg_cnt,
                   unsigned long long* __restrict__ arena_count, unsigned long long arena_cap,
                   int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t s_unique, s_ins, s_full;
    __shared__ unsigned long long s_base;
    const unsigned int n = *spill_n;
    for (unsigned int k = blockIdx.x; k < n; k += gridDim.x) {
        candidates_of<BLOCK>(o, r, td, slots, values, sig, first, spill_list[k], set_log2, nullptr, nullptr,
                             cand_ids, cand_anchor, seg_off, seg_cnt, arena_count, arena_cap, status, smem,
                             s_unique, s_ins, s_full, s_base);
        __syncthreads();                            // the next anchor reuses the shared state
    }
}

// ---------------------------------------------------------------------------
// Stage 2: alignment of every (anchor, candidate) pair, both strands.
//   getCandidateAlignments            include/corrector.hpp:925-979
//   cpuShiftedHammingDistance...      src/cpu_alignment.cpp:32-323
//   chooseBestAlignmentOrientation    include/alignmentorientation.hpp:72-92
//   computePairFlags                  include/corrector.hpp:763-807 (PE)
// ---------------------------------------------------------------------------
constexpr uint32_t kNoMirror = 0xffffffffu;

// Mirror pairs. When candidate c of anchor a is itself an anchor of the
// batch, has a's length and holds a among its candidates, the pairs (a, c)
// and (c, a) share their scans: the reverse-complement alignments are the
// same (same shift, overlap and mismatches) and both forward alignments come
// from one tie-aware scan (shifted_hamming_pair). The pair with a < c leads
// and computes both results; its mirror is skipped. Work list: leaders
// {pair, mirror} from the front, single pairs {pair, kNoMirror} from the
// back (index total-1 down), counts in work_n[0] and work_n[1].
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK)
k_pair_mirror(DevReads r, uint32_t first, uint32_t count, const uint32_t* __restrict__ cand_ids,
              const uint32_t* __restrict__ cand_anchor, const uint32_t* __restrict__ seg_off,
              const uint32_t* __restrict__ seg_cnt, const unsigned long long* __restrict__ total_ptr,
              unsigned long long arena_cap, const int* __restrict__ status, const uint32_t* __restrict__ pair_order,
              uint2* __restrict__ work, unsigned int* __restrict__ work_n) {
    if (*status & kStatusCandOverflow) return;
    const unsigned long long total = *total_ptr;
    if (total > arena_cap) return;
    const unsigned long long slot = (unsigned long long)blockIdx.x * BLOCK + threadIdx.x;
    if (slot - (threadIdx.x & 31) >= total) return;          // whole warp past the end
    int kind = 0;                                            // 1 leader, 2 single
    uint32_t i = 0, j = kNoMirror;
    if (slot < total) {
        i = pair_order ? pair_order[slot] : (uint32_t)slot;
        const uint32_t a = first + cand_anchor[i];
        const uint32_t c = cand_ids[i];
        kind = 2;
        if (c - first < count && r.len[a] == r.len[c]) {
            const uint32_t ci = c - first, off = seg_off[ci], cnt = seg_cnt[ci];
            uint32_t lo = 0, hi = cnt;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (cand_ids[off + mid] < a) lo = mid + 1; else hi = mid;
            }
            if (lo < cnt && cand_ids[off + lo] == a) {
                j = off + lo;
                kind = a < c ? 1 : 0;
            }
        }
    }
    const unsigned ln = threadIdx.x & 31, below = (1u << ln) - 1u;
    const unsigned ml = __ballot_sync(0xffffffffu, kind == 1), ms = __ballot_sync(0xffffffffu, kind == 2);
    unsigned bl = 0, bs = 0;
    if (ln == 0) {
        if (ml) bl = atomicAdd(&work_n[0], (unsigned)__popc(ml));
        if (ms) bs = atomicAdd(&work_n[1], (unsigned)__popc(ms));
    }
    bl = __shfl_sync(0xffffffffu, bl, 0);
    bs = __shfl_sync(0xffffffffu, bs, 0);
    if (kind == 1) work[bl + __popc(ml & below)] = make_uint2(i, j);
    if (kind == 2) work[total - 1 - (bs + __popc(ms & below))] = make_uint2(i, kNoMirror);
}

// Candidate c's pair flag: c's mate is a candidate of the anchor's mate
// (equivalent to flagPairedCandidates, include/util.hpp:1016-1197).
__device__ __forceinline__ uint8_t mate_flag(const uint32_t* __restrict__ cand_ids, const uint32_t* __restrict__ seg_off,
                       const uint32_t* __restrict__ seg_cnt, uint32_t ai, uint32_t c) {
    const uint32_t mi = ai ^ 1u;
    const uint32_t moff = seg_off[mi], mcnt = seg_cnt[mi];
    const uint32_t target = c ^ 1u;
    uint32_t lo2 = 0, hi2 = mcnt;
    while (lo2 < hi2) {
        const uint32_t mid = (lo2 + hi2) >> 1;
        if (cand_ids[moff + mid] < target) lo2 = mid + 1; else hi2 = mid;
    }
    return (lo2 < mcnt && cand_ids[moff + lo2] == target) ? 1 : 0;
}

// CNT: the statistics form, which also adds the 32-bit word compares its
// scans actually run (after the early exits) to run_count.
// One alignment work item (slot of the mirror work list, of pair_order from
// `base`, or the pair itself): both orientations, the orientation choice and
// the AlignRes (a mirrored pair writes both). false past the work list.
template <int NW, bool CNT>
__device__ __forceinline__ bool
align_item(const DevOptions& o, const DevReads& r, uint32_t first, const uint32_t* __restrict__ cand_ids,
           const uint32_t* __restrict__ cand_anchor, const uint32_t* __restrict__ seg_off,
           const uint32_t* __restrict__ seg_cnt, unsigned long long total, AlignRes* __restrict__ out,
           unsigned long long* __restrict__ work_count, const uint32_t* __restrict__ pair_order,
           unsigned long long base, const uint2* __restrict__ work, const unsigned int* __restrict__ work_n,
           unsigned long long* __restrict__ run_count, const int* s_mex, unsigned long long slot) {
    using Cnt = typename std::conditional<CNT, WordCount, NoCount>::type;
    Cnt wc;
    unsigned long long i;
    uint32_t j = kNoMirror;
    if (work) {                        // mirror work list (k_pair_mirror)
        const unsigned nl = work_n[0], ns = work_n[1];
        if (slot >= (unsigned long long)nl + ns) return false;
        const uint2 w = slot < nl ? work[slot] : work[total - 1 - (slot - nl)];
        i = w.x;
        j = w.y;
    } else {
        i = pair_order ? pair_order[base + slot] : slot;
    }
    const uint32_t ai = cand_anchor[i];
    const uint32_t a = first + ai;
    const uint32_t c = cand_ids[i];
    const int La = r.len[a], Lc = r.len[c];
    uint32_t Ah[NW + 2], Al[NW + 2], Ch[NW + 2], Cl[NW + 2];
    load_planes<NW>(r.seq + (size_t)a * r.seq_pitch, La, Ah, Al);
    load_planes<NW>(r.seq + (size_t)c * r.seq_pitch, Lc, Ch, Cl);
    const int lo = __float2int_rz(__fmul_rn((float)La, o.min_overlap_ratio));
    const int minov = o.min_overlap > lo ? o.min_overlap : lo;
    if (work_count) {                 // un-pruned word compares of the scans run here (roofline work)
        const unsigned m = __activemask();
        const unsigned ws = __reduce_add_sync(m, (unsigned)(2 * unpruned_words(La, Lc, minov)));
        if ((int)(threadIdx.x & 31) == __ffs(m) - 1) atomicAdd(work_count, (unsigned long long)ws);
    }
    ShdResult f, g;                   // g: forward alignment of the mirror pair (c, a)
    if (j != kNoMirror) shifted_hamming_pair<NW, Cnt>(Ah, Al, Ch, Cl, La, minov, s_mex, f, g, &wc);
    else f = shifted_hamming<NW, Cnt>(Ah, Al, La, Ch, Cl, Lc, minov, s_mex, &wc);
    uint32_t Rh[NW + 2], Rl[NW + 2];
    revcomp_planes<NW>(Ch, Cl, Lc, Rh, Rl);
    const ShdResult rc = shifted_hamming<NW, Cnt>(Ah, Al, La, Rh, Rl, Lc, minov, s_mex, &wc);
    if constexpr (CNT) {
        const unsigned m = __activemask();
        const unsigned ws = __reduce_add_sync(m, (unsigned)wc.n);
        if ((int)(threadIdx.x & 31) == __ffs(m) - 1) atomicAdd(run_count, (unsigned long long)ws);
    }
    const float ler = __fmul_rn(o.estimated_errorrate, 4.0f);
    auto result = [&](const ShdResult& fw, uint32_t anchor_index, uint32_t cand) {
        const int orient = choose_orientation(fw, rc, La, o.min_overlap_ratio, o.min_overlap, ler);
        AlignRes res;
        const ShdResult& b = orient == 2 ? rc : fw;
        res.shift = (int16_t)b.shift;
        res.overlap = (int16_t)b.overlap;
        res.nops = (int16_t)b.nops;
        res.orient = (uint8_t)orient;
        res.paired = o.paired_end ? mate_flag(cand_ids, seg_off, seg_cnt, anchor_index, cand) : 0;
        return res;
    };
    out[i] = result(f, ai, c);
    if (j != kNoMirror) out[j] = result(g, c - first, a);
    return true;
}

template <int BLOCK>
__device__ __forceinline__ void align_mex_table(const DevOptions& o, int* s_mex) {
    // int(float(ov) * maxErrorRate), the first term of max_errors_excl
    for (int i = threadIdx.x; i <= kMaxLen; i += BLOCK) s_mex[i] = __float2int_rz(__fmul_rn((float)i, o.max_error_rate));
    __syncthreads();
}

template <int BLOCK, int NW, bool CNT = false>
__global__ void __launch_bounds__(BLOCK)
k_align(DevOptions o, DevReads r, uint32_t first, const uint32_t* __restrict__ cand_ids,
        const uint32_t* __restrict__ cand_anchor, const uint32_t* __restrict__ seg_off,
        const uint32_t* __restrict__ seg_cnt, const unsigned long long* __restrict__ total_ptr,
        unsigned long long arena_cap, const int* __restrict__ status, AlignRes* __restrict__ out,
        unsigned long long* __restrict__ work_count, const uint32_t* __restrict__ pair_order,
        const uint2* __restrict__ work, const unsigned int* __restrict__ work_n,
        unsigned long long* __restrict__ run_count) {
    __shared__ int s_mex[kMaxLen + 1];
    align_mex_table<BLOCK>(o, s_mex);
    // an overflowed candidate arena holds unwritten entries: the batch is
    // repeated with a larger arena, nothing here may read them
    if (*status & kStatusCandOverflow) return;
    const unsigned long long slot = (unsigned long long)blockIdx.x * BLOCK + threadIdx.x;
    const unsigned long long total = *total_ptr;
    if (total > arena_cap || slot >= total) return;
    align_item<NW, CNT>(o, r, first, cand_ids, cand_anchor, seg_off, seg_cnt, total, out, work_count, pair_order, 0,
                        work, work_n, run_count, s_mex, slot);
}

// One length class of the batch's pairs (cls = {offset in the class list,
// pairs}, k_pair_class_*): resident blocks stride over its pairs, with the
// register budget of the class's plane width.
template <int BLOCK, int NW, bool CNT = false>
__global__ void __launch_bounds__(BLOCK, (NW <= 5 ? 1024 : 768) / BLOCK)
k_align_class(DevOptions o, DevReads r, uint32_t first, const uint32_t* __restrict__ cand_ids,
              const uint32_t* __restrict__ cand_anchor, const uint32_t* __restrict__ seg_off,
              const uint32_t* __restrict__ seg_cnt, const unsigned long long* __restrict__ total_ptr,
              unsigned long long arena_cap, const int* __restrict__ status, AlignRes* __restrict__ out,
              unsigned long long* __restrict__ work_count, const uint32_t* __restrict__ class_list,
              const uint2* __restrict__ cls, unsigned long long* __restrict__ run_count) {
    __shared__ int s_mex[kMaxLen + 1];
    align_mex_table<BLOCK>(o, s_mex);
    if (*status & kStatusCandOverflow) return;
    const unsigned long long total = *total_ptr;
    if (total > arena_cap) return;
    const unsigned long long n = cls->y, base = cls->x;
#pragma unroll 1
    for (unsigned long long slot = (unsigned long long)blockIdx.x * BLOCK + threadIdx.x; slot < n;
         slot += (unsigned long long)gridDim.x * BLOCK)
        align_item<NW, CNT>(o, r, first, cand_ids, cand_anchor, seg_off, seg_cnt, total, out, work_count, class_list,
                            base, nullptr, nullptr, run_count, s_mex, slot);
}

// ---------------------------------------------------------------------------
// Warp-cooperative alignment: one warp per work item, lane r of the warp
// takes shift 32*w + r of each group w of 32 shifts (the funnel shift amount
// is the lane; the planes slide by one word per group, as in shd_scan).
// Every lane counts its shift's mismatches up to its own limit
// min(int(ov * maxErrorRate), best - total + 2*ov), with `best` the score
// found by the earlier groups, and the warp keeps the smallest key
// (score << 10 | rank of the shift in the scan order). The result is the
// first shift in scan order with the smallest score among the shifts whose
// mismatches are below int(ov * maxErrorRate): the same shift the sequential
// scan with early exits returns (src/cpu_alignment.cpp:247-316). A direction
// ends at the first group whose leading shift can no longer reach the best
// (its limit is <= 0 and the limit does not grow along a direction).
// TIES: the equal-length pair form (both directions of a mirrored pair, as
// shd_scan_ties): ties with the best are kept (limit + 1) and a second key
// ranks the shifts in the order of the (C, A) scan.
constexpr unsigned kKeyRankBits = 10;          // ranks and scores stay below 1024 (reads <= 256 bases)
constexpr unsigned kKeyRankMask = (1u << kKeyRankBits) - 1u;

// D0: shifts of the first direction (its ranks are t, the second's D0 + t - 1);
// negs: the (C, A) order's count of shifts <= 0 after 0 (TIES).
template <int NW, bool TIES, class Cnt>
__device__ __forceinline__ void shd_scan_lanes(uint32_t (&Sh)[NW + 2], uint32_t (&Sl)[NW + 2],
                                               const uint32_t (&Oh)[NW + 2], const uint32_t (&Ol)[NW + 2],
                                               int t0, int t1, int dir, int La, int Lc, int total, int D0,
                                               int negs, const int* __restrict__ mextab, unsigned& keyA,
                                               unsigned& keyB, Cnt* cnt) {
    if (t1 < t0) return;
    const int lane = threadIdx.x & 31;
    const int tie = TIES ? 1 : 0;
    auto overlap = [&](int t) { return dir == 0 ? min(La - t, Lc) : min(La, Lc - t); };
#pragma unroll 1
    for (int w = 0; w <= (t1 >> 5); ++w) {
        const int t = 32 * w + lane;
        const int best = (int)(keyA >> kKeyRankBits);
        unsigned ka = 0xFFFFFFFFu, kb = 0xFFFFFFFFu;
        if (t >= t0 && t <= t1) {
            const int ov = overlap(t);
            const int mex = min(mextab[ov], best - total + 2 * ov + tie);
            if (mex > 0) {
                const int r = lane;
                uint32_t d0 = (funnel_l(Sh[1], Sh[0], r) ^ Oh[0]) | (funnel_l(Sl[1], Sl[0], r) ^ Ol[0]);
                uint32_t d1 = (funnel_l(Sh[2], Sh[1], r) ^ Oh[1]) | (funnel_l(Sl[2], Sl[1], r) ^ Ol[1]);
                if (ov < 64) { d0 &= lead_mask(ov); d1 &= lead_mask(ov - 32); }
                int mm = popc32(d0) + popc32(d1);
                if (cnt) cnt->add(2);
                if (mm < mex && ov > 64) {
#pragma unroll
                    for (int j = 2; j < NW; ++j) {
                        if (32 * j < ov && mm < mex) {
                            uint32_t dj = (funnel_l(Sh[j + 1], Sh[j], r) ^ Oh[j]) |
                                          (funnel_l(Sl[j + 1], Sl[j], r) ^ Ol[j]);
                            dj &= lead_mask(ov - 32 * j);
                            mm += popc32(dj);
                            if (cnt) cnt->add(1);
                        }
                    }
                }
                if (mm < mex) {
                    const unsigned sc = (unsigned)(mm + total - 2 * ov) << kKeyRankBits;
                    ka = sc | (unsigned)(dir == 0 ? t : D0 + t - 1);
                    if constexpr (TIES) kb = sc | (unsigned)(dir == 0 ? (t == 0 ? 0 : negs + t) : t);
                }
            }
        }
        keyA = min(keyA, __reduce_min_sync(0xffffffffu, ka));
        if constexpr (TIES) keyB = min(keyB, __reduce_min_sync(0xffffffffu, kb));
        const int tn = 32 * (w + 1);
        if (tn > t1) break;
        {   // end of the direction: the next group's first shift cannot reach the best
            const int ovn = overlap(tn);
            if (min(mextab[ovn], (int)(keyA >> kKeyRankBits) - total + 2 * ovn + tie) <= 0) break;
        }
#pragma unroll
        for (int j = 0; j < NW + 1; ++j) { Sh[j] = Sh[j + 1]; Sl[j] = Sl[j + 1]; }
        Sh[NW + 1] = 0u; Sl[NW + 1] = 0u;
    }
}

// ShdResult of a scan from its best key: shift of rank `rank`, the overlap,
// score and mismatches (nOps) of that shift.
__device__ __forceinline__ ShdResult shd_from_shift(int shift, int score, int La, int Lc) {
    ShdResult res;
    res.valid = shift != -Lc;
    const int cb = max(-shift, 0);
    const int ce = min(Lc, La - shift);
    res.overlap = ce - cb;
    res.score = score;
    res.shift = shift;
    res.nops = score - (La + Lc) + 2 * res.overlap;
    return res;
}

// shifted_hamming with the warp: every lane returns the same result.
template <int NW, class Cnt>
__device__ __forceinline__ ShdResult shifted_hamming_lanes(const uint32_t (&Ah)[NW + 2], const uint32_t (&Al)[NW + 2],
                                                           int La, const uint32_t (&Ch)[NW + 2],
                                                           const uint32_t (&Cl)[NW + 2], int Lc, int minov,
                                                           const int* __restrict__ mextab, Cnt* cnt) {
    const int total = La + Lc;
    const int T0 = La - minov;
    const int D0 = T0 + 1 > 0 ? T0 + 1 : 0;      // shifts of the first direction: ranks 0..D0-1
    unsigned keyA = ((unsigned)total << kKeyRankBits) | kKeyRankMask, keyB = 0xFFFFFFFFu;
    uint32_t Sh[NW + 2], Sl[NW + 2];
#pragma unroll 1
    for (int dir = 0; dir < 2; ++dir) {
#pragma unroll
        for (int j = 0; j < NW + 2; ++j) { Sh[j] = dir ? Ch[j] : Ah[j]; Sl[j] = dir ? Cl[j] : Al[j]; }
        if (dir == 0) shd_scan_lanes<NW, false>(Sh, Sl, Ch, Cl, 0, T0, 0, La, Lc, total, D0, 0, mextab, keyA, keyB, cnt);
        else shd_scan_lanes<NW, false>(Sh, Sl, Ah, Al, 1, Lc - minov, 1, La, Lc, total, D0, 0, mextab, keyA, keyB, cnt);
    }
    const int score = (int)(keyA >> kKeyRankBits), rank = (int)(keyA & kKeyRankMask);
    const int shift = score >= total ? -Lc : (rank < D0 ? rank : -(rank - D0 + 1));
    return shd_from_shift(shift, score, La, Lc);
}

// shifted_hamming_pair with the warp: forward (A, C) and (C, A) of a pair of
// equal length L.
template <int NW, class Cnt>
__device__ __forceinline__ void shifted_hamming_pair_lanes(const uint32_t (&Ah)[NW + 2], const uint32_t (&Al)[NW + 2],
                                                           const uint32_t (&Ch)[NW + 2], const uint32_t (&Cl)[NW + 2],
                                                           int L, int minov, const int* __restrict__ mextab,
                                                           ShdResult& ac, ShdResult& ca, Cnt* cnt) {
    const int total = 2 * L;
    const int T = L - minov;
    unsigned keyA = ((unsigned)total << kKeyRankBits) | kKeyRankMask, keyB = keyA;
    uint32_t Sh[NW + 2], Sl[NW + 2];
#pragma unroll 1
    for (int dir = 0; dir < 2; ++dir) {
#pragma unroll
        for (int j = 0; j < NW + 2; ++j) { Sh[j] = dir ? Ch[j] : Ah[j]; Sl[j] = dir ? Cl[j] : Al[j]; }
        if (dir == 0) shd_scan_lanes<NW, true>(Sh, Sl, Ch, Cl, 0, T, 0, L, L, total, T + 1, T, mextab, keyA, keyB, cnt);
        else shd_scan_lanes<NW, true>(Sh, Sl, Ah, Al, 1, T, 1, L, L, total, T + 1, T, mextab, keyA, keyB, cnt);
    }
    const int score = (int)(keyA >> kKeyRankBits);
    const int ra = (int)(keyA & kKeyRankMask), rb = (int)(keyB & kKeyRankMask);
    const int sA = score >= total ? -L : (ra <= T ? ra : -(ra - T));
    // rank in the (C, A) order: 0 for shift 0, -s for s < 0, T + s for s > 0
    const int sB = score >= total ? -L : (rb <= T ? -rb : rb - T);
    ac = shd_from_shift(sA, score, L, L);
    ca = shd_from_shift(sB == -L ? -L : -sB, score, L, L);
}

// The alignment stage with a warp per work item (a mirrored pair or a single
// pair; the same items and outputs as k_align). Persistent: the grid's warps
// stride over the items.
template <int BLOCK, int NW, bool CNT = false>
__global__ void __launch_bounds__(BLOCK)
k_align_warp(DevOptions o, DevReads r, uint32_t first, const uint32_t* __restrict__ cand_ids,
             const uint32_t* __restrict__ cand_anchor, const uint32_t* __restrict__ seg_off,
             const uint32_t* __restrict__ seg_cnt, const unsigned long long* __restrict__ total_ptr,
             unsigned long long arena_cap, const int* __restrict__ status, AlignRes* __restrict__ out,
             unsigned long long* __restrict__ work_count, const uint32_t* __restrict__ pair_order,
             const uint2* __restrict__ work, const unsigned int* __restrict__ work_n,
             unsigned long long* __restrict__ run_count) {
    using Cnt = typename std::conditional<CNT, WordCount, NoCount>::type;
    __shared__ int s_mex[kMaxLen + 1];
    for (int i = threadIdx.x; i <= kMaxLen; i += BLOCK) s_mex[i] = __float2int_rz(__fmul_rn((float)i, o.max_error_rate));
    __syncthreads();
    if (*status & kStatusCandOverflow) return;
    const unsigned long long total = *total_ptr;
    if (total > arena_cap) return;
    const unsigned long long items = work ? (unsigned long long)work_n[0] + work_n[1] : total;
    const int lane = threadIdx.x & 31;
    const unsigned long long nwarps = (unsigned long long)gridDim.x * (BLOCK / 32);
    const float ler = __fmul_rn(o.estimated_errorrate, 4.0f);
#pragma unroll 1
    for (unsigned long long slot = (unsigned long long)blockIdx.x * (BLOCK / 32) + (threadIdx.x >> 5); slot < items;
         slot += nwarps) {
        Cnt wc;
        unsigned long long i;
        uint32_t j = kNoMirror;
        if (work) {
            const unsigned nl = work_n[0];
            const uint2 wv = slot < nl ? work[slot] : work[total - 1 - (slot - nl)];
            i = wv.x;
            j = wv.y;
        } else {
            i = pair_order ? pair_order[slot] : slot;
        }
        const uint32_t ai = cand_anchor[i];
        const uint32_t a = first + ai;
        const uint32_t c = cand_ids[i];
        const int La = r.len[a], Lc = r.len[c];
        uint32_t Ah[NW + 2], Al[NW + 2], Ch[NW + 2], Cl[NW + 2];
        load_planes<NW>(r.seq + (size_t)a * r.seq_pitch, La, Ah, Al);
        load_planes<NW>(r.seq + (size_t)c * r.seq_pitch, Lc, Ch, Cl);
        const int lo = __float2int_rz(__fmul_rn((float)La, o.min_overlap_ratio));
        const int minov = o.min_overlap > lo ? o.min_overlap : lo;
        if (work_count && lane == 0) atomicAdd(work_count, (unsigned long long)(2 * unpruned_words(La, Lc, minov)));
        ShdResult f, g;
        if (j != kNoMirror) shifted_hamming_pair_lanes<NW, Cnt>(Ah, Al, Ch, Cl, La, minov, s_mex, f, g, &wc);
        else f = shifted_hamming_lanes<NW, Cnt>(Ah, Al, La, Ch, Cl, Lc, minov, s_mex, &wc);
        uint32_t Rh[NW + 2], Rl[NW + 2];
        revcomp_planes<NW>(Ch, Cl, Lc, Rh, Rl);
        const ShdResult rc = shifted_hamming_lanes<NW, Cnt>(Ah, Al, La, Rh, Rl, Lc, minov, s_mex, &wc);
        if constexpr (CNT) {
            const unsigned ws = __reduce_add_sync(0xffffffffu, (unsigned)wc.n);
            if (lane == 0) atomicAdd(run_count, (unsigned long long)ws);
        }
        if (lane == 0) {
            auto result = [&](const ShdResult& fw, uint32_t anchor_index, uint32_t cand) {
                const int orient = choose_orientation(fw, rc, La, o.min_overlap_ratio, o.min_overlap, ler);
                AlignRes res;
                const ShdResult& b = orient == 2 ? rc : fw;
                res.shift = (int16_t)b.shift;
                res.overlap = (int16_t)b.overlap;
                res.nops = (int16_t)b.nops;
                res.orient = (uint8_t)orient;
                res.paired = o.paired_end ? mate_flag(cand_ids, seg_off, seg_cnt, anchor_index, cand) : 0;
                return res;
            };
            out[i] = result(f, ai, c);
            if (j != kNoMirror) out[j] = result(g, c - first, a);
        }
    }
}

// ---------------------------------------------------------------------------
// Stage 3: filters, MSA, refinement, correction.
//   filterCandidatesByAlignmentFlag / ...MismatchRatio(WithPairFlags)
//                                     include/corrector.hpp:982-1211
//   alignmentsComputeWeightsAndAoStoSoA :1260-1280, calculateOverlapWeight
//                                     include/hostdevicefunctions.cuh:93-97
//   MultipleSequenceAlignment::build/addSequence/findConsensus/
//   findOrigWeightAndCoverage         src/msa.cpp:9-173
//   refineMSA                         include/corrector.hpp:1307-1421
//   findCandidatesOfDifferentRegion   src/msa.cpp:532-734
//   getMSAProperties                  src/msa.cpp:304-376
//   getCorrectedAnchor                src/msa.cpp:379-453
//   getCorrectedCandidates            src/msa.cpp:457-522
//   makeOutputOfTask (edits)          include/corrector.hpp:1639-1761
//
// What the anchor's result needs of the MSA: per anchor column the consensus,
// its support and the counts. A column whose rows all hold the anchor's base
// has that base as consensus with support exactly 1 (one of the four sums is
// non-zero, and it is the column weight), whatever its sums are. So the rows
// are compared with the anchor 16 bases at a time while they are staged, and
// only the columns where some row differs (disputed columns, a quarter of
// them at 30x) get sums: one lane per column, its rows in list order, anchor
// first, with separate IEEE multiply and add (no FMA) -- the reference's order
// and rounding, so the sums are bit-identical. Coverage comes from the rows'
// ends. Columns outside the anchor are summed only for candidate correction,
// within its new_columns of the anchor.
//
// Rows are staged in shared memory as the words of the anchor's own 16-base
// grid (word g holds anchor positions 16 g .. 16 g + 15, turned into the
// aligned orientation), a thread per (row, word); the anchor is row 0. They
// stay staged across refinement rebuilds when the candidate list fits (up to
// 128 rows in 16 KB).
// Bound: instruction issue. Measured against sums of every column with the
// rows staged whole: 1M 150 bp paired-end reads at 30x 13.0 ms (20.7), 400k
// reads of 50-250 bases 8.8 ms (18.2), 1.3M reads at 50x 22.4 ms (38.4), 128
// anchors 66 us (168).
// ---------------------------------------------------------------------------
struct MsaOut {
    uint8_t* status;
    int32_t* nedits;
    char* seq;                        // count * max_len
    uint32_t* corr_id;
    uint32_t* corr_anchor;
    int32_t* corr_shift;
    uint8_t* corr_use_edits;
    char* corr_seq;                   // corr_cap * max_len
    unsigned long long* corr_count;
    unsigned long long corr_cap;
    // decision columns (EMIT): 24 features, read id, pos | orig << 16 | cons << 18
    float* feat;
    uint32_t* feat_read;
    uint32_t* feat_meta;
    unsigned long long* feat_count;
    unsigned long long feat_cap;
    // bases of the MSAs' rows (anchor and candidates, every build): the MSA
    // stage's roofline work (the sums of undisputed columns are not formed);
    // may be null
    unsigned long long* elem_count;
    // refinement statistics, may be null: [0] the rows' bases in rebuilds
    // (builds after the first), [1] anchors rebuilt at least once
    unsigned long long* rebuild_count;
};

constexpr int kNumFeatures = 24;

constexpr int kStageMax = 128;        // candidate rows held in shared memory, at most
constexpr int kStageBudget = 16384;   // bytes of staged rows

// The staged rows' grid: `words` 16-base words, `edge` of them on each side of
// the anchor (columns outside it that candidate correction reads), `wpg`
// 32-bit words per grid word: the bases, then the qualities of the same
// positions (16 1-bit codes in the high half, 16 2-bit codes, or 16
// characters); per-column arrays hold 16 * words entries.
struct MsaGrid {
    int edge, words, wpg, rw, rows;
    uint32_t magic;                   // x / words as the high word of x * magic (words > 1)
};
__host__ __device__ constexpr MsaGrid msa_grid(int max_len, int qb, int correct_candidates, int new_columns) {
    MsaGrid g{};
    const int nc = new_columns < 0 ? 0 : new_columns > kMaxLen ? kMaxLen : new_columns;
    g.edge = correct_candidates ? (nc + 15) / 16 : 0;
    g.words = (max_len + 15) / 16 + 2 * g.edge;
    g.wpg = qb == 0 ? 1 : qb == 8 ? 5 : 2;
    g.rw = g.words * g.wpg;
    const int rows = kStageBudget / (g.rw * 4);
    g.rows = rows > kStageMax ? kStageMax : (rows < 16 ? 16 : rows);
    g.magic = (uint32_t)((0x100000000ull + (uint32_t)g.words - 1) / (uint32_t)g.words);
    return g;
}

// dynamic shared memory of k_msa: the staged rows (the anchor and `rows`
// candidates), per anchor position the support and the four counts, with
// decision rows three column weights, then the coverage, the column list and
// the bases of the grid's columns. Every part starts on a 16-byte boundary.
__host__ __device__ constexpr size_t msa_round16(size_t x) { return (x + 15) & ~(size_t)15; }
__host__ __device__ constexpr size_t msa_smem_bytes(const MsaGrid& g, int max_len, bool emit) {
    const size_t cols = 16 * (size_t)g.words;
    return msa_round16((size_t)(g.rows + 1) * g.rw * 4) + msa_round16((size_t)max_len * 4) + (size_t)max_len * 8 +
           8 * (size_t)(max_len & 1) + (emit ? msa_round16((size_t)3 * max_len * 4) : 0) +
           msa_round16((size_t)max_len * 2) + msa_round16(cols * 2) + cols;
}
// the most that any read length, quality encoding and edge takes
constexpr size_t msa_smem_most() {
    size_t most = 0;
    for (int qb = 0; qb <= 8; qb = qb == 0 ? 1 : 2 * qb)
        for (int len = 1; len <= kMaxLen; ++len)
            for (int nc = 0; nc <= kMaxLen; nc += 16) {
                const size_t n = msa_smem_bytes(msa_grid(len, qb, 1, nc), len, true);
                most = n > most ? n : most;
            }
    return most;
}
// With the static part (below 10 KB) no launch needs a raised limit, which
// would be shared by all threads of the process.
static_assert(msa_smem_most() + 10240 <= 48 * 1024, "the MSA fits the default limit");

// reverse the 16 2-bit codes of a word, keeping each code's bits
__device__ __forceinline__ uint32_t rev2(uint32_t w) {
    w = __brev(w);
    return ((w >> 1) & 0x55555555u) | ((w & 0x55555555u) << 1);
}

// One element of a column: weight w added to the sum of its base (b8 = base
// * 8) and one to the base's 8-bit count in c8 (A | C << 8 | G << 16 |
// T << 24), nothing when the column lies outside the row (p, the column's
// position in the row, not below len). IEEE adds (add.rn.f32, no
// contraction), predicated on (base, in row): the sums see the same
// additions in the same order as an add per element of the base.
__device__ __forceinline__ void msa_add8(float& wA, float& wC, float& wG, float& wT, uint32_t& c8,
                                         uint32_t b8, float w, int p, int len) {
    asm("{\n\t"
        ".reg .pred pin, pa, pc, pg, pt;\n\t"
        ".reg .b32 inc;\n\t"
        "setp.lt.u32 pin, %7, %8;\n\t"
        "setp.eq.and.b32 pa, %6, 0, pin;\n\t"
        "setp.eq.and.b32 pc, %6, 8, pin;\n\t"
        "setp.eq.and.b32 pg, %6, 16, pin;\n\t"
        "setp.eq.and.b32 pt, %6, 24, pin;\n\t"
        "@pa add.rn.f32 %0, %0, %5;\n\t"
        "@pc add.rn.f32 %1, %1, %5;\n\t"
        "@pg add.rn.f32 %2, %2, %5;\n\t"
        "@pt add.rn.f32 %3, %3, %5;\n\t"
        "shl.b32 inc, %9, %6;\n\t"
        "@pin add.u32 %4, %4, inc;\n\t"
        "}"
        : "+f"(wA), "+f"(wC), "+f"(wG), "+f"(wT), "+r"(c8)
        : "f"(w), "r"(b8), "r"(p), "r"(len), "r"(1u));
}

// The whole MSA stage of one anchor (local index ai) for one CTA. Every
// early return is taken by all threads of the CTA together.
// QB: the quality encoding the sums read (0: qualities unused, else 1, 2 or
// 8 bits per quality).
template <int BLOCK, int QB, bool EMIT>
__device__ __forceinline__ void
msa_anchor(const DevOptions& o, const DevReads& r, uint32_t first, uint32_t ai, const MsaGrid& grid,
           const uint32_t* __restrict__ cand_ids, const uint32_t* __restrict__ seg_off,
           const uint32_t* __restrict__ seg_cnt, const AlignRes* __restrict__ ares,
           CandRec* __restrict__ recs, const MsaOut& out, int* __restrict__ status) {
    constexpr int NWARP = BLOCK / 32;
    extern __shared__ __align__(16) unsigned char dsm[];
    __shared__ float s_qw[QB == 8 ? 256 : 1];
    __shared__ float s_qwc[4];               // weight of a 1- or 2-bit quality code
    // by slot (0: the anchor): the row, its weight, weight * weight of a 1- or
    // 2-bit quality code
    __shared__ uint2 s_slot[kStageMax + 1];  // {id, shift (16 bits) | length << 16 | reverse complement << 31}
    __shared__ float s_w[kStageMax + 1];
    __shared__ __align__(16) float s_wq[kStageMax + 1][4];
    // the rows of the sums in list order, {byte offset of the staged row,
    // -shift, length, 16 * slot}, one entry of length 0 behind the last
    __shared__ uint4 s_ent[kStageMax + 2];
    __shared__ uint32_t s_dis[kMaxLen / 16];  // disputed columns, bit 30 - 2 * (position % 16)
    __shared__ __align__(16) int s_diff[kMaxLen + 4]; // coverage changes by anchor position
    __shared__ int s_red[NWARP + 1];
    __shared__ int s_nd, s_sig, s_min, s_mincov, s_maxcov, s_bases, s_ndec;
    __shared__ float s_avg, s_defect;
    __shared__ uint16_t s_dec[EMIT ? kMaxLen : 1];   // decision positions of the anchor (EMIT)

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t a = first + ai;
    const uint32_t off = seg_off[ai], cnt = seg_cnt[ai];
    const int La = r.len[a];
    const int mlen = r.max_len;
    char* aout = out.seq + (size_t)ai * mlen;
    const int nstage = grid.rows, rw = grid.rw, G = grid.words, E = grid.edge, wpg = grid.wpg;
    const int nwa = (La + 15) >> 4;
    // dynamic shared memory (msa_smem_bytes)
    uint32_t* s_raw = (uint32_t*)dsm;                        // [nstage + 1][rw]
    float* s_sup = (float*)(dsm + msa_round16((size_t)(nstage + 1) * rw * 4));   // support by anchor position
    ushort4* s_cnt4 = (ushort4*)((unsigned char*)s_sup + msa_round16((size_t)mlen * 4));   // counts A C G T (disputed)
    // per anchor position: column weight sum, consensus weight, weight of the
    // anchor's base (EMIT only)
    float* s_fw = (float*)((unsigned char*)s_cnt4 + (size_t)(mlen + (mlen & 1)) * 8);
    uint16_t* s_cov = (uint16_t*)((unsigned char*)s_fw + (EMIT ? msa_round16((size_t)3 * mlen * 4) : 0));
    int16_t* s_col = (int16_t*)((unsigned char*)s_cov + msa_round16((size_t)mlen * 2));   // columns of the sums
    // per grid column: consensus | plain rule's base << 2 | anchor's base << 4
    uint8_t* s_cons = (uint8_t*)s_col + msa_round16((size_t)16 * G * 2);

    if (cnt == 0) {
        if (tid == 0) { out.status[ai] = 0; out.nedits[ai] = 0; }
        return;
    }
    // block-wide rank of the threads with keep set (0/1); *tot gets their number
    auto block_rank = [&](bool keep, int* tot) {
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        __syncthreads();
        if (lane == 0) s_red[warp] = __popc(m);
        __syncthreads();
        int pre = 0, all = 0;
#pragma unroll
        for (int w = 0; w < NWARP; ++w) { const int sv = s_red[w]; if (w < warp) pre += sv; all += sv; }
        *tot = all;
        return pre + __popc(m & ((1u << lane) - 1u));
    };

    // ---- quality weights (qualityscoreweights.hpp:12-44) ----
    if constexpr (QB == 8) for (int i = tid; i < 256; i += BLOCK) s_qw[i] = c_qweight[i];
    if (tid < 4) {
        // the characters a 2- or 1-bit code stands for (qualityscorecompression.hpp:121-145)
        const uint32_t ch = QB == 2 ? (tid == 0 ? '$' : tid == 1 ? '(' : tid == 2 ? '1' : '9')
                                    : (tid == 1 ? '5' : '(');
        s_qwc[tid] = c_qweight[ch];
        s_wq[0][tid] = c_qweight[ch];                        // the anchor's factor is 1
    }
    if (tid == 0) {
        s_slot[0] = make_uint2(a, (uint32_t)La << 16);
        s_w[0] = 1.0f;
    }
    auto slot_beg = [&](int k) { return (int)(int16_t)s_slot[k].y; };
    auto slot_len = [&](int k) { return (int)((s_slot[k].y >> 16) & 0x7fffu); };

    // ---- alignment filters (corrector.hpp:982-1211), ordered compaction ----
    const float base = fmul_rn(o.estimated_errorrate, 1.0f);
    const float base2 = fmul_rn(2.0f, base), base3 = fmul_rn(3.0f, base), base4 = fmul_rn(4.0f, base);
    // the first candidate of each thread: its alignment, mismatch ratio, id
    // and length stay in registers for the compaction below (the id and
    // length loads overlap the counting)
    AlignRes ar0{};
    float mr0 = 0.0f;
    uint32_t id0 = 0;
    int len0 = 0;
    // counts below the three thresholds and of aligned candidates, 16 bits
    // each (a list holds fewer than 2^14 candidates)
    uint32_t c01 = 0, c23 = 0;
    for (uint32_t i = tid; i < cnt; i += BLOCK) {
        const AlignRes ar = ares[off + i];
        float mr = 0.0f;
        if (ar.orient != 3) {
            mr = fdiv_rn((float)ar.nops, (float)ar.overlap);
            c01 += (mr < base2 ? 1u : 0u) + (mr < base3 ? 65536u : 0u);
            c23 += (mr < base4 ? 1u : 0u) + 65536u;
        }
        if (i == (uint32_t)tid) {
            ar0 = ar;
            mr0 = mr;
            id0 = cand_ids[off + i];
            len0 = r.len[id0];
        }
    }
    c01 = __reduce_add_sync(0xffffffffu, c01);
    c23 = __reduce_add_sync(0xffffffffu, c23);
    __shared__ uint32_t s_cnt[NWARP][2];
    if (lane == 0) { s_cnt[warp][0] = c01; s_cnt[warp][1] = c23; }
    __syncthreads();
    c01 = c23 = 0;
#pragma unroll
    for (int w = 0; w < NWARP; ++w) { c01 += s_cnt[w][0]; c23 += s_cnt[w][1]; }
    if ((c23 >> 16) == 0) {
        if (tid == 0) { out.status[ai] = 0; out.nedits[ai] = 0; }
        return;
    }
    float thr = -3.402823466e+38f;
    {
        const float good = fmul_rn(o.estimated_coverage, o.m_coverage);
        const int n2 = c01 & 0xFFFF, n3 = c01 >> 16, n4 = c23 & 0xFFFF;
        if (n2 > 0 || n3 > 0 || n4 > 0) {
            if ((float)n2 >= good) thr = base2;
            else if ((float)n3 >= good) thr = base3;
            else if ((float)n4 >= good) thr = base4;
        }
    }
    // slot k of the staged rows
    auto fill_slot = [&](int k, const CandRec& rec) {
        s_slot[k] = make_uint2(rec.id, (uint32_t)(uint16_t)rec.shift | (uint32_t)rec.len << 16 |
                                           (rec.orient == 1 ? 0u : 0x80000000u));
        s_w[k] = rec.weight;
        if constexpr (QB == 1 || QB == 2)
            *reinterpret_cast<float4*>(&s_wq[k][0]) =
                make_float4(fmul_rn(rec.weight, s_qwc[0]), fmul_rn(rec.weight, s_qwc[1]),
                            fmul_rn(rec.weight, s_qwc[2]), fmul_rn(rec.weight, s_qwc[3]));
    };
    // every candidate fits the staged rows: the survivors' records go straight
    // to shared memory (else to the global records, staged chunk by chunk)
    const bool direct = cnt <= (uint32_t)nstage;
    int V = 0;
    for (uint32_t c = 0; c < cnt; c += BLOCK) {
        const uint32_t i = c + tid;
        bool keep = false;
        AlignRes ar = ar0;
        float mr = mr0;
        if (i < cnt) {
            if (c) {
                ar = ares[off + i];
                if (ar.orient != 3) mr = fdiv_rn((float)ar.nops, (float)ar.overlap);
            }
            if (ar.orient != 3)
                keep = o.paired_end ? (ar.paired || mr < o.paired_filter_threshold) : (mr < thr);
        }
        int tot;
        const int pre = block_rank(keep, &tot);
        if (keep) {
            CandRec rec;
            rec.id = c ? cand_ids[off + i] : id0;
            rec.shift = ar.shift;
            rec.len = (uint16_t)(c ? r.len[rec.id] : len0);
            // calculateOverlapWeight: 1 - sqrtf(nOps / (overlap * maxMismatchRatio))
            rec.weight = fsub_rn(1.0f, __fsqrt_rn(fdiv_rn((float)ar.nops, fmul_rn((float)ar.overlap, o.max_error_rate))));
            rec.orient = ar.orient;
            const int k = V + pre;
            if (direct) fill_slot(k + 1, rec);
            else recs[off + k] = rec;
        }
        V += tot;
    }
    if (V == 0) {
        if (tid == 0) { out.status[ai] = 0; out.nedits[ai] = 0; }
        return;
    }

    const int sp = r.seq_pitch, qp = r.qual_pitch;
    const uint32_t* arow = r.seq + (size_t)a * sp;
    // Word g of slot k, a thread each: 16 codes from row position 16 (g - E) -
    // shift on, reverse-complement rows turned into the alignment's
    // orientation (bases reversed and complemented, qualities reversed over
    // the whole quality pitch: reverseQualitiesOfRCAlignments,
    // corrector.hpp:1227-1239). load: from the read storage (else the words
    // are staged already); disputed columns are marked on the way.
    // Slots k0 .. k0 + n - 1, or with list the slots of entries 1 .. n.
    auto scan_words = [&](int n, int k0, bool load, bool list) {
#pragma unroll 1
        for (int idx = tid; idx < n * G; idx += BLOCK) {
            const int e = G > 1 ? (int)__umulhi((uint32_t)idx, grid.magic) : idx, g = idx - e * G;
            const int k = list ? (int)(s_ent[e + 1].w >> 4) : k0 + e;
            const int p0 = 16 * (g - E);                     // anchor position of the word's first code
            const uint2 slot = s_slot[k];
            const int sft = (int)(int16_t)slot.y, L = (int)((slot.y >> 16) & 0x7fffu);
            const int lo = max(sft - p0, 0), hi = min(sft + L - p0, 16);
            if (lo >= hi) continue;                          // the row does not reach the word
            uint32_t* dst = s_raw + k * rw + g * wpg;
            uint32_t ws;
            if (load) {
                const bool rev = slot.y >> 31;
                const size_t id = slot.x;
                const int q0 = p0 - sft;
                ws = window2(r.seq + id * sp, sp, staged_start(rev, L, q0, 16, 0));
                if (rev) ws = ~rev2(ws);                     // reversed, complemented: A<->T, C<->G
                if constexpr (QB == 2) {
                    uint32_t wq = window2(r.qual + id * qp, qp, staged_start(rev, mlen, q0, 16, 0));
                    if (rev) wq = rev2(wq);
                    *reinterpret_cast<uint2*>(dst) = make_uint2(ws, wq);
                } else {
                    dst[0] = ws;
                    if constexpr (QB == 1) {
                        uint32_t wq = window1(r.qual + id * qp, qp, staged_start(rev, mlen, q0, 16, 0));
                        if (rev) wq = __brev(wq) << 16;
                        dst[1] = wq;
                    } else if constexpr (QB == 8) {
#pragma unroll
                        for (int h = 0; h < 4; ++h) {
                            uint32_t wq = window8(r.qual + id * qp, qp, staged_start(rev, mlen, q0, 4, h));
                            if (rev) wq = __byte_perm(wq, 0u, 0x0123);
                            dst[1 + h] = wq;
                        }
                    }
                }
            } else {
                ws = dst[0];
            }
            if (p0 >= 0 && p0 < La) {
                const int end = min(hi, La - p0);
                uint32_t d = ws ^ __ldg(arow + (p0 >> 4));
                d = (d | (d >> 1)) & 0x55555555u & (0xFFFFFFFFu >> (2 * lo));
                if (end < 16) d &= ~(0xFFFFFFFFu >> (2 * max(end, 0)));
                if (d) atomicOr(&s_dis[p0 >> 4], d);
            }
        }
    };
    // entries of slots 1 .. n (and the anchor's, entry 0, when with_anchor)
    auto put_entry = [&](int e, int k, int len) {
        s_ent[e] = make_uint4((uint32_t)(k * rw * 4), (uint32_t)-slot_beg(k), (uint32_t)len, (uint32_t)k * 16u);
    };
    // a chunk of the global records into slots 1 .. n
    auto stage_chunk = [&](int c, int n) {
        __syncthreads();
        for (int k = tid; k < n; k += BLOCK) {
            fill_slot(k + 1, recs[off + c + k]);
            put_entry(k + 1, k + 1, slot_len(k + 1));
        }
        if (tid == 0) put_entry(n + 1, 0, 0);
        __syncthreads();
        scan_words(n, 1, true, false);
        __syncthreads();
    };
    // base (2-bit, in the candidate's aligned orientation) of staged slot k at
    // anchor position p
    auto staged_base = [&](int k, int p) -> uint32_t {
        return (s_raw[k * rw + ((p >> 4) + E) * wpg] >> (30 - 2 * (p & 15))) & 3u;
    };
    const bool persistent = V <= nstage;      // all rows stay staged across rebuilds
    const int sigThr = f2i_rz(fmul_rn((float)o.coverage_int, 0.3f));
    int nalive = V;
    bool outside = false;                     // the sums of candidate correction's columns outside the anchor
    bool hq = false;
    int iter = 0;
    if (persistent && !direct) {
        __syncthreads();
        for (int k = tid; k < V; k += BLOCK) fill_slot(k + 1, recs[off + k]);
    }
    for (int i = tid; i < G * wpg; i += BLOCK) s_raw[i] = 0u;

    for (;;) {
        int ncol;
        if (!outside) {
            // ---- disputed columns, coverage ----
            for (int i = tid; i < (kMaxLen + 4) / 4; i += BLOCK) reinterpret_cast<int4*>(s_diff)[i] = make_int4(0, 0, 0, 0);
            if (tid < kMaxLen / 16) s_dis[tid] = tid == 0 && sigThr <= 0 ? 0x40000000u : 0u;   // counts of 0 are significant
            if (tid == 0) { s_sig = 0x7fffffff; s_bases = 0; s_defect = 0.0f; s_ndec = 0; s_red[NWARP] = 0; }
            __syncthreads();
            if (iter == 0) scan_words(1, 0, true, false);    // the anchor
            int sl = 0;
            auto add_cover = [&](int sft, int L) {
                const int b = max(sft, 0), e = min(sft + L, La);
                if (b < e) { atomicAdd(&s_diff[b], 1); atomicAdd(&s_diff[e], -1); }
                sl += L;
            };
            if (persistent) {
                scan_words(nalive, 1, iter == 0, iter > 0);
                for (int i = tid; i < nalive; i += BLOCK) {
                    const int k = iter == 0 ? i + 1 : (int)(s_ent[i + 1].w >> 4);
                    if (iter == 0) put_entry(i + 1, k, slot_len(k));
                    add_cover(slot_beg(k), slot_len(k));
                }
                if (tid == 0) { put_entry(0, 0, La); put_entry(nalive + 1, 0, 0); }
            } else {
                for (int c = 0; c < nalive; c += nstage) {
                    const int n = min(nstage, nalive - c);
                    stage_chunk(c, n);
                    for (int k = tid; k < n; k += BLOCK) add_cover(slot_beg(k + 1), slot_len(k + 1));
                }
                if (tid == 0) {
                    put_entry(0, 0, La);
                    if (nalive == 0) put_entry(1, 0, 0);
                }
            }
            if (out.elem_count) {
                sl = __reduce_add_sync(0xffffffffu, sl);
                if (lane == 0) atomicAdd(&s_bases, sl);
            }
            __syncthreads();
            if (warp == 0) {                                  // the list of disputed columns
                uint32_t d = lane < nwa ? s_dis[lane] : 0u;
                const int n = __popc(d);
                int x = n;
#pragma unroll
                for (int q = 1; q < 32; q <<= 1) { const int y = __shfl_up_sync(0xffffffffu, x, q); if (lane >= q) x += y; }
                if (lane == 31) { s_nd = x; s_min = x < La ? __float_as_int(1.0f) : 0x7f7fffff; }
                int at = x - n;
                while (d) {
                    const int bit = 31 - __clz(d);
                    d &= ~(1u << bit);
                    s_col[at++] = (int16_t)(16 * lane + (30 - bit) / 2);
                }
            } else if (warp == 1) {                           // coverage: prefix sums, 8 positions a lane
                int v[8], sum = 0;
                const int4 lo4 = *reinterpret_cast<const int4*>(&s_diff[8 * lane]);
                const int4 hi4 = *reinterpret_cast<const int4*>(&s_diff[8 * lane + 4]);
                v[0] = lo4.x; v[1] = lo4.y; v[2] = lo4.z; v[3] = lo4.w; v[4] = hi4.x; v[5] = hi4.y; v[6] = hi4.z; v[7] = hi4.w;
#pragma unroll
                for (int q = 0; q < 8; ++q) { sum += v[q]; v[q] = sum; }
                int x = sum;
#pragma unroll
                for (int q = 1; q < 32; q <<= 1) { const int y = __shfl_up_sync(0xffffffffu, x, q); if (lane >= q) x += y; }
                const int before = x - sum + 1;               // the anchor itself
                int mn = 0x7fffffff, mx = 0;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int p = 8 * lane + q, cv = before + v[q];
                    if (p < La) {
                        mn = min(mn, cv);
                        mx = max(mx, cv);
                        if constexpr (EMIT) s_cov[p] = (uint16_t)cv;
                    }
                }
                mn = __reduce_min_sync(0xffffffffu, mn);
                mx = __reduce_max_sync(0xffffffffu, mx);
                if (lane == 0) { s_mincov = mn; s_maxcov = mx; }
            } else {                                          // undisputed until summed
                for (int p = tid - 64; p < La; p += BLOCK - 64) {
                    const uint32_t ob = staged_base(0, p);
                    s_cons[p + 16 * E] = (uint8_t)(ob * 21u);
                    s_sup[p] = 1.0f;
                }
            }
            if (tid == 0 && out.elem_count) {
                const unsigned long long tot = (unsigned long long)(La + s_bases);
                atomicAdd(out.elem_count, tot);
                if (iter > 0 && out.rebuild_count) {
                    atomicAdd(out.rebuild_count, tot);
                    if (iter == 1) atomicAdd(out.rebuild_count + 1, 1ull);
                }
            }
            __syncthreads();
            ncol = s_nd;
        } else {
            ncol = s_nd;
        }

        // ---- column sums (anchor first, then candidates in list order) and
        //      consensus (findConsensus, msa.cpp:135-157): 32 listed columns
        //      a warp, lane = column ----
        int mism = 0;
        float defect = 0.0f;                                 // 1 - support of the lane's columns
        const int nblk = (ncol + 31) >> 5;
        const int nchunk = persistent ? 1 : max(1, (nalive + nstage - 1) / nstage);
#pragma unroll 1
        for (int b0 = 0; b0 < nblk; b0 += NWARP) {
            const int ci = 32 * (b0 + warp) + lane;
            const bool act = ci < ncol;
            const int p = act ? s_col[ci] : 0;               // anchor position of the lane's column
            uint32_t cAC = 0u, cGT = 0u;                     // 16-bit counts: A | C << 16, G | T << 16
            float wA = 0.0f, wC = 0.0f, wG = 0.0f, wT = 0.0f;
            // the lane's word in every staged row (byte offset) and its bits
            // there, as rotations that bring the base to bits 3-4 (base * 8)
            // and the quality code to bits 2-3 (2-bit) or bit 2 (1-bit), i.e.
            // the byte offset of its weight
            const int gw = (p >> 4) + E;
            const uint32_t rb8 = (uint32_t)(59 - 2 * (p & 15)) & 31u;
            const int loff = gw * wpg * 4;
            uint32_t rq = 0u;
            int qoff = 0;
            if constexpr (QB == 2) rq = (uint32_t)(60 - 2 * (p & 15)) & 31u;
            if constexpr (QB == 1) rq = (uint32_t)(61 - (p & 15)) & 31u;
            if constexpr (QB == 8) { rq = 8u * (uint32_t)(p & 3); qoff = 4 + 4 * ((p & 15) >> 2); }
            const unsigned char* rawb = reinterpret_cast<const unsigned char*>(s_raw) + loff;
            const unsigned char* wqb = reinterpret_cast<const unsigned char*>(&s_wq[0][0]);
#pragma unroll 1
            for (int ch = 0; ch < nchunk; ++ch) {
                int n = nalive;
                if (!persistent) {
                    n = min(nstage, nalive - ch * nstage);
                    if (nchunk > 1) stage_chunk(ch * nstage, n);
                }
                if (32 * (b0 + warp) >= ncol) continue;      // warp-uniform (no barrier below)
                uint32_t c8 = 0u;       // the chunk's 8-bit counts A | C << 8 | G << 16 | T << 24: at most 129 rows
#pragma unroll 1
                for (int i = ch == 0 ? 0 : 1; i <= n; i += 2) {
                    uint32_t bb[2];
                    float ww[2];
                    int pp[2], ll[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const uint4 e = s_ent[i + u];
                        const unsigned char* wp = rawb + e.x;
                        uint32_t sw, qv = 0u;
                        if constexpr (QB == 2) {
                            const uint2 t2 = *reinterpret_cast<const uint2*>(wp);
                            sw = t2.x;
                            qv = t2.y;
                        } else {
                            sw = *reinterpret_cast<const uint32_t*>(wp);
                            if constexpr (QB == 1) qv = *reinterpret_cast<const uint32_t*>(wp + 4);
                            if constexpr (QB == 8) qv = *reinterpret_cast<const uint32_t*>(wp + qoff);
                        }
                        bb[u] = __funnelshift_r(sw, sw, rb8) & 24u;
                        if constexpr (QB == 0) ww[u] = s_w[e.w >> 4];
                        else if constexpr (QB == 2)
                            ww[u] = *reinterpret_cast<const float*>(wqb + (e.w + (__funnelshift_r(qv, qv, rq) & 12u)));
                        else if constexpr (QB == 1)
                            ww[u] = *reinterpret_cast<const float*>(wqb + (e.w + (__funnelshift_r(qv, qv, rq) & 4u)));
                        else ww[u] = fmul_rn(s_w[e.w >> 4], s_qw[(qv >> rq) & 0xFFu]);
                        pp[u] = p + (int)e.y;
                        ll[u] = (int)e.z;
                    }
#pragma unroll
                    for (int u = 0; u < 2; ++u) msa_add8(wA, wC, wG, wT, c8, bb[u], ww[u], pp[u], ll[u]);
                }
                cAC += (c8 & 0xFFu) | ((c8 & 0xFF00u) << 8);
                cGT += ((c8 >> 16) & 0xFFu) | ((c8 >> 24) << 16);
            }
            if (act) {
                uint32_t cs = 0; float cw = wA;
                if (wC > cw) { cs = 1; cw = wC; }
                if (wG > cw) { cs = 2; cw = wG; }
                if (wT > cw) { cs = 3; cw = wT; }
                if (outside) {
                    s_cons[p + 16 * E] = (uint8_t)cs;
                } else {
                    const float colw = __fadd_rn(__fadd_rn(__fadd_rn(wA, wC), wG), wT);
                    const float sup = fdiv_rn(cw, colw);
                    const uint32_t nA = cAC & 0xFFFFu, nC = cAC >> 16, nG = cGT & 0xFFFFu, nT = cGT >> 16;
                    const uint32_t ob = staged_base(0, p);
                    // origCoverages: count of the anchor's base
                    const uint32_t oc = ob == 0 ? nA : ob == 1 ? nC : ob == 2 ? nG : nT;
                    const uint32_t rule = sup > 0.90f && oc <= 2u ? cs : ob;
                    s_cons[p + 16 * E] = (uint8_t)(cs | rule << 2 | ob << 4);
                    s_sup[p] = sup;
                    s_cnt4[p] = make_ushort4((uint16_t)nA, (uint16_t)nC, (uint16_t)nG, (uint16_t)nT);
                    mism |= cs != ob;
                    defect = __fadd_rn(defect, fsub_rn(1.0f, sup));
                    const bool sig = (cs != 0 && sigThr <= (int)nA) || (cs != 1 && sigThr <= (int)nC) ||
                                     (cs != 2 && sigThr <= (int)nG) || (cs != 3 && sigThr <= (int)nT);
                    if (sig) atomicMin(&s_sig, p);
                    atomicMin(&s_min, __float_as_int(sup));   // supports are positive
                    if constexpr (EMIT) {
                        s_fw[p] = colw;
                        s_fw[mlen + p] = cw;
                        s_fw[2 * mlen + p] = ob == 0 ? wA : ob == 1 ? wC : ob == 2 ? wG : wT;
                    }
                }
            }
        }
        if (!outside && 32 * warp < ncol) {                  // warp-uniform
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) defect = __fadd_rn(defect, __shfl_xor_sync(0xffffffffu, defect, d));
            if (lane == 0) atomicAdd(&s_defect, defect);
        }
        mism = __syncthreads_or(mism);
        if (outside) break;

        // ---- refinement: findCandidatesOfDifferentRegion (msa.cpp:532-734) ----
        const int col = s_sig;                               // first column with a significant other base
        if (iter < 5 && mism && col != 0x7fffffff) {
            int foundBase = -1;               // the last qualifying base index wins (:591-601)
            {
                const ushort4 c4 = s_cnt4[col];
                const int cs = s_cons[col + 16 * E] & 3;
                if (cs != 0 && sigThr <= (int)c4.x) foundBase = 0;
                if (cs != 1 && sigThr <= (int)c4.y) foundBase = 1;
                if (cs != 2 && sigThr <= (int)c4.z) foundBase = 2;
                if (cs != 3 && sigThr <= (int)c4.w) foundBase = 3;
            }
            const bool keepMatching = (int)staged_base(0, col) == foundBase;
            // per candidate: remove? (discard_rows :622-665); veto by weight >= 0.90 (:672-689)
            auto removes = [&](int b) { return keepMatching ? (b != foundBase) : (b == foundBase); };
            auto record_removed = [&](const CandRec& rc) {
                const int q = col - rc.shift;
                if (q < 0 || q >= (int)rc.len) return false;
                const uint32_t* row = r.seq + (size_t)rc.id * sp;
                return removes(rc.orient == 1 ? (int)base_at(row, q) : (int)(base_at(row, rc.len - 1 - q) ^ 3u));
            };
            auto slot_removed = [&](int k) {
                const int q = col - slot_beg(k);
                return q >= 0 && q < slot_len(k) && removes((int)staged_base(k, col));
            };
            int nrem = 0, veto = 0;
            for (int i = tid; i < nalive; i += BLOCK) {
                bool rem;
                float w;
                if (persistent) {
                    const int k = (int)(s_ent[i + 1].w >> 4);
                    rem = slot_removed(k);
                    w = s_w[k];
                } else {
                    const CandRec rc = recs[off + i];
                    rem = record_removed(rc);
                    w = rc.weight;
                }
                nrem |= rem;
                veto |= rem && w >= 0.90f;
            }
            const int anyVeto = __syncthreads_or(veto);
            const int anyRem = __syncthreads_or(nrem);
            if (!anyVeto && anyRem) {             // else the rebuilt MSA would be identical
                // ordered compaction of the survivors
                int newV = 0;
                for (int c = 0; c < nalive; c += BLOCK) {
                    const int i = c + tid;
                    bool keep = false;
                    uint4 ent = make_uint4(0u, 0u, 0u, 0u);
                    CandRec rc{};
                    if (i < nalive) {
                        if (persistent) { ent = s_ent[i + 1]; keep = !slot_removed((int)(ent.w >> 4)); }
                        else { rc = recs[off + i]; keep = !record_removed(rc); }
                    }
                    int tot;
                    const int pre = block_rank(keep, &tot);
                    __syncthreads();
                    if (keep) {
                        if (persistent) s_ent[1 + newV + pre] = ent;
                        else recs[off + newV + pre] = rc;
                    }
                    newV += tot;
                    __syncthreads();
                }
                nalive = newV;
                ++iter;
                __syncthreads();
                continue;
            }
        }

        // ---- MSA properties (getMSAProperties, msa.cpp:304-376) ----
        // The reference's average support is one serial chain of float adds
        // over the anchor's columns. What it decides are comparisons with two
        // thresholds, so the average from the disputed columns' defects
        // settles them unless it comes within 1e-4 of one: both averages are
        // within 1e-5 of the exact one (256 adds below 256, each half an ulp
        // of 2^-16 at most). Otherwise, and for the decision rows' features,
        // the chain is added up. (1,200 of 9,500 warp instructions per anchor
        // and a wait of the whole CTA for one lane: 13.0 -> 12.6 ms per 1M
        // reads.)
        auto serial_average = [&]() {         // into s_avg, by warp 0; the supports read four at a time
            float sum = 0.0f;
            if (warp == 0 && lane == 0) {
                const float4* v4 = reinterpret_cast<const float4*>(s_sup);
                int p = 0;
                for (; p + 4 <= La; p += 4) {
                    const float4 v = v4[p >> 2];
                    sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, v.x), v.y), v.z), v.w);
                }
                for (; p < La; ++p) sum = __fadd_rn(sum, s_sup[p]);
                s_avg = fdiv_rn(sum, (float)La);
            }
        };
        const float minSup = __int_as_float(s_min);
        const int minCov = s_mincov;
        bool allGood;
        {
            const float e = o.estimated_errorrate;
            const float avgThr = fsub_rn(1.0f, fmul_rn(1.0f, e));
            const float minThr = fsub_rn(1.0f, fmul_rn(3.0f, e));
            const float covThr = fmul_rn(fdiv_rn(o.m_coverage, 6.0f), o.estimated_coverage);
            // HQ: the smallest percentage pc in [0, pct] whose thresholds hold
            // is at most half of pct; they loosen as pc grows, so the largest
            // such pc decides
            const int pct = (int)ceilf(fmul_rn(e, 100.0f));
            const float fac = fdiv_rn((float)(pct >> 1), 100.0f);
            const float hqAvg = fsub_rn(1.0f, fmul_rn(1.0f, fac)), hqMin = fsub_rn(1.0f, fmul_rn(3.0f, fac));
            float avg = fdiv_rn(fsub_rn((float)La, s_defect), (float)La);
            if (!(fabsf(avg - avgThr) > 1e-4f && fabsf(avg - hqAvg) > 1e-4f)) {      // block-uniform
                serial_average();
                __syncthreads();
                avg = s_avg;
            }
            allGood = fgeq(avg, avgThr) && fgeq(minSup, minThr) && fgeq((float)minCov, covThr);
            hq = allGood && pct >= 0 && fgeq(avg, hqAvg) && fgeq(minSup, hqMin);
        }

        // ---- anchor correction (getCorrectedAnchor, msa.cpp:379-453) ----
        if (nalive == 0) {
            if (tid == 0) { out.status[ai] = 0; out.nedits[ai] = 0; }
            return;   // nCandidates == 0: not corrected; no candidate corrections either
        }
        int diffs = 0;
        for (int p = tid; p < La; p += BLOCK) {
            const uint32_t e = s_cons[p + 16 * E];
            const uint32_t cb = allGood ? e & 3u : (e >> 2) & 3u;
            aout[p] = "ACGT"[cb];
            diffs += cb != e >> 4;
        }
        diffs = __reduce_add_sync(0xffffffffu, diffs);
        if (lane == 0 && diffs) atomicAdd(&s_red[NWARP], diffs);
        __syncthreads();
        if (tid == 0) {
            const int nd = s_red[NWARP];
            const bool useEdits = !r.ambig[a] && nd <= La / 7;
            out.status[ai] = (uint8_t)(1 | (hq ? 2 : 0) | (useEdits ? 4 : 0));
            out.nedits[ai] = useEdits ? nd : 0;
        }

        // ---- decision columns (correctAnchorClf, corrector.hpp:1448-1472) ----
        // Non-HQ MSAs only: each anchor position whose base differs from the
        // consensus (and whose column reaches clf_min_coverage) becomes a row of
        // 24 features. The plain rule's base stays in aout; with the network
        // deciding, k_clf_apply overwrites it from the row's logit.
        if constexpr (EMIT) {
            if (!hq) {
                // the decision positions are listed first (any order: rows are
                // appended through a global counter), so that their features are
                // computed by consecutive threads instead of by the warps that
                // happen to hold one
                auto mismatch = [&](int p) { const uint32_t e = s_cons[p + 16 * E]; return (e & 3u) != e >> 4; };
                // the anchor's quality weight at position q
                auto anchor_weight = [&](int q) -> float {
                    const uint32_t* w = s_raw + ((q >> 4) + E) * wpg;
                    if constexpr (QB == 0) return 1.0f;
                    else if constexpr (QB == 2) return s_wq[0][(w[1] >> (30 - 2 * (q & 15))) & 3u];
                    else if constexpr (QB == 1) return s_wq[0][(w[1] >> (31 - (q & 15))) & 1u];
                    else return s_qw[(w[1 + ((q & 15) >> 2)] >> (8 * (q & 3))) & 0xFFu];
                };
                int nm = 0;
                for (int p = tid; p < La; p += BLOCK) {
                    const bool mis = mismatch(p);
                    nm += mis;
                    if (mis && (int)s_cov[p] >= o.clf_min_coverage) s_dec[atomicAdd(&s_ndec, 1)] = (uint16_t)p;
                }
                nm = __reduce_add_sync(0xffffffffu, nm);
                if (lane == 0) s_red[warp] = nm;
                serial_average();
                __syncthreads();
                int nmis = 0;
#pragma unroll
                for (int w = 0; w < NWARP; ++w) nmis += s_red[w];
                const int maxCov = s_maxcov;
                const float avgSup = s_avg;
                const float Ec = o.estimated_coverage;
                const int ndec = s_ndec;
                for (int i = tid; i < ndec; i += BLOCK) {
                    const int p = s_dec[i];
                    const uint32_t ce = s_cons[p + 16 * E];
                    const uint32_t ob = ce >> 4, cb = ce & 3u;
                    const float cov = (float)s_cov[p];
                    const ushort4 c4 = s_cnt4[p];
                    const int oc = ob == 0 ? c4.x : ob == 1 ? c4.y : ob == 2 ? c4.z : c4.w;
                    const int cc = cb == 0 ? c4.x : cb == 1 ? c4.y : cb == 2 ? c4.z : c4.w;
                    const float wsum = s_fw[p], wc = s_fw[mlen + p], wo = s_fw[2 * mlen + p];
                    float x[kNumFeatures];
                    x[0] = fdiv_rn((float)oc, cov);
                    x[1] = fdiv_rn(wo, wsum);
                    x[2] = fdiv_rn(wo, (float)oc);
                    x[3] = fdiv_rn((float)cc, cov);
                    x[4] = s_sup[p];
                    x[5] = fdiv_rn(wc, (float)cc);
                    x[6] = fdiv_rn(wsum, cov);
                    x[7] = fdiv_rn(cov, Ec);
                    x[8] = fdiv_rn(wsum, Ec);
                    x[9] = avgSup;
                    x[10] = minSup;
                    x[11] = fdiv_rn((float)maxCov, Ec);
                    x[12] = fdiv_rn((float)minCov, Ec);
                    x[13] = anchor_weight(p);
                    x[14] = fdiv_rn((float)min(p, La - 1 - p), (float)La);
                    x[15] = fdiv_rn(fsub_rn(fsub_rn(wsum, wc), wo), wsum);
                    const int lo = max(p - 3, 0), hi = min(p + 3, La - 1);
                    float ssum = 0.0f, smin = s_sup[lo], qsum = 0.0f;
                    for (int q = lo; q <= hi; ++q) {
                        const float sv = s_sup[q];
                        ssum = __fadd_rn(ssum, sv);
                        if (sv < smin) smin = sv;
                        qsum = __fadd_rn(qsum, anchor_weight(q));
                    }
                    const float nwin = (float)(hi - lo + 1);
                    x[16] = fdiv_rn(ssum, nwin);
                    x[17] = smin;
                    x[18] = fdiv_rn((float)nmis, (float)La);
                    int nloc = 0;
                    for (int q = max(p - 5, 0); q <= min(p + 5, La - 1); ++q) nloc += q != p && mismatch(q);
                    x[19] = fdiv_rn((float)nloc, 10.0f);
                    x[20] = fdiv_rn((float)nalive, Ec);
                    x[21] = allGood ? 1.0f : 0.0f;
                    x[22] = (allGood || (s_sup[p] > 0.90f && oc <= 2)) ? 1.0f : 0.0f;
                    x[23] = fdiv_rn(qsum, nwin);
                    const unsigned long long slot = atomicAdd(out.feat_count, 1ull);
                    if (slot >= out.feat_cap) { atomicOr(status, kStatusFeatOverflow); continue; }
                    float4* dst = reinterpret_cast<float4*>(out.feat + slot * kNumFeatures);
#pragma unroll
                    for (int q = 0; q < kNumFeatures / 4; ++q) dst[q] = make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
                    out.feat_read[slot] = a;
                    out.feat_meta[slot] = (uint32_t)p | (ob << 16) | (cb << 18);
                }
            }
        }
        if (!hq || !o.correct_candidates) return;

        // ---- columns outside the anchor that its candidates' corrections
        //      read: up to new_columns on each side, as far as rows reach ----
        int mn = 0, mx = La;
        for (int i = tid; i < nalive; i += BLOCK) {
            int sft, L;
            if (persistent) { const int k = (int)(s_ent[i + 1].w >> 4); sft = slot_beg(k); L = slot_len(k); }
            else { const CandRec rc = recs[off + i]; sft = rc.shift; L = rc.len; }
            mn = min(mn, sft);
            mx = max(mx, sft + L);
        }
        mn = __reduce_min_sync(0xffffffffu, mn);
        mx = __reduce_max_sync(0xffffffffu, mx);
        __syncthreads();
        if (lane == 0) { s_cnt[warp][0] = (uint32_t)mn; s_cnt[warp][1] = (uint32_t)mx; }
        __syncthreads();
#pragma unroll
        for (int w = 0; w < NWARP; ++w) { mn = min(mn, (int)s_cnt[w][0]); mx = max(mx, (int)s_cnt[w][1]); }
        const int left = min(-mn, 16 * E), right = min(mx - La, 16 * E);
        for (int i = tid; i < left + right; i += BLOCK) s_col[i] = (int16_t)(i < left ? i - left : La + i - left);
        if (tid == 0) s_nd = left + right;
        outside = true;
        __syncthreads();
    }

    // ---- candidate correction (getCorrectedCandidates, msa.cpp:457-522) ----
    {
        const int ncc = o.new_columns;
        for (int i = tid; i < nalive; i += BLOCK) {
            uint32_t id; int shift, L; bool fwd;
            if (persistent) {
                const int k = (int)(s_ent[i + 1].w >> 4);
                id = s_slot[k].x; shift = slot_beg(k); L = slot_len(k); fwd = !(s_slot[k].y >> 31);
            } else {
                const CandRec rc = recs[off + i];
                id = rc.id; shift = rc.shift; L = rc.len; fwd = rc.orient == 1;
            }
            if (!(-ncc <= shift && shift <= ncc && shift + L <= La + ncc)) continue;
            const unsigned long long slot = atomicAdd(out.corr_count, 1ull);
            if (slot >= out.corr_cap) { atomicOr(status, kStatusCorrOverflow); continue; }
            char* dst = out.corr_seq + slot * mlen;
            const uint32_t* row = r.seq + (size_t)id * sp;
            const uint8_t* cons = s_cons + shift + 16 * E;
            int nd = 0;
            for (int p = 0; p < L; ++p) {
                // forward orientation of the corrected candidate
                const uint32_t cs = fwd ? cons[p] & 3u : (cons[L - 1 - p] & 3u) ^ 3u;
                dst[p] = "ACGT"[cs];
                nd += cs != base_at(row, p);
            }
            for (int p = L; p < mlen; ++p) dst[p] = 0;   // rows read as zero past the read
            out.corr_id[slot] = id;
            out.corr_anchor[slot] = a;
            out.corr_shift[slot] = shift;
            out.corr_use_edits[slot] = (!r.ambig[id] && nd <= L / 7) ? 1 : 0;
        }
    }
}

// One CTA per anchor, in `order` (e.g. most candidates first) when given;
// the hardware block scheduler hands out the anchors.
// CTAS: CTAs that share an SM. With rows short enough for ten of them and
// anchors enough to fill them, the register limit of ten is taken (48
// registers, a few spills): 12.6 -> 12.0 ms per 1M 150 bp reads. Reads of
// 50-250 bases, which shared memory holds to eight, lose by it (8.5 -> 8.9 ms
// per 400k), and so do 128 anchors, one per SM (66 -> 88 us).
constexpr int kMsaManyCtas = 10;
inline bool msa_many_ctas(size_t dynamic_smem, uint32_t anchors, int sms) {
    return (dynamic_smem + 8192) * kMsaManyCtas <= 228 * 1024 && anchors >= (uint32_t)(16 * sms);
}
template <int BLOCK, int QB, bool EMIT = false, int CTAS = (EMIT ? 768 : 1024) / BLOCK>
__global__ void __launch_bounds__(BLOCK, CTAS)
k_msa(DevOptions o, DevReads r, uint32_t first, uint32_t count, MsaGrid grid, const uint32_t* __restrict__ order,
      const uint32_t* __restrict__ cand_ids, const uint32_t* __restrict__ seg_off,
      const uint32_t* __restrict__ seg_cnt, const AlignRes* __restrict__ ares,
      CandRec* __restrict__ recs, MsaOut out, int* __restrict__ status) {
    if (blockIdx.x >= count) return;
    if (*status & kStatusIncomplete) return;     // unwritten candidates or alignments
    msa_anchor<BLOCK, QB, EMIT>(o, r, first, order ? order[blockIdx.x] : blockIdx.x, grid, cand_ids, seg_off,
                                seg_cnt, ares, recs, out, status);
}

// Persistent form: a grid of resident CTAs pulls anchors from a device work
// queue (an atomic cursor over `order`) until the batch is done.
template <int BLOCK, int QB, bool EMIT = false>
__global__ void __launch_bounds__(BLOCK, (EMIT ? 768 : 1024) / BLOCK)
k_msa_queue(DevOptions o, DevReads r, uint32_t first, uint32_t count, MsaGrid grid, const uint32_t* __restrict__ order,
            unsigned int* __restrict__ cursor, const uint32_t* __restrict__ cand_ids,
            const uint32_t* __restrict__ seg_off, const uint32_t* __restrict__ seg_cnt,
            const AlignRes* __restrict__ ares, CandRec* __restrict__ recs, MsaOut out,
            int* __restrict__ status) {
    __shared__ uint32_t s_item;
    if (*status & kStatusIncomplete) return;
    for (;;) {
        __syncthreads();                      // the previous anchor is done with shared memory
        if (threadIdx.x == 0) s_item = atomicAdd(cursor, 1u);
        __syncthreads();
        const uint32_t it = s_item;
        if (it >= count) return;
        msa_anchor<BLOCK, QB, EMIT>(o, r, first, order ? order[it] : it, grid, cand_ids, seg_off, seg_cnt, ares,
                                    recs, out, status);
    }
}

// Longest-processing-time order of a batch's anchors: a counting sort by
// candidate count, most candidates first (order within a count arbitrary:
// anchors are independent, results are written by anchor index).
constexpr int kLptBins = 4096;
static __global__ void k_lpt_hist(const uint32_t* __restrict__ seg_cnt, uint32_t count,
                                  unsigned int* __restrict__ bins) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
        atomicAdd(&bins[kLptBins - 1 - min(seg_cnt[i], (uint32_t)(kLptBins - 1))], 1u);
}
// exclusive scan of the bins in place (one CTA of 1024 threads)
static __global__ void k_lpt_scan(unsigned int* __restrict__ bins) {
    __shared__ unsigned int s_part[1024];
    constexpr int per = kLptBins / 1024;
    const int t = threadIdx.x;
    unsigned int loc[per], sum = 0;
#pragma unroll
    for (int k = 0; k < per; ++k) { loc[k] = bins[t * per + k]; sum += loc[k]; }
    s_part[t] = sum;
    __syncthreads();
    for (int d = 1; d < 1024; d <<= 1) {
        const unsigned int v = t >= d ? s_part[t - d] : 0u;
        __syncthreads();
        s_part[t] += v;
        __syncthreads();
    }
    unsigned int run = s_part[t] - sum;
#pragma unroll
    for (int k = 0; k < per; ++k) { bins[t * per + k] = run; run += loc[k]; }
}
static __global__ void k_lpt_scatter(const uint32_t* __restrict__ seg_cnt, uint32_t count,
                                     unsigned int* __restrict__ bins, uint32_t* __restrict__ order) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
        order[atomicAdd(&bins[kLptBins - 1 - min(seg_cnt[i], (uint32_t)(kLptBins - 1))], 1u)] = i;
}

// Per-alignment order of each anchor's candidate segment by candidate length
// (a counting sort over 16-base length classes, one CTA per anchor): warps of
// k_align then hold pairs of similar scan length. Results stay at their pair
// index, so the MSA still sees candidates in id order.
static __global__ void k_pair_order(const DevReads r, const uint32_t* __restrict__ cand_ids,
                                    const uint32_t* __restrict__ seg_off, const uint32_t* __restrict__ seg_cnt,
                                    uint32_t count, const int* __restrict__ status,
                                    uint32_t* __restrict__ pair_order) {
    constexpr int NB = kMaxLen / 16 + 1;
    __shared__ unsigned int s_bin[NB];
    const uint32_t ai = blockIdx.x;
    if (ai >= count || (*status & kStatusCandOverflow)) return;
    const uint32_t off = seg_off[ai], cnt = seg_cnt[ai];
    for (int b = threadIdx.x; b < NB; b += blockDim.x) s_bin[b] = 0;
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < cnt; k += blockDim.x) atomicAdd(&s_bin[r.len[cand_ids[off + k]] >> 4], 1u);
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int run = 0;
        for (int b = 0; b < NB; ++b) { const unsigned int c = s_bin[b]; s_bin[b] = run; run += c; }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < cnt; k += blockDim.x)
        pair_order[off + atomicAdd(&s_bin[r.len[cand_ids[off + k]] >> 4], 1u)] = off + k;
}

// Length classes of the alignment pairs: the plane width (32-base words) the
// longer read of a pair needs, 4 / 5 / 6 / 8, so that each class runs the
// k_align instance of its width (fewer registers for short pairs, lanes of
// similar lengths). cls[c] = {offset in the class list, pairs}; within a
// class, warps keep the pair order they read (warp-aggregated cursors).
constexpr int kAlignClasses = 4;
__host__ __device__ inline int align_class_width(int c) { return c == 0 ? 4 : c == 1 ? 5 : c == 2 ? 6 : 8; }
__device__ __forceinline__ int align_class_of(int L) {
    const int nw = (L + 31) >> 5;
    return nw <= 4 ? 0 : nw == 5 ? 1 : nw == 6 ? 2 : 3;
}
__device__ __forceinline__ int pair_class(const DevReads& r, uint32_t first, const uint32_t* cand_ids,
                                          const uint32_t* cand_anchor, unsigned long long i) {
    return align_class_of(max(r.len[first + cand_anchor[i]], r.len[cand_ids[i]]));
}
static __global__ void k_pair_class_count(DevReads r, uint32_t first, const uint32_t* __restrict__ cand_ids,
                                          const uint32_t* __restrict__ cand_anchor,
                                          const unsigned long long* __restrict__ total_ptr, unsigned long long cap,
                                          const int* __restrict__ status, const uint32_t* __restrict__ pair_order,
                                          uint2* __restrict__ cls) {
    if (*status & kStatusCandOverflow) return;
    const unsigned long long total = *total_ptr;
    if (total > cap) return;
    const int lane = threadIdx.x & 31;
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long s0 = (unsigned long long)blockIdx.x * blockDim.x; s0 < total; s0 += stride) {
        const unsigned long long slot = s0 + threadIdx.x;
        const bool act = slot < total;
        const int c = act ? pair_class(r, first, cand_ids, cand_anchor, pair_order ? pair_order[slot] : slot) : -1;
#pragma unroll
        for (int k = 0; k < kAlignClasses; ++k) {
            const unsigned m = __ballot_sync(0xffffffffu, c == k);
            if (m && lane == 0) atomicAdd(&cls[k].y, (unsigned)__popc(m));
        }
    }
}
static __global__ void k_pair_class_offsets(uint2* __restrict__ cls, unsigned int* __restrict__ cursor) {
    if (threadIdx.x != 0) return;
    unsigned run = 0;
    for (int k = 0; k < kAlignClasses; ++k) { cls[k].x = run; cursor[k] = run; run += cls[k].y; }
}
static __global__ void k_pair_class_scatter(DevReads r, uint32_t first, const uint32_t* __restrict__ cand_ids,
                                            const uint32_t* __restrict__ cand_anchor,
                                            const unsigned long long* __restrict__ total_ptr, unsigned long long cap,
                                            const int* __restrict__ status, const uint32_t* __restrict__ pair_order,
                                            unsigned int* __restrict__ cursor, uint32_t* __restrict__ list) {
    if (*status & kStatusCandOverflow) return;
    const unsigned long long total = *total_ptr;
    if (total > cap) return;
    const int lane = threadIdx.x & 31;
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long s0 = (unsigned long long)blockIdx.x * blockDim.x; s0 < total; s0 += stride) {
        const unsigned long long slot = s0 + threadIdx.x;
        const bool act = slot < total;
        const uint32_t i = act ? (pair_order ? pair_order[slot] : (uint32_t)slot) : 0u;
        const int c = act ? pair_class(r, first, cand_ids, cand_anchor, i) : -1;
#pragma unroll
        for (int k = 0; k < kAlignClasses; ++k) {
            const unsigned m = __ballot_sync(0xffffffffu, c == k);
            if (!m) continue;
            unsigned b = 0;
            if (lane == 0) b = atomicAdd(&cursor[k], (unsigned)__popc(m));
            b = __shfl_sync(0xffffffffu, b, 0);
            if (c == k) list[b + __popc(m & ((1u << lane) - 1u))] = i;
        }
    }
}

// The network's verdict on each decision column of the batch: the consensus
// base where the logit is positive, else the original base.
static __global__ void k_clf_apply(const uint32_t* __restrict__ feat_read, const uint32_t* __restrict__ feat_meta,
                            const float* __restrict__ logit, const unsigned long long* __restrict__ count,
                            unsigned long long cap, uint32_t first, int mlen, char* __restrict__ seq,
                            uint8_t* __restrict__ touched) {
    const unsigned long long n = min(*count, cap);
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        const uint32_t meta = feat_meta[i];
        const uint32_t ai = feat_read[i] - first;
        const uint32_t b = logit[i] > 0.0f ? (meta >> 18) & 3u : (meta >> 16) & 3u;
        seq[(size_t)ai * mlen + (meta & 0xFFFFu)] = "ACGT"[b];
        touched[ai] = 1;
    }
}

// Edit counts of the anchors whose corrected sequence k_clf_apply changed
// (makeOutputOfTask, corrector.hpp:1648-1675): one warp per anchor.
static __global__ void k_clf_recount(DevReads r, uint32_t first, uint32_t count, const uint8_t* __restrict__ touched,
                              const char* __restrict__ seq, uint8_t* __restrict__ status,
                              int32_t* __restrict__ nedits) {
    const int lane = threadIdx.x & 31;
    const uint32_t ai = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (ai >= count || !touched[ai]) return;
    const uint32_t a = first + ai;
    const int La = r.len[a];
    const uint32_t* row = r.seq + (size_t)a * r.seq_pitch;
    const char* s = seq + (size_t)ai * r.max_len;
    int nd = 0;
    for (int p = lane; p < La; p += 32) nd += "ACGT"[base_at(row, p)] != s[p];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) nd += __shfl_xor_sync(0xffffffffu, nd, d);
    if (lane == 0) {
        const bool useEdits = !r.ambig[a] && nd <= La / 7;
        status[ai] = (uint8_t)((status[ai] & ~4u) | (useEdits ? 4u : 0u));
        nedits[ai] = useEdits ? nd : 0;
    }
}

// Signatures of all reads (for table construction): one warp per read.
static __global__ void k_signatures(DevOptions o, DevReads r, uint32_t first, uint32_t count,
                             unsigned long long* __restrict__ sig) {
    const int lane = threadIdx.x & 31;
    const uint32_t ri = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (ri >= count) return;
    const uint32_t id = first + ri;
    const int L = r.len[id];
    const int h = o.num_maps;
    const uint32_t* row = r.seq + (size_t)id * r.seq_pitch;
    unsigned long long mine[2] = {~0ull, ~0ull};  // maps lane and lane+32
    unsigned long long alt[2] = {~0ull, ~0ull};
    if (L >= o.k) {
        const int npos = L - o.k + 1;
        const int rcshift = 64 - 2 * o.k;
        for (int p0 = 0; p0 < npos; p0 += 32) {
            // each lane builds one canonical k-mer, then all lanes hash all 32
            unsigned long long cn = 0;
            const int p = p0 + lane;
            if (p < npos) {
                const int w = p >> 4, of = p & 15;
                const uint32_t s0 = __ldg(row + w);
                const uint32_t s1 = (w + 1 < r.seq_pitch) ? __ldg(row + w + 1) : 0u;
                const uint32_t s2 = (w + 2 < r.seq_pitch) ? __ldg(row + w + 2) : 0u;
                const unsigned long long hi = ((unsigned long long)s0 << 32) | s1;
                const unsigned long long top = of ? (hi << (2 * of)) | ((unsigned long long)s2 >> (32 - 2 * of)) : hi;
                const unsigned long long fw = top >> (64 - 2 * o.k);
                const unsigned long long rv = revcomp64(fw) >> rcshift;
                cn = fw < rv ? fw : rv;
            }
            // two k-mers per step into separate minima (the min chains of a
            // lane overlap; an odd count hashes the last k-mer twice)
            const int nv = min(32, npos - p0);
            for (int q = 0; q < nv; q += 2) {
                const unsigned long long k0 = __shfl_sync(0xffffffffu, cn, q);
                const unsigned long long k1 = __shfl_sync(0xffffffffu, cn, q + 1 < nv ? q + 1 : q);
                if (lane < h) {
                    const unsigned long long v0 = murmur64(k0 + lane), v1 = murmur64(k1 + lane);
                    mine[0] = v0 < mine[0] ? v0 : mine[0];
                    alt[0] = v1 < alt[0] ? v1 : alt[0];
                }
                if (lane + 32 < h) {
                    const unsigned long long v0 = murmur64(k0 + lane + 32), v1 = murmur64(k1 + lane + 32);
                    mine[1] = v0 < mine[1] ? v0 : mine[1];
                    alt[1] = v1 < alt[1] ? v1 : alt[1];
                }
            }
        }
    }
    mine[0] = alt[0] < mine[0] ? alt[0] : mine[0];
    mine[1] = alt[1] < mine[1] ? alt[1] : mine[1];
    if (lane < h) sig[(size_t)ri * h + lane] = mine[0] & o.kmer_mask;
    if (lane + 32 < h) sig[(size_t)ri * h + lane + 32] = mine[1] & o.kmer_mask;
}

}  // namespace careb200
