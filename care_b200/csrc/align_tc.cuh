// align_tc.cuh -- the shifted Hamming alignment of an anchor with all its
// candidates as a contraction on the tensor cores.
//
//   cpuShiftedHammingDistancePopcount2BitHiLo  src/cpu_alignment.cpp:32-323
//   chooseBestAlignmentOrientation             include/alignmentorientation.hpp:72-92
//
// The reference's scan returns the first shift, in scan order, with the
// smallest score among the shifts whose mismatches are below
// int(overlap * maxErrorRate) (see shd_scan in device.cuh). Nearly every
// shift of nearly every pair is far above that limit, so the work is to rule
// shifts out. One bit per base does that: with x(b) = +1 / -1 by the high bit
// of the 2-bit code, sum_p x(A[s + p]) x(C[p]) = overlap - 2 * (bases whose
// high bits differ), and a base whose high bits differ is a mismatch. These
// sums for every shift s and every candidate are one matrix product per
// anchor: rows = shifts (the anchor's Toeplitz matrix), columns = candidates
// in both orientations, K = candidate positions. The few (shift, column) that
// stay possible are then counted exactly on the packed 2-bit words, and the
// result is the same shift the scan returns.
//
// Operands are e4m3 bytes (0x38 = 1.0, 0xB8 = -1.0, 0 outside a read), the
// sums exact in fp32. The Toeplitz matrix is not stored: in the K-major
// no-swizzle layout row i of an 8-row group lies 16 bytes after row i - 1 and
// K chunk c (16 elements) LBO bytes after chunk c - 1, so with LBO = 16 a
// region of (7 + K/16) * 16 bytes holding the anchor's bytes from base b on
// reads as eight rows of shifts b, b + 16, ..., b + 112. Sixteen regions with
// b = s0 .. s0 + 15 (SBO = the region's size) are the 128 shifts s0 .. s0+127
// of one M = 128 tile: 4.3 KB instead of 20 KB at K = 160, and the copy that
// would write them.
//
// Bound: instruction issue and barriers (57 % issue active and 13K warp
// instructions per anchor of 47 candidates, with mirrors 69 % and 8.8K; the
// products take a tenth of the tensor pipe, 46 cycles per 128 x 64 x 32 step,
// the same as with a stored Toeplitz matrix). Measured against the thread scan
// (k_align) and its pair mirroring: 1M 150 bp paired-end reads at 30x 14.3 ms
// (18.8), 1.3M at 50x 24.3 ms (36.3), 400k reads of 50-250 bases 11.8 ms with
// mirrors, 18.0 ms without (34.1), 300k 100 bp reads 3.1 and 4.1 ms (5.6), 128
// anchors 26 us (58). Where the scan is faster: tc_faster.
#pragma once
#include "kernels.cuh"
#include "tc05.cuh"
#include "tc_math.cuh"

namespace careb200 {

constexpr uint32_t kTcWaitLimit = 1u << 22;
constexpr int kTcGaveUp = 1 << 30;      // in place of the number of listed shifts: the wait ran out

// Whether the tensor-core alignment takes these options.
inline bool tc_applies(float max_error_rate, int min_overlap, float min_overlap_ratio) {
    return max_error_rate >= 0.0f && max_error_rate <= kTcMaxErrorRate && min_overlap >= 1 &&
           min_overlap_ratio >= 0.0f && min_overlap_ratio <= 1.0f;
}

// Mirror of each pair of the batch: its mirror's index when it leads,
// kMirrorSkip when its mirror answers it; the caller has set every entry to
// kMirrorSingle. The shorter read leads (the smaller id of equal lengths): its
// minimum overlap is the smaller one, so its shifts include the mirror's.
// Only leaders search (the mirror of a
// pair exists exactly when the leader finds it) and write both entries, and
// the pair flag of the mirror's result, whose search through global memory
// would hold up a whole CTA of the alignment. With a search per pair and the
// flags searched there, the alignment of 1.3M reads at 50x took 29.8 ms.
static __global__ void __launch_bounds__(256)
k_mirror_index(DevReads r, int paired_end, uint32_t first, uint32_t count, const uint32_t* __restrict__ cand_ids,
               const uint32_t* __restrict__ cand_anchor, const uint32_t* __restrict__ seg_off,
               const uint32_t* __restrict__ seg_cnt, const unsigned long long* __restrict__ total_ptr,
               unsigned long long arena_cap, const int* __restrict__ status, uint32_t* __restrict__ mirror,
               AlignRes* __restrict__ out) {
    if (*status & kStatusCandOverflow) return;
    const unsigned long long total = *total_ptr;
    if (total > arena_cap) return;
    const unsigned long long i = (unsigned long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= total) return;
    const uint32_t a = first + cand_anchor[i], c = cand_ids[i];
    if (c - first >= count) return;
    const int La = r.len[a], Lc = r.len[c];
    if (La > Lc || (La == Lc && c <= a)) return;
    const uint32_t ci = c - first, off = seg_off[ci], cnt = seg_cnt[ci];
    uint32_t lo = 0, hi = cnt;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (cand_ids[off + mid] < a) lo = mid + 1; else hi = mid;
    }
    if (lo < cnt && cand_ids[off + lo] == a) {
        mirror[i] = off + lo;
        mirror[off + lo] = kMirrorSkip;
        out[off + lo].paired = paired_end ? mate_flag(cand_ids, seg_off, seg_cnt, ci, a) : 0;
    }
}

// D[tmem] (+)= A x B^T, e4m3 operands, fp32 sums, K = 32; the matrix
// descriptors as halves (only the start addresses in the low ones change)
__device__ __forceinline__ void mma_e4m3(uint32_t d_tmem, uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi,
                                         uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
        "mov.b64 a, {%1, %2};\n\t"
        "mov.b64 b, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a, b, %5, p;\n\t}"
        :: "r"(d_tmem), "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// 8 consecutive fp32 columns of this thread's tensor-memory lane
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
// true in one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
    return p != 0u;
}
// halves of a K-major no-swizzle matrix descriptor
__device__ __forceinline__ uint32_t tc_desc_lo(uint32_t saddr, uint32_t lbo) { return ((saddr >> 4) & 0x3FFFu) | (lbo >> 4) << 16; }
__device__ __forceinline__ uint32_t tc_desc_hi(uint32_t sbo) { return (sbo >> 4) | 1u << 14; }

// Persistent CTAs, one anchor at a time. Per anchor: the Toeplitz regions of
// its shifts, then per product of up to 32 candidates (i) their packed rows,
// both orientations, as operand columns, (ii) one tcgen05 product per
// 128-shift tile, (iii) every sum against its shift's threshold (a warp reads
// its 32 shifts of all columns), the possible ones listed (in a bit each when
// there are too many), (iv) their exact counts and a minimum per column, (v) the orientation, the pair flag and the
// AlignRes. The next anchor's segment, ids and lengths load meanwhile.
// mirror (may be null): k_mirror_index's array; a leading pair also writes
// its mirror's result. splits: parts that an anchor's candidates are handed
// out in (tc_splits). wait_limit: polls of a product's completion (kTcWaitLimit;
// a test lets it run out), after which kStatusTensorWait is set.
static __global__ void __launch_bounds__(kTcBlock, kTcCtas)
k_align_tc(DevOptions o, DevReads r, uint32_t first, uint32_t count, const uint32_t* __restrict__ cand_ids,
           const uint32_t* __restrict__ seg_off, const uint32_t* __restrict__ seg_cnt,
           const unsigned long long* __restrict__ total_ptr, unsigned long long arena_cap, int* __restrict__ status,
           AlignRes* __restrict__ out, unsigned long long* __restrict__ work_count,
           const uint32_t* __restrict__ mirror, unsigned int* __restrict__ cursor, uint32_t splits, TcLayout lay,
           uint32_t wait_limit) {
    extern __shared__ __align__(128) unsigned char tsm[];
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ uint32_t s_tmem, s_next;
    __shared__ int s_nh;
    __shared__ int s_win[2][3];                        // per parity: items, shortest and longest candidate
    __shared__ float s_thr[kMaxLen + 1];               // by overlap
    // by parity of the window: what the results need while the next one loads
    __shared__ uint32_t s_idb[2][kTcWindow], s_mirb[2][kTcWindow], s_mateb[2][kTcMate];
    __shared__ uint16_t s_lenb[2][kTcWindow];
    __shared__ uint8_t s_pib[2][kTcWindow];
    __shared__ uint32_t s_hit[kTcHits];                // column | (shift + 512) << 16
    __shared__ uint32_t s_key[4][kTcMaxItems];         // best of (A, C), (A, rc C), (C, A), (C, rc A)
    __shared__ __align__(16) float s_kl[kTcMaxItems];  // kappa * length
    if (*status & kStatusCandOverflow) return;         // arena entries past the overflow are unwritten
    if (*total_ptr > arena_cap) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int W = lay.W, RS = lay.RS, XL = lay.XL;
    uint32_t* s_aw = reinterpret_cast<uint32_t*>(tsm + lay.aw);     // the anchor's packed row
    uint4* s_q = reinterpret_cast<uint4*>(tsm + lay.q);
    uint4* s_top = reinterpret_cast<uint4*>(tsm + lay.top);
    unsigned char* s_b = tsm + lay.b;
    uint32_t* s_fw = reinterpret_cast<uint32_t*>(tsm + lay.fw);
    uint32_t* s_ar = reinterpret_cast<uint32_t*>(tsm + lay.ar);     // and its reverse complement
    auto minov_of = [&](int L) { return max(o.min_overlap, f2i_rz(fmul_rn((float)L, o.min_overlap_ratio))); };
    auto mex_of = [&](int ov) { return f2i_rz(fmul_rn((float)ov, o.max_error_rate)); };
    for (int i = tid; i <= kMaxLen; i += kTcBlock) s_thr[i] = tc_threshold(i, mex_of(i));
    for (int it = tid; it < kTcMaxItems; it += kTcBlock)
        for (int w = W; w < RS; ++w) s_fw[it * RS + w] = 0u;
    if (tid < 2) { s_win[tid][0] = 0; s_win[tid][1] = kMaxLen; s_win[tid][2] = 0; }
    if (tid == 0) {
        s_nh = 0;
        tc05::mbar_init(&s_bar, 1);
    }
    if (warp == 0) tc05::tmem_alloc(&s_tmem, kTcCols);
    tc05::fence_before_sync();
    __syncthreads();
    tc05::fence_after_sync();
    const uint32_t tmem = s_tmem;
    uint32_t phase = 0u;
    bool bad = false;
    unsigned long long words = 0;
    const float kappa = 1.0f - 2.0f * o.max_error_rate;       // thresholds are above kappa * overlap + kTcSlack
    const float ler = __fmul_rn(o.estimated_errorrate, 4.0f);
    // this lane's row of a tile, as a shift relative to the tile's first
    const int srow = tc_row_shift(32 * warp + lane);
    int par = 0;

    // the anchor at hand: segment, length, this thread's candidate of its
    // first window, its length and mirror
    // (unit = anchor * splits + part: part p takes windows p, p + splits, ...)
    const uint32_t units = count * splits;
    const uint32_t win = splits > 1 ? 32u : (uint32_t)kTcWindow;
    uint32_t unit = blockIdx.x, ai = splits > 1 ? unit / splits : unit, off = 0, cnt = 0, c = 0, mir = kMirrorSkip;
    int La = 0, Lc = 0;
    auto load_cand = [&](uint32_t off_, uint32_t w0_, uint32_t cnt_, uint32_t& c_, uint32_t& m_) {
        const uint32_t i = w0_ + (uint32_t)tid;
        c_ = 0;
        m_ = kMirrorSkip;
        if (i < cnt_ && (uint32_t)tid < win) {
            c_ = cand_ids[off_ + i];
            m_ = mirror ? mirror[off_ + i] : kMirrorSingle;
        }
    };
    if (unit < units) {
        off = seg_off[ai];
        cnt = seg_cnt[ai];
        La = r.len[first + ai];
        load_cand(off, (unit - ai * splits) * win, cnt, c, mir);
        if (mir != kMirrorSkip) Lc = r.len[c];
    }
    while (unit < units) {
        const uint32_t a = first + ai;
        const int minov = minov_of(La);
        const int smax = La - minov;
        const int nwa = (La + 15) >> 4;
        const int q0 = smax - 127 - 128 * (lay.tiles - 1);    // base of the first operand chunk
        uint32_t* s_mate = s_mateb[par];                      // (a later window of the anchor writes it again)
        uint32_t mcnt = 0;
        // the next anchor
        uint32_t unitn = units, ain = 0, w0n = 0, offn = 0, cntn = 0, cn = 0, mirn = kMirrorSkip;
        int Lan = 0, Lcn = 0;
        if (tid == 0) s_next = gridDim.x + atomicAdd(cursor, 1u);
        bool have_top = false, have_cand = false, have_len = false;
        const uint32_t wf = (unit - ai * splits) * win;
        for (uint32_t w0 = wf;; w0 += win * splits) {
            // ---- the window's items (the first window's are in registers) ----
            uint32_t* s_id = s_idb[par];
            uint32_t* s_mir = s_mirb[par];
            uint16_t* s_len = s_lenb[par];
            uint8_t* s_pi = s_pib[par];
            s_mate = s_mateb[par];
            if (w0 != wf) {
                load_cand(off, w0, cnt, c, mir);
                if (mir != kMirrorSkip) Lc = r.len[c];
            }
            {
                const bool item = mir != kMirrorSkip;
                const unsigned bm = __ballot_sync(0xffffffffu, item);
                if (bm) {
                    const int mnl = __reduce_min_sync(0xffffffffu, item ? Lc : kMaxLen);
                    const int mxl = __reduce_max_sync(0xffffffffu, item ? Lc : 0);
                    int base = 0;
                    if (lane == 0) {
                        base = atomicAdd(&s_win[par][0], __popc(bm));
                        atomicMin(&s_win[par][1], mnl);
                        atomicMax(&s_win[par][2], mxl);
                    }
                    base = __shfl_sync(0xffffffffu, base, 0);
                    if (item) {
                        const int p = base + __popc(bm & ((1u << lane) - 1u));
                        s_id[p] = c;
                        s_mir[p] = mir;
                        s_pi[p] = (uint8_t)tid;
                        s_len[p] = (uint16_t)Lc;
                    }
                }
            }
            if (w0 == wf && tid < kMaxLen / 16 + 2) s_aw[tid] = tid < nwa ? __ldg(r.seq + (size_t)a * r.seq_pitch + tid) : 0u;
            if (o.paired_end) {
                const uint32_t moff = seg_off[ai ^ 1u];
                mcnt = seg_cnt[ai ^ 1u];
                if (mcnt <= (uint32_t)kTcMate)
                    for (uint32_t i = tid; i < mcnt; i += kTcBlock) s_mate[i] = cand_ids[moff + i];
            }
            __syncthreads();
            if (w0 == wf) {
                unitn = s_next;
                if (unitn < units) {
                    ain = splits > 1 ? unitn / splits : unitn;
                    w0n = (unitn - ain * splits) * win;
                    offn = seg_off[ain];
                    cntn = seg_cnt[ain];
                    Lan = r.len[first + ain];
                }
            }
            const int nwin = s_win[par][0], minl = s_win[par][1], maxl = s_win[par][2];
            if (tid < 3) s_win[par ^ 1][tid] = tid == 1 ? kMaxLen : 0;      // the next window's
            const bool uniform = minl == maxl;
            const int smin = minov - maxl;                    // lowest shift of the window's longest read
            const int ntiles = (nwin == 0 || smax < 0 || maxl < minov) ? 0 : (smax - smin + 128) >> 7;
            const int ksteps = (maxl + 31) >> 5;
            if (work_count) {
                if (tid < (uniform ? min(nwin, 1) : nwin))
                    words += (unsigned long long)(uniform ? 2 * nwin : 2) * (unsigned)unpruned_words(La, s_len[tid], minov);
            }
            const int nprod = (nwin + kTcMaxItems - 1) / kTcMaxItems;
            const int per = nprod ? (((nwin + nprod - 1) / nprod) + 7) & ~7 : kTcMaxItems;
            for (int i0 = 0; i0 < nwin; i0 += per) {
                const int n = min(per, nwin - i0), nI = (n + 7) & ~7;
                // ---- packed rows; the anchor's operand bytes ----
#pragma unroll 1
                for (int idx = tid; idx < n * W; idx += kTcBlock) {
                    const int it = (int)(((uint32_t)idx * lay.magic_w) >> 16), w = idx - it * W;
                    const int L = s_len[i0 + it];
                    s_fw[it * RS + w] = 16 * w < L ? __ldg(r.seq + (size_t)s_id[i0 + it] * r.seq_pitch + w) : 0u;
                }
                if (!have_top && warp == kTcWarps - 1)
#pragma unroll 1
                    for (int x = lane; x <= XL; x += 32) {
                        uint32_t w[4];
                        tc_q_chunk(s_aw, nwa, La, q0 + 16 * x, w);
                        s_q[x] = make_uint4(w[0], w[1], w[2], w[3]);
                        if (x < kMaxLen / 16 + 2) s_ar[x] = x < nwa ? tc_rc_word(s_aw, nwa, La, x) : 0u;
                    }
                __syncthreads();
                // ---- operands (a warp per 16-base chunk, a lane per row) ----
                if (tid < kTcMaxItems) {
                    s_key[0][tid] = s_key[1][tid] = s_key[2][tid] = s_key[3][tid] = 0xFFFFFFFFu;
                    s_kl[tid] = tid < n ? kappa * (float)s_len[i0 + tid] : 0.0f;
                }
                if (tid == 0) s_nh = 0;
                if (ntiles > 0) {
                    const uint32_t magic_n = (65535u + (uint32_t)nI) / (uint32_t)nI;
#pragma unroll 1
                    for (int idx = tid; idx < nI * W; idx += kTcBlock) {      // rows n .. nI - 1 are zeros
                        const int ch = (int)(((uint32_t)idx * magic_n) >> 16), it = idx - ch * nI;
                        const int left = (it < n ? (int)s_len[i0 + it] : 0) - 16 * ch;
                        const uint32_t* row = s_fw + it * RS;
                        uint32_t w[4], y[4];
                        tc_expand(row[ch], w);
                        tc_expand_rc(tc_rc_window(row, left + 16 * ch, ch), y);
                        if (left < 16) {
                            uint32_t mk[4] = {~0u, ~0u, ~0u, ~0u};
                            tc_mask(mk, 0, left);
#pragma unroll
                            for (int i = 0; i < 4; ++i) { w[i] &= mk[i]; y[i] &= mk[i]; }
                        }
                        const int rr = nI + it;
                        unsigned char* bc = s_b + ch * 128;
                        *reinterpret_cast<uint4*>(bc + (it >> 3) * (128 * W) + (it & 7) * 16) = make_uint4(w[0], w[1], w[2], w[3]);
                        *reinterpret_cast<uint4*>(bc + (rr >> 3) * (128 * W) + (rr & 7) * 16) = make_uint4(y[0], y[1], y[2], y[3]);
                    }
                    if (!have_top) {                          // warp w: the regions of bytes 4 w .. 4 w + 3
#pragma unroll 1
                        for (int x = lane; x < XL; x += 32) {
                            const uint4 l = s_q[x], h = s_q[x + 1];
                            const uint32_t q8[8] = {l.x, l.y, l.z, l.w, h.x, h.y, h.z, h.w};
                            uint32_t e[5];
#pragma unroll
                            for (int i = 0; i < 5; ++i)
                                e[i] = warp < 2 ? (warp == 0 ? q8[i] : q8[i + 1]) : (warp == 2 ? q8[i + 2] : q8[i + 3]);
#pragma unroll
                            for (int rb = 0; rb < 4; ++rb) {
                                uint32_t w[4];
                                tc_shift16(e, rb, w);
                                s_top[(4 * warp + rb) * XL + x] = make_uint4(w[0], w[1], w[2], w[3]);
                            }
                        }
                        have_top = true;
                    }
                }
                if (!have_cand) {
                    load_cand(offn, w0n, cntn, cn, mirn);
                    have_cand = true;
                }
                tc05::fence_smem_to_async();
                __syncthreads();
                // ---- products, thresholds ----
                const int nbuf = 2 * nI <= kTcCols / 2 ? 2 : 1;
                int kept = 0;
#pragma unroll 1
                for (int t0 = 0; t0 < ntiles; t0 += nbuf) {
                    const int nt = min(nbuf, ntiles - t0);
                    if (warp == 0 && elect_one()) {
                        tc05::fence_after_sync();
                        const uint32_t idesc = (1u << 4) | ((uint32_t)(2 * nI >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
                        const uint32_t blo = tc_desc_lo(tc05::smem_addr(s_b), 128u), bhi = tc_desc_hi(128u * W);
                        const uint32_t ahi = tc_desc_hi(16u * XL);
#pragma unroll 1
                        for (int t = 0; t < nt; ++t) {
                            const uint32_t alo = tc_desc_lo(tc05::smem_addr(s_top) + 128u * (uint32_t)(lay.tiles - 1 - t0 - t), 16u);
                            const uint32_t d = tmem + (uint32_t)(t * (kTcCols / 2));
                            // K = 32 a step: two chunks further in both operands
#pragma unroll 4
                            for (uint32_t k = 0; k < (uint32_t)ksteps; ++k)
                                mma_e4m3(d, alo + 2 * k, ahi, blo + 16 * k, bhi, idesc, k);
                        }
                        tc05::commit(&s_bar);
                    }
                    if (!have_len) {
                        if (mirn != kMirrorSkip) Lcn = r.len[cn];
                        have_len = true;
                    }
                    // one warp polls; after a wait that ran out no product
                    // follows: the barrier's parity tells one unfinished
                    // product only
                    if (warp == 0 && !tc05::mbar_wait(&s_bar, phase, wait_limit)) s_nh = kTcGaveUp;
                    phase ^= 1u;
                    __syncthreads();
                    tc05::fence_after_sync();
#pragma unroll 1
                    for (int t = 0; t < nt; ++t) {
                        const int s = smax - 127 - 128 * (t0 + t) + srow;
                        // threshold of this lane's shift: its own with one
                        // length, else a bound per column from the length
                        const int u = max(s, 0);
                        float thr = uniform ? 1e9f : 0.0f;
                        if (uniform && s >= smin) {
                            const int ov = tc_overlap(s, La, minl);
                            if (ov >= minov) thr = s_thr[ov];
                        }
                        const float c1 = kappa * (float)(La - u) + kTcSlack, c2 = kappa * (float)(s - u) + kTcSlack;
                        const float cmin = s >= smin ? kappa * (float)minov + kTcSlack : 1e9f;
                        const uint32_t col0 = tmem + ((uint32_t)warp << 21) + (uint32_t)(t * (kTcCols / 2));
                        auto scan_tile = [&](auto same) {
#pragma unroll 1
                            for (int q = 0; q < 2 * nI; q += 16) {
                                float v[16];
                                tc05::tmem_ld16(col0 + q, v);
                                if constexpr (!decltype(same)::value) {    // each column's sum against its own bound: thr = 0
#pragma unroll
                                    for (int e = 0; e < 16; e += 4) {
                                        const int it0 = q + e - (q + (e & 8) >= nI ? nI : 0);
                                        const float4 kl = *reinterpret_cast<const float4*>(&s_kl[it0]);
                                        v[e] -= fmaxf(fminf(c1, kl.x + c2), cmin);
                                        v[e + 1] -= fmaxf(fminf(c1, kl.y + c2), cmin);
                                        v[e + 2] -= fmaxf(fminf(c1, kl.z + c2), cmin);
                                        v[e + 3] -= fmaxf(fminf(c1, kl.w + c2), cmin);
                                    }
                                }
                                float m[2];
#pragma unroll
                                for (int g = 0; g < 2; ++g) {
                                    const float* x = v + 8 * g;
                                    m[g] = fmaxf(max3(max3(max3(x[0], x[1], x[2]), x[3], x[4]), x[5], x[6]), x[7]);
                                }
                                if (fmaxf(m[0], m[1]) >= thr) {
                                    float limit = thr;        // opaque: or the masks below are formed ahead of the branch
                                    asm volatile("" : "+f"(limit));
#pragma unroll
                                    for (int g = 0; g < 2; ++g) {
                                        if (m[g] < limit) continue;
                                        uint32_t hits = 0u;
#pragma unroll
                                        for (int e = 0; e < 8; ++e) if (v[8 * g + e] >= limit) hits |= 1u << e;
                                        if (*(volatile int*)&s_nh > kTcHits) continue;    // the list has overflowed
                                        int p = atomicAdd(&s_nh, __popc(hits));
                                        do {
                                            const int e = __ffs(hits) - 1;
                                            hits &= hits - 1u;
                                            if (p < kTcHits)
                                                s_hit[p] = (uint32_t)(q + 8 * g + e) | (uint32_t)(s + 512) << 16;
                                            ++p;
                                        } while (hits);
                                    }
                                }
                            }
                        };
                        if (uniform) scan_tile(std::true_type{});
                        else scan_tile(std::false_type{});
                    }
                    tc05::fence_before_sync();
                    __syncthreads();
                    // ---- exact counts of the listed shifts, once the last
                    //      sums are read (of an overflowing round, of those
                    //      kept from the rounds before): four lanes per shift,
                    //      each every fourth word ----
                    const int nh = s_nh;
                    if (nh <= kTcHits && t0 + nbuf < ntiles) { kept = nh; continue; }
                    if (nh >= kTcGaveUp) { bad = true; goto done; }
                    const int work = nh > kTcHits ? kept : nh;
                    kept = 0;
#pragma unroll 1
                    for (int k0 = 8 * warp; k0 < work; k0 += kTcBlock / 4) {
                        const uint32_t hv = s_hit[min(k0 + (lane >> 2), work - 1)];
                        const int col = (int)(hv & 0xFFFFu), sh = (int)(hv >> 16) - 512;
                        const int rev = col >= nI;
                        const int it = col - rev * nI;
                        const int L = s_len[i0 + it];
                        const int ov = tc_overlap(sh, La, L);
                        // A against the candidate's reverse complement is A's
                        // reverse complement against the candidate
                        const uint32_t ca = lay.fw + 4u * (uint32_t)(it * RS), an = rev ? lay.ar : lay.aw;
                        const int sv = rev ? La - L - sh : sh;
                        const bool pos = sv >= 0;
                        int mm = tc_mismatches(reinterpret_cast<const uint32_t*>(tsm + (pos ? an : ca)),
                                               reinterpret_cast<const uint32_t*>(tsm + (pos ? ca : an)),
                                               pos ? sv : -sv, ov, lane & 3, 4);
                        mm += __shfl_xor_sync(0xffffffffu, mm, 1);
                        mm += __shfl_xor_sync(0xffffffffu, mm, 2);
                        if ((lane & 3) == 0 && ov >= minov && mm < mex_of(ov)) {
                            const uint32_t sc = (uint32_t)(mm + La + L - 2 * ov) << 10;
                            atomicMin(&s_key[rev][it], sc | tc_rank(sh));
                            if (mirror && ov >= minov_of(L)) atomicMin(&s_key[2 + rev][it], sc | tc_rank(tc_mirror_shift(sh, rev, La, L)));
                        }
                    }
                    if (nh <= kTcHits) continue;
                    // ---- more possible shifts than the list holds (reads of
                    //      short tandem repeats): the round's possible shifts
                    //      as a bit each, from the sums, then each column's
                    //      groups of 32 shifts by falling overlap, a lane per
                    //      shift, up to the mismatches that still improve on
                    //      the column's best. Against counts of all shifts of
                    //      the product, alignment ms with 2, 20 and 60 % of the
                    //      genome in repeats of 1-6 bases: 300k reads of 100
                    //      bases 7.9 -> 4.9 and 31.5 -> 7.6, 200k of 150 bases
                    //      146 -> 24 (thread scan 5.7, 6.3, 12.9) ----
                    __syncthreads();                          // the list's words become the bits
                    if (tid == 0) s_nh = 0;
#pragma unroll 1
                    for (int t = 0; t < nt; ++t) {
                        const int s = smax - 127 - 128 * (t0 + t) + srow;
                        const int u = max(s, 0);
                        const float c1 = kappa * (float)(La - u) + kTcSlack, c2 = kappa * (float)(s - u) + kTcSlack;
                        const float cmin = s >= smin ? kappa * (float)minov + kTcSlack : 1e9f;
                        const uint32_t col0 = tmem + ((uint32_t)warp << 21) + (uint32_t)(t * (kTcCols / 2));
#pragma unroll 1
                        for (int q = 0; q < 2 * nI; q += 8) {
                            float v[8];
                            tmem_ld8(col0 + q, v);
                            const float* kl = &s_kl[q - (q >= nI ? nI : 0)];
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                const uint32_t b = __ballot_sync(0xffffffffu, v[e] >= fmaxf(fminf(c1, kl[e] + c2), cmin));
                                if (lane == 0) s_hit[4 * (t * 2 * nI + q + e) + warp] = b;
                            }
                        }
                    }
                    tc05::fence_before_sync();
                    __syncthreads();
#pragma unroll 1
                    for (int en = warp; en < nt * 2 * nI; en += kTcWarps) {
                        const uint32_t bits = s_hit[4 * en + tc_shift_word(lane)] >> tc_shift_bit(lane, 0) & 0x55u;
                        if (!__any_sync(0xffffffffu, bits != 0u)) continue;
                        const int t = en >= 2 * nI, col = en - t * 2 * nI, rev = col >= nI, it = col - rev * nI;
                        const int L = s_len[i0 + it], minl2 = mirror ? minov_of(L) : 0;
                        const int s0 = smax - 127 - 128 * (t0 + t);
                        const uint32_t ca = lay.fw + 4u * (uint32_t)(it * RS), an = rev ? lay.ar : lay.aw;
#pragma unroll 1
                        for (int k = 0; k < 7; ++k) {
                            const int g = tc_group(s0, k);
                            if ((unsigned)g > 3u || !__any_sync(0xffffffffu, (bits >> 2 * g) & 1u)) continue;
                            const int sh = s0 + 32 * g + lane, ov = tc_overlap(sh, La, L);
                            const bool mirrored = mirror && ov >= minl2;
                            const int cap = ov < minov ? 0 : tc_cap(ov, mex_of(ov), La, L, *(volatile uint32_t*)&s_key[rev][it],
                                                                    mirrored, *(volatile uint32_t*)&s_key[2 + rev][it]);
                            if (((bits >> 2 * g) & 1u) && cap > 0) {
                                const int sv = rev ? La - L - sh : sh;
                                const bool pos = sv >= 0;
                                const int mm = tc_mismatches_below(reinterpret_cast<const uint32_t*>(tsm + (pos ? an : ca)),
                                                                   reinterpret_cast<const uint32_t*>(tsm + (pos ? ca : an)),
                                                                   pos ? sv : -sv, ov, cap);
                                if (mm < cap) {
                                    const uint32_t sc = (uint32_t)(mm + La + L - 2 * ov) << 10;
                                    atomicMin(&s_key[rev][it], sc | tc_rank(sh));
                                    if (mirrored) atomicMin(&s_key[2 + rev][it], sc | tc_rank(tc_mirror_shift(sh, rev, La, L)));
                                }
                            }
                            __syncwarp();
                        }
                    }
                }
                __syncthreads();
                // ---- orientation and results. With mirrors eight items a
                //      warp, lanes 0-7 the pair, lanes 8-15 its mirror (its
                //      pair flag is written already); else by one warp, while
                //      the others go on (four warps: 0.7 ms more per 1M reads).
                //      Nothing read here is written before the next two
                //      barriers ----
                {
                    const int it = mirror ? 8 * warp + (lane & 7) : lane;
                    const int side = mirror ? lane >> 3 : warp == 1 ? 0 : 2;
                    if (it < n && side < 2 && (side == 0 || s_mir[i0 + it] != kMirrorSingle)) {
                        const int L = s_len[i0 + it];
                        const int L1 = side ? L : La, L2 = side ? La : L;
                        const ShdResult fw = tc_result(s_key[2 * side][it], L1, L2);
                        const ShdResult rc = tc_result(s_key[2 * side + 1][it], L1, L2);
                        const int orr = choose_orientation(fw, rc, L1, o.min_overlap_ratio, o.min_overlap, ler);
                        const ShdResult& b = orr == 2 ? rc : fw;
                        AlignRes* dst = out + (side ? (size_t)s_mir[i0 + it] : (size_t)off + w0 + s_pi[i0 + it]);
                        dst->shift = (int16_t)b.shift;
                        dst->overlap = (int16_t)b.overlap;
                        dst->nops = (int16_t)b.nops;
                        dst->orient = (uint8_t)orr;
                        if (side == 0) {
                            uint8_t paired = 0;
                            if (o.paired_end && orr != 3) {
                                const uint32_t target = s_id[i0 + it] ^ 1u;
                                if (mcnt <= (uint32_t)kTcMate) {
                                    uint32_t l = 0, h = mcnt;
                                    while (l < h) {
                                        const uint32_t mid = (l + h) >> 1;
                                        if (s_mate[mid] < target) l = mid + 1; else h = mid;
                                    }
                                    paired = l < mcnt && s_mate[l] == target;
                                } else {
                                    paired = mate_flag(cand_ids, seg_off, seg_cnt, ai, s_id[i0 + it]);
                                }
                            }
                            dst->paired = paired;
                        }
                    }
                }
            }
            par ^= 1;
            const bool more = w0 + win * splits < cnt;
            if (nwin == 0 || more) __syncthreads();           // no barrier since s_win was set; the results read s_id
            if (!more) break;
        }
        if (!have_cand) load_cand(offn, w0n, cntn, cn, mirn);
        if (!have_len && mirn != kMirrorSkip) Lcn = r.len[cn];
        unit = unitn;
        ai = ain;
        off = offn;
        cnt = cntn;
        La = Lan;
        c = cn;
        mir = mirn;
        Lc = Lcn;
    }
done:
    if (bad) {
        if (tid == 0) atomicOr(status, kStatusTensorWait | kStatusIncomplete);
        tc05::mbar_wait(&s_bar, phase ^ 1u);            // the product in flight ends before its memory is released
    }
    if (work_count) {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) words += __shfl_xor_sync(0xffffffffu, words, d);
        if (lane == 0) atomicAdd(work_count, words);
    }
    tc05::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc05::fence_after_sync();
        tc05::tmem_dealloc(tmem, kTcCols);
    }
}

}  // namespace careb200
