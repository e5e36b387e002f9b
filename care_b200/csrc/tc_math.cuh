// tc_math.cuh -- index and operand arithmetic of the tensor-core alignment
// (align_tc.cuh), __host__ __device__ so that a host build can check it
// against the CPU oracle.
#pragma once
#include "device.cuh"

namespace careb200 {

constexpr int kTcBlock = 128;
constexpr int kTcWarps = kTcBlock / 32;
constexpr int kTcMaxItems = 32;         // candidates per product: N = 2 * 32 columns
constexpr int kTcWindow = kTcBlock;     // candidates looked at at a time
constexpr int kTcCols = 64;             // tensor-memory columns of a CTA
constexpr int kTcCtas = 512 / kTcCols;  // CTAs that the tensor memory of an SM holds
constexpr int kTcMate = 192;            // ids of the mate's list held in shared memory
// Possible (shift, column) waiting for their exact count; with more of them the
// same words hold a bit for each shift of a round's sums.
constexpr int kTcHits = 256;
static_assert(kTcHits == 4 * kTcCols, "four words of shifts per column of sums");
// A random pair of bases differs in its high bit with probability 1/2, so up
// to this rate a possible shift is rare; above it the thread scan runs.
constexpr float kTcMaxErrorRate = 0.30f;

constexpr uint32_t kMirrorSingle = 0xffffffffu;   // k_mirror_index: no mirror in the batch
constexpr uint32_t kMirrorSkip = 0xfffffffeu;     // answered by its mirror

// Shared-memory layout, in bytes from the start of the dynamic part.
struct TcLayout {
    int W;                              // 16-base chunks of a row (even): K = 16 * W
    int RS;                             // words of a packed row (odd, > W)
    int tiles;                          // 128-shift tiles of the widest anchor
    int XL;                             // 16-byte chunks of a Toeplitz region
    uint32_t magic_w;                   // x / W as (x * magic) >> 16, x < 4096
    uint32_t aw, ar, q, top, b, fw, total;
};

// Shifts of the widest scan of one orientation.
constexpr int tc_span(int max_len, int min_overlap, float min_overlap_ratio) {
    int span = 1;
    for (int la = 1; la <= max_len; ++la) {
        const int lo = (int)((float)la * min_overlap_ratio);
        const int m = lo > min_overlap ? lo : min_overlap, mo = m < max_len ? m : max_len;
        const int n = la + max_len - 2 * mo + 1;
        span = n > span ? n : span;
    }
    return span;
}

constexpr TcLayout tc_layout(int max_len, int min_overlap, float min_overlap_ratio) {
    TcLayout t{};
    t.W = 2 * ((max_len + 31) / 32);
    t.RS = (t.W + 1) | 1;
    const int span = tc_span(max_len, min_overlap, min_overlap_ratio);
    t.tiles = (span + 127) / 128;
    t.XL = 7 + t.W + 8 * (t.tiles - 1);
    t.magic_w = (65536u + (uint32_t)t.W - 1) / (uint32_t)t.W;
    t.aw = 0;
    t.ar = 4u * (kMaxLen / 16 + 4);
    uint32_t at = 2u * t.ar;
    t.q = at;
    at += (uint32_t)(t.XL + 1) * 16u;
    t.top = (at + 127u) & ~127u;
    at = t.top + 16u * (uint32_t)t.XL * 16u;
    t.b = (at + 127u) & ~127u;
    at = t.b + 2u * kTcMaxItems * 16u * (uint32_t)t.W;
    t.fw = at;
    at += kTcMaxItems * 4u * (uint32_t)t.RS;
    t.total = at;
    return t;
}

// The widest layout, with the static part, needs no raised shared-memory limit.
// Such a limit belongs to the function on the device, not to a context: one set
// per call to the call's own size could fall below another thread's between
// that thread's setting and its launch.
static_assert(tc_layout(kMaxLen, 1, 0.0f).total + 8192 <= 48 * 1024, "the alignment fits the default limit");

// CTAs of the alignment that share an SM: its tensor memory, its shared memory
// (8 KB of a CTA's part is static or reserved).
inline int tc_ctas(const TcLayout& t) {
    const int n = (int)(228u * 1024u / (t.total + 8192u));
    return n < 1 ? 1 : n > kTcCtas ? kTcCtas : n;
}

// Parts per anchor: with fewer anchors than resident CTAs an anchor's
// candidates go to several of them.
inline uint32_t tc_splits(uint32_t anchors, uint32_t resident) {
    const uint32_t n = anchors ? resident / anchors : 1u;
    return n < 1u ? 1u : n > 8u ? 8u : n;
}

// Whether the tensor-core alignment is the faster one, from what the host
// knows: an anchor costs it a chain of loads and barriers whatever its
// candidates, and a product costs the same for few shifts as for many, so the
// thread scan (k_align) is ahead where pairs are few or shifts are: short
// reads, low coverage, a minimum overlap near the read's length. Costs fitted
// to 200k reads of 36 to 250 bases at 5x to 40x (1.25 pairs per anchor and unit
// of coverage) and to 128 to 4,000 anchors. Alignment ms, thread scan and
// tensor cores: 36 bases 5x 0.16, 0.91; 50 bases 20x 0.89, 1.33; 60 bases 40x
// 2.20, 2.17; 100 bases 5x 0.70, 1.18, 10x 1.31, 1.40, 20x 2.54, 1.95; 150
// bases 5x 1.02, 1.26, 10x 1.95, 1.55; 150 bases 30x with a minimum overlap of
// 135 1.18, 2.09, of 90 3.29, 2.40; 250 bases 5x 2.47, 1.91, 30x with a minimum
// overlap of 225 4.33, 2.88; 1,000 anchors of 50 bases 5x 0.018, 0.022, of 70
// bases 0.029, 0.022. fixed_us: what the scan's route adds to a call.
inline bool tc_faster(int max_len, int min_overlap, float min_overlap_ratio, float coverage, uint32_t anchors,
                      bool mirror, float fixed_us) {
    const int lo = (int)((float)max_len * min_overlap_ratio), mo = lo > min_overlap ? lo : min_overlap;
    const float pairs = 1.25f * coverage, shifts = mo < max_len ? (float)(4 * (max_len - mo) + 2) : 2.0f;
    // ns per pair on a full chip, by the words of a bit plane (registers of the scan)
    const float pair = max_len <= 160 ? 0.03f + 0.00165f * shifts : max_len <= 192 ? 0.1f + 0.00175f * shifts
                                                                                : 0.25f + 0.0019f * shifts;
    const float column = 0.12f + 0.0004f * (float)max_len + 0.085f * (float)((int)(0.5f * shifts + 127.0f) / 128 - 1);
    const float scan = pairs * (mirror ? 0.07f + 0.58f * pair : pair);
    const float tc = 4.2f + pairs * (mirror ? 0.68f * column : column);
    // us: the longest pair, the chain, and the anchors
    const float n = 1e-3f * (float)anchors;
    return !(fixed_us + 0.115f * shifts + n * scan < 12.5f + n * tc);
}

// 16 bases of a packed word -> 16 e4m3 bytes by their high bits, first base in
// the lowest byte of w[0]. A byte of the word holds four bases with their high
// bits at 7, 5, 3, 1; the product moves them to bits 7, 15, 23, 31 (the four
// copies do not overlap, so nothing carries).
CB_HD void tc_expand(uint32_t x, uint32_t (&w)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#ifdef __CUDA_ARCH__
        const uint32_t b = __byte_perm(x, 0u, 0x4443u - (uint32_t)i);
#else
        const uint32_t b = (x >> (24 - 8 * i)) & 0xFFu;
#endif
        w[i] = ((b * 0x40100401u) & 0x80808080u) ^ 0x38383838u;
    }
}

// zeroes the bytes outside [lo, hi) of 16 (a row's end, the anchor's both ends)
CB_HD void tc_mask(uint32_t (&w)[4], int lo, int hi) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int l = lo - 4 * i, h = hi - 4 * i;
        const uint32_t mh = h >= 4 ? 0xFFFFFFFFu : (h <= 0 ? 0u : (1u << (8 * h)) - 1u);
        const uint32_t ml = l <= 0 ? 0xFFFFFFFFu : (l >= 4 ? 0u : 0xFFFFFFFFu << (8 * l));
        w[i] &= mh & ml;
    }
}

// The 16 bases from base b on (b may be negative: zeros) of a packed row of n
// words.
CB_HD uint32_t tc_window(const uint32_t* row, int n, int b) {
    const int wi = b >> 4;                             // floor
    const uint32_t hi = wi >= 0 && wi < n ? row[wi] : 0u;
    const uint32_t lo = wi >= -1 && wi + 1 < n ? row[wi + 1] : 0u;
    return funnel_l(lo, hi, 2 * (b & 15));
}

// The window of a row of length L whose reverse complement is chunk c of the
// row's reverse complement; bases past its end are arbitrary (row[-1] is read
// there: it has to be readable).
CB_HD uint32_t tc_rc_window(const uint32_t* row, int L, int c) {
    const int b = L - 16 - 16 * c;
    const int wi = b >= -16 ? b >> 4 : -1;
    return funnel_l(row[wi + 1], row[wi], 2 * (b & 15));
}

// tc_expand of a window's reverse complement: bytes in reverse order, signs
// flipped. The high bits of a byte go from 1, 3, 5, 7 to 7, 15, 23, 31; the
// four copies meet only at bits 13, 19 and 25, whose carries stop one bit up.
CB_HD void tc_expand_rc(uint32_t x, uint32_t (&w)[4]) {
    x &= 0xAAAAAAAAu;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#ifdef __CUDA_ARCH__
        const uint32_t b = __byte_perm(x, 0u, 0x4440u + (uint32_t)i);
#else
        const uint32_t b = (x >> (8 * i)) & 0xFFu;
#endif
        w[i] = ((b * 0x01041040u) & 0x80808080u) ^ 0xB8B8B8B8u;
    }
}

// Word c of the packed reverse complement of a row of n words and length L
// (the high bases of the last word's tail are arbitrary).
CB_HD uint32_t tc_rc_word(const uint32_t* row, int n, int L, int c) {
    uint32_t w = brev32(tc_window(row, n, L - 16 - 16 * c));
    w = ((w >> 1) & 0x55555555u) | ((w & 0x55555555u) << 1);
    return ~w;
}

// Bases shared at shift s.
CB_HD int tc_overlap(int s, int La, int Lc) { return s >= 0 ? min(La - s, Lc) : min(La, Lc + s); }

// Smallest possible value of the one-bit sum at a shift that the scan could
// accept: mismatches <= mex - 1 bounds the differing high bits.
CB_HD float tc_threshold(int ov, int mex) { return mex > 0 ? (float)(ov - 2 * mex + 2) : 1e9f; }

// Mismatches of the overlap of `ov` bases, row y from its first base against
// row x from base t on: those of 16-base words first, first + step, ...
CB_HD int tc_mismatches(const uint32_t* x, const uint32_t* y, int t, int ov, int first, int step) {
    const int w0 = t >> 4, r = 2 * (t & 15);
    int mm = 0;
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
    for (int j = first; 16 * j < ov; j += step) {
        uint32_t d = funnel_l(x[w0 + j + 1], x[w0 + j], r) ^ y[j];
        d = (d | (d >> 1)) & 0x55555555u;
        const int left = ov - 16 * j;
        if (left < 16) d &= ~(0xFFFFFFFFu >> (2 * left));
        mm += popc32(d);
    }
    return mm;
}

// The same, but any value from cap on when they are not below cap.
CB_HD int tc_mismatches_below(const uint32_t* x, const uint32_t* y, int t, int ov, int cap) {
    const int w0 = t >> 4, r = 2 * (t & 15);
    int mm = 0;
    const uint32_t* xp = x + w0;
    uint32_t hi = xp[0];
    int left = ov;
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
    for (; left >= 32 && mm < cap; left -= 32) {       // two words a step
        const uint32_t m = xp[1], lo = xp[2];
        uint32_t d0 = funnel_l(m, hi, r) ^ y[0], d1 = funnel_l(lo, m, r) ^ y[1];
        hi = lo;
        xp += 2;
        y += 2;
        d0 = (d0 | (d0 >> 1)) & 0x55555555u;
        d1 = (d1 | (d1 >> 1)) & 0x55555555u;
        mm += popc32(d0 | d1 << 1);
    }
    if (left >= 32) return mm;
    for (; left > 0 && mm < cap; left -= 16) {
        const uint32_t lo = xp[1];
        uint32_t d = funnel_l(lo, hi, r) ^ y[0];
        hi = lo;
        ++xp;
        ++y;
        d = (d | (d >> 1)) & 0x55555555u;
        if (left < 16) d &= ~(0xFFFFFFFFu >> (2 * left));
        mm += popc32(d);
    }
    return mm;
}

// Mismatches from which on a shift of overlap ov can no longer improve a column
// whose best keys are `key` (for the mirror, where the overlap is long enough
// for it, `mkey`): a shift of as many mismatches and a lower rank still can.
CB_HD int tc_cap(int ov, int mex, int La, int Lc, uint32_t key, bool mirrored, uint32_t mkey) {
    const uint32_t best = max(key >> 10, mirrored ? mkey >> 10 : 0u);
    return min(mex, (int)best - (La + Lc - 2 * ov) + 1);
}

// Rank of shift s in the scan order 0, 1, ..., then -1, -2, ... (A's shift s
// is -s for (C, A)). Keys are score << 10 | rank; ranks and scores stay below
// 1024.
CB_HD uint32_t tc_rank(int s) { return (uint32_t)(s >= 0 ? s : 512 - s); }
CB_HD int tc_rank_shift(uint32_t r) { return r < 512u ? (int)r : 512 - (int)r; }

// The shift of the mirrored pair (C as anchor, A or its reverse complement as
// candidate) that compares the same bases as (A, C) or (A, rc C) at s.
CB_HD int tc_mirror_shift(int s, int rev, int La, int Lc) { return rev ? s - (La - Lc) : -s; }

// ShdResult of a scan from its best key (all ones: no shift).
CB_HD ShdResult tc_result(uint32_t key, int La, int Lc) {
    ShdResult res;
    const bool ok = key != 0xFFFFFFFFu;
    const int s = ok ? tc_rank_shift(key & 1023u) : -Lc;
    res.valid = ok;
    res.shift = s;
    res.overlap = ok ? tc_overlap(s, La, Lc) : 0;
    res.score = ok ? (int)(key >> 10) : La + Lc;
    res.nops = ok ? res.score - (La + Lc) + 2 * res.overlap : 0;
    return res;
}

// The row of a 128-shift tile as a shift relative to the tile's first: the
// 8-row group m / 8 holds shifts m / 8 + 16 * (m % 8).
CB_HD int tc_row_shift(int m) { return (m >> 3) + 16 * (m & 7); }

// Its bit in a column's four words (one per warp) as the shift's place in the
// tile: lane l of group g (the shifts 32 g + l) finds it in word (l % 16) / 4.
CB_HD int tc_shift_word(int l) { return (l & 15) >> 2; }
CB_HD int tc_shift_bit(int l, int g) { return 8 * (l & 3) + (l >> 4) + 2 * g; }
// The k-th of a tile's four groups from the one nearest shift 0 outwards (the
// overlaps fall that way); outside 0 .. 3 there is none. s0: the first shift.
CB_HD int tc_group(int s0, int k) {
    const int at = -s0 >> 5;
    return (at < 0 ? 0 : at > 3 ? 3 : at) + ((k & 1) ? (k + 1) >> 1 : -(k >> 1));
}

// Chunk x of the anchor's operand bytes: 16 bytes from base q0 + 16 * x on,
// q0 = smax - 127 - 128 * (tiles - 1), zeros outside the read.
CB_HD void tc_q_chunk(const uint32_t* aw, int nwa, int La, int b, uint32_t (&w)[4]) {
    w[0] = w[1] = w[2] = w[3] = 0u;
    if (b <= -16 || b >= La) return;
    tc_expand(tc_window(aw, nwa, b), w);
    if (b < 0 || b + 16 > La) tc_mask(w, -b, La - b);
}

// 16 bytes from byte `r` (0..3) on of the 20 in e.
CB_HD void tc_shift16(const uint32_t (&e)[5], int r, uint32_t (&w)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#ifdef __CUDA_ARCH__
        w[i] = __funnelshift_r(e[i], e[i + 1], 8 * r);
#else
        w[i] = r ? (e[i] >> (8 * r)) | (e[i + 1] << (32 - 8 * r)) : e[i];
#endif
    }
}

// Bound below the threshold of any length: for int(ov * rate) <= ov * rate the
// smallest possible sum is at least (1 - 2 * rate) * ov + 2; the quarter
// covers the rounding of the float expressions.
constexpr float kTcSlack = 1.75f;

}  // namespace careb200
