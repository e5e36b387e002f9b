// Host emulation of the tensor-core alignment (care_b200/csrc/align_tc.cuh)
// for one anchor and its candidates: the operand images and the addresses the
// matrix descriptors form, the sums, both threshold forms, the exact counts
// and the keys. Test infrastructure only.
#include "../../care_b200/csrc/tc_math.cuh"

#include <cstring>
#include <vector>

using namespace careb200;

static float e4m3(uint8_t b) { return b == 0x38 ? 1.0f : b == 0xB8 ? -1.0f : b == 0 ? 0.0f : 1e30f; }

// rows: n candidates of `pitch` words. out: 22 ints per candidate -- score,
// overlap, shift, nops, valid of (A, C), of (A, rc C), of (C, A) and of (C, rc
// A) (for a candidate not shorter than the anchor), then the orientations of
// (A, C) and (C, A). per_column: 1 the threshold form of mixed lengths, 2 that
// form and the counts of a list that overflows (a bit per possible shift,
// counted in groups of 32 by falling overlap, up to what still improves on the
// best). Returns the possible shifts listed, -1 on a byte no operand holds, -2 on an index past
// a buffer.
extern "C" int hd_tc(const uint32_t* a, int La, const uint32_t* rows, int pitch, const int* len, int n, int max_len,
                     int min_overlap, float rate, float ratio, float est, int per_column, int* out) {
    const TcLayout lay = tc_layout(max_len, min_overlap, ratio);
    const int W = lay.W, RS = lay.RS, XL = lay.XL;
    if (n > kTcMaxItems) return -2;
    const int lo = f2i_rz(fmul_rn((float)La, ratio));
    const int minov = min_overlap > lo ? min_overlap : lo;
    const int smax = La - minov, nwa = (La + 15) / 16, nI = (n + 7) & ~7;
    int maxl = 0;
    for (int i = 0; i < n; ++i) maxl = len[i] > maxl ? len[i] : maxl;
    const int smin = minov - maxl;
    const int ntiles = (smax < 0 || maxl < minov) ? 0 : (smax - smin + 128) >> 7;
    if (ntiles > lay.tiles) return -2;
    std::vector<uint32_t> aw(kMaxLen / 16 + 2, 0u), fwp((size_t)kTcMaxItems * RS + 1, 0x5a5a5a5au), ar(kMaxLen / 16 + 2, 0u);
    uint32_t* fw = fwp.data() + 1;                     // a word before the first row is read
    for (int i = 0; i < nwa; ++i) aw[i] = a[i];
    for (int i = 0; i < nwa; ++i) ar[i] = tc_rc_word(aw.data(), nwa, La, i);
    std::vector<uint8_t> top(lay.b - lay.top), b((size_t)2 * kTcMaxItems * 16 * W, 0x7f);
    for (int i = 0; i < n; ++i)
        for (int w = 0; w < W; ++w) fw[i * RS + w] = 16 * w < len[i] ? rows[(size_t)i * pitch + w] : 0u;
    for (int i = 0; i < n; ++i)
        for (int c = 0; c < W; ++c)
            for (int rev = 0; rev < 2; ++rev) {
                uint32_t w[4];
                if (rev) tc_expand_rc(tc_rc_window(&fw[i * RS], len[i], c), w);
                else tc_expand(fw[i * RS + c], w);
                if (len[i] - 16 * c < 16) tc_mask(w, 0, len[i] - 16 * c);
                const int row = rev * nI + i;
                std::memcpy(&b[(size_t)(row >> 3) * (128 * W) + c * 128 + (row & 7) * 16], w, 16);
            }
    std::vector<uint32_t> q((size_t)(XL + 1) * 4);
    if ((uint32_t)q.size() * 4 > lay.top - lay.q) return -2;
    for (int x = 0; x <= XL; ++x) {
        uint32_t w[4];
        tc_q_chunk(aw.data(), nwa, La, smax - 127 - 128 * (lay.tiles - 1) + 16 * x, w);
        std::memcpy(&q[4 * x], w, 16);
    }
    for (int rho = 0; rho < 16; ++rho)
        for (int x = 0; x < XL; ++x) {
            uint32_t e[5], w[4];
            std::memcpy(e, &q[4 * x + (rho >> 2)], 20);
            tc_shift16(e, rho & 3, w);
            if ((size_t)(rho * XL + x) * 16 + 16 > top.size()) return -2;
            std::memcpy(&top[(size_t)(rho * XL + x) * 16], w, 16);
        }
    for (int idx = 0; idx < kTcMaxItems * W; ++idx)
        if ((int)(((uint32_t)idx * lay.magic_w) >> 16) != idx / W) return -2;
    std::vector<uint32_t> key((size_t)4 * n, 0xFFFFFFFFu);
    const float kappa = 1.0f - 2.0f * rate;
    int hits = 0;
    const int K = 32 * ((maxl + 31) / 32);
    for (int t = 0; t < ntiles; ++t) {
        std::vector<uint32_t> bits((size_t)4 * 2 * n, 0u);       // a column's words, one per warp
        for (int m = 0; m < 128; ++m) {
            const int s = smax - 127 - 128 * t + tc_row_shift(m);
            for (int col = 0; col < 2 * n; ++col) {
                const int rev = col >= n, it = col - rev * n, row = rev * nI + it, Lc = len[it];
                float d = 0.0f;
                for (int k = 0; k < K; ++k) {
                    const size_t ea = (size_t)8 * (lay.tiles - 1 - t) * 16 + (size_t)(m >> 3) * (16 * XL) + (k >> 4) * 16 + (m & 7) * 16 + (k & 15);
                    const size_t eb = (size_t)(row >> 3) * (128 * W) + (k >> 4) * 128 + (row & 7) * 16 + (k & 15);
                    if (ea >= top.size() || eb >= b.size()) return -2;
                    d += e4m3(top[ea]) * e4m3(b[eb]);
                }
                if (d > 1e6f || d < -1e6f) return -1;
                if (s < smin) continue;
                float thr = 1e9f;
                if (!per_column) {
                    const int ov = tc_overlap(s, La, Lc);
                    if (ov >= minov) thr = tc_threshold(ov, f2i_rz(fmul_rn((float)ov, rate)));
                } else {
                    const int u = s > 0 ? s : 0;
                    const float c1 = kappa * (float)(La - u) + kTcSlack, c2 = kappa * (float)(s - u) + kTcSlack;
                    const float cm = kappa * (float)minov + kTcSlack;
                    const float e = kappa * (float)Lc + c2;
                    thr = e < c1 ? e : c1;
                    thr = thr > cm ? thr : cm;
                }
                if (!(d >= thr)) continue;
                ++hits;
                if (per_column == 2) {
                    bits[(size_t)4 * col + (m >> 5)] |= 1u << (m & 31);
                    continue;
                }
                const int ov = tc_overlap(s, La, Lc);
                if (ov < minov) continue;
                // the reverse complement's shift, seen from the anchor's reverse complement
                const uint32_t *cr = &fw[it * RS], *an = rev ? ar.data() : aw.data();
                const int sv = rev ? La - Lc - s : s;
                const int mex = f2i_rz(fmul_rn((float)ov, rate));
                int mm = 0;
                for (int part = 0; part < 4; ++part)
                    mm += sv >= 0 ? tc_mismatches(an, cr, sv, ov, part, 4) : tc_mismatches(cr, an, -sv, ov, part, 4);
                if (mm >= mex) continue;
                const uint32_t sc = (uint32_t)(mm + La + Lc - 2 * ov) << 10;
                uint32_t& ka = key[rev * n + it];
                ka = ka < (sc | tc_rank(s)) ? ka : sc | tc_rank(s);
                const int lc = f2i_rz(fmul_rn((float)Lc, ratio));
                if (ov < (min_overlap > lc ? min_overlap : lc)) continue;
                uint32_t& kc = key[(2 + rev) * n + it];
                const uint32_t m = sc | tc_rank(tc_mirror_shift(s, rev, La, Lc));
                kc = kc < m ? kc : m;
            }
        }
        const int s0 = smax - 127 - 128 * t;
        for (int col = 0; per_column == 2 && col < 2 * n; ++col) {
            const int rev = col >= n, it = col - rev * n, Lc = len[it];
            const uint32_t *cr = &fw[it * RS], *an = rev ? ar.data() : aw.data();
            const int lc = f2i_rz(fmul_rn((float)Lc, ratio)), minlc = min_overlap > lc ? min_overlap : lc;
            int seen = 0;
            for (int k = 0; k < 7; ++k) {
                const int g = tc_group(s0, k);
                if ((unsigned)g > 3u) continue;
                seen |= 1 << g;
                uint32_t ka = key[rev * n + it], kc = key[(2 + rev) * n + it];
                const uint32_t ka0 = ka, kc0 = kc;               // what the group's lanes see
                for (int lane = 0; lane < 32; ++lane) {
                    const int s = s0 + 32 * g + lane, ov = tc_overlap(s, La, Lc);
                    if (tc_row_shift(32 * tc_shift_word(lane) + tc_shift_bit(lane, g)) != 32 * g + lane) return -2;
                    if (!((bits[(size_t)4 * col + tc_shift_word(lane)] >> tc_shift_bit(lane, g)) & 1u)) continue;
                    const bool mirrored = ov >= minlc;
                    const int cap = ov < minov ? 0 : tc_cap(ov, f2i_rz(fmul_rn((float)ov, rate)), La, Lc, ka0, mirrored, kc0);
                    if (cap <= 0) continue;
                    const int sv = rev ? La - Lc - s : s;
                    const int mm = sv >= 0 ? tc_mismatches_below(an, cr, sv, ov, cap) : tc_mismatches_below(cr, an, -sv, ov, cap);
                    if (mm >= cap) continue;
                    const uint32_t sc = (uint32_t)(mm + La + Lc - 2 * ov) << 10;
                    const uint32_t x = sc | tc_rank(s), y = sc | tc_rank(tc_mirror_shift(s, rev, La, Lc));
                    ka = ka < x ? ka : x;
                    if (mirrored) kc = kc < y ? kc : y;
                }
                key[rev * n + it] = ka;
                key[(2 + rev) * n + it] = kc;
            }
            if (seen != 15) return -2;
        }
    }
    for (int it = 0; it < n; ++it) {
        const int L = len[it];
        const ShdResult rs[4] = {tc_result(key[it], La, L), tc_result(key[n + it], La, L),
                                 tc_result(key[2 * n + it], L, La), tc_result(key[3 * n + it], L, La)};
        int* o = out + 22 * it;
        for (int k = 0; k < 4; ++k) {
            o[5 * k] = rs[k].score; o[5 * k + 1] = rs[k].overlap; o[5 * k + 2] = rs[k].shift;
            o[5 * k + 3] = rs[k].nops; o[5 * k + 4] = rs[k].valid;
        }
        o[20] = choose_orientation(rs[0], rs[1], La, ratio, min_overlap, fmul_rn(est, 4.0f));
        o[21] = choose_orientation(rs[2], rs[3], L, ratio, min_overlap, fmul_rn(est, 4.0f));
    }
    return hits;
}

extern "C" int hd_tc_faster(int max_len, int min_overlap, float ratio, float coverage, unsigned anchors, int mirror) {
    return tc_faster(max_len, min_overlap, ratio, coverage, anchors, mirror != 0, 0.0f);
}
