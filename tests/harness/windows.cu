// Host build of the row windows that the MSA stages its words with
// (care_b200/csrc/device.cuh), over every grid word that a row reaches: which
// words of the row are read, and which codes arrive. Test infrastructure only.
#include "../../care_b200/csrc/device.cuh"

#include <cstring>
#include <vector>

using namespace careb200;

namespace {

// A row that records the indexes asked for; those outside it give a fixed word.
struct CheckedRow {
    const uint32_t* p;
    int n;
    int* range;                                        // lowest and highest index
    const uint32_t* operator+(int i) const {
        static const uint32_t outside = 0xA5C33C5Au;
        if (i < range[0]) range[0] = i;
        if (i > range[1]) range[1] = i;
        return i < 0 || i >= n ? &outside : p + i;
    }
};

uint32_t code_of(const std::vector<uint32_t>& row, int bits, int q) {
    if (bits == 2) return base_at(row.data(), q);
    if (bits == 1) return (row[q >> 5] >> (31 - (q & 31))) & 1u;
    return (row[q >> 2] >> (8 * (q & 3))) & 0xFFu;
}

}  // namespace

// A row of `span` codes of `bits` bits, read by a read of length L at every
// shift against an anchor of up to 256 bases with edge grid words on each
// side. range: lowest and highest word index asked for. Returns the codes that
// arrived wrong.
extern "C" int hd_windows(int bits, int span, int L, int edge, int* range) {
    const int per = 32 / bits, n = (span + per - 1) / per;
    std::vector<uint32_t> row((size_t)n);
    for (int i = 0; i < n; ++i) row[i] = (uint32_t)murmur64((unsigned long long)(i + 1) * 977u + (unsigned)span);
    const CheckedRow cr{row.data(), n, range};
    int wrong = 0;
    for (int shift = -kMaxLen; shift <= kMaxLen; ++shift)
        for (int g = -edge; g < kMaxLen / 16 + edge; ++g) {
            const int p0 = 16 * g, q0 = p0 - shift;
            const int lo = shift - p0 > 0 ? shift - p0 : 0, hi = shift + L - p0 < 16 ? shift + L - p0 : 16;
            if (lo >= hi) continue;                    // the row does not reach the word
            for (int rev = 0; rev < 2; ++rev) {
                const int codes = bits == 8 ? 4 : 16;
                for (int part = 0; part < 16 / codes; ++part) {
                    const int b = staged_start(rev, span, q0, codes, part);
                    const uint32_t w = bits == 2 ? window2(cr, n, b) : bits == 1 ? window1(cr, n, b) : window8(cr, n, b);
                    for (int e = 0; e < codes; ++e) {
                        const int at = codes * part + (rev ? codes - 1 - e : e);      // code of the grid word
                        if (at < lo || at >= hi) continue;
                        const uint32_t got = bits == 2 ? (w >> (30 - 2 * e)) & 3u : bits == 1 ? (w >> (31 - e)) & 1u
                                                                                            : (w >> (8 * e)) & 0xFFu;
                        wrong += got != code_of(row, bits, rev ? span - 1 - (q0 + at) : q0 + at);
                    }
                }
            }
        }
    return wrong;
}
