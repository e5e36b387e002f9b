// The tensor-core alignment with a given limit of its completion waits and the
// MSA behind it, on n reads of length L that are all candidates of one another.
// Test infrastructure only.
#include "../../care_b200/csrc/align_tc.cuh"

#include <vector>

using namespace careb200;

namespace {

struct Buf {
    void* p = nullptr;
    ~Buf() { cudaFree(p); }
    template <class T> T* as() const { return static_cast<T*>(p); }
    bool fill(const void* src, size_t n) {
        return cudaMalloc(&p, n) == cudaSuccess && cudaMemcpy(p, src, n, cudaMemcpyHostToDevice) == cudaSuccess;
    }
    bool set(int byte, size_t n) {
        return cudaMalloc(&p, n) == cudaSuccess && cudaMemset(p, byte, n) == cudaSuccess;
    }
};

}  // namespace

// rows: n rows of (L + 15) / 16 words. ares: 8 bytes per pair. corrected: the
// MSA's status byte of each read, 0x5a before. queue: the MSA's persistent
// form. status: the status word after the kernels. Returns 0, or -1 on a CUDA
// error.
extern "C" int gpu_align_with_limit(const uint32_t* rows, int n, int L, uint32_t limit, int grid, int queue,
                                    void* ares, void* corrected, int* status) {
    const int pitch = (L + 15) / 16;
    const size_t pairs = (size_t)n * (n - 1);
    std::vector<uint32_t> ids, off, cnt;
    for (int i = 0; i < n; ++i) {
        off.push_back((uint32_t)ids.size());
        cnt.push_back((uint32_t)n - 1);
        for (int j = 0; j < n; ++j) if (j != i) ids.push_back((uint32_t)j);
    }
    const std::vector<int> len((size_t)n, L);
    const unsigned long long total = pairs;
    Buf d_seq, d_len, d_ids, d_off, d_cnt, d_total, d_status, d_ares, d_cursor, d_recs, d_ambig, d_out, d_edits, d_cseq;
    if (!d_seq.fill(rows, (size_t)n * pitch * 4) || !d_len.fill(len.data(), (size_t)n * 4) ||
        !d_ids.fill(ids.data(), pairs * 4) || !d_off.fill(off.data(), (size_t)n * 4) ||
        !d_cnt.fill(cnt.data(), (size_t)n * 4) || !d_total.fill(&total, 8) || !d_status.set(0, 16) ||
        !d_ares.set(0x5a, pairs * sizeof(AlignRes)) || !d_cursor.set(0, 16) ||
        !d_recs.set(0, pairs * sizeof(CandRec)) || !d_ambig.set(0, (size_t)n) || !d_out.set(0x5a, (size_t)n) ||
        !d_edits.set(0, (size_t)n * 4) || !d_cseq.set(0, (size_t)n * L))
        return -1;
    DevOptions o{};
    o.min_overlap = 30;
    o.min_overlap_ratio = 0.3f;
    o.max_error_rate = 0.2f;
    o.estimated_errorrate = 0.06f;
    o.estimated_coverage = 30.0f;
    o.m_coverage = 0.6f;
    o.coverage_int = 30;
    DevReads r{};
    r.seq = d_seq.as<uint32_t>();
    r.len = d_len.as<int32_t>();
    r.ambig = d_ambig.as<uint8_t>();
    r.seq_pitch = pitch;
    r.max_len = L;
    r.n = (uint32_t)n;
    const TcLayout lay = tc_layout(L, o.min_overlap, o.min_overlap_ratio);
    k_align_tc<<<grid, kTcBlock, lay.total>>>(o, r, 0, (uint32_t)n, d_ids.as<uint32_t>(), d_off.as<uint32_t>(),
                                              d_cnt.as<uint32_t>(), d_total.as<unsigned long long>(), pairs,
                                              d_status.as<int>(), d_ares.as<AlignRes>(), nullptr, nullptr,
                                              d_cursor.as<unsigned int>(), 1, lay, limit);
    if (cudaGetLastError() != cudaSuccess) return -1;
    MsaOut mo{};
    mo.status = d_out.as<uint8_t>();
    mo.nedits = d_edits.as<int32_t>();
    mo.seq = d_cseq.as<char>();
    const MsaGrid mg = msa_grid(L, 0, 0, 0);
    const size_t smem = msa_smem_bytes(mg, L, false);
    if (smem > 48 * 1024) return -1;
    if (queue)
        k_msa_queue<128, 0><<<grid, 128, smem>>>(o, r, 0, (uint32_t)n, mg, nullptr, d_cursor.as<unsigned int>() + 1,
                                                 d_ids.as<uint32_t>(), d_off.as<uint32_t>(), d_cnt.as<uint32_t>(),
                                                 d_ares.as<AlignRes>(), d_recs.as<CandRec>(), mo, d_status.as<int>());
    else
        k_msa<128, 0><<<n, 128, smem>>>(o, r, 0, (uint32_t)n, mg, nullptr, d_ids.as<uint32_t>(), d_off.as<uint32_t>(),
                                        d_cnt.as<uint32_t>(), d_ares.as<AlignRes>(), d_recs.as<CandRec>(), mo,
                                        d_status.as<int>());
    if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) return -1;
    if (cudaMemcpy(corrected, d_out.p, (size_t)n, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    if (cudaMemcpy(status, d_status.p, 4, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    return cudaMemcpy(ares, d_ares.p, pairs * sizeof(AlignRes), cudaMemcpyDeviceToHost) == cudaSuccess ? 0 : -1;
}
