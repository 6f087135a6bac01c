// qz_sweep.cu -- stand-alone sweep launch: one CTA runs the whole xi sweep of one time step
// (the sweep itself is in qz_sweep_body.cuh).
#include "qz_sweep_body.cuh"

namespace qzb {

// EXT: the variant for decks with the smoothing filter, static (analytic) beam sources or adaptive sub-slicing (sweep_ext)
template <int ORD, bool REG, int kMaxR, bool EXT>
__global__ void __launch_bounds__(kSweepThreads, 1) sweep_m0_kernel(const SweepArgs A) {
    extern __shared__ double smem_raw[];
    NoGate g;
    sweep_body<ORD, REG, kMaxR, NoGate, EXT>(A, smem_raw, g);
}

size_t sweep_m0_smem_bytes(int M, bool dbuf, bool const_smem, bool filter, int pcache) {
    size_t d = (size_t)(3 + 2 + 6 + (dbuf ? 18 : 9)) * M + sweep_detail::kTot;
    if (const_smem) d += (size_t)consts0_arrays(M) * M;
    if (filter) d += 4 * (size_t)M + 2 * 14 * (kSweepThreads / 32);
    // + the words from Smem::lost on, and with the particle copy 6 doubles and a cell index per particle
    return sizeof(double) * d + sweep_detail::kMiscBytes + (pcache > 0 ? (size_t)pcache * (6 * sizeof(double) + sizeof(int)) : 0);
}

static int hist_of(const SweepArgs& A, bool ext) {
    return sweep_detail::hist_doubles(A.ord, A.np <= kSweepThreads, A.rows_per_thread == 1 ? 1 : 3, ext);
}

bool sweep_m0_dbuf(const SweepArgs& A, bool ext) { return A.dbuf && !hist_of(A, ext); }

size_t sweep_m0_smem_bytes(const SweepArgs& A, bool ext) {
    const int hist = hist_of(A, ext);
    // (the variant with the history lays its arrays out kSweepThreads nodes apart: carve)
    return sweep_m0_smem_bytes(hist ? kSweepThreads : A.M, sweep_m0_dbuf(A, ext), consts_in_smem(A), A.filter != 0, A.pcache) +
           sizeof(double) * hist * kSweepThreads;
}

namespace {
template <int ORD, bool REG, int RM, bool EXT>
cudaError_t launch_t(const SweepArgs& A, size_t smem, cudaStream_t stream) {
    cudaError_t e = cudaFuncSetAttribute(sweep_m0_kernel<ORD, REG, RM, EXT>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    sweep_m0_kernel<ORD, REG, RM, EXT><<<1, kSweepThreads, smem, stream>>>(A);
    return cudaGetLastError();
}

template <int ORD, bool EXT>
cudaError_t launch_e(const SweepArgs& A, size_t smem, cudaStream_t stream) {
    const bool reg = A.np <= kSweepThreads;
    if (A.rows_per_thread == 1)
        return reg ? launch_t<ORD, true, 1, EXT>(A, smem, stream) : launch_t<ORD, false, 1, EXT>(A, smem, stream);
    return reg ? launch_t<ORD, true, 3, EXT>(A, smem, stream) : launch_t<ORD, false, 3, EXT>(A, smem, stream);
}

template <int ORD>
cudaError_t launch_o(const SweepArgs& A, size_t smem, cudaStream_t stream) {
    return sweep_ext(A) ? launch_e<ORD, true>(A, smem, stream) : launch_e<ORD, false>(A, smem, stream);
}
}  // namespace

cudaError_t launch_sweep_m0(const SweepArgs& A, cudaStream_t stream) {
    if (A.rows_per_thread < 1 || A.rows_per_thread > 3) return cudaErrorInvalidValue;
    const size_t smem = sweep_m0_smem_bytes(A, sweep_ext(A));
    switch (A.ord) {
        case 1: return launch_o<1>(A, smem, stream);
        case 2: return launch_o<2>(A, smem, stream);
        case 3: return launch_o<3>(A, smem, stream);
        case 4: return launch_o<4>(A, smem, stream);
        case 5: return launch_o<5>(A, smem, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace qzb
