// Launches of the row-band kernels and of whole steps (band.cuh, steps.cuh), for one precision.
#pragma once
#include <algorithm>

#include "nse2d_internal.h"
#include "steps.cuh"

namespace nse2d {

#define NSE_BAND512_DISPATCH(FN, ...)                                          \
    switch (c->M) {                                                            \
        case 32: return FN<T, 32>(__VA_ARGS__);                                \
        case 64: return FN<T, 64>(__VA_ARGS__);                                \
        case 128: return FN<T, 128>(__VA_ARGS__);                              \
        case 256: return FN<T, 256>(__VA_ARGS__);                              \
        case 512: return FN<T, 512>(__VA_ARGS__);                              \
        default: set_error("no band kernel for M = %d", c->M); return -1;      \
    }
#define NSE_BAND_DISPATCH(FN, ...)                                             \
    if (c->M == 1024) return FN<T, 1024>(__VA_ARGS__);                         \
    NSE_BAND512_DISPATCH(FN, __VA_ARGS__)

template <typename T, int M, bool INV> int band_kernel_t(Context* c, BandParams<T>& p, cudaStream_t s) {
    // rows per band: one band per SM while it fits, so that a launch is one wave; the bands of channels that run
    // together are counted together, since every band transforms two halo rows more than its own (an ensemble step of 4,
    // 8 and 12 channels of 256 to 1024 points by 129 to 513 rows: 118, 139 and 210 us without, 111, 115 and 183 with it)
    const int R = std::max(1, (int)std::min<long long>(Band<M>::RMAX, ((long long)c->Ni * c->band_share + c->num_sms - 1) / c->num_sms));
    const size_t sm = band_smem_bytes<T, M>(R);
    NSE_CUDA_TRY(cudaFuncSetAttribute(k_band<T, M, INV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)band_smem_bytes<T, M>(Band<M>::RMAX)));
    return launch_step_kernel(c, k_band<T, M, INV>, dim3((c->Ni + R - 1) / R), dim3((R + 2) * Band<M>::TPR), sm, s, nullptr, p);
}
template <typename T, int M> int band_inv_t(Context* c, BandParams<T>& p, cudaStream_t s) { return band_kernel_t<T, M, true>(c, p, s); }
template <typename T, int M> int band_psi_t(Context* c, BandParams<T>& p, cudaStream_t s) { return band_kernel_t<T, M, false>(c, p, s); }
template <typename T, int M> int rows_fwd_t(Context* c, BandParams<T>& p, cudaStream_t s) {
    constexpr size_t sm = band_rows_smem_bytes<T, M>();
    NSE_CUDA_TRY(cudaFuncSetAttribute(k_rows_fwd<T, M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    constexpr int G = Band<M>::ROWS_G;
    return launch_step_kernel(c, k_rows_fwd<T, M>, dim3((p.nrows + G - 1) / G), dim3(G * Band<M>::TPR), sm, s, nullptr, p);
}
template <typename T, int M> int rows_inv_t(Context* c, BandParams<T>& p, cudaStream_t s) {
    constexpr size_t sm = band_rows_smem_bytes<T, M>();
    NSE_CUDA_TRY(cudaFuncSetAttribute(k_rows_inv<T, M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    constexpr int G = Band<M>::ROWS_G;
    return launch_step_kernel(c, k_rows_inv<T, M>, dim3((c->Ni + G - 1) / G), dim3(G * Band<M>::TPR), sm, s, nullptr, p);
}

// Whether a channel steps by bands: while all of them, of the most rows, are resident at once; of rows of up to 256
// points, whose bands are the short ones, in two rounds. Beyond that line a band is a second (third) wave in which most
// SMs idle, its two halo rows are transformed by CTAs that have no time left over, and psi-hat's own buffer is one more
// in L2; the separate kernels have finer tiles. A step by bands and by separate kernels either side of it, us: FP64
// 1024x594 65 and 76, 1024x600 87 and 84; 512x890 58 and 70, 512x900 78 and 70; 128x1778 57 and 59, 128x1800 66 and 60;
// FP32 58 and 68, 75 and 72; 50 and 62, 66 and 60; 128x3552 64 and 70, 128x3600 72 and 70. Far beyond: FP64 1024x4097
// 322 and 264, FP32 251 and 207, 512x8193 413 and 351.
template <typename T, int M> int band_setup_t(Context* c) {
    using B = Band<M>;
    int per_sm = 0;
    NSE_CUDA_TRY(cudaFuncSetAttribute(k_band<T, M, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)band_smem_bytes<T, M>(B::RMAX)));
    NSE_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_band<T, M, true>, B::MAXT, band_smem_bytes<T, M>(B::RMAX)));
    if (per_sm < 1) return 0;                                // separate kernels
    c->band_load = (double)((c->Ni + B::RMAX - 1) / B::RMAX) / ((double)per_sm * c->num_sms);
    c->band_fit = c->band_load <= (M <= 128 ? 2.0 : 1.0);
    return 0;
}
template <typename T> int band_setup_impl(Context* c) {
    if (!band_stage_ok(c->M)) return 0;
    NSE_BAND512_DISPATCH(band_setup_t, c)
}

// Stage `stage` of the step and the forward transform of its omega^(s+1); inv: the inverse transform of
// psi-hat and the wall closure of w_in before it (else psi is read from the context's psi).
template <typename T>
int band_stage_impl(Context* c, BandParams<T> p, int stage, bool inv, T* w_in, const T* w_n, T* w_out, T* rhs_out, const double* closure,
                    cudaStream_t s) {
    p.stage = stage; p.w_in = w_in; p.w_n = w_n; p.w_out = w_out; p.rhs_out = rhs_out; p.closure = closure;
    if (inv) { NSE_BAND512_DISPATCH(band_inv_t, c, p, s) }
    NSE_BAND512_DISPATCH(band_psi_t, c, p, s)
}
template <typename T> int band_rows_fwd_impl(Context* c, BandParams<T> p, const T* src, int row0, int nrows, cudaStream_t s) {
    p.src = src; p.row0 = row0; p.nrows = nrows;
    NSE_BAND_DISPATCH(rows_fwd_t, c, p, s)
}
template <typename T> int band_rows_inv_impl(Context* c, BandParams<T> p, T* psi, T* w, bool thom, bool advance, cudaStream_t s) {
    p.psi_out = psi; p.w_in = w; p.do_thom = thom ? 1 : 0; p.advance = advance ? 1 : 0;
    NSE_BAND_DISPATCH(rows_inv_t, c, p, s)
}

template <typename T, int M> int steps_setup_t(Context* c) {
    const int R = std::max(1, (c->Ni + c->num_sms - 1) / c->num_sms);
    if (R > Steps<M>::RMAX || c->Ni > SC_MAX_NI) return 0;
    if ((c->H + Steps<M>::KX - 1) / Steps<M>::KX > std::min(c->num_sms, c->Ni)) return 0;      // a group of columns per CTA
    const size_t sm = steps_smem_bytes<T, M>(R, c->Ni);
    int per_sm = 0;
    if (cudaFuncSetAttribute(k_steps<T, M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)steps_smem_bytes<T, M>(Steps<M>::RMAX, SC_MAX_NI)) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_steps<T, M>, steps_threads<M>(R), sm) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();                                  // the step by launches
        return 0;
    }
    c->steps_R = R;
    return 0;
}
// Whether the context's steps can be taken in one launch: one band per SM, all resident.
template <typename T> int steps_setup_impl(Context* c) {
    int dev = 0, coop = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop || !band_stage_ok(c->M)) return 0;
    NSE_BAND512_DISPATCH(steps_setup_t, c)
}

template <typename T, int M> int steps_t(Context* c, const StepsParams<T>& p, cudaStream_t s) {
    cudaLaunchConfig_t lc{};
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    lc.gridDim = dim3(std::min(c->num_sms, c->Ni));         // bands of floor or ceil(Ni / grid) <= R rows
    lc.blockDim = dim3(steps_threads<M>(p.R));
    lc.dynamicSmemBytes = steps_smem_bytes<T, M>(p.R, c->Ni);
    lc.stream = s;
    lc.attrs = &at;
    lc.numAttrs = 1;
    NSE_CUDA_TRY(cudaLaunchKernelEx(&lc, k_steps<T, M>, p));
    return 0;
}
template <typename T> int steps_impl(Context* c, StepsParams<T> p, int nsteps, int run, int store, cudaStream_t s) {
    p.mx = max_params(c);
    p.nsteps = nsteps; p.R = c->steps_R; p.run = run; p.store = store;
    NSE_BAND512_DISPATCH(steps_t, c, p, s)
}

}  // namespace nse2d
