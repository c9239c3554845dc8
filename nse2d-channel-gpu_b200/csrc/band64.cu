// Launches of the FP64 row-band kernels (band.cuh).
#include <algorithm>

#include "nse2d_internal.h"
#include "band.cuh"

namespace nse2d {

// The transforms of rows of 64 to 2048 points: longer rows have their own kernels (prefetched rows at 4096),
// shorter ones have fewer points than a warp. Bands: see band.cuh for where the line lies.
bool band_rows_ok(int M) { return M >= 32 && M <= 1024; }
bool band_stage_ok(int M) { return M >= 32 && M <= 512; }

// Rows per band: one band per SM while it fits, so that a launch is one wave.
static int band_R(const Context* c, int rmax) { return std::max(1, std::min(rmax, (c->Ni + c->num_sms - 1) / c->num_sms)); }

BandParams<double> band_params64(const Context* c) {
    BandParams<double> p{};
    p.hat_in = c->hat2 ? c->hat2 : c->hat; p.hat_out = c->hat; p.psi_in = c->psi; p.tw = c->tw_band; p.wN = c->wN; p.rt = c->rt; p.ctl = c->ctl;
    p.Nx = c->Nx; p.Ny = c->Ny; p.Hp = c->Hp; p.free_slip = c->cfg.free_slip;
    p.nu_dx2 = c->nu * c->inv_dx2; p.lin_drag = c->cfg.lin_drag;
    p.psi_bot = c->psi_bot; p.psi_top = c->psi_top;
    return p;
}

#define NSE_BAND512_DISPATCH(FN)                                               \
    switch (c->M) {                                                            \
        case 32: return FN<32>(c, p, s);     case 64: return FN<64>(c, p, s);   \
        case 128: return FN<128>(c, p, s);   case 256: return FN<256>(c, p, s); \
        case 512: return FN<512>(c, p, s);                                      \
        default: set_error("no band kernel for M = %d", c->M); return -1;       \
    }
#define NSE_BAND_DISPATCH(FN)                                                  \
    switch (c->M) {                                                            \
        case 32: return FN<32>(c, p, s);     case 64: return FN<64>(c, p, s);   \
        case 128: return FN<128>(c, p, s);   case 256: return FN<256>(c, p, s); \
        case 512: return FN<512>(c, p, s);   case 1024: return FN<1024>(c, p, s); \
        default: set_error("no band kernel for M = %d", c->M); return -1;       \
    }

template <int M, bool INV> static int band_t(Context* c, BandParams<double>& p, cudaStream_t s) {
    const int R = band_R(c, Band<M>::RMAX);
    const size_t sm = band_smem_bytes<double, M>(R);
    NSE_CUDA_TRY(cudaFuncSetAttribute(k_band<double, M, INV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)band_smem_bytes<double, M>(Band<M>::RMAX)));
    return launch_step_kernel(c, k_band<double, M, INV>, dim3((c->Ni + R - 1) / R), dim3((R + 2) * Band<M>::TPR), sm, s, nullptr, p);
}
template <int M> static int band_inv_t(Context* c, BandParams<double>& p, cudaStream_t s) { return band_t<M, true>(c, p, s); }
template <int M> static int band_psi_t(Context* c, BandParams<double>& p, cudaStream_t s) { return band_t<M, false>(c, p, s); }
template <int M> static int rows_fwd_t(Context* c, BandParams<double>& p, cudaStream_t s) {
    constexpr size_t sm = band_rows_smem_bytes<double, M>();
    NSE_CUDA_TRY(cudaFuncSetAttribute(k_rows_fwd<double, M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    constexpr int G = Band<M>::ROWS_G;
    return launch_step_kernel(c, k_rows_fwd<double, M>, dim3((p.nrows + G - 1) / G), dim3(G * Band<M>::TPR), sm, s, nullptr, p);
}
template <int M> static int rows_inv_t(Context* c, BandParams<double>& p, cudaStream_t s) {
    constexpr size_t sm = band_rows_smem_bytes<double, M>();
    NSE_CUDA_TRY(cudaFuncSetAttribute(k_rows_inv<double, M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    constexpr int G = Band<M>::ROWS_G;
    return launch_step_kernel(c, k_rows_inv<double, M>, dim3((c->Ni + G - 1) / G), dim3(G * Band<M>::TPR), sm, s, nullptr, p);
}

// Stage `stage` of the step and the forward transform of its omega^(s+1); inv: the inverse transform of
// psi-hat and the wall closure of w_in before it (else psi is read from the context's psi).
int band_stage(Context* c, int stage, bool inv, double* w_in, const double* w_n, double* w_out, double* rhs_out,
               const double* closure, cudaStream_t s) {
    BandParams<double> p = band_params64(c);
    p.stage = stage; p.w_in = w_in; p.w_n = w_n; p.w_out = w_out; p.rhs_out = rhs_out; p.closure = closure;
    if (inv) { NSE_BAND512_DISPATCH(band_inv_t) }
    NSE_BAND512_DISPATCH(band_psi_t)
}

int band_rows_fwd(Context* c, const double* src, int row0, int nrows, cudaStream_t s) {
    BandParams<double> p = band_params64(c);
    p.src = src; p.row0 = row0; p.nrows = nrows;
    NSE_BAND_DISPATCH(rows_fwd_t)
}

int band_rows_inv(Context* c, double* psi, double* w, bool thom, bool advance, cudaStream_t s) {
    BandParams<double> p = band_params64(c);
    p.psi_out = psi; p.w_in = w; p.do_thom = thom ? 1 : 0; p.advance = advance ? 1 : 0;
    NSE_BAND_DISPATCH(rows_inv_t)
}

}  // namespace nse2d
