// Launches of whole FP64 steps (steps.cuh).
#include <algorithm>

#include "nse2d_internal.h"
#include "steps.cuh"

namespace nse2d {

template <int M> static int steps_setup_t(Context* c) {
    const int R = std::max(1, (c->Ni + c->num_sms - 1) / c->num_sms);
    if (R > Steps<M>::RMAX || c->Ni > SC_MAX_NI) return 0;
    const size_t sm = steps_smem_bytes<double, M>(R, c->Ni);
    if ((c->H + Steps<M>::KX - 1) / Steps<M>::KX > std::min(c->num_sms, c->Ni)) return 0;      // a group of columns per CTA
    int per_sm = 0;
    if (cudaFuncSetAttribute(k_steps<double, M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)steps_smem_bytes<double, M>(Steps<M>::RMAX, SC_MAX_NI)) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_steps<double, M>, steps_threads<M>(R), sm) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();                                  // the step by launches
        return 0;
    }
    c->steps_R = R;
    return 0;
}

// Whether the context's steps can be taken in one launch: one band per SM, all resident.
int steps_setup(Context* c) {
    int dev = 0, coop = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop || !band_stage_ok(c->M)) return 0;
    switch (c->M) {
        case 32: return steps_setup_t<32>(c);
        case 64: return steps_setup_t<64>(c);
        case 128: return steps_setup_t<128>(c);
        case 256: return steps_setup_t<256>(c);
        case 512: return steps_setup_t<512>(c);
        default: return 0;
    }
}

template <int M> static int steps_t(Context* c, const StepsParams<double>& p, cudaStream_t s) {
    cudaLaunchConfig_t lc{};
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    lc.gridDim = dim3(std::min(c->num_sms, c->Ni));         // bands of floor or ceil(Ni / grid) <= R rows
    lc.blockDim = dim3(steps_threads<M>(p.R));
    lc.dynamicSmemBytes = steps_smem_bytes<double, M>(p.R, c->Ni);
    lc.stream = s;
    lc.attrs = &at;
    lc.numAttrs = 1;
    NSE_CUDA_TRY(cudaLaunchKernelEx(&lc, k_steps<double, M>, p));
    return 0;
}

int launch_steps(Context* c, int nsteps, int run, int store, cudaStream_t s) {
    StepsParams<double> p{};
    p.b = band_params64(c);
    p.th = thomas_params(c);
    p.mx = max_params(c);
    p.w[0] = c->w; p.w[1] = c->w1; p.w[2] = c->w2;
    p.psi = c->psi; p.rhs = c->rhs;
    p.nsteps = nsteps; p.R = c->steps_R; p.run = run; p.store = store;
    switch (c->M) {
        case 32: return steps_t<32>(c, p, s);
        case 64: return steps_t<64>(c, p, s);
        case 128: return steps_t<128>(c, p, s);
        case 256: return steps_t<256>(c, p, s);
        case 512: return steps_t<512>(c, p, s);
        default: set_error("no step kernel for M = %d", c->M); return -1;
    }
}

}  // namespace nse2d
