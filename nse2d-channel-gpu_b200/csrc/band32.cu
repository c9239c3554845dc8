// The FP32-bulk step's row-band kernels and whole steps.
#include "band_host.cuh"

namespace nse2d {

static BandParams<float> band_params(const Context* c) {
    BandParams<float> p{};
    p.hat_in = c->hat32b ? c->hat32b : c->hat32; p.hat_out = c->hat32; p.psi_in = c->psif; p.tw = c->twf_band; p.wN = c->wNf; p.rt = c->rt;
    p.rc = c->rc32;
    p.ctl = c->ctl;
    p.Nx = c->Nx; p.Ny = c->Ny; p.Hp = c->Hp; p.free_slip = c->cfg.free_slip;
    p.nu_dx2 = c->nu * c->inv_dx2; p.lin_drag = c->cfg.lin_drag;
    p.wall_bot = c->wall_bot32; p.wall_top = c->wall_top32;
    return p;
}

int band32_stage(Context* c, int stage, bool inv, float* w_in, const float* w_n, float* w_out, float* rhs_out, cudaStream_t s) {
    return band_stage_impl<float>(c, band_params(c), stage, inv, w_in, w_n, w_out, rhs_out, nullptr, s);
}
int band32_rows_fwd(Context* c, const float* src, cudaStream_t s) { return band_rows_fwd_impl(c, band_params(c), src, 1, c->Ni, s); }
int band32_rows_inv(Context* c, float* w, bool advance, cudaStream_t s) {
    return band_rows_inv_impl(c, band_params(c), c->psif, w, true, advance, s);
}

int band_setup32(Context* c) { return band_setup_impl<float>(c); }
int steps_setup32(Context* c) { return steps_setup_impl<float>(c); }
int launch_steps32(Context* c, int nsteps, int run, int store, cudaStream_t s) {
    StepsParams<float> p{};
    p.b = band_params(c);
    p.th = thomas_params(c, true);
    p.dpsibar = c->rc32 + (size_t)RC_DPB * c->Ny;
    p.w[0] = c->wf; p.w[1] = c->w1f; p.w[2] = c->w2f;
    p.psi = c->psif; p.rhs = c->rhsf;
    return steps_impl(c, p, nsteps, run, store, s);
}

}  // namespace nse2d
