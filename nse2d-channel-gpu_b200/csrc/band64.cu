// The FP64 row-band kernels and whole steps.
#include "band_host.cuh"

namespace nse2d {

// The transforms of rows of 64 to 2048 points: longer rows have their own kernels (prefetched rows at 4096),
// shorter ones have fewer points than a warp. Bands: of rows of up to 1024 points (see band.cuh), by band_setup.
bool band_rows_ok(int M) { return M >= 32 && M <= 1024; }
bool band_stage_ok(int M) { return M >= 32 && M <= 512; }

static BandParams<double> band_params(const Context* c) {
    BandParams<double> p{};
    p.hat_in = c->hat2 ? c->hat2 : c->hat; p.hat_out = c->hat; p.psi_in = c->psi; p.tw = c->tw_band; p.wN = c->wN; p.rt = c->rt;
    p.ctl = c->ctl;
    p.Nx = c->Nx; p.Ny = c->Ny; p.Hp = c->Hp; p.free_slip = c->cfg.free_slip;
    p.nu_dx2 = c->nu * c->inv_dx2; p.lin_drag = c->cfg.lin_drag;
    p.psi_bot = c->psi_bot; p.psi_top = c->psi_top;
    return p;
}

int band_stage(Context* c, int stage, bool inv, double* w_in, const double* w_n, double* w_out, double* rhs_out, const double* closure,
               cudaStream_t s) {
    return band_stage_impl(c, band_params(c), stage, inv, w_in, w_n, w_out, rhs_out, closure, s);
}
int band_rows_fwd(Context* c, const double* src, int row0, int nrows, cudaStream_t s) {
    return band_rows_fwd_impl(c, band_params(c), src, row0, nrows, s);
}
int band_rows_inv(Context* c, double* psi, double* w, bool thom, bool advance, cudaStream_t s) {
    return band_rows_inv_impl(c, band_params(c), psi, w, thom, advance, s);
}

int band_setup(Context* c) { return band_setup_impl<double>(c); }
int steps_setup(Context* c) { return c->prec32 ? steps_setup32(c) : steps_setup_impl<double>(c); }
int launch_steps(Context* c, int nsteps, int run, int store, cudaStream_t s) {
    if (c->prec32) return launch_steps32(c, nsteps, run, store, s);
    StepsParams<double> p{};
    p.b = band_params(c);
    p.th = thomas_params(c);
    p.w[0] = c->w; p.w[1] = c->w1; p.w[2] = c->w2;
    p.psi = c->psi; p.rhs = c->rhs;
    return steps_impl(c, p, nsteps, run, store, s);
}

}  // namespace nse2d
