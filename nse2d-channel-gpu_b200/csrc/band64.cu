// The FP64 row-band kernels and whole steps.
#include "band_host.cuh"

namespace nse2d {

// The transforms of rows of 64 to 2048 points: longer rows have their own kernels (prefetched rows at 4096),
// shorter ones have fewer points than a warp. Bands: of rows of up to 1024 points (see band.cuh), by band_setup.
bool band_rows_ok(int M) { return M >= 32 && M <= 1024; }
bool band_stage_ok(int M) { return M >= 32 && M <= 512; }
// Rows of 2048 points have four to a CTA of 256 threads, and two (FP32: three) CTAs to an SM: a launch takes as long as
// its last round over the SMs. Where that round is less than a quarter full (the fourth, which begins the next wave in
// FP32: half) the transforms of one row per CTA are faster. A step by four rows and by one, us: FP64 2048x600 123 and
// 117, x1184 166 and 182, x1200 193 and 187, x1800 254 and 249, x2300 293 and 316; FP32 x600 96 and 94, x1184 119 and
// 126, x1200 133 and 129, x1800 184 and 170, x2049 193 and 182, x2300 214 and 225.
static int row_round(const Context* c) { return Band<1024>::ROWS_G * c->num_sms; }
bool rows_by_band(const Context* c) {
    if (!band_rows_ok(c->M)) return false;
    if (c->M < 1024) return true;
    const int round = row_round(c), full = c->Ni / round, rest = c->Ni % round;
    return full < 1 || full > 3 || rest == 0 || rest >= (full == 3 ? round / 2 : round / 4);
}
// The Poisson solve alone, three launches from the host, also while the rows of 2048 points are fewer than a round:
// 2048x33 20.7 and 16.6 us, 2048x300 24.7 and 21.8 (in a step the four rows to a CTA are the faster there too, 66 and 68).
bool solve_rows_by_band(const Context* c) { return c->band && !(c->M == 1024 && c->Ni < row_round(c)); }

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
