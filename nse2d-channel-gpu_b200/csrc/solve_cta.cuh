// The tridiagonal solve of a few columns by one CTA, for grids of up to 514 rows. Written for this project.
//
// The arithmetic is k_thomas_cluster's (segments of rows in registers, joined through their affine carries), with
// all interior rows of KX columns in one CTA of 256 threads: 256 / KX segments of L rows, so the carries cross a
// warp by shuffles and eight warps through shared memory, with two barriers, and nothing crosses CTAs. On a short
// grid the cluster form's start-up, its exchanges between CTAs (about 1000 clocks each way) and its tensor-map
// loads were most of its time. Step with the cluster form and with this one: 128x129 34.9 and 30.7 us, 256x257
// 39.4 and 32.8, 1024x513 66.4 and 59.4. From 515 rows on a segment would be 16 rows (or the columns fewer than a
// 32-byte sector); those grids keep the cluster form.
#pragma once
#include "step_kernels.cuh"

namespace nse2d {

constexpr int SC_NT = 256;
constexpr int SC_NW = SC_NT / 32;
template <int KX> struct SolveSmem {
    double2 D[2][SC_NW][KX];
    double P[2][SC_NW][KX];
};

// threads 0 .. 255 of a CTA (bar.sync 15)
__device__ __forceinline__ void sc_sync() { asm volatile("bar.sync 15, %0;\n" ::"n"(SC_NT) : "memory"); }

// Where the coefficients come from: global memory (one solve), or the CTA's own columns in shared memory (a launch of
// many solves, k_steps): cp[Ni][KX] and rc[Ni] = {asub, 1 / csup}.
template <int KX> struct SolveCoefGlobal {
    const ThomasParams& p;
    int kx;
    __device__ __forceinline__ double cp(int r) const { return __ldg(&p.cp[(size_t)r * p.Hp + kx]); }
    __device__ __forceinline__ double2 row(int r) const { return make_double2(__ldg(&p.asub[r + 1]), __ldg(&p.inv_csup[r + 1])); }
};
template <int KX> struct SolveCoefShared {
    const double* c;
    const double2* rc;
    int k;
    __device__ __forceinline__ double cp(int r) const { return c[r * KX + k]; }
    __device__ __forceinline__ double2 row(int r) const { return rc[r]; }
};

template <int KX, int L, bool F32, typename Coef>
__device__ __forceinline__ void solve_columns(const ThomasParams& p, int g, SolveSmem<KX>& sm, const Coef& coef) {
    using ST2 = typename SpecT<F32>::T2;
    const int tid = threadIdx.x, k = tid % KX, q = tid / KX, lane = tid & 31, w = tid >> 5;
    const int kx = g * KX + k, lo = q * L, Ni = p.Ni;
    const bool valid = kx < p.H;
    const size_t Hp = (size_t)p.Hp;
    const ST2* hat = F32 ? reinterpret_cast<const ST2*>(p.hat32) : reinterpret_cast<const ST2*>(p.hat);
    ST2* out = F32 ? reinterpret_cast<ST2*>(p.out32) : reinterpret_cast<ST2*>(p.out);
    double2 x[L];
    double cpv[L], be[L];
#pragma unroll
    for (int i = 0; i < L; ++i) {                            // kx < Hp: the padding columns hold zeros
        x[i] = make_double2(0.0, 0.0);
        if (lo + i < Ni) x[i] = spec_wide(__ldcg(hat + (size_t)(lo + i + 1) * Hp + kx));
    }
    // the coefficients while the spectra are on their way (be: 1 / c_i until the sweep)
#pragma unroll
    for (int i = 0; i < L; ++i) {
        cpv[i] = 0.0;
        be[i] = 0.0;
        if (lo + i < Ni) {
            cpv[i] = coef.cp(lo + i);
            be[i] = coef.row(lo + i).y;
        }
    }
    // rhs = -omega-hat, with the k = 0 Dirichlet wall terms of src/poisson.cu:91-95,109-114
    if (kx == 0) {
#pragma unroll
        for (int i = 0; i < L; ++i) {
            if (lo + i == 0) x[i].x += p.asub[1] * p.psi_bot * (double)p.Nx;
            if (lo + i == Ni - 1) x[i].x += p.csup[p.Ny - 2] * p.psi_top * (double)p.Nx;
        }
    }
    // forward sweep from c = 0
    AffMap m{make_double2(0.0, 0.0), 1.0};
#pragma unroll
    for (int i = 0; i < L; ++i) {
        if (lo + i < Ni) {
            const double alpha = cpv[i] * be[i];
            be[i] = -coef.row(lo + i).x * alpha;
            m.D.x = fma(be[i], m.D.x, -alpha * x[i].x);
            m.D.y = fma(be[i], m.D.y, -alpha * x[i].y);
            x[i] = m.D;
            m.P = be[i] * m.P;
        }
    }
    // the warp's segments, then the warps below (dp before the first row is 0)
    AffMap s = m;
#pragma unroll
    for (int off = KX; off < 32; off *= 2) {
        const AffMap o = aff_shfl_up(s, off);
        if (lane >= off) s = aff_after(s, o);
    }
    AffMap ex = aff_shfl_up(s, KX);
    if (lane < KX) ex = AffMap{make_double2(0.0, 0.0), 1.0};
    if (lane >= 32 - KX) { sm.D[0][w][k] = s.D; sm.P[0][w][k] = s.P; }
    sc_sync();
    double2 A = make_double2(0.0, 0.0);
#pragma unroll
    for (int v = 0; v < SC_NW - 1; ++v)
        if (v < w) {
            const double2 d = sm.D[0][v][k];
            const double P = sm.P[0][v][k];
            A = make_double2(fma(P, A.x, d.x), fma(P, A.y, d.y));
        }
    const double2 c = make_double2(fma(ex.P, A.x, ex.D.x), fma(ex.P, A.y, ex.D.y));
    // carry term, backward sweep from X = 0
    double Pc = 1.0;
#pragma unroll
    for (int i = 0; i < L; ++i)
        if (lo + i < Ni) {
            Pc = be[i] * Pc;
            x[i].x = fma(Pc, c.x, x[i].x);
            x[i].y = fma(Pc, c.y, x[i].y);
        }
    m = AffMap{make_double2(0.0, 0.0), 1.0};
#pragma unroll
    for (int i = L - 1; i >= 0; --i)
        if (lo + i < Ni) {
            m.D.x = fma(-cpv[i], m.D.x, x[i].x);
            m.D.y = fma(-cpv[i], m.D.y, x[i].y);
            x[i] = m.D;
            m.P = -cpv[i] * m.P;
        }
    s = m;
#pragma unroll
    for (int off = KX; off < 32; off *= 2) {
        const AffMap o = aff_shfl_down(s, off);
        if (lane + off < 32) s = aff_after(s, o);
    }
    ex = aff_shfl_down(s, KX);
    if (lane >= 32 - KX) ex = AffMap{make_double2(0.0, 0.0), 1.0};
    if (lane < KX) { sm.D[1][w][k] = s.D; sm.P[1][w][k] = s.P; }
    sc_sync();
    A = make_double2(0.0, 0.0);
#pragma unroll
    for (int v = SC_NW - 1; v > 0; --v)
        if (v > w) {
            const double2 d = sm.D[1][v][k];
            const double P = sm.P[1][v][k];
            A = make_double2(fma(P, A.x, d.x), fma(P, A.y, d.y));
        }
    const double2 X = make_double2(fma(ex.P, A.x, ex.D.x), fma(ex.P, A.y, ex.D.y));
    // carry term; psi-hat out
    double Qc = 1.0;
#pragma unroll
    for (int i = L - 1; i >= 0; --i)
        if (lo + i < Ni) {
            Qc = -cpv[i] * Qc;
            if (valid) out[(size_t)(lo + i + 1) * Hp + kx] = spec_narrow<F32>(fma(Qc, X.x, x[i].x), fma(Qc, X.y, x[i].y));
        }
    // wall rows of psi-hat: Nx psi_bot / Nx psi_top at kx = 0, else 0 (poisson.cu:130-132)
    if (valid && q == 0) {
        out[kx] = spec_narrow<F32>(kx == 0 ? (double)p.Nx * p.psi_bot : 0.0, 0.0);
        out[(size_t)(p.Ny - 1) * Hp + kx] = spec_narrow<F32>(kx == 0 ? (double)p.Nx * p.psi_top : 0.0, 0.0);
    }
}

// Two columns per CTA while those CTAs fit the device about once, else four: 128 or 64 segments, of the fewest
// rows that hold the grid.
constexpr int SC_MAX_NI = 512;
inline int solve_kx(int H, int num_sms) { return H <= 2 * num_sms ? 2 : 4; }
inline int solve_L(int Ni, int kx) {
    int L = 1;
    while (L * (SC_NT / kx) < Ni) L *= 2;
    return L;
}

template <int KX, int L, bool F32>
static __global__ void __launch_bounds__(SC_NT) k_thomas_cta(ThomasParams p) {
    __shared__ SolveSmem<KX> sm;
    pdl_begin();
    solve_columns<KX, L, F32>(p, blockIdx.x, sm, SolveCoefGlobal<KX>{p, (int)blockIdx.x * KX + (int)threadIdx.x % KX});
}

}  // namespace nse2d
