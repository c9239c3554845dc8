// The tridiagonal solve of a few columns by one CTA, for grids of up to 514 rows (up to 1026: k_thomas_wide). Written for this project.
//
// The arithmetic is k_thomas_cluster's (segments of rows in registers, joined through their affine carries), with
// all interior rows of KX columns in one CTA of 256 threads: 256 / KX segments of L rows, so the carries cross a
// warp by shuffles and eight warps through shared memory, with two barriers, and nothing crosses CTAs. On a short
// grid the cluster form's start-up, its exchanges between CTAs (about 1000 clocks each way) and its tensor-map
// loads were most of its time. Step with the cluster form and with this one: 128x129 34.9 and 30.7 us, 256x257
// 39.4 and 32.8, 1024x513 66.4 and 59.4. From 515 rows on a segment would be 16 rows (or the columns fewer than a
// 32-byte sector): k_thomas_wide takes twice the threads.
#pragma once
#include "step_kernels.cuh"

namespace nse2d {

constexpr int SC_NT = 256;
template <int KX, int NT = SC_NT> struct SolveSmem {
    double2 D[2][NT / 32][KX];
    double P[2][NT / 32][KX];
};

// threads 0 .. NT-1 of a CTA (bar.sync 15)
template <int NT> __device__ __forceinline__ void sc_sync() { asm volatile("bar.sync 15, %0;\n" ::"n"(NT) : "memory"); }

// Where the coefficients of row lo + i come from: global memory (one solve), the CTA's own columns in shared memory
// (a launch of many solves, k_steps): cp[Ni][KX] and rc[Ni] = {asub, 1 / csup}; kKeep: held in registers by the sweeps.
template <int KX> struct SolveCoefGlobal {
    static constexpr bool kKeep = true;
    const ThomasParams& p;
    int kx;
    __device__ __forceinline__ double cp(int lo, int i) const { return __ldg(&p.cp[(size_t)(lo + i) * p.Hp + kx]); }
    __device__ __forceinline__ double2 row(int lo, int i) const { return make_double2(__ldg(&p.asub[lo + i + 1]), __ldg(&p.inv_csup[lo + i + 1])); }
};
template <int KX> struct SolveCoefShared {
    static constexpr bool kKeep = true;
    const double* c;
    const double2* rc;
    int k;
    __device__ __forceinline__ double cp(int lo, int i) const { return c[(lo + i) * KX + k]; }
    __device__ __forceinline__ double2 row(int lo, int i) const { return rc[lo + i]; }
};
// The same in shared memory with the rows of segment q exchanged by q (row lo + i at lo + (i ^ q mod L)), so that
// the segments of a warp, L rows apart, read different banks; read again by each sweep (registers are the limit).
template <int KX, int L> struct SolveCoefSwizzled {
    static constexpr bool kKeep = false;
    const double* c;
    const double2* rc;
    int k, sw;
    __device__ __forceinline__ double cp(int lo, int i) const { return c[(lo + (i ^ sw)) * KX + k]; }
    __device__ __forceinline__ double2 row(int lo, int i) const { return rc[lo + (i ^ sw)]; }
};

// Ready: called once the loads of the spectra are on their way, before the first coefficient is read.
struct SolveReady { __device__ __forceinline__ void operator()() const {} };
template <int KX, int L, bool F32, int NT = SC_NT, typename Coef, typename Ready = SolveReady>
__device__ __forceinline__ void solve_columns(const ThomasParams& p, int g, SolveSmem<KX, NT>& sm, const Coef& coef, const Ready& ready = Ready{}) {
    constexpr int NW = NT / 32;
    using ST2 = typename SpecT<F32>::T2;
    const int tid = threadIdx.x, k = tid % KX, q = tid / KX, lane = tid & 31, w = tid >> 5;
    const int kx = g * KX + k, lo = q * L, Ni = p.Ni;
    const bool valid = kx < p.H;
    const size_t Hp = (size_t)p.Hp;
    const ST2* hat = F32 ? reinterpret_cast<const ST2*>(p.hat32) : reinterpret_cast<const ST2*>(p.hat);
    ST2* out = F32 ? reinterpret_cast<ST2*>(p.out32) : reinterpret_cast<ST2*>(p.out);
    double2 x[L];
    double cpv[L], be[L];                                    // kKeep
#pragma unroll
    for (int i = 0; i < L; ++i) {                            // kx < Hp: the padding columns hold zeros
        x[i] = make_double2(0.0, 0.0);
        if (lo + i < Ni) x[i] = spec_wide(__ldcg(hat + (size_t)(lo + i + 1) * Hp + kx));
    }
    ready();
    // the coefficients while the spectra are on their way (be: 1 / c_i until the sweep)
    if constexpr (Coef::kKeep) {
#pragma unroll
        for (int i = 0; i < L; ++i) {
            cpv[i] = 0.0;
            be[i] = 0.0;
            if (lo + i < Ni) {
                cpv[i] = coef.cp(lo, i);
                be[i] = coef.row(lo, i).y;
            }
        }
    }
    auto cp_at = [&](int i) {
        if constexpr (Coef::kKeep) return cpv[i];
        else return coef.cp(lo, i);
    };
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
            const double2 rc = coef.row(lo, i);
            const double alpha = cp_at(i) * (Coef::kKeep ? be[i] : rc.y);
            const double beta = -rc.x * alpha;
            if constexpr (Coef::kKeep) be[i] = beta;
            m.D.x = fma(beta, m.D.x, -alpha * x[i].x);
            m.D.y = fma(beta, m.D.y, -alpha * x[i].y);
            x[i] = m.D;
            m.P = beta * m.P;
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
    sc_sync<NT>();
    double2 A = make_double2(0.0, 0.0);
    if constexpr (NW <= 8) {
#pragma unroll
        for (int v = 0; v < NW - 1; ++v)
            if (v < w) {
                const double2 d = sm.D[0][v][k];
                const double P = sm.P[0][v][k];
                A = make_double2(fma(P, A.x, d.x), fma(P, A.y, d.y));
            }
    } else {                                                 // column w's warps scanned by warp w
        if (w < KX) {
            AffMap a{make_double2(0.0, 0.0), 1.0};
            if (lane < NW) a = AffMap{sm.D[0][lane][w], sm.P[0][lane][w]};
#pragma unroll
            for (int off = 1; off < NW; off *= 2) {
                const AffMap o = aff_shfl_up(a, off);
                if (lane >= off) a = aff_after(a, o);
            }
            a.D = make_double2(__shfl_up_sync(0xffffffffu, a.D.x, 1), __shfl_up_sync(0xffffffffu, a.D.y, 1));
            if (lane < NW) sm.D[0][lane][w] = lane ? a.D : make_double2(0.0, 0.0);
        }
        sc_sync<NT>();
        A = sm.D[0][w][k];
    }
    const double2 c = make_double2(fma(ex.P, A.x, ex.D.x), fma(ex.P, A.y, ex.D.y));
    // carry term, backward sweep from X = 0
    double Pc = 1.0;
#pragma unroll
    for (int i = 0; i < L; ++i)
        if (lo + i < Ni) {
            double beta;
            if constexpr (Coef::kKeep) {
                beta = be[i];
            } else {
                const double2 rc = coef.row(lo, i);
                beta = -rc.x * (cp_at(i) * rc.y);
            }
            Pc = beta * Pc;
            x[i].x = fma(Pc, c.x, x[i].x);
            x[i].y = fma(Pc, c.y, x[i].y);
        }
    m = AffMap{make_double2(0.0, 0.0), 1.0};
#pragma unroll
    for (int i = L - 1; i >= 0; --i)
        if (lo + i < Ni) {
            m.D.x = fma(-cp_at(i), m.D.x, x[i].x);
            m.D.y = fma(-cp_at(i), m.D.y, x[i].y);
            x[i] = m.D;
            m.P = -cp_at(i) * m.P;
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
    sc_sync<NT>();
    A = make_double2(0.0, 0.0);
    if constexpr (NW <= 8) {
#pragma unroll
        for (int v = NW - 1; v > 0; --v)
            if (v > w) {
                const double2 d = sm.D[1][v][k];
                const double P = sm.P[1][v][k];
                A = make_double2(fma(P, A.x, d.x), fma(P, A.y, d.y));
            }
    } else {
        if (w < KX) {                                        // lane l: warp NW-1-l, from the top
            AffMap a{make_double2(0.0, 0.0), 1.0};
            if (lane < NW) a = AffMap{sm.D[1][NW - 1 - lane][w], sm.P[1][NW - 1 - lane][w]};
#pragma unroll
            for (int off = 1; off < NW; off *= 2) {
                const AffMap o = aff_shfl_up(a, off);
                if (lane >= off) a = aff_after(a, o);
            }
            a.D = make_double2(__shfl_up_sync(0xffffffffu, a.D.x, 1), __shfl_up_sync(0xffffffffu, a.D.y, 1));
            if (lane < NW) sm.D[1][NW - 1 - lane][w] = lane ? a.D : make_double2(0.0, 0.0);
        }
        sc_sync<NT>();
        A = sm.D[1][w][k];
    }
    const double2 X = make_double2(fma(ex.P, A.x, ex.D.x), fma(ex.P, A.y, ex.D.y));
    // carry term; psi-hat out
    double Qc = 1.0;
#pragma unroll
    for (int i = L - 1; i >= 0; --i)
        if (lo + i < Ni) {
            Qc = -cp_at(i) * Qc;
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

// Grids of 515 to 1026 rows: 512 threads, so that a segment has no more than eight rows, and the coefficients in
// shared memory, so that two CTAs fit an SM (64 registers; the columns' 32 bytes of cp a row by cp.async, while the
// spectra travel to registers). The 16 warps are joined by a scan of one warp per column: folding up to 31 maps in
// every thread, as the eight warps above do, was 500 of 1500 instructions at 32 warps. The same on the cluster form
// and here, us a solve: 2048x1025 16.0 and 11.1 (FP32 15.7 and 9.6), 1024x777 9.6 and 7.3, 512x1000 9 and 5.5.
// What bounds it at 2048x1025: one wave of 257 CTAs, latency; shared-memory reads of the sweeps are the most
// frequent stall. From 1027 rows on the same with 1024 threads fills an SM with one CTA and loses to the clusters
// (4096x2049 50 us against 38; FP32 45 against 36).
constexpr int SC_WIDE_NT = 512;
constexpr int SC_WIDE_MAX_NI = 1024;
template <int KX, int L> __host__ __device__ constexpr size_t solve_wide_smem() { return (size_t)(SC_WIDE_NT / KX) * L * (16 + 8 * KX); }
template <int KX, int L, bool F32>
static __global__ void __launch_bounds__(SC_WIDE_NT, 2) k_thomas_wide(ThomasParams p) {
    constexpr int NT = SC_WIDE_NT;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SolveSmem<KX, NT> sm;
    pdl_begin();
    constexpr int R = NT / KX * L;                           // rows that the CTA can hold
    double2* rc = reinterpret_cast<double2*>(smem_raw);
    double* cps = reinterpret_cast<double*>(rc + R);
    const int kx0 = blockIdx.x * KX, Ni = p.Ni;
    auto at = [](int r) { return r ^ ((r / L) & (L - 1)); };
    auto ready = [&]() {
        for (int e = threadIdx.x; e < Ni * (KX / 2); e += NT) {
            const int r = e / (KX / 2), c = 2 * (e % (KX / 2));
            cp_async16(cps + at(r) * KX + c, p.cp + (size_t)r * p.Hp + kx0 + c);
        }
        for (int r = threadIdx.x; r < Ni; r += NT) rc[at(r)] = make_double2(__ldg(&p.asub[r + 1]), __ldg(&p.inv_csup[r + 1]));
        cp_async_wait_all();
        __syncthreads();
    };
    solve_columns<KX, L, F32, NT>(p, blockIdx.x, sm,
                                  SolveCoefSwizzled<KX, L>{cps, rc, (int)threadIdx.x % KX, ((int)threadIdx.x / KX) & (L - 1)}, ready);
}

}  // namespace nse2d
