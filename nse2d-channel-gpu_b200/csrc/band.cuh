// Row-band kernels: the row transforms and the stage of a band of rows in one launch, for rows of up to
// 1024 points, and the row transforms alone for rows of 64 to 2048 points (M = Nx / 2 from 32 to 1024),
// in FP64 and for the FP32-bulk step. Written for this project.
//
// The step's row work is inverse transform -> wall closure -> stage -> forward transform. On grids
// whose fields stay in L2 each of those was a launch of about 4 us with a round trip of its rows
// through L2, and the transforms kept 8 to 64 of a CTA's 128 threads busy. Here
//   k_band<.., INV>: a CTA owns the rows [j0, j1) and holds psi of rows j0-1 .. j1 in shared memory: INV
//     transforms them from psi-hat there (the two halo rows are transformed by the neighbours too: at
//     most R + 2 instead of R rows, cheaper than a launch and a round trip), or they are read from psi
//     (stage 1, whose psi is the step's). The wall closure of omega^(s), the stage and the forward
//     transform of the band's rows follow in the same launch: a stage is two launches (this one and the
//     tridiagonal solve) instead of four.
//   k_rows_fwd, k_rows_inv: the transforms alone (Poisson solve, spectra, the end of a step).
// A row is transformed by a group of one warp (M <= 128) or two, so that its passes need only that group's
// barrier and the groups of a CTA run independently; the stage is spread over all threads of the CTA.
// What bounds a band at 1024x513 (128 CTAs of 12 warps): the latency of its phases, in clocks of an SM:
// inverse 3800, stage 6000, forward 3800 of 16800, the FP64 pipe 30% busy. Steps, before and after: 128x129
// 55.3 -> 34.9 us, 256x257 58.8 -> 39.4, 1024x513 86.0 -> 66.4.
// Rows of 2048 points keep the separate stage kernel: a band of 7 rows and its halo (one per SM, 576
// threads) took 36.8 us against 34 for the three kernels, bound by its registers (96) and shared memory.
//
// psi-hat and omega-hat are different buffers, because a CTA reads halo rows of psi-hat while its
// neighbours write omega-hat. The per-point arithmetic is the stage kernels' (stage_rhs_interior,
// stage32_rhs_interior) and the transforms (band_fft.cuh) write their multiply-adds out: every split of the
// work gives the same bits.
#pragma once
#include "band_fft.cuh"
#include "bulk32.cuh"

namespace nse2d {

template <int M> struct Band {
    static constexpr int R0 = band_plan<M>::R(0);
    static constexpr int NB0 = M / R0;                       // pass-0 butterflies of a row
    static constexpr int TPR = M <= 128 ? 32 : 64;           // threads of a row group
    // elements of a row buffer: 0 .. M, padded; even, so that what follows the buffers is 16-byte aligned in FP32 too
    static constexpr int ROW = (M + (M >> ip_shift_a(M)) + (M >> ip_shift_b(M)) + 2) & ~1;
    static constexpr int RMAX = M <= 256 ? 6 : 4;            // rows of a band of k_band (M <= 512)
    static constexpr int MAXT = (RMAX + 2) * TPR;
    static constexpr int ROWS_G = 4;                         // row groups per CTA of the transforms alone
    static_assert(NB0 <= TPR, "one pass-0 butterfly per thread");
};
// Shared memory: the twiddles (pass tables, then W_2M^k, k <= M / 2), the row constants, the row buffers,
// the omega rows, omega^n and omega^(s+1) of the band.
template <int M> __host__ __device__ constexpr int band_ntw() { return band_plan<M>::off(band_plan<M>::P); }
template <int M> __host__ __device__ constexpr int band_ntab() { return band_ntw<M>() + M / 2 + 2; }
constexpr int BAND_RC = 10;                                  // row constants kept per row (RC32_N in FP32)
template <typename T, int M> __host__ __device__ constexpr size_t band_head_bytes(int R) {
    return (band_ntab<M>() * sizeof(cpx<T>) + (size_t)(R + 2) * BAND_RC * sizeof(T) + 15) / 16 * 16;
}
template <typename T, int M> __host__ __device__ constexpr size_t band_smem_bytes(int R) {
    return band_head_bytes<T, M>(R) + ((size_t)(R + 2) * Band<M>::ROW + (size_t)(3 * R + 2) * M) * sizeof(cpx<T>);
}
template <typename T, int M> __host__ __device__ constexpr size_t band_rows_smem_bytes() {
    return band_head_bytes<T, M>(0) + (size_t)Band<M>::ROWS_G * Band<M>::ROW * sizeof(cpx<T>);
}

template <typename T> struct BandParams {
    const cpx<T>* hat_in;    // psi-hat [Ny][Hp] (INV)
    cpx<T>* hat_out;         // omega-hat [Ny][Hp]
    const T* psi_in;         // psi [Ny][Nx] (no INV)
    T* psi_out;              // k_rows_inv: psi [Ny][Nx]
    const T* src;            // k_rows_fwd: real rows
    T* w_in;                 // omega^(s); with INV its wall rows are set here
    const T* w_n;            // omega^n; may be w_out in stage 3
    T* w_out;                // omega^(s+1)
    T* rhs_out;              // optional
    const double* closure;   // optional: tau, rhs -= tau on interior rows (FP64)
    const cpx<T>* tw;
    const cpx<T>* wN;
    RowTables rt;
    const float* rc;         // row constants of the FP32 stage
    Ctl* ctl;
    int Nx, Ny, Hp, stage, row0, nrows;
    int do_thom, advance, free_slip;
    double nu_dx2, lin_drag;
    double psi_bot, psi_top;     // psi on the walls (FP32: 0)
    double wall_bot, wall_top;   // FP32: the constant part of the wall vorticity
};

template <int TPR> __device__ __forceinline__ void row_sync(int group) {
    if constexpr (TPR == 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;\n" ::"r"(group + 1), "n"(TPR) : "memory");
}

// element copy to shared memory (16 bytes in FP64, past L1; 8 in FP32, through it: after a barrier across the grid
// L1 holds nothing stale)
__device__ __forceinline__ void cp_async_cpx(cpx<double>* d, const cpx<double>* g) { cp_async16(d, g); }
__device__ __forceinline__ void cp_async_cpx(cpx<float>* d, const cpx<float>* g) { cp_async8(d, g); }

// The twiddles to shared memory (no kernel writes them, so this may precede the wait for the previous
// kernel): every pass of every row reads them, and a table read from global memory would wait on L2
// once per pass and CTA.
template <typename T, int M> __device__ __forceinline__ void band_load_tables(cpx<T>* tab, const BandParams<T>& p) {
    constexpr int NTW = band_ntw<M>();
    for (int i = threadIdx.x; i < NTW + M / 2 + 1; i += blockDim.x) cp_async_cpx(tab + i, i < NTW ? p.tw + i : p.wN + (i - NTW));
}

// Passes Q .. P-1 by a row group; the last pass hands its outputs to out(position, value).
template <typename T, int M, int Q, bool INV, typename Out>
__device__ __forceinline__ void band_passes(cpx<T>* buf, const SmemTw<T>& tw, int t, int group, Out out) {
    constexpr int TPR = Band<M>::TPR, R = band_plan<M>::R(Q), LP = band_plan<M>::LP(Q), NB = M / R;
#pragma unroll 1
    for (int b0 = 0; b0 < NB; b0 += TPR) {
        const int b = b0 + t;
        if (NB % TPR != 0 && b >= NB) break;
        cpx<T> v[R];
        const int base = plan_bfly<T, band_plan<M>, Q, INV>(buf, tw, b, v);
        if constexpr (Q == band_plan<M>::P - 1) {
#pragma unroll
            for (int r = 0; r < R; ++r) out(base + r * LP, v[r]);
        } else {
#pragma unroll
            for (int r = 0; r < R; ++r) buf[ip_idx<M>(base + r * LP)] = v[r];
        }
    }
    row_sync<TPR>(group);
    if constexpr (Q < band_plan<M>::P - 1) band_passes<T, M, Q + 1, INV>(buf, tw, t, group, out);
}

// A spectral row X_0 .. X_M into buf (cp.async past L1; natural order, padded). Pass 0 needs X_n and X_{M-n}: from
// shared memory they cost one read of the row, and none of the registers that two loads per point in flight do.
template <typename T, int M> __device__ __forceinline__ void band_load_spec(const cpx<T>* X, cpx<T>* buf, int t) {
    for (int n = t; n <= M; n += Band<M>::TPR) cp_async_cpx(buf + ip_idx<M>(n), X + n);
}
// Inverse transform of the spectral row in buf (all of it arrived, and a barrier of the group since) into
// out(n, z_n), z_n = x_2n + i x_2n+1, times 2M: the merge of k_ifft_thom, then the passes.
template <typename T, int M, typename Out>
__device__ __forceinline__ void band_inverse(cpx<T>* buf, const SmemTw<T>& tw, const SmemTw<T>& wN, int t, int group, Out out) {
    constexpr int NB0 = Band<M>::NB0, TPR = Band<M>::TPR, R0 = Band<M>::R0;
    const bool on = NB0 >= TPR || t < NB0;
    cpx<T> v[R0];
    if (on) {
        const cpx<T> wt = ldtw(wN, t);
#pragma unroll
        for (int r = 0; r < R0; ++r) {
            const int n = t + NB0 * r;
            const cpx<T> a = buf[ip_idx<M>(n)], c = buf[ip_idx<M>(M - n)];
            const cpx<T> sm = {a.x + c.x, a.y - c.y};
            const cpx<T> df = {a.x - c.x, a.y + c.y};
            const cpx<T> wn = (r == 0) ? wt : fmul_c(wt, w32<T>(r * (16 / R0)));
            v[r] = cadd(sm, mul_pi(fmul_cc(df, wn)));
        }
        fdftR<T, R0, true>(v);
    }
    row_sync<TPR>(group);                                     // the spectral row is read
    if (on) {
        const int p0 = dit_pos<band_plan<M>>(t);
#pragma unroll
        for (int q = 0; q < R0; ++q) buf[ip_idx<M>(p0 + q)] = v[q];
    }
    row_sync<TPR>(group);
    band_passes<T, M, 1, true>(buf, tw, t, group, out);
}

// The forward transform from pass 0's registers on (v: the points t + NB0 r, r < R0, of thread t < NB0),
// through buf (free when called): X_k, k = 0 .. M, to dst.
template <typename T, int M>
__device__ __forceinline__ void band_forward(cpx<T> (&v)[Band<M>::R0], cpx<T>* buf, const SmemTw<T>& tw, const SmemTw<T>& wN, int t, int group,
                                             cpx<T>* __restrict__ dst) {
    constexpr int NB0 = Band<M>::NB0, TPR = Band<M>::TPR, R0 = Band<M>::R0;
    if (NB0 >= TPR || t < NB0) {
        fdftR<T, R0, false>(v);
        const int p0 = dit_pos<band_plan<M>>(t);
#pragma unroll
        for (int q = 0; q < R0; ++q) buf[ip_idx<M>(p0 + q)] = v[q];
    }
    row_sync<TPR>(group);
    band_passes<T, M, 1, false>(buf, tw, t, group, [&](int n, const cpx<T>& z) { buf[ip_idx<M>(n)] = z; });
    // the split step of k_fft_fwd: X_k and X_{M-k} from Z_k and Z_{M-k}
#pragma unroll 2
    for (int k = t; k <= M / 2; k += TPR) {
        const cpx<T> w1 = ldtw(wN, k);
        const cpx<T> wk = {(T)0.5 * w1.x, (T)0.5 * w1.y};
        const cpx<T> a = buf[ip_idx<M>(k)];
        const cpx<T> b = buf[ip_idx<M>(k == 0 ? 0 : M - k)];
        const cpx<T> sm = {(T)0.5 * (a.x + b.x), (T)0.5 * (a.y - b.y)};
        const cpx<T> df = {a.x - b.x, a.y + b.y};
        dst[k] = cadd(sm, fmul_c(wk, mul_mi(df)));
        if (k < M / 2) {
            const cpx<T> wm = {-wk.x, wk.y};
            dst[M - k] = cadd(cpx<T>{sm.x, -sm.y}, fmul_c(wm, cpx<T>{df.y, df.x}));
        }
    }
}

// Wall vorticity at one point of one wall from psi at the first two interior rows.
struct WallConst {
    double A, B, pw;         // FP64
    float Af, Bf, base;      // FP32
};
template <typename T> __device__ __forceinline__ WallConst wall_const(const BandParams<T>& p, bool top) {
    const double d1 = __ldg(&p.rt.dy_edge[top ? p.Ny - 2 : 0]);
    const double d2 = __ldg(&p.rt.dy_edge[top ? p.Ny - 3 : 1]);
    WallConst c;
    c.A = 2.0 * (1.0 / (d1 * d1) + 1.0 / (d1 * d2));
    c.B = (-2.0) * d1 / (d2 * (d1 + d2) * (d1 + d2));
    c.pw = top ? p.psi_top : p.psi_bot;
    c.Af = (float)c.A; c.Bf = (float)c.B;
    c.base = (float)(top ? p.wall_top : p.wall_bot);
    return c;
}
template <typename T> __device__ __forceinline__ T wall_value(const BandParams<T>& p, const WallConst& c, T p1, T p2) {
    if constexpr (sizeof(T) == 8) return p.free_slip ? 0.0 : thom_value(c.A, c.B, p1 - c.pw, p2 - c.pw);
    else return p.free_slip ? c.base : thom32_value(c.base, c.Af, c.Bf, p1, p2);
}
// The wall row of w (and of ws, when given) from the psi row buffers b1, b2, by all threads of the CTA.
template <typename T, int M>
__device__ __forceinline__ void band_wall_row(const BandParams<T>& p, bool top, const cpx<T>* b1, const cpx<T>* b2, T* w, cpx<T>* ws) {
    const WallConst c = wall_const(p, top);
    cpx<T>* wr = reinterpret_cast<cpx<T>*>(w + (size_t)(top ? p.Ny - 1 : 0) * p.Nx);
    for (int n = threadIdx.x; n < M; n += blockDim.x) {
        const cpx<T> u = b1[ip_idx<M>(n)], v = b2[ip_idx<M>(n)];
        const cpx<T> o = {wall_value(p, c, u.x, v.x), wall_value(p, c, u.y, v.y)};
        wr[n] = o;
        if (ws) ws[n] = o;
    }
}

// One row of the window of the points 2n, 2n + 1: x = 2n - 1 .. 2n + 2, from a row of cpx elements
// (PAD: the padded layout of the transforms' buffers).
template <typename T, int M, bool PAD>
__device__ __forceinline__ void band_window(const cpx<T>* row, int n, T (&v)[4]) {
    const int nl = (n - 1) & (M - 1), nr = (n + 1) & (M - 1);
    const cpx<T> c = row[PAD ? ip_idx<M>(n) : n];
    v[0] = row[PAD ? ip_idx<M>(nl) : nl].y;
    v[1] = c.x; v[2] = c.y;
    v[3] = row[PAD ? ip_idx<M>(nr) : nr].x;
}

// Row constants of the stage, copied to shared memory with the tables.
struct BandRow64 { double f, ap, am, cj; };
struct BandRow32 { Rc32Row k; float f; };
__device__ __forceinline__ void band_load_rows(double* rc, const BandParams<double>& p, int j0, int n) {
    for (int e = threadIdx.x; e < 4 * n; e += blockDim.x) {
        const int q = e & 3, r = e >> 2, j = j0 + r;
        rc[r * BAND_RC + q] = __ldg((q == 0 ? p.rt.frow : q == 1 ? p.rt.st_ap : q == 2 ? p.rt.st_am : p.rt.st_cj) + j);
    }
}
__device__ __forceinline__ void band_load_rows(float* rc, const BandParams<float>& p, int j0, int n) {
    static_assert(RC32_N <= BAND_RC, "row constants of the FP32 stage");
    for (int e = threadIdx.x; e < RC32_N * n; e += blockDim.x) {
        const int q = e / n, r = e - q * n;
        rc[r * BAND_RC + q] = __ldg(&p.rc[(size_t)q * p.Ny + j0 + r]);
    }
}
__device__ __forceinline__ BandRow64 band_row(const double* rc) { return {rc[0], rc[1], rc[2], rc[3]}; }
__device__ __forceinline__ BandRow32 band_row(const float* rc) {
    return {Rc32Row{rc[RC_DPB], rc[RC_DPP], rc[RC_DPM], rc[RC_DWB], rc[RC_DWP], rc[RC_DWM], rc[RC_AP], rc[RC_AM], rc[RC_CJ]}, rc[RC_R]};
}
__device__ __forceinline__ double band_rhs(const BandRow64& k, double rhs, double wc, double pxm, double pxp, double pym, double pyp,
                                           double dpm, double dpc, double dpp, const double (&dxp)[3], double oxm, double oxp,
                                           double oym, double oyp, double dom, double doc, double dop, const double (&dxo)[3],
                                           double nu_dx2) {
    return stage_rhs_interior(rhs, wc, pxm, pxp, pym, pyp, dpm, dpc, dpp, dxp, oxm, oxp, oym, oyp, dom, doc, dop, dxo, nu_dx2,
                              k.ap, k.am, k.cj);
}
__device__ __forceinline__ float band_rhs(const BandRow32& k, float rhs, float wc, float pxm, float pxp, float pym, float pyp, float dpm,
                                          float dpc, float dpp, const float (&dxp)[3], float oxm, float oxp, float oym, float oyp,
                                          float dom, float doc, float dop, const float (&dxo)[3], float nu_dx2) {
    return stage32_rhs_interior(rhs, wc, pxm, pxp, pym, pyp, dpm, dpc, dpp, dxp, oxm, oxp, oym, oyp, dom, doc, dop, dxo, nu_dx2, k.k);
}
__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }

// A window row of the points 2n, 2n + 1: x = 2n - 1 .. 2n + 2 of psi and omega, and their x differences.
template <typename T> struct BandWin {
    T p[4], o[4], dp[2], dop[2];
};
template <typename T, int M> __device__ __forceinline__ void band_window_row(const cpx<T>* prow, const cpx<T>* orow, int n, BandWin<T>& w) {
    band_window<T, M, true>(prow, n, w.p);
    band_window<T, M, false>(orow, n, w.o);
}
template <typename T> __device__ __forceinline__ void band_diffs(BandWin<T>& w) {
#pragma unroll
    for (int e = 0; e < 2; ++e) { w.dp[e] = w.p[e + 2] - w.p[e]; w.dop[e] = w.o[e + 2] - w.o[e]; }
}
// Stage of the points 2n, 2n + 1 of interior row j: their omega^(s+1), from the window rows a, b, c = j-1, j, j+1.
template <typename T, int M, typename Row>
__device__ __forceinline__ cpx<T> band_pair(const BandParams<T>& p, const Row& k, T dt, T mdrag, T nu_dx2, int j, int n, const cpx<T>& wn,
                                            const BandWin<T>& a, const BandWin<T>& b, const BandWin<T>& c) {
    T dyo[4], dyp[4], dxp[3], dxo[3];
#pragma unroll
    for (int i = 0; i < 4; ++i) { dyo[i] = c.o[i] - a.o[i]; dyp[i] = c.p[i] - a.p[i]; }
    T w[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const T wc = b.o[e + 1];
        dxp[0] = a.dp[e]; dxp[1] = b.dp[e]; dxp[2] = c.dp[e];
        dxo[0] = a.dop[e]; dxo[1] = b.dop[e]; dxo[2] = c.dop[e];
        w[e] = band_rhs(k, fma_t(mdrag, wc, k.f), wc, b.p[e], b.p[e + 2], a.p[e + 1], c.p[e + 1], dyp[e], dyp[e + 1], dyp[e + 2], dxp,
                        b.o[e], b.o[e + 2], a.o[e + 1], c.o[e + 1], dyo[e], dyo[e + 1], dyo[e + 2], dxo, nu_dx2);
    }
    const int id = j * M + n;
    if constexpr (sizeof(T) == 8) {
        if (p.closure) {
            const double2 tau = __ldg(reinterpret_cast<const double2*>(p.closure) + id);
            w[0] -= tau.x;
            w[1] -= tau.y;
        }
    }
    if (p.rhs_out) reinterpret_cast<cpx<T>*>(p.rhs_out)[id] = cpx<T>{w[0], w[1]};
    w[0] = fma_t(dt, w[0], b.o[1]);
    w[1] = fma_t(dt, w[1], b.o[2]);
    if (p.stage > 1) {
        w[0] = rk_combine(p.stage, wn.x, w[0]);
        w[1] = rk_combine(p.stage, wn.y, w[1]);
    }
    return {w[0], w[1]};
}

// A CTA's band of rows and its shared memory: the pieces below are the row work of one CTA, by all of its threads.
template <typename T, int M> struct BandCta {
    using B = Band<M>;
    cpx<T> *tab, *rows, *ws, *wns, *zs;      // tables, psi rows j0 - 1 .. j1, omega rows, omega^n and omega^(s+1) of the band
    T* rc;                                   // row constants of rows j0 - 1 .. j1
    SmemTw<T> tw, wN;
    int t, group, j0, nr;                    // thread of a row group; rows [j0, j0 + nr) of the band
    bool bot, top;                           // the band lies at a wall

    // R: most rows of a band (the row groups 0 .. R + 1 take the rows j0 - 1 .. j1)
    __device__ __forceinline__ BandCta(const BandParams<T>& p, unsigned char* smem, int R) {
        tab = reinterpret_cast<cpx<T>*>(smem);
        rc = reinterpret_cast<T*>(tab + band_ntab<M>());
        rows = reinterpret_cast<cpx<T>*>(smem + band_head_bytes<T, M>(R));
        ws = rows + (size_t)(R + 2) * B::ROW;
        wns = ws + (size_t)(R + 2) * M;
        zs = wns + (size_t)R * M;
        tw.p = tab;
        wN.p = tab + band_ntw<M>();
        t = (int)threadIdx.x % B::TPR;
        group = (int)threadIdx.x / B::TPR;
        const int Ni = p.Ny - 2;
        j0 = 1 + (int)(((long long)blockIdx.x * Ni) / gridDim.x);
        const int j1 = 1 + (int)(((long long)(blockIdx.x + 1) * Ni) / gridDim.x);
        nr = j1 - j0;
        bot = (j0 == 1);
        top = (j1 == p.Ny - 1);
    }
    __device__ __forceinline__ bool rowed() const { return group < nr + 2; }
    __device__ __forceinline__ int row() const { return j0 - 1 + group; }                // the group's psi row
    __device__ __forceinline__ bool wallrow() const { return (bot && group == 0) || (top && group == nr + 1); }
    __device__ __forceinline__ cpx<T>* buf() const { return rows + (size_t)group * B::ROW; }

    // tables and row constants, which no step kernel writes (a commit group of its own)
    __device__ __forceinline__ void load_consts(const BandParams<T>& p) {
        band_load_tables<T, M>(tab, p);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        band_load_rows(rc, p, j0 - 1, nr + 2);
    }
    // psi rows j0 - 1 .. j1 (cp.async)
    __device__ __forceinline__ void load_psi(const T* psi) {
        if (!rowed()) return;
        const cpx<T>* src = reinterpret_cast<const cpx<T>*>(psi) + (size_t)row() * M;
        for (int n = t; n < M; n += B::TPR) cp_async_cpx(buf() + ip_idx<M>(n), src + n);
    }
    // omega rows j0 - 1 .. j1, without the wall rows when the closure sets them (cp.async)
    __device__ __forceinline__ void load_omega(const T* w, bool walls) {
        constexpr int CH = M * (int)sizeof(cpx<T>) / 16, CE = 16 / (int)sizeof(cpx<T>);
        if (!rowed() || (!walls && wallrow())) return;
        const cpx<T>* src = reinterpret_cast<const cpx<T>*>(w) + (size_t)row() * M;
        for (int c = t; c < CH; c += B::TPR) cp_async16(ws + (size_t)group * M + CE * c, src + CE * c);
    }
    // omega^n of the band's rows (cp.async)
    __device__ __forceinline__ void load_omega_n(const T* w) {
        constexpr int CH = M * (int)sizeof(cpx<T>) / 16, CE = 16 / (int)sizeof(cpx<T>);
        if (group < 1 || group > nr) return;
        const cpx<T>* src = reinterpret_cast<const cpx<T>*>(w) + (size_t)row() * M;
        for (int c = t; c < CH; c += B::TPR) cp_async16(wns + (size_t)(group - 1) * M + CE * c, src + CE * c);
    }
    // psi-hat rows j0 - 1 .. j1 into the row buffers (cp.async)
    __device__ __forceinline__ void load_spec(const BandParams<T>& p) {
        if (rowed() && !wallrow()) band_load_spec<T, M>(p.hat_in + (size_t)row() * p.Hp, buf(), t);
    }
    // psi rows j0 - 1 .. j1 from them, once they have arrived
    __device__ __forceinline__ void inverse(const BandParams<T>& p) {
        if (!rowed()) return;
        cpx<T>* b = buf();
        if (wallrow()) {
            const T v = (T)(group == 0 ? p.psi_bot : p.psi_top);
            for (int n = t; n < M; n += B::TPR) b[ip_idx<M>(n)] = cpx<T>{v, v};
        } else {
            constexpr T scale = (T)0.5 / (T)M;                // the merge forms 2 Z_n
            band_inverse<T, M>(b, tw, wN, t, group, [&](int n, const cpx<T>& z) { b[ip_idx<M>(n)] = cpx<T>{z.x * scale, z.y * scale}; });
        }
    }
    // wall rows of w (and of the omega rows) from the psi rows; between barriers
    __device__ __forceinline__ void walls(const BandParams<T>& p, T* w) {
        if (bot) band_wall_row<T, M>(p, false, rows + B::ROW, rows + 2 * (size_t)B::ROW, w, ws);
        if (top) band_wall_row<T, M>(p, true, rows + (size_t)nr * B::ROW, rows + (size_t)(nr - 1) * B::ROW, w, ws + (size_t)(nr + 1) * M);
    }
    // omega^(s+1) of the band into zs and w_out. save_n: omega^(s) of the band's rows into wns (stage 1, whose
    // omega^(s) is omega^n)
    __device__ __forceinline__ void stage(const BandParams<T>& p, T dt, bool save_n) {
        if (p.rhs_out && (bot || top)) {
            // the walls' rhs is f - r omega (their omega is the closure's)
            for (int side = 0; side < 2; ++side) {
                if (!(side ? top : bot)) continue;
                const int j = side ? p.Ny - 1 : 0, q = side ? nr + 1 : 0;
                const auto k = band_row(rc + q * BAND_RC);
                for (int n = threadIdx.x; n < M; n += blockDim.x) {
                    const cpx<T> wc = ws[(size_t)q * M + n];
                    reinterpret_cast<cpx<T>*>(p.rhs_out)[(size_t)j * M + n] =
                        cpx<T>{fma_t(-(T)p.lin_drag, wc.x, k.f), fma_t(-(T)p.lin_drag, wc.y, k.f)};
                }
            }
        }
        // an item is a pair n and the rows [qa, qb) of the band (all of them, or half where that evens out the
        // threads); a thread walks down its rows with j-1, j, j+1 of its window in registers
        cpx<T>* w_out = reinterpret_cast<cpx<T>*>(p.w_out);
        const T mdrag = -(T)p.lin_drag, nu_dx2 = (T)p.nu_dx2;
        const int NT = (int)blockDim.x;
        const int half = (nr + 1) / 2;
        const bool split = ((2 * M + NT - 1) / NT) * half < ((M + NT - 1) / NT) * nr;
        for (int item = threadIdx.x; item < (split ? 2 * M : M); item += NT) {
            const int n = item & (M - 1);
            const int qa = item < M ? 0 : half, qb = (split && item < M) ? half : nr;
            const cpx<T>* pr = rows + (size_t)qa * B::ROW;
            const cpx<T>* orow = ws + (size_t)qa * M;
            cpx<T>* w_n = wns + (size_t)qa * M + n;
            BandWin<T> win[3];
            band_window_row<T, M>(pr, orow, n, win[0]);
            band_window_row<T, M>(pr + B::ROW, orow + M, n, win[1]);
            band_window_row<T, M>(pr + 2 * B::ROW, orow + 2 * M, n, win[2]);
            band_diffs(win[0]);
            band_diffs(win[1]);
            cpx<T> wn = {0, 0};
            if (p.stage > 1) wn = *w_n;
            // unrolled, so that the window rotates by name instead of by moves; the row after next and the next
            // omega^n are loaded before this row's arithmetic
#pragma unroll
            for (int u = 0; u < B::RMAX; ++u) {
                const int q = qa + u;
                if (q >= qb) break;
                BandWin<T>&wa = win[u % 3], &wb = win[(u + 1) % 3], &wc = win[(u + 2) % 3];
                band_diffs(wc);
                const cpx<T> wnq = wn;
                BandWin<T> nx;
                const bool more = q + 1 < qb;
                if (more) {
                    band_window_row<T, M>(pr + (u + 3) * B::ROW, orow + (u + 3) * M, n, nx);
                    if (p.stage > 1) wn = w_n[(u + 1) * M];
                }
                const int j = j0 + q;
                const cpx<T> z = band_pair<T, M>(p, band_row(rc + (q + 1) * BAND_RC), dt, mdrag, nu_dx2, j, n, wnq, wa, wb, wc);
                w_out[j * M + n] = z;
                zs[q * M + n] = z;
                if (save_n) w_n[u * M] = cpx<T>{wb.o[1], wb.o[2]};
                if (more) wa = nx;
            }
        }
    }
    // forward transform of the band's omega^(s+1), after a barrier: group g transforms row j0 + g in row buffer
    // g + 1, which ends the psi rows
    __device__ __forceinline__ void forward(const BandParams<T>& p) {
        if (group >= nr) return;
        const cpx<T>* src = zs + (size_t)group * M;
        cpx<T> z[B::R0];
        if (B::NB0 >= B::TPR || t < B::NB0) {
#pragma unroll
            for (int r = 0; r < B::R0; ++r) z[r] = src[t + B::NB0 * r];
        }
        band_forward<T, M>(z, buf() + B::ROW, tw, wN, t, group, p.hat_out + (size_t)(j0 + group) * p.Hp);
    }
};

// The stage and the forward transform of a band of rows, with (INV) the inverse transform and the
// wall closure before it. Grid: an even split of the interior rows; blockDim = (R + 2) TPR for bands
// of at most R rows.
template <typename T, int M, bool INV>
static __global__ void __launch_bounds__(Band<M>::MAXT, 1) k_band(BandParams<T> p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BandCta<T, M> c(p, smem_raw, (int)blockDim.x / Band<M>::TPR - 2);
    c.load_consts(p);                                         // before the wait for the previous kernel
    pdl_begin();
    const T dt = (T)p.ctl->dt;
    if constexpr (INV) c.load_spec(p);
    else c.load_psi(p.psi_in);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    c.load_omega(p.w_in, !INV);                               // in flight while psi is transformed
    if (p.stage > 1) c.load_omega_n(p.w_n);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    if constexpr (INV) {
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();                                      // the tables and the spectral rows
        c.inverse(p);
    }
    cp_async_wait_all();
    __syncthreads();
    if constexpr (INV) {
        if (c.bot || c.top) {
            c.walls(p, p.w_in);
            __syncthreads();
        }
    }
    c.stage(p, dt, false);
    __syncthreads();
    c.forward(p);
}

// Forward transforms of rows row0 .. row0 + nrows - 1, ROWS_G rows per CTA.
template <typename T, int M>
static __global__ void __launch_bounds__(Band<M>::ROWS_G * Band<M>::TPR) k_rows_fwd(BandParams<T> p) {
    using B = Band<M>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int t = (int)threadIdx.x % B::TPR, group = (int)threadIdx.x / B::TPR;
    cpx<T>* tab = reinterpret_cast<cpx<T>*>(smem_raw);
    cpx<T>* buf = reinterpret_cast<cpx<T>*>(smem_raw + band_head_bytes<T, M>(0)) + (size_t)group * B::ROW;
    band_load_tables<T, M>(tab, p);
    pdl_begin();
    const int r0 = (int)blockIdx.x * B::ROWS_G + group;
    const int j = p.row0 + r0;
    cpx<T> z[B::R0];
    if (r0 < p.nrows && (B::NB0 >= B::TPR || t < B::NB0)) {
        const cpx<T>* src = reinterpret_cast<const cpx<T>*>(p.src) + (size_t)j * M;
#pragma unroll
        for (int r = 0; r < B::R0; ++r) z[r] = ldtw(src, t + B::NB0 * r);
    }
    cp_async_wait_all();
    __syncthreads();
    if (r0 < p.nrows)
        band_forward<T, M>(z, buf, SmemTw<T>{tab}, SmemTw<T>{tab + band_ntw<M>()}, t, group, p.hat_out + (size_t)j * p.Hp);
}

// Inverse transforms of every row, ROWS_G interior rows per CTA (an even split; at least two when there
// is more than one CTA), with the wall rows of psi, and (do_thom) the wall closure of w_in by the first
// and last CTA, which hold the rows next to the walls. With advance the last CTA to finish advances the time.
template <typename T, int M>
static __global__ void __launch_bounds__(Band<M>::ROWS_G * Band<M>::TPR) k_rows_inv(BandParams<T> p) {
    using B = Band<M>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cpx<T>* tab = reinterpret_cast<cpx<T>*>(smem_raw);
    cpx<T>* rows = reinterpret_cast<cpx<T>*>(smem_raw + band_head_bytes<T, M>(0));
    const int t = (int)threadIdx.x % B::TPR, group = (int)threadIdx.x / B::TPR;
    const int Ni = p.Ny - 2;
    const int j0 = 1 + (int)(((long long)blockIdx.x * Ni) / gridDim.x);
    const int j1 = 1 + (int)(((long long)(blockIdx.x + 1) * Ni) / gridDim.x);
    const bool bot = (j0 == 1), top = (j1 == p.Ny - 1), wall = (bot || top) && p.do_thom;
    cpx<T>* psi = reinterpret_cast<cpx<T>*>(p.psi_out);
    band_load_tables<T, M>(tab, p);
    pdl_begin();
    cpx<T>* buf = rows + (size_t)group * B::ROW;
    if (j0 + group < j1) band_load_spec<T, M>(p.hat_in + (size_t)(j0 + group) * p.Hp, buf, t);
    cp_async_wait_all();
    __syncthreads();
    if (j0 + group < j1) {
        cpx<T>* dst = psi + (size_t)(j0 + group) * M;
        constexpr T scale = (T)0.5 / (T)M;
        band_inverse<T, M>(buf, SmemTw<T>{tab}, SmemTw<T>{tab + band_ntw<M>()}, t, group, [&](int n, const cpx<T>& z) {
            const cpx<T> o = {z.x * scale, z.y * scale};
            dst[n] = o;
            if (wall) buf[ip_idx<M>(n)] = o;
        });
    }
    if (bot) for (int n = threadIdx.x; n < M; n += blockDim.x) psi[n] = cpx<T>{(T)p.psi_bot, (T)p.psi_bot};
    if (top) for (int n = threadIdx.x; n < M; n += blockDim.x) psi[(size_t)(p.Ny - 1) * M + n] = cpx<T>{(T)p.psi_top, (T)p.psi_top};
    if (wall) {
        __syncthreads();
        const int nr = j1 - j0;
        if (bot) band_wall_row<T, M>(p, false, rows, rows + B::ROW, p.w_in, (cpx<T>*)nullptr);
        if (top) band_wall_row<T, M>(p, true, rows + (size_t)(nr - 1) * B::ROW, rows + (size_t)(nr - 2) * B::ROW, p.w_in, (cpx<T>*)nullptr);
    }
    if (p.advance) {
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(&p.ctl->ifft_done, 1u) == gridDim.x - 1) {
                __threadfence();
                p.ctl->ifft_done = 0;
                advance_time(p.ctl);
            }
        }
    }
}

}  // namespace nse2d
