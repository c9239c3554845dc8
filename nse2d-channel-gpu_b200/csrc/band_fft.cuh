// The transforms of the row-band kernels: plans and butterflies. Written for this project.
//
// The scheme is fft_rows.cuh's (in-place decimation-in-time passes, pass 0 from registers in digit-reversed
// order, per-pass twiddle tables), with the radix chosen per length and with every multiply-add written out, so
// that a transform gives the same bits in every kernel it is compiled into: a step by bands, a step by separate
// kernels and the transforms alone agree to the bit. (fft_rows.cuh leaves the contraction to the compiler.)
//
// Radix 16 at 1024 points (two warps a row), 8 at 512 and 4 below, where a row has 2 to 16 points per thread and
// the length of a thread's own chain counts: a radix-16 pass of a 128-point row would run on 8 threads. The last
// pass takes what is left (with radix 4, up to 3 bits). Bands at 1024x513 with radix 16 throughout: 84 us a step
// against 70.
#pragma once
#include "fft_rows.cuh"

namespace nse2d {

__host__ __device__ constexpr int plan_log2(int M) {
    int m = 0;
    while ((1 << m) < M) ++m;
    return m;
}
__host__ __device__ constexpr int plan_passes(int M, int rb) { return rb == 2 ? plan_log2(M) / 2 : (plan_log2(M) + rb - 1) / rb; }
__host__ __device__ constexpr int plan_bits(int M, int rb, int q) {
    return q < plan_passes(M, rb) - 1 ? rb : plan_log2(M) - rb * (plan_passes(M, rb) - 1);
}
template <int M_, int RB> struct RowPlan {
    static constexpr int M = M_;
    static constexpr int P = plan_passes(M, RB);
    static constexpr int bits(int q) { return plan_bits(M, RB, q); }
    static constexpr int R(int q) { return 1 << bits(q); }
    static constexpr int sh(int q) { return RB * q; }      // log2 of LP(q)
    static constexpr int LP(int q) { return 1 << sh(q); }
    static constexpr int off(int q) {           // first table entry of pass q >= 1
        int o = 0;
        for (int i = 1; i < q; ++i) o += 4 * LP(i);
        return o;
    }
};
__host__ __device__ constexpr int band_radix_bits(int M) { return M >= 1024 ? 4 : (M == 512 ? 3 : 2); }
template <int M> using band_plan = RowPlan<M, band_radix_bits(M)>;

template <typename PL> __host__ __device__ __forceinline__ int dit_pos(int n) {
    int p = 0, sn = 0;
#pragma unroll
    for (int q = PL::P - 1; q >= 0; --q) {
        const int b = PL::bits(q);
        p |= ((n >> sn) & ((1 << b) - 1)) << PL::sh(q);
        sn += b;
    }
    return p;
}

// the tables of every pass of the plan with rb bits of radix, from tw[m] = W_M^m
template <typename C>
inline void plan_twiddle_table(int M, int rb, const C* tw, std::vector<C>& out) {
    out.clear();
    for (int q = 1; q < plan_passes(M, rb); ++q) {
        const int LP = 1 << (rb * q), R = 1 << plan_bits(M, rb, q), L = R * LP, step = M / L;
        for (int e = 1; e <= 8; e *= 2)
            for (int k = 0; k < LP; ++k) out.push_back(tw[((long long)e * step * k) % M]);
    }
    if (out.empty()) out.push_back(tw[0]);
}

// a twiddle table that a kernel has copied to shared memory
template <typename T> struct SmemTw { const cpx<T>* p; };
template <typename T> __device__ __forceinline__ cpx<T> ldtw(const SmemTw<T>& tw, int i) { return tw.p[i]; }

template <typename T> NSE_HD T fmadd(T a, T b, T c) { return ::fma(a, b, c); }
template <typename T> NSE_HD cpx<T> fmul_c(cpx<T> a, cpx<T> b) { return {fmadd(a.x, b.x, -(a.y * b.y)), fmadd(a.x, b.y, a.y * b.x)}; }
template <typename T> NSE_HD cpx<T> fmul_cc(cpx<T> a, cpx<T> b) { return {fmadd(a.x, b.x, a.y * b.y), fmadd(a.y, b.x, -(a.x * b.y))}; }  // a * conj(b)
template <typename T, bool INV> NSE_HD cpx<T> fmul_tw(cpx<T> a, cpx<T> w) { return INV ? fmul_cc(a, w) : fmul_c(a, w); }

template <typename T, bool INV> NSE_HD void fdft8(cpx<T>* v) {
    // radix-2 split into even/odd 4-point DFTs, then combine with e^{-/+ 2 pi i k/8}, whose factor 1/sqrt(2)
    // goes into the multiply-adds of the combine
    const T s = (T)0.70710678118654752440084436210484903928;
    cpx<T> e[4] = {v[0], v[2], v[4], v[6]};
    cpx<T> o[4] = {v[1], v[3], v[5], v[7]};
    dft4<T, INV>(e); dft4<T, INV>(o);
    const cpx<T> o1 = INV ? cpx<T>{o[1].x - o[1].y, o[1].x + o[1].y} : cpx<T>{o[1].x + o[1].y, o[1].y - o[1].x};
    const cpx<T> o2 = INV ? mul_pi(o[2]) : mul_mi(o[2]);
    const cpx<T> o3 = INV ? cpx<T>{-(o[3].x + o[3].y), o[3].x - o[3].y} : cpx<T>{o[3].y - o[3].x, -(o[3].x + o[3].y)};
    v[0] = cadd(e[0], o[0]); v[4] = csub(e[0], o[0]);
    v[1] = {fmadd(s, o1.x, e[1].x), fmadd(s, o1.y, e[1].y)};
    v[5] = {fmadd(-s, o1.x, e[1].x), fmadd(-s, o1.y, e[1].y)};
    v[2] = cadd(e[2], o2);   v[6] = csub(e[2], o2);
    v[3] = {fmadd(s, o3.x, e[3].x), fmadd(s, o3.y, e[3].y)};
    v[7] = {fmadd(-s, o3.x, e[3].x), fmadd(-s, o3.y, e[3].y)};
}
// as dft16, 4 x 4
template <typename T, bool INV> NSE_HD void fdft16(cpx<T>* v) {
    cpx<T> y[4][4];
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
        cpx<T> q[4] = {v[n2], v[4 + n2], v[8 + n2], v[12 + n2]};
        dft4<T, INV>(q);
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) {
            const int j = n2 * k1;                             // W16^j = e^{-i pi (2 j) / 16}
            if (j == 0) y[n2][k1] = q[k1];
            else if (j == 4) y[n2][k1] = INV ? mul_pi(q[k1]) : mul_mi(q[k1]);
            else y[n2][k1] = fmul_tw<T, INV>(q[k1], w32<T>(2 * j >= 16 ? 2 * j - 16 : 2 * j));
            if (2 * j >= 16) y[n2][k1] = {-y[n2][k1].x, -y[n2][k1].y};
        }
    }
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
        cpx<T> q[4] = {y[0][k1], y[1][k1], y[2][k1], y[3][k1]};
        dft4<T, INV>(q);
#pragma unroll
        for (int k2 = 0; k2 < 4; ++k2) v[k1 + 4 * k2] = q[k2];
    }
}
template <typename T, int R, bool INV> NSE_HD void fdftR(cpx<T>* v) {
    if constexpr (R == 2) dft2<T, INV>(v);
    else if constexpr (R == 4) dft4<T, INV>(v);
    else if constexpr (R == 8) fdft8<T, INV>(v);
    else fdft16<T, INV>(v);
}

// Butterfly b of pass q >= 1: loads its R points from the buffer, applies the twiddles and the
// R-point DFT; v[r] is then the output at position base + r LP (returned in base).
template <typename T, typename PL, int Q, bool INV, typename TW>
__device__ __forceinline__ int plan_bfly(const cpx<T>* __restrict__ buf, const TW& tw, int b, cpx<T> (&v)[PL::R(Q)]) {
    constexpr int M = PL::M, R = PL::R(Q), LP = PL::LP(Q), OFF = PL::off(Q);
    const int mm = b & (LP - 1);
    const int base = (b - mm) * R + mm;
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = buf[ip_idx<M>(base + r * LP)];
    if (mm > 0) {
        const int t = OFF + mm;
        const cpx<T> w1 = ldtw(tw, t);
        if constexpr (R == 2) {
            v[1] = fmul_tw<T, INV>(v[1], w1);
        } else {
            const cpx<T> w2 = ldtw(tw, t + LP), w3 = fmul_c(w1, w2);
#pragma unroll
            for (int r = 1; r < R; ++r) {                  // low digit a = r mod 4
                const int a = r & 3;
                if (a) v[r] = fmul_tw<T, INV>(v[r], a == 1 ? w1 : (a == 2 ? w2 : w3));
            }
            if constexpr (R >= 8) {                        // high digit r / 4
                const cpx<T> w4 = ldtw(tw, t + 2 * LP);
                cpx<T> w8 = w4, w12 = w4;
                if constexpr (R == 16) {
                    w8 = ldtw(tw, t + 3 * LP);
                    w12 = fmul_c(w4, w8);
                }
#pragma unroll
                for (int r = 4; r < R; ++r) {
                    const int hb = r >> 2;
                    v[r] = fmul_tw<T, INV>(v[r], hb == 1 ? w4 : (hb == 2 ? w8 : w12));
                }
            }
        }
    }
    fdftR<T, R, INV>(v);
    return base;
}

}  // namespace nse2d
