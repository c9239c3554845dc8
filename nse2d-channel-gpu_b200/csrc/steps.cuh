// Whole steps in one launch, for grids of up to 514 rows of up to 1024 points. Written for this project.
//
// On such a grid a step by launches is eight kernels of 2 to 3 us each and as much again between them. Here one
// cooperative launch takes any number of steps (run_steps asks for 64 at most, so that other streams come in between, and
// steps beside those of another channel by launches): a CTA keeps its band of rows (band.cuh) in shared memory from step
// to step, the tridiagonal solve (solve_cta.cuh) is dealt over the same CTAs, and a barrier across the grid
// separates the two: seven barriers a step (six without an adaptive dt). Per step
//   3 x { stage of the band; forward transform -> omega-hat | barrier | solve of the CTA's columns -> psi-hat, the
//         next omega rows in flight | barrier | inverse transform of the band and its halo, wall closure }
//   psi out, time advanced by every CTA alike, max |u|, |v| of the band | barrier | dt.
// The fields and the control block end as by the same number of steps by launches, to the bit: the row work and the
// solve are the same functions. omega^n of the band stays in shared memory for the three stages, psi is not
// written between them.
//
// What is written by one CTA and read by another in the same launch (spectra, omega halo rows) is read past L1
// (ld.cg, cp.async.cg), or through an L1 that the barrier's acquire has emptied. Every wait is bounded: a barrier that
// gives up sets bit 1 of the non-finite flag and the CTA returns; the others then give up too, and later launches do
// nothing until a state is set. The launch is cooperative, so all CTAs are resident.
//
// What bounds it: at 128x129 (127 CTAs of one row) the barriers, about 3000 clocks each of 42000 a step (drain of
// the stores, arrival, poll: three trips to L2); at 1024x513 the latency of the phases (stage 6000 clocks, solve
// 6600, inverse 5500, forward 3400, barriers 3000 to 6000 with their skew, of 103000). Steps by launches and here:
// 128x129 30.7 and 21.2 us, 256x257 32.8 and 25.1, 1024x513 59.4 and 52.3; FP32 512x301 48 and 28.9. Polling with
// relaxed loads and one fence at the end: 0.3 us a barrier more. The rhs of stage 1, which needs no dt, between arriving
// at the maxima's barrier and waiting there: a second copy of the stage in the kernel, 128x129 23.0 us.
#pragma once
#include "band.cuh"
#include "solve_cta.cuh"

namespace nse2d {

template <int M> struct Steps {
    static constexpr int RMAX = 4;                           // rows of a band: 512 interior rows over the SMs
    static constexpr int NT = (RMAX + 2) * Band<M>::TPR > SC_NT ? (RMAX + 2) * Band<M>::TPR : SC_NT;   // most threads
    static constexpr int KX = M <= 256 ? 2 : 4;              // columns of a solve
};
// threads of a CTA for bands of R rows: the row groups, and the 256 of the solve
template <int M> __host__ __device__ constexpr int steps_threads(int R) {
    return (R + 2) * Band<M>::TPR > SC_NT ? (R + 2) * Band<M>::TPR : SC_NT;
}

template <typename T> struct StepsParams {
    BandParams<T> b;
    ThomasParams th;
    MaxParams mx;            // constants of dt (adapt) and of the maxima
    const float* dpsibar;    // FP32: psibar_{j+1} - psibar_{j-1}
    T* w[3];                 // omega^n, omega^(1), omega^(2)
    T* psi;
    T* rhs;
    int nsteps, R, run;
    int store;               // the stage-3 rhs: 0 never, 1 in the last step, 2 in every step
};

// A barrier across the grid; false when it gave up. `target` counts the arrivals due so far (thread 0).
__device__ __forceinline__ bool grid_barrier(unsigned* arrive, unsigned& target) {
    __syncthreads();
    bool ok = true;
    if (threadIdx.x == 0) {
        target += gridDim.x;
        asm volatile("fence.acq_rel.gpu;\n" ::: "memory");
        atomicAdd(arrive, 1u);
        unsigned it = 0, v;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(arrive) : "memory");
        } while ((int)(v - target) < 0 && ++it < kTmaWaitLimit);
        ok = (int)(v - target) >= 0;
    }
    return __syncthreads_and(ok);
}

// max |u|, |v|, |v| a of the band's rows (k_maxuv_dt, k_maxuv32: the same per-point values) into acc[3], and bit 0 of
// the non-finite flag
template <typename T, int M>
__device__ __forceinline__ void band_maxima(const BandCta<T, M>& c, const StepsParams<T>& p, unsigned long long* acc) {
    using B = Band<M>;
    __shared__ double red[3][16];
    double um = 0.0, vm = 0.0, vmm = 0.0;
    T probe = 0;
    const double cy = 0.5 * p.mx.inv_deta, cx = 0.5 * p.mx.inv_dx;
    for (int item = threadIdx.x; item < c.nr * M; item += blockDim.x) {
        const int n = item & (M - 1), q = item / M, j = c.j0 + q;
        const cpx<T>* b = c.rows + (size_t)q * B::ROW;
        T v[4];
        band_window<T, M, true>(b + B::ROW, n, v);
        const cpx<T> lo = b[ip_idx<M>(n)], hi = b[2 * B::ROW + ip_idx<M>(n)];
        const double a = __ldg(&p.mx.a_node[j]);
        T e0 = hi.x - lo.x, e1 = hi.y - lo.y;
        if constexpr (sizeof(T) == 4) {
            const float d = __ldg(&p.dpsibar[j]);
            e0 += d;
            e1 += d;
        }
        const T f0 = v[2] - v[0], f1 = v[3] - v[1];
        probe += (e0 + f0) + (e1 + f1);
        const double dym = nn_max((double)fabs(e0), (double)fabs(e1)), dxm = nn_max((double)fabs(f0), (double)fabs(f1));
        const double av = dxm * cx;
        um = nn_max(um, a * (dym * cy));
        vm = nn_max(vm, av);
        vmm = nn_max(vmm, av * a);
    }
    um = warp_max_nn(um); vm = warp_max_nn(vm); vmm = warp_max_nn(vmm);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)blockDim.x >> 5;
    if (lane == 0) { red[0][warp] = um; red[1][warp] = vm; red[2][warp] = vmm; }
    const int anynf = __syncthreads_or(!(probe - probe == (T)0) || !(um <= 1e300) || !(vm <= 1e300));
    if (threadIdx.x < 3) {
        double m = 0.0;
        for (int w = 0; w < nw; ++w) m = nn_max(m, red[threadIdx.x][w]);
        atomicMax(&acc[threadIdx.x], (unsigned long long)__double_as_longlong(m));
        if (threadIdx.x == 0 && anynf) atomicOr(&p.b.ctl->nonfinite, 1);
    }
}

// The solve of the CTA's columns (at most one group of KX per CTA), by its first 256 threads.
template <int KX, bool F32>
__device__ __forceinline__ void solve_own(const ThomasParams& p, SolveSmem<KX>& sm, const double* cp, const double2* rc) {
    const int g = blockIdx.x;
    if (threadIdx.x >= SC_NT || g * KX >= p.H) return;
    const SolveCoefShared<KX> coef{cp, rc, (int)threadIdx.x % KX};
    if (p.Ni <= 1 * (SC_NT / KX)) solve_columns<KX, 1, F32>(p, g, sm, coef);
    else if (p.Ni <= 2 * (SC_NT / KX)) solve_columns<KX, 2, F32>(p, g, sm, coef);
    else if (p.Ni <= 4 * (SC_NT / KX)) solve_columns<KX, 4, F32>(p, g, sm, coef);
    else solve_columns<KX, 8, F32>(p, g, sm, coef);
}
template <typename T, int M> __host__ __device__ constexpr size_t steps_smem_bytes(int R, int Ni) {
    return (band_smem_bytes<T, M>(R) + 15) / 16 * 16 + (size_t)Ni * (16 + 8 * Steps<M>::KX);
}

template <typename T, int M>
static __global__ void __launch_bounds__(Steps<M>::NT, 1) k_steps(const __grid_constant__ StepsParams<T> p) {
    using B = Band<M>;
    constexpr int KX = Steps<M>::KX;
    constexpr bool F32 = sizeof(T) == 4;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SolveSmem<KX> solve_sm;
    BandParams<T> b = p.b;
    BandCta<T, M> c(b, smem_raw, p.R);
    Ctl* ctl = b.ctl;
    // the control block: every CTA advances its own copy alike, CTA 0 writes it back
    StepClock k;
    k.load(ctl);
    double mu = ctl->umax, mv = ctl->vmax, mvm = ctl->vmaxm;
    long long budget = ctl->run_budget;
    const int adapt = p.mx.adapt;
    if (*(volatile const int*)&ctl->nonfinite & 2) return;   // after a wait that gave up the state is void, and the counters are
    unsigned target = 0;
    c.load_consts(b);
    // the coefficients of the CTA's columns and rows of the solve, for every solve of the launch
    const int Ni = p.th.Ni;
    double2* rcs = reinterpret_cast<double2*>(smem_raw + (band_smem_bytes<T, M>(p.R) + 15) / 16 * 16);
    double* cps = reinterpret_cast<double*>(rcs + Ni);
    if ((int)blockIdx.x * KX < p.th.H) {
        for (int e = threadIdx.x; e < Ni * KX; e += blockDim.x) cps[e] = __ldg(&p.th.cp[(size_t)(e / KX) * p.th.Hp + blockIdx.x * KX + e % KX]);
        for (int r = threadIdx.x; r < Ni; r += blockDim.x) rcs[r] = make_double2(__ldg(&p.th.asub[r + 1]), __ldg(&p.th.inv_csup[r + 1]));
    }
    c.load_psi(p.psi);
    c.load_omega(p.w[0], true);
    cp_async_wait_all();
    __syncthreads();
    if (adapt) band_maxima<T, M>(c, p, ctl->mx2[0]);
    if (!grid_barrier(&ctl->bar_arrive, target)) {
        if (threadIdx.x == 0) atomicOr(&ctl->nonfinite, 2);
        return;
    }
    for (int n = 0;; ++n) {
        const int nf = *(volatile const int*)&ctl->nonfinite;
        if (adapt) {
            const unsigned long long* acc = ctl->mx2[n & 1];
            mu = __longlong_as_double((long long)__ldcg(acc));
            mv = __longlong_as_double((long long)__ldcg(acc + 1));
            mvm = __longlong_as_double((long long)__ldcg(acc + 2));
            k.dt = adaptive_dt(mu, mvm, k.t, k.next_out, p.mx.cfl, p.mx.dx, p.mx.deta, p.mx.cvisc, p.mx.nu, p.mx.inv_dx2, p.mx.inv_dymin2,
                               p.mx.dt_max);
        }
        const T dt = (T)k.dt;
        const bool last = n + 1 == p.nsteps;
        // the spectra and the rows of a stage cross CTAs twice
#pragma unroll 1
        for (int st = 1; st <= 3; ++st) {
            b.stage = st;
            b.w_out = st == 3 ? p.w[0] : p.w[st];
            b.rhs_out = (st == 3 && (p.store == 2 || (p.store == 1 && last))) ? p.rhs : nullptr;
            c.stage(b, dt, st == 1);
            __syncthreads();
            c.forward(b);
            bool ok = grid_barrier(&ctl->bar_arrive, target);
            if (ok) {
                if (adapt && st == 1 && blockIdx.x == 0 && threadIdx.x < 3) ctl->mx2[(n + 1) & 1][threadIdx.x] = 0ull;
                c.load_omega(b.w_out, false);                // in flight during the solve
                solve_own<KX, F32>(p.th, solve_sm, cps, rcs);
                ok = grid_barrier(&ctl->bar_arrive, target);
            }
            if (!ok) {
                if (threadIdx.x == 0) atomicOr(&ctl->nonfinite, 2);
                cp_async_wait_all();
                return;
            }
            c.load_spec(b);
            cp_async_wait_all();                             // the omega rows too
            __syncthreads();
            c.inverse(b);
            __syncthreads();
            if (c.bot || c.top) {
                c.walls(b, b.w_out);
                __syncthreads();
            }
        }
        // psi^(n+1) out
        cpx<T>* psi = reinterpret_cast<cpx<T>*>(p.psi);
        const int q0 = c.bot ? 0 : 1, q1 = c.top ? c.nr + 1 : c.nr;     // a band at a wall writes the wall's row too
        for (int item = threadIdx.x; item < (q1 - q0 + 1) * M; item += blockDim.x) {
            const int q = q0 + item / M, i = item & (M - 1);
            psi[(size_t)(c.j0 - 1 + q) * M + i] = c.rows[(size_t)q * B::ROW + ip_idx<M>(i)];
        }
        int reason = k.advance(p.run, nf);
        if (p.run) {
            budget -= 1;
            if (!reason && budget <= 0) reason = 16;
        }
        if (reason || last) {
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                k.store(ctl);
                ctl->umax = mu; ctl->vmax = mv; ctl->vmaxm = mvm;
                ctl->run_budget = budget;
                if (reason) {
                    ctl->halt = 1;
                    ctl->halt_reason = reason;
                }
            }
            break;
        }
        if (adapt) {
            band_maxima<T, M>(c, p, ctl->mx2[(n + 1) & 1]);
            if (!grid_barrier(&ctl->bar_arrive, target)) {
                if (threadIdx.x == 0) atomicOr(&ctl->nonfinite, 2);
                return;
            }
        }
    }
    // the last CTA out leaves the barrier and the accumulators as it found them
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&ctl->bar_exit, 1u) == gridDim.x - 1) {
            ctl->bar_arrive = 0;
            ctl->bar_exit = 0;
            for (int q = 0; q < 6; ++q) ctl->mx2[q / 3][q % 3] = 0ull;
        }
    }
}

}  // namespace nse2d
