// The learned subgrid closure: a small CNN whose 3x3 convolutions run as BF16 GEMMs on the
// tensor cores (tcgen05, FP32 accumulate), its backward pass, AdamW, and the coarse-grid data
// generator (box filter). Written for this project; the reference has no closure model.
//
// Model. Inputs per point: the coarse omega, psi, u, v (each divided by a fixed scale) and y,
// 5 channels. Four 3x3 convolutions 5 -> H -> H -> H -> 1, GELU (tanh form) after the first
// three, periodic in x and zero-padded beyond the walls. Output: tau / tau_scale, the subgrid
// term of the Jacobian,
//   tau = filter(J(psi, omega)) - J(filter psi, filter omega),
// which the coarse solver subtracts from its rhs on interior rows. A batch is B whole coarse
// fields side by side; every field keeps its own periodic x and its own walls.
//
// Layout. A pixel p = b Nx Ny + j Nx + i; activations are BF16 [P][C] (channels contiguous; the input's 5
// channels padded to 8). A convolution is k_conv (conv_tc.cuh), Z = A . W^T + b with W [N_pad][K] (K = tap C +
// c, tap = 3 (dy + 1) + dx + 1, padded to a multiple of 64; N_pad a multiple of 16), whose epilogue writes Z
// (FP32, kept for the backward pass) and GELU(Z) in BF16, the next layer's input.
//
// Backward (loss = mean over interior pixels of (z - tau/tau_scale)^2):
//   dW[n][k] = sum_p dZ[p][n] A[p][k] with dZ in FP32 (k_wgrad; k_wgrad_out for the one output channel),
//   db[n] = sum_p dZ[p][n]; per-block partials folded in a fixed order, so the gradients do not depend on
//   scheduling;
//   dZ of the layer below = GELU'(z) times the convolution of dZ (BF16) with the flipped taps (k_conv again;
//   k_dgrad_out for the output layer).
// AdamW updates FP32 master weights and re-exports the BF16 W and the flipped W.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "nse2d_internal.h"
#include "conv_tc.cuh"
#include "../../include/nse2d.h"

namespace nse2d {

__device__ int g_tc_err;                  // error flag of the tensor-core GEMM's bounded waits

namespace {

constexpr int CN_LAYERS = 4;
constexpr int CN_CIN = 5;                 // omega, psi, u, v, y
constexpr int CN_C0 = 8;                  // channels of the stored input (padded: 16 bytes a pixel)
constexpr int CN_NT = 256;
constexpr int CN_OUT_PX = 512;           // pixels per block of the output layer's weight gradient

int round_up(int x, int m) { return (x + m - 1) / m * m; }

}  // namespace

struct Cnn {
    int Nx = 0, Ny = 0, nxy = 0, hidden = 0, max_batch = 0;
    int nb = 1, P = 0, Ppad = 0;          // the current batch
    int cin[CN_LAYERS], cout[CN_LAYERS], npad[CN_LAYERS], K[CN_LAYERS];
    float* w32[CN_LAYERS] = {};           // [npad][K] master weights (padding stays zero)
    float* b32[CN_LAYERS] = {};           // [npad]
    float* gw[CN_LAYERS] = {};
    float* gb[CN_LAYERS] = {};
    float* mw[CN_LAYERS] = {};
    float* vw[CN_LAYERS] = {};
    float* mb[CN_LAYERS] = {};
    float* vb[CN_LAYERS] = {};
    __nv_bfloat16* wbf[CN_LAYERS] = {};   // [npad][K]
    __nv_bfloat16* wtbf[CN_LAYERS] = {};  // layers 1, 2: [cin][9 npad], tap-major, for the gradient of the input
    __nv_bfloat16* h[CN_LAYERS] = {};     // layer input: h[0] [Ppad][8], h[l] [Ppad][npad[l-1]]
    float* z[CN_LAYERS] = {};             // pre-activations [Ppad][npad]; the output layer's [Ppad]
    float* dz[2] = {};                    // dZ of two layers [Ppad][hidden]
    __nv_bfloat16* dzb[2] = {};           // the same in BF16
    float* dz_out = nullptr;              // dZ of the output layer [Ppad]
    int sms = 0;                          // SMs of the device
    int wg_blocks = 0;                    // blocks of the weight-gradient reductions
    float* part = nullptr;                // their partials
    float* lpart = nullptr;               // loss partials [ceil(Ppad / CN_NT)]
    float* loss = nullptr;                // [1]
    double* y = nullptr;                  // [Ny] wall-normal coordinate (the fifth input)
    int* idx = nullptr;                   // [max_batch] sample of every batch slot
    int* err = nullptr;
    double in_scale[CN_CIN - 1] = {1.0, 1.0, 1.0, 1.0};
    double out_tau = 1.0;
    int wall_rows = 1;                    // rows next to each wall (the wall row included) with tau = 0
    double gain = 1.0;                    // factor on the applied tau
    bool row_mean = false;                // apply the x-mean of tau on every row (the mean-flow part)
    long long step = 0;
    unsigned settings = 0;                // changes of the scales and of the application
};

int tc_gemm_launch(const TcGemmParams& p0, cudaStream_t s);

namespace {

template <typename T> int cn_alloc(T** p, size_t n) {
    NSE_CUDA_TRY(cudaMalloc((void**)p, n * sizeof(T) + 16));
    NSE_CUDA_TRY(cudaMemset(*p, 0, n * sizeof(T) + 16));
    return 0;
}

struct PackSrc {
    const double* w;         // [S][Ny][Nx]; batch slot b reads sample idx[b]
    const double* psi;
    const double* u;
    const double* v;
    const int* idx;          // [nb]
    const double* y;         // [Ny]
    double s0, s1, s2, s3;   // 1 / scale of omega, psi, u, v
};

// The 5 input channels of every pixel of the batch, padded to 8. UV: u and v of the fields' psi (one field;
// src/ops.cu:47-70) instead of given ones, as the solver's coupling needs them.
struct PackUv {
    const double* a_node;
    double inv_dx, inv_deta;
};
template <bool UV>
__global__ void k_pack_input(PackSrc q, PackUv g, __nv_bfloat16* h0, int nxy, int Nx, int Ny, int P) {
    cv_wait_for_last_layer();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P) return;
    const int b = p / nxy, r = p - b * nxy;
    const size_t src = (size_t)q.idx[b] * nxy + r;
    double u, v;
    const int j = r / Nx;
    if constexpr (UV) {
        const int i = r - j * Nx, xm = i == 0 ? Nx - 1 : i - 1, xp = i == Nx - 1 ? 0 : i + 1;
        const int ym = j == 0 ? 0 : j - 1, yp = j == Ny - 1 ? j : j + 1;
        const double dpsideta = (q.psi[(size_t)yp * Nx + i] - q.psi[(size_t)ym * Nx + i]) * 0.5 * g.inv_deta;
        const double dpsidx = (q.psi[(size_t)j * Nx + xp] - q.psi[(size_t)j * Nx + xm]) * 0.5 * g.inv_dx;
        u = g.a_node[j] * dpsideta;
        v = -dpsidx;
    } else {
        u = q.u[src];
        v = q.v[src];
    }
    const float f[CN_CIN] = {(float)(q.w[src] * q.s0), (float)(q.psi[src] * q.s1), (float)(u * q.s2), (float)(v * q.s3), (float)q.y[j]};
    *reinterpret_cast<uint4*>(h0 + (size_t)p * CN_C0) = make_uint4(cv_pack2(f[0], f[1]), cv_pack2(f[2], f[3]), cv_pack2(f[4], 0.f), 0u);
}

// the x-mean of tau on every row: one CTA per row
__global__ void __launch_bounds__(CN_NT) k_unpack_row_mean(const float* z, double* tau, int Nx, int Ny, double ts, int wall_rows) {
    __shared__ double red[CN_NT];
    cv_wait_for_last_layer();
    const int j = blockIdx.x;
    double sum = 0.0;
    for (int i = threadIdx.x; i < Nx; i += CN_NT) sum += (double)z[(size_t)j * Nx + i];
    red[threadIdx.x] = sum;
    __syncthreads();
    for (int st = CN_NT / 2; st > 0; st >>= 1) {
        if ((int)threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
        __syncthreads();
    }
    const double m = (j < wall_rows || j >= Ny - wall_rows) ? 0.0 : ts * red[0] / (double)Nx;
    for (int i = threadIdx.x; i < Nx; i += CN_NT) tau[(size_t)j * Nx + i] = m;
}

// loss partials and dZ of the output layer: d = z - tau / tau_scale on interior pixels
__global__ void __launch_bounds__(CN_NT) k_loss(const float* z, const double* tau, const int* idx, double inv_ts, int Nx, int Ny, int P,
                                                int wall_rows, float inv_pint, float* dz, float* lpart) {
    __shared__ float red[CN_NT];
    const int p = blockIdx.x * CN_NT + threadIdx.x;
    const int nxy = Nx * Ny;
    float l = 0.f;
    if (p < P) {
        float g = 0.f;
        const int b = p / nxy, r = p - b * nxy, j = r / Nx;
        if (j >= wall_rows && j < Ny - wall_rows) {
            const float d = z[p] - (float)(tau[(size_t)idx[b] * nxy + r] * inv_ts);
            l = d * d;
            g = 2.f * d * inv_pint;
        }
        dz[p] = g;
    }
    red[threadIdx.x] = l;
    __syncthreads();
    for (int st = CN_NT / 2; st > 0; st >>= 1) {
        if ((int)threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0) lpart[blockIdx.x] = red[0];
}
__global__ void __launch_bounds__(CN_NT) k_fold_loss(const float* lpart, int n, float scale, float* loss) {
    __shared__ float red[CN_NT];
    float s = 0.f;
    for (int i = threadIdx.x; i < n; i += CN_NT) s += lpart[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int st = CN_NT / 2; st > 0; st >>= 1) {
        if ((int)threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0) *loss = red[0] * scale;
}

// Weight-gradient partials [nblk][nk][nn] and bias partials [nblk][nn] (after them) -> gw[n][k] (row stride K)
// and gb[n]. A block folds 32 outputs in eight slices of the partials' blocks; the order is fixed.
__global__ void __launch_bounds__(256) k_fold_grads(const float* part, int nblk, int nk, int nn, int K, float* gw, float* gb) {
    __shared__ float red[8][33];
    const int lane = threadIdx.x & 31, sl = threadIdx.x >> 5;
    const int nout = (nk + 1) * nn, o = blockIdx.x * 32 + lane;
    const bool bias = o >= nk * nn;
    const float* src = bias ? part + (size_t)nblk * nk * nn + (o - nk * nn) : part + o;
    const size_t stride = bias ? nn : (size_t)nk * nn;
    float s = 0.f;
    if (o < nout) {
        const int b0 = (int)((long long)sl * nblk / 8), b1 = (int)((long long)(sl + 1) * nblk / 8);
#pragma unroll 8
        for (int b = b0; b < b1; ++b) s += src[(size_t)b * stride];
    }
    red[sl][lane] = s;
    __syncthreads();
    if (sl == 0 && o < nout) {
#pragma unroll
        for (int q = 1; q < 8; ++q) s += red[q][lane];
        if (bias) gb[o - nk * nn] = s;
        else gw[(size_t)(o % nn) * K + o / nn] = s;
    }
}

// dZ of the layer below the output layer: the one output channel's dZ (BF16) times the flipped taps of W, times
// GELU'(z). A thread takes eight channels of a pixel. Products of two BF16 values are exact in FP32.
__global__ void __launch_bounds__(CN_NT) k_dgrad_out(const float* dz, const __nv_bfloat16* w, int C, const float* zprev, int Nx, int Ny, int P,
                                                     float* dzo, __nv_bfloat16* dzb) {
    extern __shared__ __align__(16) float ws[];                    // [9][C]
    for (int e = threadIdx.x; e < 9 * C; e += CN_NT) ws[e] = __bfloat162float(w[e]);
    __syncthreads();
    const int nq = C >> 3;
    const long long t = (long long)blockIdx.x * CN_NT + threadIdx.x;
    const int p = (int)(t / nq), c = (int)(t - (long long)p * nq) * 8;
    if (p >= P) return;
    const size_t o = (size_t)p * C + c;
    const float4 z0 = __ldg(reinterpret_cast<const float4*>(zprev + o)), z1 = __ldg(reinterpret_cast<const float4*>(zprev + o) + 1);
    const CvPix q = cv_pix(p, P, Nx, Ny);
    float d[9], s[8] = {};
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
        int src;
        d[tap] = cv_tap(q, 1 - tap / 3, 1 - tap % 3, Nx, Ny, src) ? __bfloat162float(__float2bfloat16_rn(__ldg(dz + src))) : 0.f;
    }
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
        const float4 a = *reinterpret_cast<const float4*>(ws + tap * C + c), b = *reinterpret_cast<const float4*>(ws + tap * C + c + 4);
        s[0] = fmaf(d[tap], a.x, s[0]); s[1] = fmaf(d[tap], a.y, s[1]); s[2] = fmaf(d[tap], a.z, s[2]); s[3] = fmaf(d[tap], a.w, s[3]);
        s[4] = fmaf(d[tap], b.x, s[4]); s[5] = fmaf(d[tap], b.y, s[5]); s[6] = fmaf(d[tap], b.z, s[6]); s[7] = fmaf(d[tap], b.w, s[7]);
    }
    s[0] *= tg_gelu_grad(z0.x); s[1] *= tg_gelu_grad(z0.y); s[2] *= tg_gelu_grad(z0.z); s[3] *= tg_gelu_grad(z0.w);
    s[4] *= tg_gelu_grad(z1.x); s[5] *= tg_gelu_grad(z1.y); s[6] *= tg_gelu_grad(z1.z); s[7] *= tg_gelu_grad(z1.w);
    reinterpret_cast<float4*>(dzo + o)[0] = make_float4(s[0], s[1], s[2], s[3]);
    reinterpret_cast<float4*>(dzo + o)[1] = make_float4(s[4], s[5], s[6], s[7]);
    *reinterpret_cast<uint4*>(dzb + o) = make_uint4(cv_pack2(s[0], s[1]), cv_pack2(s[2], s[3]), cv_pack2(s[4], s[5]), cv_pack2(s[6], s[7]));
}

// The output layer's weight gradient: dW[tap C + c] = sum_q h[q][c] dZ[q - offset of the tap], db = sum dZ, as
// partials [nblk][9 C] and [nblk]. A warp takes 32 pixels at a time: every lane gathers the nine dZ of its own
// pixel into shared memory, then the lanes are the channels (one or two each) and walk over the 32 pixels, whose
// dZ they read as broadcasts. Gathering per pixel by the whole warp took 95 us for 264192 pixels.
__global__ void __launch_bounds__(CN_NT) k_wgrad_out(const __nv_bfloat16* h, const float* dz, int C, int Nx, int Ny, int P, float* part) {
    __shared__ float red[8][9 * 64 + 1];
    __shared__ __align__(16) float sd[8][32][12];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int p1 = min(P, ((int)blockIdx.x + 1) * CN_OUT_PX);
    float a[2][9] = {}, sb = 0.f;
    for (int p0 = blockIdx.x * CN_OUT_PX + warp * 32; p0 < p1; p0 += 8 * 32) {
        const CvPix q = cv_pix(p0 + lane, p1, Nx, Ny);             // beyond p1: zeros
        float d[9];
#pragma unroll
        for (int tap = 0; tap < 9; ++tap) {
            int src;
            d[tap] = cv_tap(q, 1 - tap / 3, 1 - tap % 3, Nx, Ny, src) ? __ldg(dz + src) : 0.f;
        }
        sb += d[4];
        __syncwarp();
        float4* w = reinterpret_cast<float4*>(sd[warp][lane]);
        w[0] = make_float4(d[0], d[1], d[2], d[3]);
        w[1] = make_float4(d[4], d[5], d[6], d[7]);
        w[2] = make_float4(d[8], 0.f, 0.f, 0.f);
        __syncwarp();
        const int n = min(32, p1 - p0);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const int c = lane + 32 * g;
            if (c >= C) continue;
            const __nv_bfloat16* hp = h + (size_t)p0 * C + c;
#pragma unroll 16
            for (int k = 0; k < n; ++k) {
                const float x = __bfloat162float(hp[(size_t)k * C]);
                const float4* v = reinterpret_cast<const float4*>(sd[warp][k]);
                const float4 u0 = v[0], u1 = v[1];
                const float u8 = sd[warp][k][8];
                a[g][0] = fmaf(u0.x, x, a[g][0]); a[g][1] = fmaf(u0.y, x, a[g][1]); a[g][2] = fmaf(u0.z, x, a[g][2]);
                a[g][3] = fmaf(u0.w, x, a[g][3]); a[g][4] = fmaf(u1.x, x, a[g][4]); a[g][5] = fmaf(u1.y, x, a[g][5]);
                a[g][6] = fmaf(u1.z, x, a[g][6]); a[g][7] = fmaf(u1.w, x, a[g][7]); a[g][8] = fmaf(u8, x, a[g][8]);
            }
        }
    }
#pragma unroll
    for (int g = 0; g < 2; ++g)
        if (lane + 32 * g < C)
            for (int tap = 0; tap < 9; ++tap) red[warp][tap * C + lane + 32 * g] = a[g][tap];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sb += __shfl_down_sync(0xffffffffu, sb, o);
    if (lane == 0) red[warp][9 * C] = sb;
    __syncthreads();
    for (int o = threadIdx.x; o <= 9 * C; o += CN_NT) {
        float s = red[0][o];
        for (int w = 1; w < 8; ++w) s += red[w][o];
        if (o < 9 * C) part[(size_t)blockIdx.x * 9 * C + o] = s;
        else part[(size_t)gridDim.x * 9 * C + blockIdx.x] = s;
    }
}

// One layer's parameters (AdamW and the export of the BF16 copies).
struct LayerParams {
    float *w, *gw, *mw, *vw, *b, *gb, *mb, *vb;
    __nv_bfloat16 *wbf, *wt;               // wt: [cin][9 npad] or null
    int npad, K, cin;
};
struct AllLayers { LayerParams l[CN_LAYERS]; };

__device__ __forceinline__ void adamw_one(float* w, const float* g, float* m, float* v, int e, float lr, float b1, float b2, float eps,
                                          float wd, float bc1, float bc2) {
    const float gg = g[e];
    const float mm = b1 * m[e] + (1.f - b1) * gg;
    const float vv = b2 * v[e] + (1.f - b2) * gg * gg;
    m[e] = mm;
    v[e] = vv;
    const float mh = mm / bc1, vh = vv / bc2;
    w[e] -= lr * (mh / (sqrtf(vh) + eps) + wd * w[e]);
}
// W (BF16), and the flipped-tap gradient's [cin][tap npad + n]
__device__ __forceinline__ void export_one(const LayerParams& q, int e) {
    const int n = e / q.K, k = e - n * q.K;
    const __nv_bfloat16 b = __float2bfloat16_rn(q.w[e]);
    q.wbf[e] = b;
    if (q.wt && k < 9 * q.cin) {
        const int tap = k / q.cin, c = k - tap * q.cin;
        q.wt[(size_t)c * 9 * q.npad + tap * q.npad + n] = b;
    }
}
// grid: (blocks of the largest layer, layers). err: a wait of the passes before timed out, and the gradients are void.
__global__ void __launch_bounds__(CN_NT) k_adamw(AllLayers all, const int* err, float lr, float b1, float b2, float eps, float wd, float bc1, float bc2) {
    if (*err) return;
    const LayerParams& q = all.l[blockIdx.y];
    const int e = blockIdx.x * CN_NT + threadIdx.x;
    if (e < q.npad * q.K) {
        adamw_one(q.w, q.gw, q.mw, q.vw, e, lr, b1, b2, eps, wd, bc1, bc2);
        export_one(q, e);
    }
    if (e < q.npad) adamw_one(q.b, q.gb, q.mb, q.vb, e, lr, b1, b2, eps, 0.f, bc1, bc2);
}
__global__ void __launch_bounds__(CN_NT) k_export_w(LayerParams q) {
    const int e = blockIdx.x * CN_NT + threadIdx.x;
    if (e < q.npad * q.K) export_one(q, e);
}

// Top-hat filter of a fine field onto a coarse grid whose nodes are every rx-th column and
// ry-th row of the fine one: the mean over fine columns rx i + d and rows ry j + e, |d| <= rx/2,
// |e| <= ry/2, with half weight at |d| = rx/2 and |e| = ry/2; periodic in x; rows beyond the
// walls are left out and the weights renormalised.
__global__ void k_box_filter(const double* f, int Nxf, int Nyf, double* c, int Nxc, int Nyc) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= Nxc * Nyc) return;
    const int j = p / Nxc, i = p - j * Nxc;
    const int rx = Nxf / Nxc, ry = (Nyf - 1) / (Nyc - 1);
    const int hx = rx / 2, hy = ry / 2;
    double s = 0.0, ws = 0.0;
    for (int e = -hy; e <= hy; ++e) {
        const int jf = ry * j + e;
        if (jf < 0 || jf >= Nyf) continue;
        const double we = (hy > 0 && (e == -hy || e == hy)) ? 0.5 : 1.0;
        for (int d = -hx; d <= hx; ++d) {
            int ifn = rx * i + d;
            ifn = ((ifn % Nxf) + Nxf) % Nxf;
            const double wd = (hx > 0 && (d == -hx || d == hx)) ? 0.5 : 1.0;
            s += we * wd * f[(size_t)jf * Nxf + ifn];
            ws += we * wd;
        }
    }
    c[p] = s / ws;
}

int grid_of(long long n, int nt = CN_NT) { return (int)((n + nt - 1) / nt); }

LayerParams layer_params(const Cnn* n, int l) {
    return LayerParams{n->w32[l], n->gw[l], n->mw[l], n->vw[l], n->b32[l], n->gb[l], n->mb[l], n->vb[l],
                       n->wbf[l], n->wtbf[l], n->npad[l], n->K[l], n->cin[l]};
}

int export_layer(Cnn* n, int l, cudaStream_t s) {
    k_export_w<<<grid_of((long long)n->npad[l] * n->K[l]), CN_NT, 0, s>>>(layer_params(n, l));
    NSE_CUDA_TRY(cudaGetLastError());
    return 0;
}

// a CTA's strip: up to 128 columns, two rows, or one while the strips do not fill the device twice (32 channels, 264192
// pixels, us with one, two and four rows: forward 47, 37, 38; input gradient 52, 44, 50)
void conv_strip(ConvParams& p, int sms) {
    const int sx = (p.Nx + 127) / 128, nb = p.P / (p.Nx * p.Ny);
    p.W = (p.Nx + sx - 1) / sx;
    p.R = 2;
    while (p.R > 1 && (long long)nb * sx * ((p.Ny + p.R - 1) / p.R) < 2 * sms) p.R /= 2;
}
// A kernel that begins with cv_wait_for_last_layer, launched before the one before it has ended.
template <typename... KArgs, typename... Args>
int launch_layer(void (*kern)(KArgs...), int blocks, int threads, size_t smem, cudaStream_t s, Args&&... args) {
    cudaLaunchConfig_t lc{};
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    lc.gridDim = dim3(blocks); lc.blockDim = dim3(threads); lc.dynamicSmemBytes = smem; lc.stream = s;
    lc.attrs = &at; lc.numAttrs = 1;
    NSE_CUDA_TRY(cudaLaunchKernelEx(&lc, kern, std::forward<Args>(args)...));
    return 0;
}
template <int C, int MODE> int conv_t(ConvParams p, int sms, bool setup, cudaStream_t s) {
    if (setup) {
        NSE_CUDA_TRY(cudaFuncSetAttribute(k_conv<C, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)cv_smem_bytes<C>(64, 128, 2)));
        return 0;
    }
    conv_strip(p, sms);
    const int blocks = p.P / (p.Nx * p.Ny) * ((p.Nx + p.W - 1) / p.W) * ((p.Ny + p.R - 1) / p.R);
    return launch_layer(k_conv<C, MODE>, blocks, CV_NT, cv_smem_bytes<C>(p.N, p.W, p.R), s, p);
}
// the input layer
int conv_in(const ConvParams& p, cudaStream_t s) {
    const int blocks = (p.P + TG_BM - 1) / TG_BM;
    const size_t sm = cv_in_smem_bytes(p.N);
    switch (p.N) {
        case 16: return launch_layer(k_conv_in<16>, blocks, CV_NT, sm, s, p);
        case 32: return launch_layer(k_conv_in<32>, blocks, CV_NT, sm, s, p);
        case 48: return launch_layer(k_conv_in<48>, blocks, CV_NT, sm, s, p);
        case 64: return launch_layer(k_conv_in<64>, blocks, CV_NT, sm, s, p);
        default: set_error("no input convolution to %d channels", p.N); return -1;
    }
}
// a convolution of C input channels; setup: only the kernel's shared-memory limit
template <int MODE> int conv(const ConvParams& p, int C, int sms, bool setup, cudaStream_t s) {
    switch (C) {
        case 16: return conv_t<16, MODE>(p, sms, setup, s);
        case 32: return conv_t<32, MODE>(p, sms, setup, s);
        case 48: return conv_t<48, MODE>(p, sms, setup, s);
        case 64: return conv_t<64, MODE>(p, sms, setup, s);
        default: set_error("no convolution of %d channels", C); return -1;
    }
}

template <int C, int N, int TG> int wgrad_t(const WgradParams& p, int blocks, bool setup, cudaStream_t s) {
    constexpr size_t sm = wg_smem_bytes<C, N, TG>();
    if (setup) {
        NSE_CUDA_TRY(cudaFuncSetAttribute(k_wgrad<C, N, TG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        return 0;
    }
    k_wgrad<C, N, TG><<<dim3(blocks, C == CN_C0 ? 1 : 9 / TG), WG_NT, sm, s>>>(p);
    NSE_CUDA_TRY(cudaGetLastError());
    return 0;
}
// weight gradient of the input layer (input = true) or of a hidden layer of H channels; all nine taps in a CTA
// while its accumulators fit the registers
int wgrad(const WgradParams& p, bool input, int H, int blocks, bool setup, cudaStream_t s) {
    switch (H) {
        case 16: return input ? wgrad_t<CN_C0, 16, 9>(p, blocks, setup, s) : wgrad_t<16, 16, 9>(p, blocks, setup, s);
        case 32: return input ? wgrad_t<CN_C0, 32, 9>(p, blocks, setup, s) : wgrad_t<32, 32, 9>(p, blocks, setup, s);
        case 48: return input ? wgrad_t<CN_C0, 48, 9>(p, blocks, setup, s) : wgrad_t<48, 48, 3>(p, blocks, setup, s);
        case 64: return input ? wgrad_t<CN_C0, 64, 9>(p, blocks, setup, s) : wgrad_t<64, 64, 3>(p, blocks, setup, s);
        default: set_error("no weight gradient of %d channels", H); return -1;
    }
}
// blocks of a weight gradient over P pixels: tiles of 64 pixels strided over the resident CTAs
int wgrad_blocks(const Cnn* n) { return std::max(1, std::min((n->P + WG_PX - 1) / WG_PX, n->wg_blocks)); }

void set_batch(Cnn* n, int nb) {
    n->nb = nb;
    n->P = nb * n->nxy;
    n->Ppad = round_up(n->P, 128);
}

}  // namespace

// ---- shared with the solver and the ABI ----

int tc_gemm_launch(const TcGemmParams& p0, cudaStream_t s) {
    TcGemmParams p = p0;
    if (p.M <= 0 || p.M % TG_BM != 0 || p.N < 16 || p.N > 256 || p.N % 16 != 0 || p.K < TG_BK || p.K % TG_BK != 0 ||
        p.ldc < p.N) {
        set_error("tensor-core GEMM: M = %d (multiple of 128), N = %d (16..256, multiple of 16), K = %d (multiple of 64), "
                  "ldc = %d (>= N)", p.M, p.N, p.K, p.ldc);
        return -1;
    }
    if ((reinterpret_cast<uintptr_t>(p.A) | reinterpret_cast<uintptr_t>(p.B)) % 16 != 0) {
        set_error("tensor-core GEMM: A and B must be 16-byte aligned");
        return -1;
    }
    if (!p.err) {
        void* e = nullptr;
        NSE_CUDA_TRY(cudaGetSymbolAddress(&e, g_tc_err));
        p.err = static_cast<int*>(e);
    }
    k_tc_gemm<<<p.M / TG_BM, TG_THREADS, tg_smem_bytes(p.N), s>>>(p);
    NSE_CUDA_TRY(cudaGetLastError());
    return 0;
}

int tc_gemm_setup() {
    NSE_CUDA_TRY(cudaFuncSetAttribute(k_tc_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tg_smem_bytes(256)));
    return 0;
}

// Forward pass of the current batch from the packed sources. keep: the pre-activations of every layer (for the
// backward pass); else only the output layer's, and tau directly when it is given.
static int cnn_forward_batch(Cnn* n, const PackSrc& src, const PackUv* uv, bool keep, double* tau, cudaStream_t s) {
    if (uv)
        k_pack_input<true><<<grid_of(n->P), CN_NT, 0, s>>>(src, *uv, n->h[0], n->nxy, n->Nx, n->Ny, n->P);
    else
        k_pack_input<false><<<grid_of(n->P), CN_NT, 0, s>>>(src, PackUv{}, n->h[0], n->nxy, n->Nx, n->Ny, n->P);
    NSE_CUDA_TRY(cudaGetLastError());
    for (int l = 0; l < CN_LAYERS; ++l) {
        const bool last = (l == CN_LAYERS - 1);
        ConvParams p{};
        p.h = n->h[l]; p.wt = n->wbf[l]; p.bias = n->b32[l]; p.err = n->err;
        p.Nx = n->Nx; p.Ny = n->Ny; p.P = n->P; p.N = n->npad[l]; p.ldw = n->K[l];
        if (last) {
            p.z = tau ? nullptr : n->z[l];
            p.tau = tau;
            p.wall_rows = n->wall_rows;
            p.ts = n->out_tau * n->gain;
            if (conv<CV_OUT>(p, n->cin[l], n->sms, false, s)) return -1;
        } else {
            p.z = keep ? n->z[l] : nullptr;
            p.hn = n->h[l + 1];
            if (l == 0 ? conv_in(p, s) : conv<CV_FWD>(p, n->cin[l], n->sms, false, s)) return -1;
        }
    }
    return 0;
}

static PackSrc pack_src(const Cnn* n, const double* w, const double* psi, const double* u, const double* v) {
    PackSrc q{};
    q.w = w; q.psi = psi; q.u = u; q.v = v; q.idx = n->idx; q.y = n->y;
    q.s0 = 1.0 / n->in_scale[0]; q.s1 = 1.0 / n->in_scale[1]; q.s2 = 1.0 / n->in_scale[2]; q.s3 = 1.0 / n->in_scale[3];
    return q;
}

// Inference on one field (slot 0 of the index table is always sample 0); graph-capturable.
static int cnn_forward_field(Cnn* n, const PackSrc& src, const PackUv* uv, double* tau, cudaStream_t s) {
    set_batch(n, 1);
    if (cnn_forward_batch(n, src, uv, false, n->row_mean ? nullptr : tau, s)) return -1;
    if (n->row_mean) {
        if (launch_layer(k_unpack_row_mean, n->Ny, CN_NT, 0, s, n->z[CN_LAYERS - 1], tau, n->Nx, n->Ny, n->out_tau * n->gain, n->wall_rows))
            return -1;
    }
    return 0;
}
int cnn_forward(Cnn* n, const double* w, const double* psi, const double* u, const double* v, double* tau, cudaStream_t s) {
    return cnn_forward_field(n, pack_src(n, w, psi, u, v), nullptr, tau, s);
}
// the same with u and v of psi
int cnn_forward_psi(Cnn* n, const double* w, const double* psi, const double* a_node, double inv_dx, double inv_deta, double* tau,
                    cudaStream_t s) {
    const PackUv uv{a_node, inv_dx, inv_deta};
    return cnn_forward_field(n, pack_src(n, w, psi, nullptr, nullptr), &uv, tau, s);
}

// Loss against tau (samples idx of the batch) and the gradients of every layer (after the forward pass).
static int cnn_backward(Cnn* n, const double* tau, cudaStream_t s) {
    constexpr int L = CN_LAYERS - 1;
    const int nlb = grid_of(n->P), H = n->npad[0];
    const int pint = n->nb * n->Nx * (n->Ny - 2 * n->wall_rows);
    k_loss<<<nlb, CN_NT, 0, s>>>(n->z[L], tau, n->idx, 1.0 / n->out_tau, n->Nx, n->Ny, n->P, n->wall_rows, 1.f / (float)pint, n->dz_out,
                                 n->lpart);
    k_fold_loss<<<1, CN_NT, 0, s>>>(n->lpart, nlb, 1.f / (float)pint, n->loss);
    NSE_CUDA_TRY(cudaGetLastError());
    auto fold = [&](int l, int nblk, int nk, int nn) {
        k_fold_grads<<<((nk + 1) * nn + 31) / 32, 256, 0, s>>>(n->part, nblk, nk, nn, n->K[l], n->gw[l], n->gb[l]);
        return cudaGetLastError();
    };
    // the output layer: its one channel on the CUDA cores
    const int nob = (n->P + CN_OUT_PX - 1) / CN_OUT_PX;
    k_wgrad_out<<<nob, CN_NT, 0, s>>>(n->h[L], n->dz_out, n->cin[L], n->Nx, n->Ny, n->P, n->part);
    NSE_CUDA_TRY(cudaGetLastError());
    NSE_CUDA_TRY(fold(L, nob, 9 * n->cin[L], 1));
    int cur = 0;
    k_dgrad_out<<<grid_of((long long)n->P * (H / 8)), CN_NT, 9 * H * sizeof(float), s>>>(n->dz_out, n->wbf[L], H, n->z[L - 1], n->Nx, n->Ny,
                                                                                      n->P, n->dz[cur], n->dzb[cur]);
    NSE_CUDA_TRY(cudaGetLastError());
    const int nwb = wgrad_blocks(n);
    for (int l = L - 1; l >= 0; --l) {
        const int nk = l == 0 ? 48 : 9 * n->cin[l];
        WgradParams wp{n->h[l], n->dz[cur], n->part, n->Nx, n->Ny, n->P, nk};
        if (wgrad(wp, l == 0, H, nwb, false, s)) return -1;
        NSE_CUDA_TRY(fold(l, nwb, nk, H));
        if (l == 0) break;
        ConvParams p{};
        p.h = n->dzb[cur]; p.wt = n->wtbf[l]; p.zprev = n->z[l - 1]; p.z = n->dz[cur ^ 1]; p.hn = n->dzb[cur ^ 1]; p.err = n->err;
        p.Nx = n->Nx; p.Ny = n->Ny; p.P = n->P; p.N = n->cin[l]; p.ldw = 9 * n->npad[l];
        if (conv<CV_DGRAD>(p, n->npad[l], n->sms, false, s)) return -1;
        cur ^= 1;
    }
    return 0;
}

static int cnn_adamw(Cnn* n, float lr, float wd, cudaStream_t s) {
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    n->step += 1;
    const float bc1 = 1.f - powf(b1, (float)n->step), bc2 = 1.f - powf(b2, (float)n->step);
    AllLayers all;
    int most = 0;
    for (int l = 0; l < CN_LAYERS; ++l) {
        all.l[l] = layer_params(n, l);
        most = std::max(most, n->npad[l] * n->K[l]);
    }
    k_adamw<<<dim3(grid_of(most), CN_LAYERS), CN_NT, 0, s>>>(all, n->err, lr, b1, b2, eps, wd, bc1, bc2);
    NSE_CUDA_TRY(cudaGetLastError());
    return 0;
}

unsigned cnn_settings(const Cnn* n) { return n->settings; }
int* cnn_wait_flag(Cnn* n) { return n->err; }
bool cnn_matches(const Cnn* n, int Nx, int Ny) { return n && n->Nx == Nx && n->Ny == Ny; }

void cnn_free(Cnn* n) {
    if (!n) return;
    for (int l = 0; l < CN_LAYERS; ++l) {
        cudaFree(n->w32[l]); cudaFree(n->gw[l]);          // each with its bias behind it
        cudaFree(n->mw[l]); cudaFree(n->vw[l]); cudaFree(n->mb[l]); cudaFree(n->vb[l]);
        cudaFree(n->wbf[l]); cudaFree(n->wtbf[l]); cudaFree(n->h[l]); cudaFree(n->z[l]);
    }
    for (int k = 0; k < 2; ++k) { cudaFree(n->dz[k]); cudaFree(n->dzb[k]); }
    cudaFree(n->dz_out); cudaFree(n->part); cudaFree(n->lpart);
    cudaFree(n->loss); cudaFree(n->y); cudaFree(n->idx);
    delete n;
}

static int cnn_create(int Nx, int Ny, int hidden, int max_batch, const double* y_host, Cnn** out) {
    *out = nullptr;
    if (Nx < 4 || Ny < 5 || hidden < 16 || hidden > 64 || hidden % 16 != 0 || max_batch < 1 || !y_host) {
        set_error("nse2d_cnn_create: Nx >= 4, Ny >= 5, hidden a multiple of 16 in [16, 64], max_batch >= 1, y given");
        return -1;
    }
    if ((long long)max_batch * Nx * Ny > (1ll << 30)) { set_error("nse2d_cnn_create: batch too large"); return -1; }
    if (tc_gemm_setup()) return -1;
    Cnn* n = new Cnn();
    n->Nx = Nx; n->Ny = Ny; n->nxy = Nx * Ny; n->hidden = hidden; n->max_batch = max_batch;
    set_batch(n, max_batch);
    const int Pmax = n->Ppad;
    const int ch[CN_LAYERS + 1] = {CN_CIN, hidden, hidden, hidden, 1};
    for (int l = 0; l < CN_LAYERS; ++l) {
        n->cin[l] = (l == 0) ? CN_CIN : round_up(ch[l], 16);
        n->cout[l] = ch[l + 1];
        n->npad[l] = round_up(ch[l + 1], 16);
        n->K[l] = round_up(9 * n->cin[l], 64);
    }
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int H = n->npad[0];
    n->sms = sms > 0 ? sms : 148;
    n->wg_blocks = 2 * n->sms;                       // resident CTAs of k_wgrad
    auto fail = [&]() { cnn_free(n); return -1; };
    for (int l = 0; l < CN_LAYERS; ++l) {
        const size_t nw = (size_t)n->npad[l] * n->K[l];
        // weights and biases, and their gradients, in one piece each: one copy takes a layer to the host
        if (cn_alloc(&n->w32[l], nw + n->npad[l]) || cn_alloc(&n->gw[l], nw + n->npad[l]) || cn_alloc(&n->mw[l], nw) || cn_alloc(&n->vw[l], nw) ||
            cn_alloc(&n->mb[l], n->npad[l]) || cn_alloc(&n->vb[l], n->npad[l]) || cn_alloc(&n->wbf[l], nw) ||
            cn_alloc(&n->h[l], (size_t)Pmax * (l == 0 ? CN_C0 : n->cin[l])) ||
            cn_alloc(&n->z[l], (size_t)Pmax * (l == CN_LAYERS - 1 ? 1 : n->npad[l])))
            return fail();
        n->b32[l] = n->w32[l] + nw;
        n->gb[l] = n->gw[l] + nw;
        if (l >= 1 && l < CN_LAYERS - 1 && cn_alloc(&n->wtbf[l], (size_t)n->cin[l] * 9 * n->npad[l])) return fail();
    }
    for (int k = 0; k < 2; ++k)
        if (cn_alloc(&n->dz[k], (size_t)Pmax * H) || cn_alloc(&n->dzb[k], (size_t)Pmax * H)) return fail();
    const size_t npart = std::max((size_t)wgrad_blocks(n) * (9 * H + 1) * H, (size_t)((Pmax + CN_OUT_PX - 1) / CN_OUT_PX) * (9 * H + 1));
    if (cn_alloc(&n->dz_out, Pmax) || cn_alloc(&n->part, npart) || cn_alloc(&n->lpart, (size_t)(Pmax + CN_NT - 1) / CN_NT) ||
        cn_alloc(&n->loss, 2) || cn_alloc(&n->y, Ny) || cn_alloc(&n->idx, max_batch))
        return fail();
    n->err = reinterpret_cast<int*>(n->loss + 1);                  // read with the loss
    if (cudaMemcpy(n->y, y_host, sizeof(double) * Ny, cudaMemcpyHostToDevice) != cudaSuccess) {
        set_error("nse2d_cnn_create: y upload");
        return fail();
    }
    {
        ConvParams p{};
        bool bad = false;
        p.N = H;
        bad |= conv<CV_FWD>(p, H, 0, true, 0) || conv<CV_DGRAD>(p, H, 0, true, 0);
        p.N = n->npad[CN_LAYERS - 1];
        bad |= conv<CV_OUT>(p, H, 0, true, 0) != 0;
        bad |= wgrad(WgradParams{}, true, H, 0, true, 0) || wgrad(WgradParams{}, false, H, 0, true, 0);
        if (bad) return fail();
    }
    set_batch(n, 1);
    *out = n;
    return 0;
}

}  // namespace nse2d

using namespace nse2d;

extern "C" {

int nse2d_gemm_bf16(const void* A, const void* B, const float* bias, float* Cf, void* Cb, int M, int N, int K, int ldc,
                    int relu, cudaStream_t s) {
    if (tc_gemm_setup()) return -1;
    void* e = nullptr;
    NSE_CUDA_TRY(cudaGetSymbolAddress(&e, g_tc_err));
    NSE_CUDA_TRY(cudaMemsetAsync(e, 0, sizeof(int), s));
    TcGemmParams p{};
    p.A = static_cast<const __nv_bfloat16*>(A);
    p.B = static_cast<const __nv_bfloat16*>(B);
    p.bias = bias;
    p.Cf = Cf;
    p.Cb = static_cast<__nv_bfloat16*>(Cb);
    p.err = static_cast<int*>(e);
    p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.relu = relu ? 1 : 0;
    if (tc_gemm_launch(p, s)) return -1;
    int h = 0;
    NSE_CUDA_TRY(cudaMemcpyAsync(&h, e, sizeof(int), cudaMemcpyDeviceToHost, s));
    NSE_CUDA_TRY(cudaStreamSynchronize(s));
    if (h) { set_error("tensor-core GEMM: an mbarrier wait ran out"); return -1; }
    return 0;
}

int nse2d_box_filter(const double* fine, int Nxf, int Nyf, double* coarse, int Nxc, int Nyc, cudaStream_t s) {
    if (!fine || !coarse || Nxc <= 0 || Nyc < 2 || Nxf % Nxc != 0 || (Nyf - 1) % (Nyc - 1) != 0) {
        set_error("nse2d_box_filter: Nxf must be a multiple of Nxc and Nyf - 1 of Nyc - 1");
        return -1;
    }
    k_box_filter<<<grid_of((long long)Nxc * Nyc), CN_NT, 0, s>>>(fine, Nxf, Nyf, coarse, Nxc, Nyc);
    NSE_CUDA_TRY(cudaGetLastError());
    return 0;
}

int nse2d_cnn_create(int Nx, int Ny, int hidden, int max_batch, const double* y, nse2d_cnn** out) {
    if (!out) { set_error("nse2d_cnn_create: null output"); return -1; }
    *out = nullptr;
    Cnn* n = nullptr;
    if (cnn_create(Nx, Ny, hidden, max_batch, y, &n)) return -1;
    *out = new nse2d_cnn{n};
    return 0;
}

int nse2d_cnn_destroy(nse2d_cnn* c) {
    if (!c) return 0;
    cnn_free(c->n);
    delete c;
    return 0;
}

int nse2d_cnn_layer_shape(nse2d_cnn* c, int layer, int* cin, int* cout) {
    if (!c || layer < 0 || layer >= CN_LAYERS) { set_error("nse2d_cnn_layer_shape: bad layer"); return -1; }
    if (cin) *cin = layer == 0 ? CN_CIN : c->n->cout[layer - 1];
    if (cout) *cout = c->n->cout[layer];
    return 0;
}

int nse2d_cnn_set_params(nse2d_cnn* c, int layer, const float* w, const float* b) {
    if (!c || layer < 0 || layer >= CN_LAYERS || !w || !b) { set_error("nse2d_cnn_set_params: bad arguments"); return -1; }
    Cnn* n = c->n;
    const int ci = layer == 0 ? CN_CIN : n->cout[layer - 1], co = n->cout[layer], K = n->K[layer], np = n->npad[layer];
    std::vector<float> wp((size_t)np * K, 0.f), bp(np, 0.f);
    for (int o = 0; o < co; ++o) {
        for (int tap = 0; tap < 9; ++tap)
            for (int ch = 0; ch < ci; ++ch) wp[(size_t)o * K + tap * n->cin[layer] + ch] = w[((size_t)o * 9 + tap) * ci + ch];
        bp[o] = b[o];
    }
    NSE_CUDA_TRY(cudaMemcpy(n->w32[layer], wp.data(), wp.size() * 4, cudaMemcpyHostToDevice));
    NSE_CUDA_TRY(cudaMemcpy(n->b32[layer], bp.data(), bp.size() * 4, cudaMemcpyHostToDevice));
    NSE_CUDA_TRY(cudaMemset(n->mw[layer], 0, wp.size() * 4));
    NSE_CUDA_TRY(cudaMemset(n->vw[layer], 0, wp.size() * 4));
    NSE_CUDA_TRY(cudaMemset(n->mb[layer], 0, bp.size() * 4));
    NSE_CUDA_TRY(cudaMemset(n->vb[layer], 0, bp.size() * 4));
    n->step = 0;
    if (export_layer(n, layer, 0)) return -1;
    NSE_CUDA_TRY(cudaDeviceSynchronize());
    return 0;
}

// dw: a layer's weights [npad][K] and, behind them, its biases
static int get_layer(Cnn* n, int layer, const float* dw, float* w, float* b) {
    const int ci = layer == 0 ? CN_CIN : n->cout[layer - 1], co = n->cout[layer], K = n->K[layer], np = n->npad[layer];
    std::vector<float> wp((size_t)np * (K + 1));
    NSE_CUDA_TRY(cudaDeviceSynchronize());
    NSE_CUDA_TRY(cudaMemcpy(wp.data(), dw, wp.size() * 4, cudaMemcpyDeviceToHost));
    for (int o = 0; o < co; ++o) {
        if (w)
            for (int tap = 0; tap < 9; ++tap)
                for (int ch = 0; ch < ci; ++ch) w[((size_t)o * 9 + tap) * ci + ch] = wp[(size_t)o * K + tap * n->cin[layer] + ch];
        if (b) b[o] = wp[(size_t)np * K + o];
    }
    return 0;
}

int nse2d_cnn_get_params(nse2d_cnn* c, int layer, float* w, float* b) {
    if (!c || layer < 0 || layer >= CN_LAYERS) { set_error("nse2d_cnn_get_params: bad layer"); return -1; }
    return get_layer(c->n, layer, c->n->w32[layer], w, b);
}

int nse2d_cnn_get_grads(nse2d_cnn* c, int layer, float* w, float* b) {
    if (!c || layer < 0 || layer >= CN_LAYERS) { set_error("nse2d_cnn_get_grads: bad layer"); return -1; }
    return get_layer(c->n, layer, c->n->gw[layer], w, b);
}

int nse2d_cnn_set_scales(nse2d_cnn* c, const double* in_scales, double tau_scale) {
    if (!c || !in_scales || !(tau_scale > 0)) { set_error("nse2d_cnn_set_scales: bad arguments"); return -1; }
    for (int k = 0; k < CN_CIN - 1; ++k) {
        if (!(in_scales[k] > 0)) { set_error("nse2d_cnn_set_scales: scales must be > 0"); return -1; }
        c->n->in_scale[k] = in_scales[k];
    }
    c->n->out_tau = tau_scale;
    c->n->settings += 1;
    return 0;
}

int nse2d_cnn_set_application(nse2d_cnn* c, int wall_rows, double gain, int row_mean) {
    if (!c || wall_rows < 1 || 2 * wall_rows >= c->n->Ny - 1 || !(gain >= 0.0)) {
        set_error("nse2d_cnn_set_application: wall_rows in [1, (Ny - 1) / 2), gain >= 0");
        return -1;
    }
    c->n->wall_rows = wall_rows;
    c->n->gain = gain;
    c->n->row_mean = row_mean != 0;
    c->n->settings += 1;
    return 0;
}

int nse2d_set_closure(nse2d_ctx* ctx, nse2d_cnn* net, int every_stage) {
    if (!ctx || !ctx->c) { set_error("nse2d_set_closure: null context"); return -1; }
    Context* c = ctx->c;
    if (c->run_exec) { cudaGraphExecDestroy(c->run_exec); c->run_exec = nullptr; }
    if (c->graph_exec) { cudaGraphExecDestroy(c->graph_exec); c->graph_exec = nullptr; }
    c->closure_changes += 1;
    if (!net) { c->closure_net = nullptr; return 0; }
    if (!cnn_matches(net->n, c->Nx, c->Ny)) {
        set_error("nse2d_set_closure: the model is for %dx%d, the context is %dx%d", net->n->Nx, net->n->Ny, c->Nx, c->Ny);
        return -1;
    }
    if (c->prec32) { set_error("nse2d_set_closure: the closure runs with precision 64"); return -1; }
    if (!c->closure_tau) {
        NSE_CUDA_TRY(cudaMalloc((void**)&c->closure_tau, c->N * sizeof(double)));
        NSE_CUDA_TRY(cudaMemset(c->closure_tau, 0, c->N * sizeof(double)));
    }
    c->closure_net = net->n;
    c->closure_every_stage = every_stage != 0;
    return 0;
}

int nse2d_cnn_forward(nse2d_cnn* c, const double* w, const double* psi, const double* u, const double* v, double* tau,
                      cudaStream_t s) {
    if (!c || !w || !psi || !u || !v || !tau) { set_error("nse2d_cnn_forward: null argument"); return -1; }
    return cnn_forward(c->n, w, psi, u, v, tau, s);
}

static int batch_setup(Cnn* n, const int* idx, int nb, cudaStream_t s) {
    if (!idx || nb < 1 || nb > n->max_batch) { set_error("nse2d_cnn: batch of %d (1..%d)", nb, n->max_batch); return -1; }
    for (int b = 0; b < nb; ++b)
        if (idx[b] < 0) { set_error("nse2d_cnn: negative sample index"); return -1; }
    set_batch(n, nb);
    NSE_CUDA_TRY(cudaMemcpyAsync(n->idx, idx, sizeof(int) * nb, cudaMemcpyHostToDevice, s));
    return 0;
}

// The forward and backward pass of a batch, without waiting for them.
static int enqueue_gradients(nse2d_cnn* c, const double* w, const double* psi, const double* u, const double* v, const double* tau,
                             const int* idx, int nb, cudaStream_t s) {
    if (!c || !w || !psi || !u || !v || !tau) { set_error("nse2d_cnn_gradients: null argument"); return -1; }
    Cnn* n = c->n;
    if (batch_setup(n, idx, nb, s)) return -1;
    const int rc = (cnn_forward_batch(n, pack_src(n, w, psi, u, v), nullptr, true, nullptr, s) || cnn_backward(n, tau, s)) ? -1 : 0;
    // slot 0 back to sample 0 for inference
    NSE_CUDA_TRY(cudaMemsetAsync(n->idx, 0, sizeof(int), s));
    return rc;
}
// the loss and the error flag, once the stream has come to them. A wait that timed out, in this call or in a forward
// pass since the last one, is reported once: the flag is then cleared
static int finish_gradients(Cnn* n, const char* who, float* loss, cudaStream_t s) {
    struct { float loss; int err; } r{};
    static_assert(sizeof(r) == 8, "the flag lies behind the loss");
    NSE_CUDA_TRY(cudaMemcpyAsync(&r, n->loss, sizeof(r), cudaMemcpyDeviceToHost, s));
    NSE_CUDA_TRY(cudaStreamSynchronize(s));
    if (loss) *loss = r.loss;
    if (!r.err) return 0;
    NSE_CUDA_TRY(cudaMemsetAsync(n->err, 0, sizeof(int), s));
    NSE_CUDA_TRY(cudaStreamSynchronize(s));
    set_error("%s: a tensor-core wait ran out", who);
    return -1;
}

int nse2d_cnn_gradients(nse2d_cnn* c, const double* w, const double* psi, const double* u, const double* v,
                        const double* tau, const int* idx, int nb, float* loss, cudaStream_t s) {
    const int rc = enqueue_gradients(c, w, psi, u, v, tau, idx, nb, s);
    if (rc) {
        cudaStreamSynchronize(s);
        return -1;
    }
    return finish_gradients(c->n, "nse2d_cnn_gradients", loss, s);
}

int nse2d_cnn_train_step(nse2d_cnn* c, const double* w, const double* psi, const double* u, const double* v,
                         const double* tau, const int* idx, int nb, float lr, float weight_decay, float* loss,
                         cudaStream_t s) {
    if (enqueue_gradients(c, w, psi, u, v, tau, idx, nb, s)) {
        cudaStreamSynchronize(s);
        return -1;
    }
    if (cnn_adamw(c->n, lr, weight_decay, s)) return -1;
    if (finish_gradients(c->n, "nse2d_cnn_train_step", loss, s)) {
        c->n->step -= 1;                          // no update was made
        return -1;
    }
    return 0;
}

}  // extern "C"
