// The closure model's 3x3 convolutions on the 5th-generation tensor cores (tcgen05), BF16 operands with FP32
// accumulate, and the weight gradients; written for this project.
//
// k_conv<C, MODE>: 128 consecutive pixels x N output channels per CTA of 8 warps, K = 9 C (tap-major). The
// taps are gathered straight into the MMA's core-matrix layout by 16-byte cp.async (8 channels of one tap of
// one pixel; zero-filled beyond the walls), so there is no im2col matrix in memory: that one was written and
// read back at 9 times the size of the layer's input. The whole K of a tile is staged at once and the
// accumulator in TMEM takes the K steps in order, so the sums are those of a blocked GEMM over the same K.
// The epilogue crosses shared memory, so that the pre-activations, the next layer's input and (backward) the
// gradients leave as whole 16-byte chunks of consecutive channels; one thread per row storing its own
// channels 4 bytes at a time was most of the old GEMM's time. Two to three CTAs per SM overlap the gather of
// one with the MMAs and the epilogue of another; what bounds it is latency, of the gather (9 reads of the input
// from L1/L2) and of the epilogue, with 16 warps per SM. A convolution 32 -> 32 of 264192 pixels (eight 256x129
// fields): im2col + GEMM 268 us, now 57 (66 with 4 warps per CTA); of one field 47 us, now 13.
//
// MODE CV_FWD: z = acc + bias (FP32, stored when z is given) and GELU(z) in BF16, the next layer's input.
// MODE CV_OUT: the output layer, of whose N = 16 padded channels only channel 0 exists: z [P], tau.
// MODE CV_DGRAD: the gradient of the layer's input as a convolution of dZ with the flipped taps (K = 9 npad,
// N = cin), times GELU' of the layer below's pre-activation: dZ of that layer in FP32 and BF16.
// C = 8 stands for the input layer: 5 channels, padded to one 16-byte load per tap and packed to K = 45 (48).
//
// k_wgrad<C, N, TG>: dW[n][k] = sum_p dZ[p][n] A[p][k], a contraction over the pixels, on the tensor cores
// through mma.sync (both operands are stored pixel-major and transposed on the way by ldmatrix; the
// contraction is bound by the gather of A, not by the MMA rate). dZ stays FP32: it is split into three BF16
// terms whose sum is its 24-bit significand, so every product is exact, and the sums of each 64 pixels are
// added to FP32 accumulators by ordinary additions. Per-CTA partials are folded in a fixed order. Hidden layer of
// 32 channels, 264192 pixels: im2col, CUDA-core products and a serial fold 975 us, now 69 and 9 for the fold.
#pragma once
#include "tc_gemm.cuh"

namespace nse2d {

enum { CV_FWD, CV_OUT, CV_DGRAD };
constexpr int CV_NT = 256;                 // threads of a convolution's CTA

struct ConvParams {
    const __nv_bfloat16* h;      // [P][C]
    const __nv_bfloat16* W;      // [N][ldw]
    const float* bias;           // [N]
    const float* zprev;          // CV_DGRAD: [P][N]
    float* z;                    // CV_FWD: [P][N] or null; CV_OUT: [P] or null; CV_DGRAD: dZ [P][N]
    __nv_bfloat16* hn;           // [P][N]
    double* tau;                 // CV_OUT: [P] or null
    int* err;
    int Nx, Ny, P, N, ldw;
    int wall_rows;
    double ts;                   // tau = ts z away from the walls
};

template <int C> __host__ __device__ constexpr int cv_nch() { return C == 8 ? 6 : 9 * C / 8; }   // 16-byte chunks of K
template <int C> __host__ __device__ constexpr size_t cv_smem_bytes(int N) {
    const size_t ab = (size_t)(128 + N) * cv_nch<C>() * 16, st = (size_t)128 * (N + 1) * 4;
    return (ab > st ? ab : st) + 128;
}

// 16 bytes to shared memory, zeros when !ok (the address is then not read)
__device__ __forceinline__ void cv_cp16(uint32_t s, const void* g, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(g), "r"(ok ? 16 : 0) : "memory");
}

// a pixel of the batch: its field's first pixel, row and column
struct CvPix {
    int base, j, i;
    bool in;
};
__device__ __forceinline__ CvPix cv_pix(int p, int P, int Nx, int Ny) {
    CvPix q;
    q.in = p < P;
    const int nxy = Nx * Ny, b = p / nxy, r = p - b * nxy;
    q.base = b * nxy;
    q.j = r / Nx;
    q.i = r - q.j * Nx;
    return q;
}
// the pixel (j + dy, i + dx) of the same field (x periodic); false beyond the walls
__device__ __forceinline__ bool cv_tap(const CvPix& q, int dy, int dx, int Nx, int Ny, int& src) {
    const int jj = q.j + dy;
    int ii = q.i + dx;
    ii = ii < 0 ? ii + Nx : (ii >= Nx ? ii - Nx : ii);
    src = q.base + jj * Nx + ii;
    return q.in && jj >= 0 && jj < Ny;
}

// The packed K = 45 (48) values of one pixel of the input layer: 5 of the 8 channels of every tap.
__device__ __forceinline__ void cv_gather5(const __nv_bfloat16* h, const CvPix& q, int Nx, int Ny, unsigned short (&k)[48]) {
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
        int src;
        const bool ok = cv_tap(q, tap / 3 - 1, tap % 3 - 1, Nx, Ny, src);
        uint4 v = make_uint4(0, 0, 0, 0);
        if (ok) v = *reinterpret_cast<const uint4*>(h + (size_t)src * 8);
        k[tap * 5 + 0] = (unsigned short)(v.x & 0xffffu); k[tap * 5 + 1] = (unsigned short)(v.x >> 16);
        k[tap * 5 + 2] = (unsigned short)(v.y & 0xffffu); k[tap * 5 + 3] = (unsigned short)(v.y >> 16);
        k[tap * 5 + 4] = (unsigned short)(v.z & 0xffffu);
    }
    k[45] = k[46] = k[47] = 0;
}
__device__ __forceinline__ uint4 cv_chunk(const unsigned short* k) {
    return make_uint4(k[0] | ((uint32_t)k[1] << 16), k[2] | ((uint32_t)k[3] << 16), k[4] | ((uint32_t)k[5] << 16), k[6] | ((uint32_t)k[7] << 16));
}
__device__ __forceinline__ uint32_t cv_pack2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}

template <int C, int MODE>
static __global__ void __launch_bounds__(CV_NT) k_conv(ConvParams p) {
    extern __shared__ __align__(16) unsigned char cv_smem[];
    __shared__ __align__(8) uint64_t mma_bar;
    __shared__ uint32_t tmem_base;
    constexpr int NCH = cv_nch<C>();
    unsigned char* sm = cv_smem + ((128u - (tg_smem_u32(cv_smem) & 127u)) & 127u);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * TG_BM;
    const uint32_t sA = tg_smem_u32(sm), sB = sA + 128 * NCH * 16;
    const uint32_t ncols = p.N <= 32 ? 32u : 64u;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tg_smem_u32(&tmem_base)), "r"(ncols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        tg_bar_init(&mma_bar);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    // core matrices of 8 rows x 16 bytes, [row group][k chunk]
    for (int e = tid; e < p.N * NCH; e += CV_NT) {
        const int n = e / NCH, kc = e - n * NCH;
        tg_cp16(sB + (uint32_t)((((n >> 3) * NCH + kc) << 7) + ((n & 7) << 4)), p.W + (size_t)n * p.ldw + kc * 8);
    }
    if constexpr (C == 8) {
        if (tid < 128) {
            unsigned short k[48];
            cv_gather5(p.h, cv_pix(m0 + tid, p.P, p.Nx, p.Ny), p.Nx, p.Ny, k);
#pragma unroll
            for (int kc = 0; kc < NCH; ++kc)
                *reinterpret_cast<uint4*>(sm + ((((tid >> 3) * NCH + kc) << 7) + ((tid & 7) << 4))) = cv_chunk(k + 8 * kc);
        }
    } else {
        constexpr int C8 = C / 8, IT = 128 * C8 / CV_NT;           // chunks of a tap per thread
        static_assert(128 * C8 % CV_NT == 0, "whole chunks");
        CvPix q[IT];
#pragma unroll
        for (int it = 0; it < IT; ++it) q[it] = cv_pix(m0 + (tid + CV_NT * it) / C8, p.P, p.Nx, p.Ny);
#pragma unroll
        for (int tap = 0; tap < 9; ++tap) {
            const int dy = (MODE == CV_DGRAD) ? 1 - tap / 3 : tap / 3 - 1, dx = (MODE == CV_DGRAD) ? 1 - tap % 3 : tap % 3 - 1;
#pragma unroll
            for (int it = 0; it < IT; ++it) {
                const int e = tid + CV_NT * it, row = e / C8, ch = e - row * C8;
                int src;
                const bool ok = cv_tap(q[it], dy, dx, p.Nx, p.Ny, src);
                cv_cp16(sA + (uint32_t)((((row >> 3) * NCH + tap * C8 + ch) << 7) + ((row & 7) << 4)), p.h + (ok ? (size_t)src * C + ch * 8 : 0), ok);
            }
        }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");        // copies visible to the tensor core
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_base;
    if (tid == 0) {
        const uint32_t idesc = tg_idesc(p.N);
#pragma unroll 1
        for (int kk = 0; kk < NCH / 2; ++kk) {
            const uint64_t da = tg_desc(sA + kk * 256, 128, NCH * 128);
            const uint64_t db = tg_desc(sB + kk * 256, 128, NCH * 128);
            asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                         " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                         ::"r"(tmem), "l"(da), "l"(db), "r"(idesc), "r"(kk > 0 ? 1u : 0u) : "memory");
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(tg_smem_u32(&mma_bar)) : "memory");
    }
    if (!tg_bar_wait(&mma_bar, 0)) {
        atomicOr(p.err, 1);
        tg_bar_wait(&mma_bar, 0);
    }
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    float* st = reinterpret_cast<float*>(sm);                              // [128][N + 1]: the operands are read
    const int ld = p.N + 1;
    // warps w and w + 4 read the TMEM lanes 32 (w mod 4) .., every other 16 columns each
    for (int c0 = (warp >> 2) * 16; c0 < (MODE == CV_OUT ? 16 : p.N); c0 += 32) {
        uint32_t v[16];
        const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0;
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                       "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                     : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        const int row = (warp & 3) * 32 + lane;
        if constexpr (MODE == CV_OUT) {
            const int px = m0 + row;
            if (px < p.P) {
                const float z = __uint_as_float(v[0]) + p.bias[0];
                if (p.z) p.z[px] = z;
                if (p.tau) {
                    const int j = (px / p.Nx) % p.Ny;
                    p.tau[px] = (j < p.wall_rows || j >= p.Ny - p.wall_rows) ? 0.0 : p.ts * (double)z;
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) st[row * ld + c0 + i] = __uint_as_float(v[i]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(ncols) : "memory");
    if constexpr (MODE != CV_OUT) {
        const int nq = p.N >> 2;
        for (int e = tid; e < 128 * nq; e += CV_NT) {
            const int row = e / nq, c = (e - row * nq) * 4, px = m0 + row;
            if (px >= p.P) break;                                          // e and with it the row only grow
            const size_t o = (size_t)px * p.N + c;
            float a[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = st[row * ld + c + i];
            if constexpr (MODE == CV_FWD) {
                const float4 b = __ldg(reinterpret_cast<const float4*>(p.bias + c));
                a[0] += b.x; a[1] += b.y; a[2] += b.z; a[3] += b.w;
                if (p.z) *reinterpret_cast<float4*>(p.z + o) = make_float4(a[0], a[1], a[2], a[3]);
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = tg_gelu(a[i]);
            } else {
                const float4 zp = __ldg(reinterpret_cast<const float4*>(p.zprev + o));
                a[0] *= tg_gelu_grad(zp.x); a[1] *= tg_gelu_grad(zp.y); a[2] *= tg_gelu_grad(zp.z); a[3] *= tg_gelu_grad(zp.w);
                *reinterpret_cast<float4*>(p.z + o) = make_float4(a[0], a[1], a[2], a[3]);
            }
            if (p.hn) *reinterpret_cast<uint2*>(p.hn + o) = make_uint2(cv_pack2(a[0], a[1]), cv_pack2(a[2], a[3]));
        }
    }
}

// ---- weight gradients ----
constexpr int WG_NT = 192, WG_PX = 64;      // threads (6 warps) and pixels of a tile

struct WgradParams {
    const __nv_bfloat16* h;      // the layer's input [P][C]
    const float* dz;             // [P][N]
    float* part;                 // [gridDim.x][K][N] then [gridDim.x][N] (db; by blockIdx.y == 0)
    int Nx, Ny, P, K;            // K = 9 C (48 for the input layer)
};
template <int C, int TG> __host__ __device__ constexpr int wg_rows() { return C == 8 ? 48 : TG * C; }   // rows of dW^T per CTA
template <int C, int N, int TG> __host__ __device__ constexpr size_t wg_smem_bytes() {
    return (size_t)WG_PX * ((wg_rows<C, TG>() + 8) + (3 * N + 8)) * 2;
}

__device__ __forceinline__ void wg_ldsm4t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void wg_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int C, int N, int TG>
static __global__ void __launch_bounds__(WG_NT, 2) k_wgrad(WgradParams p) {
    constexpr int ROWS = wg_rows<C, TG>(), MT = ROWS / 16, MPW = (MT + 5) / 6, N8 = N / 8;
    constexpr int LDA = ROWS + 8, LDB = 3 * N + 8;                     // odd multiples of 16 bytes: conflict-free ldmatrix
    extern __shared__ __align__(16) unsigned char wg_smem[];
    __nv_bfloat16* sA = reinterpret_cast<__nv_bfloat16*>(wg_smem);     // [64][LDA]: the taps of every pixel
    __nv_bfloat16* sB = sA + WG_PX * LDA;                              // [64][LDB]: dZ as hi | mid | lo
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tap0 = blockIdx.y * TG;
    float acc[MPW][N8][4] = {};
    float4 db = make_float4(0.f, 0.f, 0.f, 0.f);                       // channels 4 (tid mod N / 4) ..: WG_NT is a multiple of N / 4
    static_assert(WG_NT % (N / 4) == 0, "a thread keeps its channels");
    // lane's row of an ldmatrix.x4.trans: matrices (pixels 0-7, 0-7, 8-15, 8-15) x (columns 0-7, 8-15, 0-7, 8-15)
    const int lpx = (lane & 7) + ((lane >> 4) << 3), lcol = ((lane >> 3) & 1) * 8;
    const int ntiles = (p.P + WG_PX - 1) / WG_PX;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int p0 = t * WG_PX;
        if constexpr (C == 8) {
            if (tid < WG_PX) {
                unsigned short k[48];
                cv_gather5(p.h, cv_pix(p0 + tid, p.P, p.Nx, p.Ny), p.Nx, p.Ny, k);
#pragma unroll
                for (int kc = 0; kc < 6; ++kc) *reinterpret_cast<uint4*>(sA + tid * LDA + kc * 8) = cv_chunk(k + 8 * kc);
            }
        } else {
            constexpr int C8 = C / 8;
            for (int e = tid; e < WG_PX * C8; e += WG_NT) {
                const int px = e / C8, ch = e - px * C8;
                const CvPix q = cv_pix(p0 + px, p.P, p.Nx, p.Ny);
#pragma unroll
                for (int g = 0; g < TG; ++g) {
                    const int tap = tap0 + g;
                    int src;
                    const bool ok = cv_tap(q, tap / 3 - 1, tap % 3 - 1, p.Nx, p.Ny, src);
                    cv_cp16(tg_smem_u32(sA + px * LDA + g * C + ch * 8), p.h + (ok ? (size_t)src * C + ch * 8 : 0), ok);
                }
            }
        }
        for (int e = tid; e < WG_PX * (N / 4); e += WG_NT) {
            const int px = e / (N / 4), c = (e % (N / 4)) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (p0 + px < p.P) v = __ldg(reinterpret_cast<const float4*>(p.dz + (size_t)(p0 + px) * N + c));
            db.x += v.x; db.y += v.y; db.z += v.z; db.w += v.w;
            float x[4] = {v.x, v.y, v.z, v.w}, y[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float hi = __bfloat162float(__float2bfloat16_rn(x[i]));
                const float r1 = x[i] - hi;                            // exact
                const float mid = __bfloat162float(__float2bfloat16_rn(r1));
                w[i] = r1 - mid;                                       // exact, at most 8 bits
                y[i] = mid;
                x[i] = hi;
            }
            __nv_bfloat16* d = sB + px * LDB + c;
            *reinterpret_cast<uint2*>(d) = make_uint2(cv_pack2(x[0], x[1]), cv_pack2(x[2], x[3]));
            *reinterpret_cast<uint2*>(d + N) = make_uint2(cv_pack2(y[0], y[1]), cv_pack2(y[2], y[3]));
            *reinterpret_cast<uint2*>(d + 2 * N) = make_uint2(cv_pack2(w[0], w[1]), cv_pack2(w[2], w[3]));
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        float s[MPW][N8][4] = {};
#pragma unroll 1
        for (int k0 = 0; k0 < WG_PX; k0 += 16) {
            uint32_t a[MPW][4];
#pragma unroll
            for (int m = 0; m < MPW; ++m)
                if (warp + 6 * m < MT) wg_ldsm4t(a[m], tg_smem_u32(sA + (k0 + lpx) * LDA + (warp + 6 * m) * 16 + lcol));
#pragma unroll
            for (int term = 2; term >= 0; --term)                      // smallest first
#pragma unroll
                for (int n = 0; n < N8; n += 2) {
                    // two n tiles: matrices (pixels 0-7, 0-7, 8-15, 8-15) x (n, n + 8, n, n + 8)
                    uint32_t b[4];
                    wg_ldsm4t(b, tg_smem_u32(sB + (k0 + lpx) * LDB + term * N + n * 8 + lcol));
#pragma unroll
                    for (int m = 0; m < MPW; ++m)
                        if (warp + 6 * m < MT) {
                            wg_mma(s[m][n], a[m], b[0], b[2]);
                            wg_mma(s[m][n + 1], a[m], b[1], b[3]);
                        }
                }
        }
#pragma unroll
        for (int m = 0; m < MPW; ++m)
#pragma unroll
            for (int n = 0; n < N8; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[m][n][i] += s[m][n][i];
        __syncthreads();                                               // the tiles are read
    }
    // accumulator (m, n): rows lane / 4 and lane / 4 + 8 of the m tile, columns 2 (lane mod 4), + 1 of the n tile
    float* out = p.part + (size_t)blockIdx.x * p.K * N;
    const int k0 = (C == 8 ? 0 : tap0 * C);
#pragma unroll
    for (int m = 0; m < MPW; ++m) {
        if (warp + 6 * m >= MT) continue;
#pragma unroll
        for (int n = 0; n < N8; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = k0 + (warp + 6 * m) * 16 + lane / 4 + 8 * h;
                *reinterpret_cast<float2*>(out + (size_t)k * N + n * 8 + 2 * (lane & 3)) = make_float2(acc[m][n][2 * h], acc[m][n][2 * h + 1]);
            }
    }
    if (blockIdx.y == 0) {
        float4* red = reinterpret_cast<float4*>(wg_smem);              // [WG_NT]
        red[tid] = db;
        __syncthreads();
        if (tid < N / 4) {
            float4 v = red[tid];
            for (int r = tid + N / 4; r < WG_NT; r += N / 4) { v.x += red[r].x; v.y += red[r].y; v.z += red[r].z; v.w += red[r].w; }
            *reinterpret_cast<float4*>(p.part + (size_t)gridDim.x * p.K * N + (size_t)blockIdx.x * N + 4 * tid) = v;
        }
    }
}

}  // namespace nse2d
