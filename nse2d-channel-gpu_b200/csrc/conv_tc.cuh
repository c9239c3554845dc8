// The closure model's 3x3 convolutions on the 5th-generation tensor cores (tcgen05), BF16 operands with FP32
// accumulate, and the weight gradients; written for this project.
//
// k_conv<C, MODE>: a strip of R rows of up to 128 pixels x N output channels per CTA of 8 warps, K = 9 C (tap-major).
// The strip and its halo are copied once into shared memory as planes of 8 channels, 16 bytes a pixel, so that 8
// consecutive pixels are one core matrix of the MMA's A operand wherever they begin: a tap is the same planes with
// the descriptor moved by its rows and columns, and nothing is gathered per tap (nine copies of the input in shared
// memory before that, and an im2col matrix in memory before). The accumulator of each tile of 128 positions takes
// the K steps in order in TMEM, so the sums are those of a blocked GEMM over the same K.
// The epilogue crosses shared memory, so that the pre-activations, the next layer's input and (backward) the
// gradients leave as whole 16-byte chunks of consecutive channels; one thread per row storing its own
// channels 4 bytes at a time was most of the old GEMM's time. What bounds it at 32 -> 32 channels and 264192 pixels
// (eight 256x129 fields): instructions, 54% of the issue slots, most of them the GELU (FP32 tanh) and the
// epilogue's; DRAM 10 of 34 us. im2col + GEMM 268 us, taps gathered 57 (input gradient 70), strips 34 (42, with
// two accumulators 45); of one field 47, 13 and 11.
//
// MODE CV_FWD: z = acc + bias (FP32, stored when z is given) and GELU(z) in BF16, the next layer's input.
// MODE CV_OUT: the output layer, of whose N = 16 padded channels only channel 0 exists: z [P], tau.
// MODE CV_DGRAD: the gradient of the layer's input as a convolution of dZ with the flipped taps (K = 9 npad,
// N = cin), times GELU' of the layer below's pre-activation: dZ of that layer in FP32 and BF16. An accumulator in TMEM
// truncates at every K step, so the nine taps go to two accumulators (64 channels: three), which ordinary additions join:
// in one, the sums' error against 64 bits was up to twice that of a product per tap added in FP32 (64 channels, db of a
// layer below 5.0e-7, with three 1.5e-7, per tap 2.5e-7; 32 channels 2.2e-7, 1.2e-7 and 2.3e-7).
// k_conv_in, the input layer: 5 channels, padded to one 16-byte load per tap and packed to K = 45 (48).
//
// k_wgrad<C, N, TG>: dW[n][k] = sum_p dZ[p][n] A[p][k], a contraction over the pixels, on the tensor cores
// through mma.sync (both operands are stored pixel-major and transposed on the way by ldmatrix; the
// contraction is bound by the gather of A, not by the MMA rate). dZ stays FP32: it is split into three BF16
// terms whose sum is its 24-bit significand, so every product is exact, and the sums of each 32 pixels are
// added to FP32 accumulators by ordinary additions (the MMA truncates: error of dW against 64 bits 7.4e-8, with sums of
// 64 pixels 9.9e-8, by FP32 multiply-adds 2.4e-7). The taps and dZ of the next tile are on their way while one is
// multiplied. Per-CTA partials are folded in a fixed order. Hidden layer of 32 channels, 264192 pixels: im2col,
// CUDA-core products and a serial fold 975 us; 69 and 9 for the fold without the overlap, 60 with it (tensor pipe 40%,
// 12 warps an SM by their registers); input layer 55 and 34.
#pragma once
#include "tc_gemm.cuh"

namespace nse2d {

enum { CV_FWD, CV_OUT, CV_DGRAD };
constexpr int CV_NT = 256;                 // threads of a convolution's CTA

struct ConvParams {
    const __nv_bfloat16* h;      // [P][C]
    const __nv_bfloat16* wt;     // [N][ldw]
    const float* bias;           // [N]
    const float* zprev;          // CV_DGRAD: [P][N]
    float* z;                    // CV_FWD: [P][N] or null; CV_OUT: [P] or null; CV_DGRAD: dZ [P][N]
    __nv_bfloat16* hn;           // [P][N]
    double* tau;                 // CV_OUT: [P] or null
    int* err;
    int Nx, Ny, P, N, ldw;
    int wall_rows;
    double ts;                   // tau = ts z away from the walls
    int W, R;                    // a CTA's strip: columns (at most 128) and rows
};

template <int C> __host__ __device__ constexpr int cv_nch() { return C == 8 ? 6 : 9 * C / 8; }   // 16-byte chunks of K
__host__ __device__ constexpr size_t cv_in_smem_bytes(int N) {
    const size_t ab = (size_t)(128 + N) * cv_nch<8>() * 16, st = (size_t)128 * (N + 1) * 4;
    return (ab > st ? ab : st) + 128;
}
// A strip of R rows of W pixels with its halo: positions 0 .. (R + 2) (W + 2) - 1 of rows of W + 2; an MMA tile is
// 128 consecutive positions, from the start of each row of the strip or, where those are fewer tiles, end to end.
__host__ __device__ constexpr int cv_tiles(int W, int R) {
    const int t = (R * (W + 2) - 2 + 127) / 128;
    return t < R ? t : R;
}
// bytes between the planes of 8 channels: the C / 8 chunks of neighbouring pixels go to different banks
template <int C> __host__ __device__ constexpr int cv_plane(int W, int R) {
    return ((R + 2) * (W + 2) * 16 + 127) / 128 * 128 + (C == 16 ? 64 : (C == 32 ? 32 : 16));
}
__host__ __device__ constexpr int cv_cols(int N) { return N == 48 ? 64 : N; }    // TMEM columns of an accumulator
// accumulators of a tile
template <int C, int MODE> __host__ __device__ constexpr int cv_groups() { return MODE != CV_DGRAD || C == 16 ? 1 : (C == 64 ? 3 : 2); }
template <int C> __host__ __device__ constexpr size_t cv_smem_bytes(int N, int W, int R) {
    const size_t ab = ((size_t)cv_plane<C>(W, R) * (C / 8) + 127) / 128 * 128 + (size_t)N * cv_nch<C>() * 16;
    const size_t st = (size_t)cv_tiles(W, R) * 128 * (N + 1) * 4;
    return (ab > st ? ab : st) + 128;
}

// The layers follow one another by programmatic launches: a kernel is launched when every CTA of the one before has
// come past this wait, does what needs none of its results (its accumulators in TMEM, its weights) and waits here until
// that one has ended. A kernel's accumulators are allocated before it lets the next one in, so the next never keeps
// it from them. Five steps of 256x129 with the model before every stage: 765 us without, 635 with.
__device__ __forceinline__ void cv_wait_for_last_layer() {
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
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

// Pre-activations of `rows` accumulator rows in shared memory -> the layer's outputs, 16-byte chunks of consecutive
// channels; px(row): the row's pixel, or a negative number. A thread keeps its four channels from row to row.
template <int N, int MODE, typename Px>
__device__ __forceinline__ void cv_epilogue(const ConvParams& p, const float* st, int rows, const Px& px) {
    constexpr int ld = N + 1, nq = N >> 2, step = CV_NT / nq;
    const int c = (int)threadIdx.x % nq * 4;
    if ((int)threadIdx.x >= step * nq) return;
    float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (MODE == CV_FWD) b = __ldg(reinterpret_cast<const float4*>(p.bias + c));
#pragma unroll 2
    for (int row = (int)threadIdx.x / nq; row < rows; row += step) {
        const int pix = px(row);
        if (pix < 0) continue;
        const size_t o = (size_t)pix * N + c;
        float a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = st[row * ld + c + i];
        if constexpr (MODE == CV_FWD) {
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
__device__ __forceinline__ void cv_tmem_alloc(uint32_t* base, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tg_smem_u32(base)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cv_tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cv_mma(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, bool acc) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                 ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(acc ? 1u : 0u) : "memory");
}
// After the operands of the CTA have arrived: `issue` by one thread, and everyone waits for the accumulators.
template <typename Issue>
__device__ __forceinline__ void cv_mma_all(uint64_t* bar, int* err, const Issue& issue) {
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");        // copies visible to the tensor core
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (threadIdx.x == 0) {
        issue();
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(tg_smem_u32(bar)) : "memory");
    }
    if (!tg_bar_wait(bar, 0)) {
        atomicOr(err, 1);
        tg_bar_wait(bar, 0);
    }
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}

// The input layer: 128 consecutive pixels, their nine taps gathered and packed to K = 45 (48).
template <int N>
static __global__ void __launch_bounds__(CV_NT) k_conv_in(ConvParams p) {
    extern __shared__ __align__(16) unsigned char cv_smem[];
    __shared__ __align__(8) uint64_t mma_bar;
    __shared__ uint32_t tmem_base;
    constexpr int NCH = cv_nch<8>();
    unsigned char* sm = cv_smem + ((128u - (tg_smem_u32(cv_smem) & 127u)) & 127u);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * TG_BM;
    const uint32_t sA = tg_smem_u32(sm), sB = sA + 128 * NCH * 16;
    constexpr uint32_t ncols = N <= 32 ? 32u : 64u;
    if (warp == 0) cv_tmem_alloc(&tmem_base, ncols);
    if (tid == 0) {
        tg_bar_init(&mma_bar);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    // core matrices of 8 rows x 16 bytes, [row group][k chunk]
    for (int e = tid; e < N * NCH; e += CV_NT) {
        const int n = e / NCH, kc = e - n * NCH;
        tg_cp16(sB + (uint32_t)((((n >> 3) * NCH + kc) << 7) + ((n & 7) << 4)), p.wt + (size_t)n * p.ldw + kc * 8);
    }
    __syncthreads();                                                       // TMEM is allocated
    cv_wait_for_last_layer();
    if (tid < 128) {
        unsigned short k[48];
        cv_gather5(p.h, cv_pix(m0 + tid, p.P, p.Nx, p.Ny), p.Nx, p.Ny, k);
#pragma unroll
        for (int kc = 0; kc < NCH; ++kc)
            *reinterpret_cast<uint4*>(sm + ((((tid >> 3) * NCH + kc) << 7) + ((tid & 7) << 4))) = cv_chunk(k + 8 * kc);
    }
    cv_mma_all(&mma_bar, p.err, [&]() {
        const uint32_t idesc = tg_idesc(N), tmem = tmem_base;
#pragma unroll 1
        for (int kk = 0; kk < NCH / 2; ++kk) cv_mma(tmem, tg_desc(sA + kk * 256, 128, NCH * 128), tg_desc(sB + kk * 256, 128, NCH * 128), idesc, kk > 0);
    });
    const uint32_t tmem = tmem_base;
    float* st = reinterpret_cast<float*>(sm);                              // [128][N + 1]: the operands are read
    constexpr int ld = N + 1;
    const int row = (warp & 3) * 32 + lane;
    // warps w and w + 4 read the TMEM lanes 32 (w mod 4) .., every other 16 columns each
    for (int c0 = (warp >> 2) * 16; c0 < N; c0 += 32) {
        uint32_t v[16];
        cv_tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) st[row * ld + c0 + i] = __uint_as_float(v[i]);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(ncols) : "memory");
    cv_epilogue<N, CV_FWD>(p, st, 128, [&](int r) { return m0 + r < p.P ? m0 + r : -1; });
}

template <int C, int MODE>
static __global__ void __launch_bounds__(CV_NT) k_conv(ConvParams p) {
    extern __shared__ __align__(16) unsigned char cv_smem[];
    __shared__ __align__(8) uint64_t mma_bar;
    __shared__ uint32_t tmem_base;
    constexpr int NCH = cv_nch<C>(), C8 = C / 8, N = MODE == CV_OUT ? 16 : C;   // hidden layers are as wide as their inputs
    unsigned char* sm = cv_smem + ((128u - (tg_smem_u32(cv_smem) & 127u)) & 127u);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int Nx = p.Nx, Ny = p.Ny, W = p.W, R = p.R, Wp = W + 2;
    const int T = cv_tiles(W, R), plane = cv_plane<C>(W, R);
    const bool by_row = T == R;                                            // a tile per row
    // the CTA's strip: field, first row, first column
    const int sx = (Nx + W - 1) / W, rb = (Ny + R - 1) / R;
    int u = blockIdx.x;
    const int i0 = (u % sx) * W;
    u /= sx;
    const int j0 = (u % rb) * R, base = (u / rb) * Nx * Ny;
    const uint32_t sA = tg_smem_u32(sm), sB = sA + (uint32_t)((plane * C8 + 127) / 128 * 128);
    constexpr int G = cv_groups<C, MODE>(), TPG = (9 + G - 1) / G, gcol = cv_cols(N), tcol = G * gcol;
    uint32_t ncols = 32;
    while ((int)ncols < T * tcol) ncols *= 2;
    if (warp == 0) cv_tmem_alloc(&tmem_base, ncols);
    if (tid == 0) {
        tg_bar_init(&mma_bar);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    // B: core matrices of 8 rows x 16 bytes, [row group][k chunk]
    for (int e = tid; e < N * NCH; e += CV_NT) {
        const int n = e / NCH, kc = e - n * NCH;
        tg_cp16(sB + (uint32_t)((((n >> 3) * NCH + kc) << 7) + ((n & 7) << 4)), p.wt + (size_t)n * p.ldw + kc * 8);
    }
    __syncthreads();                                                       // TMEM is allocated
    cv_wait_for_last_layer();
    // the strip and its halo, [8 channels][position]: 8 consecutive positions are a core matrix of A wherever they begin
    for (int e = tid; e < (R + 2) * Wp * C8; e += CV_NT) {
        const int pos = e / C8, ch = e - pos * C8, pr = pos / Wp, j = j0 - 1 + pr;
        int i = i0 - 1 + pos - pr * Wp;
        i = i < 0 ? i + Nx : (i >= Nx ? i - Nx : i);
        const bool ok = j >= 0 && j < Ny;
        cv_cp16(sA + (uint32_t)(ch * plane + pos * 16), p.h + (ok ? (size_t)(base + j * Nx + i) * C + ch * 8 : 0), ok);
    }
    cv_mma_all(&mma_bar, p.err, [&]() {
        const uint32_t idesc = tg_idesc(N), tmem = tmem_base;
        for (int t = 0; t < T; ++t) {
            const uint32_t a0 = sA + (uint32_t)(by_row ? t * Wp : t * 128) * 16, d = tmem + (uint32_t)(t * tcol);
#pragma unroll 1
            for (int tap = 0; tap < 9; ++tap) {
                const int ty = MODE == CV_DGRAD ? 2 - tap / 3 : tap / 3, tx = MODE == CV_DGRAD ? 2 - tap % 3 : tap % 3;
#pragma unroll
                for (int c = 0; c < C8; c += 2) {
                    const uint64_t da = tg_desc(a0 + (uint32_t)((ty * Wp + tx) * 16 + c * plane), (uint32_t)plane, 128);
                    const uint64_t db = tg_desc(sB + (uint32_t)((tap * C8 + c) << 7), 128, NCH * 128);
                    if constexpr (G == 1) cv_mma(d, da, db, idesc, tap > 0 || c > 0);
                    else cv_mma(d + (uint32_t)(tap / TPG * gcol), da, db, idesc, tap % TPG > 0 || c > 0);
                }
            }
        }
    });
    const uint32_t tmem = tmem_base;
    // the pixel of accumulator row `row` of the strip's tiles
    auto px = [&](int row) {
        const int pos = by_row ? (row & 127) : row, r = by_row ? row >> 7 : pos / Wp, c = by_row ? pos : pos - r * Wp;
        return c < W && i0 + c < Nx && r < R && j0 + r < Ny ? base + (j0 + r) * Nx + i0 + c : -1;
    };
    float* st = reinterpret_cast<float*>(sm);                              // [128 T][N + 1]: the operands are read
    constexpr int ld = N + 1;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t tlane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    if constexpr (MODE == CV_OUT) {
        for (int t = warp >> 2; t < T; t += 2) {
            uint32_t v[16];
            cv_tmem_ld16(tlane + (uint32_t)(t * tcol), v);
            const int pix = px(t * 128 + row);
            if (pix >= 0) {
                const float z = __uint_as_float(v[0]) + p.bias[0];
                if (p.z) p.z[pix] = z;
                if (p.tau) {
                    const int j = (pix / Nx) % Ny;
                    p.tau[pix] = (j < p.wall_rows || j >= Ny - p.wall_rows) ? 0.0 : p.ts * (double)z;
                }
            }
        }
    } else {
        // warps w and w + 4 read the TMEM lanes 32 (w mod 4) .., every other 16 columns each
        constexpr int nc = N >> 4;
        for (int g = warp >> 2; g < T * nc; g += 2) {
            const int t = g / nc, c0 = (g - t * nc) * 16;
            uint32_t v[16];
            cv_tmem_ld16(tlane + (uint32_t)(t * tcol + c0), v);
#pragma unroll
            for (int k = 1; k < G; ++k) {
                uint32_t u[16];
                cv_tmem_ld16(tlane + (uint32_t)(t * tcol + k * gcol + c0), u);
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) + __uint_as_float(u[i]));
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) st[(t * 128 + row) * ld + c0 + i] = __uint_as_float(v[i]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(ncols) : "memory");
    if constexpr (MODE != CV_OUT) cv_epilogue<N, MODE>(p, st, T * 128, px);
}

// ---- weight gradients ----
constexpr int WG_NT = 192, WG_PX = 64;      // threads (6 warps) and pixels of a tile

struct WgradParams {
    const __nv_bfloat16* h;      // the layer's input [P][C]
    const float* dz;             // [P][N]
    float* part;                 // [gridDim.x][K][N] then [gridDim.x][N] (db; by blockIdx.y == 0)
    int Nx, Ny, P, K;            // K = 9 C (48 for the input layer)
};
// rows of dW^T per CTA (the input layer: 9 taps of 8 channels, of which 5 exist, and 8 zero rows)
template <int C, int TG> __host__ __device__ constexpr int wg_rows() { return C == 8 ? 80 : TG * C; }
template <int C, int N, int TG> __host__ __device__ constexpr size_t wg_smem_bytes() {
    return (size_t)WG_PX * (2 * (wg_rows<C, TG>() + 8) * 2 + (3 * N + 8) * 2 + N * 4);
}

__device__ __forceinline__ void wg_ldsm4t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void wg_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// the first of a sum
__device__ __forceinline__ void wg_mma0(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};\n"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

template <int C, int N, int TG>
static __global__ void __launch_bounds__(WG_NT, 2) k_wgrad(WgradParams p) {
    constexpr int ROWS = wg_rows<C, TG>(), MT = ROWS / 16, MPW = (MT + 5) / 6, N8 = N / 8;
    constexpr int LDA = ROWS + 8, LDB = 3 * N + 8;                     // odd multiples of 16 bytes: conflict-free ldmatrix
    extern __shared__ __align__(16) unsigned char wg_smem[];
    __nv_bfloat16* sA2 = reinterpret_cast<__nv_bfloat16*>(wg_smem);    // 2 x [64][LDA]: the taps of every pixel
    __nv_bfloat16* sB = sA2 + 2 * WG_PX * LDA;                         // [64][LDB]: dZ as hi | mid | lo
    float* sZ = reinterpret_cast<float*>(sB + WG_PX * LDB);            // [64][N]: dZ of the next tile
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tap0 = blockIdx.y * TG;
    float acc[MPW][N8][4] = {};
    float4 db = make_float4(0.f, 0.f, 0.f, 0.f);                       // channels 4 (tid mod N / 4) ..: WG_NT is a multiple of N / 4
    static_assert(WG_NT % (N / 4) == 0, "a thread keeps its channels");
    // lane's row of an ldmatrix.x4.trans: matrices (pixels 0-7, 0-7, 8-15, 8-15) x (columns 0-7, 8-15, 0-7, 8-15)
    const int lpx = (lane & 7) + ((lane >> 4) << 3), lcol = ((lane >> 3) & 1) * 8;
    const int ntiles = (p.P + WG_PX - 1) / WG_PX;
    // the taps of tile t (into buffer b) and its dZ, on their way while the tile before is multiplied
    auto fetch = [&](int t, int b) {
        constexpr int C8 = C / 8;
        const int p0 = t * WG_PX;
        __nv_bfloat16* sA = sA2 + b * WG_PX * LDA;
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
        for (int e = tid; e < WG_PX * (N / 4); e += WG_NT) {
            const int px = e / (N / 4), c = (e % (N / 4)) * 4;
            const bool ok = p0 + px < p.P;
            cv_cp16(tg_smem_u32(sZ + px * N + c), p.dz + (ok ? (size_t)(p0 + px) * N + c : 0), ok);
        }
    };
    if constexpr (C == 8) {                                            // the rows that no tap fills
        for (int e = tid; e < 2 * WG_PX; e += WG_NT) *reinterpret_cast<uint4*>(sA2 + e * LDA + 72) = make_uint4(0, 0, 0, 0);
    }
    if ((int)blockIdx.x < ntiles) fetch(blockIdx.x, 0);
    for (int t = blockIdx.x, b = 0; t < ntiles; t += gridDim.x, b ^= 1) {
        const __nv_bfloat16* sA = sA2 + b * WG_PX * LDA;
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        for (int e = tid; e < WG_PX * (N / 4); e += WG_NT) {           // the chunks that this thread fetched
            const int px = e / (N / 4), c = (e % (N / 4)) * 4;
            const float4 v = *reinterpret_cast<const float4*>(sZ + px * N + c);
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
            // above the largest finite BF16 value: an infinity is its own first term, a finite value is cut there instead
            // of being rounded to one
            if (fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))) > 3.38953139e38f) {
                const float t[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (!(fabsf(t[i]) > 3.38953139e38f)) continue;     // a NaN has stayed one
                    const bool inf = fabsf(t[i]) > 3.402823466e38f;
                    x[i] = __uint_as_float(__float_as_uint(t[i]) & 0xffff0000u);
                    y[i] = inf ? 0.f : __bfloat162float(__float2bfloat16_rn(t[i] - x[i]));
                    w[i] = inf ? 0.f : t[i] - x[i] - y[i];
                }
            }
            __nv_bfloat16* d = sB + px * LDB + c;
            *reinterpret_cast<uint2*>(d) = make_uint2(cv_pack2(x[0], x[1]), cv_pack2(x[2], x[3]));
            *reinterpret_cast<uint2*>(d + N) = make_uint2(cv_pack2(y[0], y[1]), cv_pack2(y[2], y[3]));
            *reinterpret_cast<uint2*>(d + 2 * N) = make_uint2(cv_pack2(w[0], w[1]), cv_pack2(w[2], w[3]));
        }
        __syncthreads();
        if (t + (int)gridDim.x < ntiles) fetch(t + gridDim.x, b ^ 1);
#pragma unroll 1
        for (int k0 = 0; k0 < WG_PX; k0 += 32) {
            float s[MPW][N8][4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k1 = k0 + 16 * h;
                uint32_t a[MPW][4];
#pragma unroll
                for (int m = 0; m < MPW; ++m)
                    if (warp + 6 * m < MT) wg_ldsm4t(a[m], tg_smem_u32(sA + (k1 + lpx) * LDA + (warp + 6 * m) * 16 + lcol));
#pragma unroll
                for (int term = 2; term >= 0; --term)                  // smallest first
#pragma unroll
                    for (int n = 0; n < N8; n += 2) {
                        // two n tiles: matrices (pixels 0-7, 0-7, 8-15, 8-15) x (n, n + 8, n, n + 8)
                        uint32_t b[4];
                        wg_ldsm4t(b, tg_smem_u32(sB + (k1 + lpx) * LDB + term * N + n * 8 + lcol));
#pragma unroll
                        for (int m = 0; m < MPW; ++m)
                            if (warp + 6 * m < MT) {
                                if (h == 0 && term == 2) {
                                    wg_mma0(s[m][n], a[m], b[0], b[2]);
                                    wg_mma0(s[m][n + 1], a[m], b[1], b[3]);
                                } else {
                                    wg_mma(s[m][n], a[m], b[0], b[2]);
                                    wg_mma(s[m][n + 1], a[m], b[1], b[3]);
                                }
                            }
                    }
            }
#pragma unroll
            for (int m = 0; m < MPW; ++m)
                if (warp + 6 * m < MT)
#pragma unroll
                    for (int n = 0; n < N8; ++n)
#pragma unroll
                        for (int i = 0; i < 4; ++i) acc[m][n][i] += s[m][n][i];
        }
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
                int k = k0 + (warp + 6 * m) * 16 + lane / 4 + 8 * h;
                if constexpr (C == 8) {                                // 5 of the 8 channels of a tap; rows 45 .. 47 are zeros
                    const int tap = k >> 3, c = k & 7;
                    if (c >= (tap == 9 ? 3 : 5)) continue;
                    k = tap * 5 + c;
                }
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
