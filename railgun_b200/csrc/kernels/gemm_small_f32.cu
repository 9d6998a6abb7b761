// y[M, N] = x[M, K] W[N, K]^T in 32-bit for products of a few rows by small matrices, where launches and latencies are all
// that counts: the library call costs 15 us of host time each, this one 7, and a small model's step outside a graph is
// bound by the host.
//
// One block of 256 threads per 32 x 32 tile of y, 2 x 2 results a thread, in one order of k whatever the other rows are.  Both
// operands' rows lie whole in shared memory (K <= 512: 132 KB; pitch 4 mod 32: eight neighbouring rows' 16-byte pieces lie in
// different banks), asked for in one batch of loads, W's without a wait for the kernel before; behind one barrier one run over k.
// Few blocks run, each once, so the latency of its parts is what counts.
//
// With a norm in front and a gated activation behind it, so that a step needs fewer launches:
//   NORM   the rows are x_new = x (+ pending), the 32-bit residual, under their RMS norm: x_new / sqrt(mean(x_new^2) + eps) * norm_w.
//          The blocks of the first column write x_new, another buffer than x, which the other blocks still read.  K <= 256.
//   GATED  W = gate [N, K] | up [N, K]; a block's 32 rows of W are 16 of each, and what comes out is silu(gate) * up.
// A block makes its 32 rows once, again in every column of blocks: three to sixteen of them.  Two portions of 32 tokens beside three
// requests that decode, three layers of width 96: 31 launches to 22, 437 to some 405 us a step launched one by one.
// Measured on the GPU (this kernel against the library's): 67 rows by 96 x 512 2.5 / 3.9 us, by 256 x 96 4.6 / 6.5; 5 rows by 96 x
// 512 2.4 / 2.5; 30 by 448 x 96 7.5 / 9.5; 256 by 512 x 576 8.9 / 10.7.  With 128 threads, the operands 32 numbers of k at a time
// between two barriers: 2.6, 5.4, 2.5, 8.8 and 10.0; only with about as many blocks as SMs or more is that a little faster at
// K < 100 (256 rows by 64 x 576 2.1, now 2.3).  SiLU-mul behind the gate and up product instead of in front of the down product
// (nine blocks of 67 rows by 256 x 96, each making 8,192 numbers first): 3.3 + 10.4 us a layer, now 3.4 + 4.6.
#include "common.cuh"

#define SG_T 32
#define SG_MAX_K 512
#define SG_MAX_NORM_K 256
#define SG_THREADS 256

template <bool NORM, bool GATED, bool VEC>
__global__ void __launch_bounds__(SG_THREADS)
small_gemm_kernel(const float* __restrict__ x, int ldx, const float* __restrict__ pending, const float* __restrict__ norm_w,
                       float eps, float* __restrict__ x_new, const float* __restrict__ W, float* __restrict__ out, int ldo, int M,
                       int N, int K) {
    extern __shared__ __align__(16) float rows[];                        // x's [SG_T][pitch], then W's
    const int KP = (K + SG_T - 1) / SG_T * SG_T, pitch = KP + 4;         // 4 mod 32
    float* sw = rows + SG_T * pitch;
    const int m0 = blockIdx.y * SG_T, n0 = blockIdx.x * (GATED ? SG_T / 2 : SG_T);
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    const int lr = threadIdx.x >> 3;                                     // loads: row lr, numbers k_first + 32 i .. + 3
    const int k_first = (threadIdx.x & 7) * 4;
    const int wn = n0 + (GATED ? lr & (SG_T / 2 - 1) : lr);               // W: gate's row, or up's N further on
    const bool xrow = m0 + lr < M, wrow = wn < N;
    auto load = [&](const float* p, int k) {                             // numbers k .. k + 3 of a row, zeros behind K
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (VEC) {
            if (k < K) v = *reinterpret_cast<const float4*>(p + k);
        } else {
            if (k < K) v.x = p[k];
            if (k + 1 < K) v.y = p[k + 1];
            if (k + 2 < K) v.z = p[k + 2];
            if (k + 3 < K) v.w = p[k + 3];
        }
        return v;
    };
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float* wp = W + (size_t)(wrow ? (GATED && lr >= SG_T / 2 ? N + wn : wn) : 0) * K;
    auto fetch = [&](float* to, const float* from, bool there) {           // a row, 256 numbers of it under way at a time
        for (int k0 = k_first; k0 < KP; k0 += SG_MAX_NORM_K) {
            float4 v[SG_MAX_NORM_K / SG_T];
#pragma unroll
            for (int i = 0; i < SG_MAX_NORM_K / SG_T; ++i) {
                v[i] = zero;
                if (there && k0 + SG_T * i < KP) v[i] = load(from, k0 + SG_T * i);
            }
#pragma unroll
            for (int i = 0; i < SG_MAX_NORM_K / SG_T; ++i)
                if (k0 + SG_T * i < KP) *reinterpret_cast<float4*>(to + k0 + SG_T * i) = v[i];
        }
    };
    fetch(sw + lr * pitch, wp, wrow);
    pdl_wait();
    pdl_trigger();
    // ---- the block's rows: eight neighbouring threads a row, all its numbers under way at once
    const size_t row = (size_t)(xrow ? m0 + lr : 0);
    float* mine = rows + lr * pitch;
    if (NORM) {
        float4 v[SG_MAX_NORM_K / SG_T], p[SG_MAX_NORM_K / SG_T];
#pragma unroll
        for (int i = 0; i < SG_MAX_NORM_K / SG_T; ++i) {
            const int k = k_first + SG_T * i;
            v[i] = p[i] = zero;
            if (xrow && k < KP) {
                v[i] = load(x + row * ldx, k);
                if (pending) p[i] = load(pending + row * K, k);
            }
        }
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < SG_MAX_NORM_K / SG_T; ++i) {
            const int k = k_first + SG_T * i;
            if (k >= KP) break;
            v[i].x += p[i].x; v[i].y += p[i].y; v[i].z += p[i].z; v[i].w += p[i].w;
            if (pending && xrow && blockIdx.x == 0) {
                float* o = x_new + row * K + k;
                if (VEC) {
                    if (k < K) *reinterpret_cast<float4*>(o) = v[i];
                } else {
                    if (k < K) o[0] = v[i].x;
                    if (k + 1 < K) o[1] = v[i].y;
                    if (k + 2 < K) o[2] = v[i].z;
                    if (k + 3 < K) o[3] = v[i].w;
                }
            }
            ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
            *reinterpret_cast<float4*>(mine + k) = v[i];
        }
        ss += __shfl_xor_sync(0xffffffffu, ss, 1);
        ss += __shfl_xor_sync(0xffffffffu, ss, 2);
        ss += __shfl_xor_sync(0xffffffffu, ss, 4);
        const float inv = rsqrtf(ss / (float)K + eps);
#pragma unroll 4
        for (int k = k_first; k < KP; k += SG_T) {                         // the thread's own numbers again
            float4 v = *reinterpret_cast<const float4*>(mine + k);
            const float4 g = load(norm_w, k);
            v.x = v.x * inv * g.x; v.y = v.y * inv * g.y; v.z = v.z * inv * g.z; v.w = v.w * inv * g.w;
            *reinterpret_cast<float4*>(mine + k) = v;
        }
    } else {
        fetch(mine, x + row * ldx, xrow);
    }
    __syncthreads();                                                      // both operands are there
    float acc[2][2] = {};
    for (int k0 = 0; k0 < K; k0 += SG_T) {
        float4 part[2][2] = {};                                           // four chains of eight, then one of steps
        const float *r0 = rows + 2 * ty * pitch + k0, *r1 = r0 + pitch, *w0 = sw + tx * pitch + k0;
#pragma unroll
        for (int k = 0; k < SG_T; k += 4) {
            const float4 a0 = *reinterpret_cast<const float4*>(r0 + k), a1 = *reinterpret_cast<const float4*>(r1 + k);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const float4 b = *reinterpret_cast<const float4*>(w0 + 16 * q * pitch + k);
                part[0][q].x += a0.x * b.x; part[0][q].y += a0.y * b.y; part[0][q].z += a0.z * b.z; part[0][q].w += a0.w * b.w;
                part[1][q].x += a1.x * b.x; part[1][q].y += a1.y * b.y; part[1][q].z += a1.z * b.z; part[1][q].w += a1.w * b.w;
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int q = 0; q < 2; ++q) acc[r][q] += (part[r][q].x + part[r][q].y) + (part[r][q].z + part[r][q].w);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int m = m0 + 2 * ty + r;
        if (GATED) {
            const float gate = acc[r][0], up = acc[r][1];
            if (m < M && n0 + tx < N) out[(size_t)m * ldo + n0 + tx] = gate / (1.f + expf(-gate)) * up;
            continue;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int n = n0 + tx + 16 * q;
            if (m < M && n < N) out[(size_t)m * ldo + n] = acc[r][q];
        }
    }
}

// norm_w [K] given: x [M, K] and pending [M, K] (or null) are rows of the residual, x_new [M, K] (another buffer; not written
// without pending) receives their sum, K <= 256; null: x are the product's rows, pending null.  gated: W [2 N, K] = gate | up,
// out [M, N] = silu(gate) * up.  W contiguous; x's rows ldx apart, out's ldo.  K <= 512.
extern "C" int rg_small_gemm_f32(const float* x, int ldx, const float* pending, const float* norm_w, float eps, float* x_new, int gated,
                                 const float* W, float* out, int ldo, int M, int N, int K, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    const int mt = (M + SG_T - 1) / SG_T, cols = gated ? SG_T / 2 : SG_T;
    if (K <= 0 || K > (norm_w ? SG_MAX_NORM_K : SG_MAX_K) || ldx < K || ldo < N || mt > 65535 || (!norm_w && pending) ||
        (pending && (!x_new || x_new == x)))
        return RG_ERR_UNSUPPORTED;
    const bool vec = K % 4 == 0 && ldx % 4 == 0 &&
                     (((uintptr_t)x | (uintptr_t)W | (uintptr_t)pending | (uintptr_t)norm_w | (uintptr_t)x_new) & 15) == 0;
    const size_t smem = (size_t)2 * SG_T * ((K + SG_T - 1) / SG_T * SG_T + 4) * sizeof(float);       // up to 132 KB
#define SG_PICK(NORM, GATED) (vec ? small_gemm_kernel<NORM, GATED, true> : small_gemm_kernel<NORM, GATED, false>)
    auto kernel = norm_w ? (gated ? SG_PICK(true, true) : SG_PICK(true, false)) : (gated ? SG_PICK(false, true) : SG_PICK(false, false));
#undef SG_PICK
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    return rg_launch(kernel, dim3((N + cols - 1) / cols, mt), dim3(SG_THREADS), smem, (cudaStream_t)stream, 1, x, ldx, pending, norm_w,
                     eps, x_new, W, out, ldo, M, N, K);
}
