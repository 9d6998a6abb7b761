// y[M, N] = x[M, K] W[N, K]^T in 32-bit for products of a few rows by small matrices, where launches and latencies are all
// that counts: the library call costs 15 us of host time each, this one 7, and a small model's step outside a graph is
// bound by the host (three requests that decode beside two portions of 32 tokens, three layers of width 96:
// 13 products in 31 launches).
//
// One block of 128 threads per 32 x 32 tile of y, 2 x 4 results a thread, in one order of k whatever the other rows are.  Both
// operands are read along their rows into shared memory (pitch 36: eight neighbouring rows' 16-byte pieces lie in different
// banks), 32 numbers of k at a time, the next ones on their way in registers; W's first do not wait for the kernel before.
// Measured on the GPU (this kernel against the library's): 67 rows by 96 x 512 2.6 / 4.0 us, by 256 x 1,024 5.4 / 6.5; 5 rows
// by 96 x 512 2.5 / 2.5, by 256 x 1,024 5.1 / 3.6 (a step of 32 numbers of k is a chain of 0.5 us), 256 by 256 x 1,024 8.7 / 7.2;
// 16 rows by 512 x 256 9.6 / 6.5.  ops.py takes it where it is no slower.
#include "common.cuh"

#define SG_T 32
#define SG_P (SG_T + 4)

template <bool VEC>
__global__ void __launch_bounds__(128)
small_gemm_kernel(const float* __restrict__ x, int ldx, const float* __restrict__ W, float* __restrict__ out, int ldo, int M,
                  int N, int K) {
    __shared__ __align__(16) float sx[SG_T][SG_P], sw[SG_T][SG_P];
    const int m0 = blockIdx.y * SG_T, n0 = blockIdx.x * SG_T;
    const int ty = threadIdx.x >> 3, tx = threadIdx.x & 7;              // rows 2 ty, 2 ty + 1; columns tx + 8 q
    const int lr = threadIdx.x >> 2, lk = (threadIdx.x & 3) * 8;         // loads: row lr, numbers lk .. + 7
    const bool xrow = m0 + lr < M, wrow = n0 + lr < N;
    const float* xp = x + (size_t)(xrow ? m0 + lr : 0) * ldx + lk;
    const float* wp = W + (size_t)(wrow ? n0 + lr : 0) * K + lk;
    float4 xv[2], wv[2];
    auto fetch = [&](float4 (&v)[2], const float* p, bool row, int k0) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = k0 + lk + 4 * h;
            v[h] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!row) continue;
            const float* q = p + k0 + 4 * h;
            if (VEC) {
                if (k < K) v[h] = *reinterpret_cast<const float4*>(q);
            } else {
                if (k < K) v[h].x = q[0];
                if (k + 1 < K) v[h].y = q[1];
                if (k + 2 < K) v[h].z = q[2];
                if (k + 3 < K) v[h].w = q[3];
            }
        }
    };
    fetch(wv, wp, wrow, 0);
    pdl_wait();
    pdl_trigger();
    fetch(xv, xp, xrow, 0);
    float acc[2][4] = {};
    for (int k0 = 0; k0 < K; k0 += SG_T) {
        __syncthreads();                                                  // the numbers before have been used
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            *reinterpret_cast<float4*>(&sx[lr][lk + 4 * h]) = xv[h];
            *reinterpret_cast<float4*>(&sw[lr][lk + 4 * h]) = wv[h];
        }
        __syncthreads();
        if (k0 + SG_T < K) {
            fetch(wv, wp, wrow, k0 + SG_T);
            fetch(xv, xp, xrow, k0 + SG_T);
        }
        float4 part[2][4] = {};                                           // four chains of eight, then one of steps
#pragma unroll
        for (int k = 0; k < SG_T; k += 4) {
            const float4 a0 = *reinterpret_cast<const float4*>(&sx[2 * ty][k]), a1 = *reinterpret_cast<const float4*>(&sx[2 * ty + 1][k]);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 b = *reinterpret_cast<const float4*>(&sw[tx + 8 * q][k]);
                part[0][q].x += a0.x * b.x; part[0][q].y += a0.y * b.y; part[0][q].z += a0.z * b.z; part[0][q].w += a0.w * b.w;
                part[1][q].x += a1.x * b.x; part[1][q].y += a1.y * b.y; part[1][q].z += a1.z * b.z; part[1][q].w += a1.w * b.w;
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[r][q] += (part[r][q].x + part[r][q].y) + (part[r][q].z + part[r][q].w);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int m = m0 + 2 * ty + r;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int n = n0 + tx + 8 * q;
            if (m < M && n < N) out[(size_t)m * ldo + n] = acc[r][q];
        }
    }
}

// The same product over rows that the kernel makes itself, so that a small model's step needs fewer launches (what bounds it: the
// host's 10 us and more each):
//   SG_NORM  x_new = x (+ pending), the 32-bit residual, and its rows' RMS norm: x_new / sqrt(mean(x_new^2) + eps) * norm_w.  The
//            blocks of the first column write x_new, another buffer than x, which the other blocks still read.
//   SG_SILU  silu(gate) * up of rows [gate K | up K]
// A block makes its 32 rows once, in shared memory (K <= 256), again in every column of blocks: three to sixteen of them; its 32
// rows of W lie there too, asked for before the wait for the kernel before this one, so that behind the rows comes one run over
// k.  Few blocks run, each once, so the latency of its parts is what counts: 256 threads, a row's numbers in one batch of loads.
// Two portions of 32 tokens beside three requests that decode, three layers of width 96: 31 launches to 22, 437 to some
// 405 us a step launched one by one.  With 128 threads, four loads under way and W a piece of 32 numbers at a time the norm's
// products took 5.05 us each and SiLU-mul and 67 rows by 256 x 96 14.1; so 3.3 and 10.4, the step replayed 120 to 108.
#define SG_NORM 1
#define SG_SILU 2
#define SG_MAX_K 256
#define SG_ROWS_T 256

template <int PRO, bool VEC>
__global__ void __launch_bounds__(SG_ROWS_T)
small_gemm_rows_kernel(const float* __restrict__ x, int ldx, const float* __restrict__ pending, const float* __restrict__ norm_w,
                       float eps, float* __restrict__ x_new, const float* __restrict__ W, float* __restrict__ out, int ldo, int M,
                       int N, int K) {
    extern __shared__ __align__(16) float rows[];                        // x's [SG_T][pitch], then W's, then SiLU's factors
    const int KP = (K + SG_T - 1) / SG_T * SG_T, pitch = KP + 4;         // pitch 4 mod 32: as SG_P
    float* sw = rows + SG_T * pitch;
    const int m0 = blockIdx.y * SG_T, n0 = blockIdx.x * SG_T;
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    const int lr = threadIdx.x >> 3;                                     // loads: row lr, numbers k_first + 32 i .. + 3
    const int k_first = (threadIdx.x & 7) * 4;
    const bool xrow = m0 + lr < M, wrow = n0 + lr < N;
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
    const float* wp = W + (size_t)(wrow ? n0 + lr : 0) * K;
#pragma unroll 8
    for (int k = k_first; k < KP; k += SG_T) *reinterpret_cast<float4*>(sw + lr * pitch + k) = wrow ? load(wp, k) : zero;
    pdl_wait();
    pdl_trigger();
    // ---- the block's rows: eight neighbouring threads a row, all its numbers under way at once
    const size_t row = (size_t)(xrow ? m0 + lr : 0);
    float* mine = rows + lr * pitch;
    float4 v[SG_MAX_K / SG_T], p[SG_MAX_K / SG_T];
#pragma unroll
    for (int i = 0; i < SG_MAX_K / SG_T; ++i) {
        const int k = k_first + SG_T * i;
        v[i] = p[i] = zero;
        if (xrow && k < KP) {
            v[i] = load(x + row * ldx, k);
            if (PRO == SG_SILU) p[i] = load(x + row * ldx + K, k);
            else if (pending) p[i] = load(pending + row * K, k);
        }
    }
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < SG_MAX_K / SG_T; ++i) {
        const int k = k_first + SG_T * i;
        if (k >= KP) break;
        if (PRO == SG_NORM) {
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
        } else {
            *reinterpret_cast<float4*>(sw + SG_T * pitch + lr * pitch + k) = p[i];
        }
        *reinterpret_cast<float4*>(mine + k) = v[i];
    }
    if (PRO == SG_SILU) {
        // the thread's own numbers, by way of shared memory: written out eight times, the exponentials and divisions are some
        // 20 KB of code that a block fetches to run once
#pragma unroll 1
        for (int k = k_first; k < KP; k += SG_T) {
            float4 g = *reinterpret_cast<const float4*>(mine + k);
            const float4 u = *reinterpret_cast<const float4*>(sw + SG_T * pitch + lr * pitch + k);
            g.x = g.x / (1.f + expf(-g.x)) * u.x; g.y = g.y / (1.f + expf(-g.y)) * u.y;
            g.z = g.z / (1.f + expf(-g.z)) * u.z; g.w = g.w / (1.f + expf(-g.w)) * u.w;
            *reinterpret_cast<float4*>(mine + k) = g;
        }
    }
    if (PRO == SG_NORM) {
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
    }
    __syncthreads();                                                      // both operands are there
    float acc[2][2] = {};
    for (int k0 = 0; k0 < K; k0 += SG_T) {
        float4 part[2][2] = {};                                           // four chains of eight, then one of steps, as above
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
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int n = n0 + tx + 16 * q;
            if (m < M && n < N) out[(size_t)m * ldo + n] = acc[r][q];
        }
    }
}

// x: rows ldx apart; W [N, K] contiguous; out: rows ldo apart.
extern "C" int rg_small_gemm_f32(const float* x, int ldx, const float* W, float* out, int ldo, int M, int N, int K, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    const int mt = (M + SG_T - 1) / SG_T;
    if (K <= 0 || ldx < K || ldo < N || mt > 65535) return RG_ERR_UNSUPPORTED;
    const bool vec = K % 4 == 0 && ldx % 4 == 0 && (((uintptr_t)x | (uintptr_t)W) & 15) == 0;
    return rg_launch(vec ? small_gemm_kernel<true> : small_gemm_kernel<false>, dim3((N + SG_T - 1) / SG_T, mt), dim3(128), 0,
                     (cudaStream_t)stream, 1, x, ldx, W, out, ldo, M, N, K);
}

// silu 0: x [M, K] and pending [M, K] (or null) are rows of the residual, x_new [M, K] (another buffer; not written without
// pending) receives their sum, norm_w [K]; silu 1: x [M, 2 K] = gate | up (rows ldx apart), the others null.  K <= 256.
extern "C" int rg_small_gemm_rows_f32(const float* x, int ldx, const float* pending, const float* norm_w, float eps, float* x_new, int silu,
                                      const float* W, float* out, int ldo, int M, int N, int K, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    const int mt = (M + SG_T - 1) / SG_T;
    if (K <= 0 || K > SG_MAX_K || ldx < (silu ? 2 * K : K) || ldo < N || mt > 65535 || (!silu && !norm_w) ||
        (pending && (!x_new || x_new == x)))
        return RG_ERR_UNSUPPORTED;
    const bool vec = K % 4 == 0 && ldx % 4 == 0 &&
                     (((uintptr_t)x | (uintptr_t)W | (uintptr_t)pending | (uintptr_t)norm_w | (uintptr_t)x_new) & 15) == 0;
    const size_t smem = (size_t)(silu ? 3 : 2) * SG_T * ((K + SG_T - 1) / SG_T * SG_T + 4) * sizeof(float);       // up to 98 KB
    auto kernel = silu ? (vec ? small_gemm_rows_kernel<SG_SILU, true> : small_gemm_rows_kernel<SG_SILU, false>)
                       : (vec ? small_gemm_rows_kernel<SG_NORM, true> : small_gemm_rows_kernel<SG_NORM, false>);
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    return rg_launch(kernel, dim3((N + SG_T - 1) / SG_T, mt), dim3(SG_ROWS_T), smem, (cudaStream_t)stream, 1, x, ldx, pending, norm_w, eps, x_new,
                     W, out, ldo, M, N, K);
}
