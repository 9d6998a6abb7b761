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

// x: rows ldx apart; W [N, K] contiguous; out: rows ldo apart.
extern "C" int rg_small_gemm_f32(const float* x, int ldx, const float* W, float* out, int ldo, int M, int N, int K, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    const int mt = (M + SG_T - 1) / SG_T;
    if (K <= 0 || ldx < K || ldo < N || mt > 65535) return RG_ERR_UNSUPPORTED;
    const bool vec = K % 4 == 0 && ldx % 4 == 0 && (((uintptr_t)x | (uintptr_t)W) & 15) == 0;
    return rg_launch(vec ? small_gemm_kernel<true> : small_gemm_kernel<false>, dim3((N + SG_T - 1) / SG_T, mt), dim3(128), 0,
                     (cudaStream_t)stream, 1, x, ldx, W, out, ldo, M, N, K);
}
