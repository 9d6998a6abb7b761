// What the chunked forms of the matrix-state recurrences share: a step's tokens, packed request by request (cu_seqlens),
// cut into chunks of 64 that start at each request's first token of the step; 64 x 64 (x 128) products in 32-bit fused
// multiply-adds; and the pass from chunk to chunk.
#pragma once
#include "common.cuh"

#define CH 64                 // tokens per chunk
#define TILE 64               // rows and columns of a block's output (columns: 64 or 128)
#define PITCH (TILE + 4)
#define NTH 256

// Chunks of a request that brings `len` tokens: none where it brings fewer than `least` (those are state_scan's).
__device__ __forceinline__ int chunks_of(int len, int least) { return len < least ? 0 : (len + CH - 1) / CH; }

// Chunk number c of the step: its request, first token and number of tokens; false beyond the last one.
__device__ __forceinline__ bool find_chunk(const int* __restrict__ cu, int R, int c, int least, int& r, int& lo, int& n) {
    for (r = 0; r < R; ++r) {
        const int len = cu[r + 1] - cu[r], k = chunks_of(len, least);
        if (c < k) {
            lo = cu[r] + c * CH;
            n = min(CH, len - c * CH);
            return true;
        }
        c -= k;
    }
    return false;
}

// c_i of the chunk's tokens for head h (64-bit), by the block's first warp; dt of the tokens (without dt: 1) into sdt.
// a_t is loga's number, or fixed's of the head, or without either -exp(A_log) dt_t.  Where a decay is 0 (its logarithm
// minus infinity) a number whose exponential is 0 takes its place, so that differences are numbers.
__device__ __forceinline__ void chunk_sums(const float* __restrict__ dt, const float* __restrict__ loga,
                                           const float* __restrict__ A_log, const double* __restrict__ fixed, int lo, int n, int H, int h,
                                           double* __restrict__ cum, float* __restrict__ sdt) {
    if (threadIdx.x < 32) {
        const int i0 = 2 * threadIdx.x, i1 = i0 + 1;
        const float d0 = i0 < n ? (dt ? dt[(size_t)(lo + i0) * H + h] : 1.f) : 0.f;
        const float d1 = i1 < n ? (dt ? dt[(size_t)(lo + i1) * H + h] : 1.f) : 0.f;
        double a0, a1;
        if (loga) {
            a0 = i0 < n ? (double)loga[(size_t)(lo + i0) * H + h] : 0.0;
            a1 = i1 < n ? (double)loga[(size_t)(lo + i1) * H + h] : 0.0;
        } else if (fixed) {
            a0 = i0 < n ? fixed[h] : 0.0;
            a1 = i1 < n ? fixed[h] : 0.0;
        } else {
            const float rate = -expf(A_log[h]);
            a0 = (double)(rate * d0);
            a1 = (double)(rate * d1);
        }
        a0 = a0 < -1e4 ? -1e4 : a0;
        a1 = a1 < -1e4 ? -1e4 : a1;
        double s = a0 + a1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, s, o);
            if ((int)threadIdx.x >= o) s += up;
        }
        cum[i0] = s - a1;
        cum[i1] = s;
        sdt[i0] = d0;
        sdt[i1] = d1;
    }
}

// dst[k][i] = src row i, number k0 + k (rows ld apart, n rows of N numbers; zeros elsewhere), for 64 x 64, times scale[i].
// A warp reads 4 rows x 8 neighbouring numbers at a time and writes 32 different banks.
__device__ __forceinline__ void load_transposed(float (*__restrict__ dst)[PITCH], const float* __restrict__ src, size_t ld,
                                                int n, int N, int k0, const float* __restrict__ scale) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int kl = lane & 7, il = lane >> 3;
#pragma unroll 4
    for (int p = warp; p < (TILE / 8) * (TILE / 4); p += NTH / 32) {
        const int k = (p & 7) * 8 + kl, i = (p >> 3) * 4 + il;
        float v = i < n && k0 + k < N ? src[(size_t)i * ld + k0 + k] : 0.f;
        if (scale) v *= scale[i];
        dst[k][i] = v;
    }
}

// acc[4][4 W] += A[k][4 rows]^T B[k][4 W columns] over kn values of k.  Thread (ty, tx): rows 4 ty .., columns 4 tx .. (+ 64)
template <int W>
__device__ __forceinline__ void multiply(float (&acc)[4][4 * W], const float (*__restrict__ A)[PITCH],
                                         const float (*__restrict__ B)[TILE * W + 4], int kn, int ty, int tx) {
#pragma unroll 4
    for (int k = 0; k < kn; ++k) {
        const float4 a = *reinterpret_cast<const float4*>(&A[k][4 * ty]);
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const float4 b = *reinterpret_cast<const float4*>(&B[k][TILE * w + 4 * tx]);
            acc[0][4 * w] += a.x * b.x; acc[0][4 * w + 1] += a.x * b.y; acc[0][4 * w + 2] += a.x * b.z; acc[0][4 * w + 3] += a.x * b.w;
            acc[1][4 * w] += a.y * b.x; acc[1][4 * w + 1] += a.y * b.y; acc[1][4 * w + 2] += a.y * b.z; acc[1][4 * w + 3] += a.y * b.w;
            acc[2][4 * w] += a.z * b.x; acc[2][4 * w + 1] += a.z * b.y; acc[2][4 * w + 2] += a.z * b.z; acc[2][4 * w + 3] += a.z * b.w;
            acc[3][4 * w] += a.w * b.x; acc[3][4 * w + 1] += a.w * b.y; acc[3][4 * w + 2] += a.w * b.z; acc[3][4 * w + 3] += a.w * b.w;
        }
    }
}

// ---- products of 64 rows by 64 or 128 columns by 128 threads of 8 x 4 or 8 x 8 results each, over rows of both operands as
// they lie in global memory.  The 4 x 4 results a thread of `multiply` read two 16-byte pieces of shared memory for 16
// multiply-adds; here 16 pieces serve 256.
#define MTH 128
#define MK 32                 // of the contraction at a time
#define MP (MK + 4)           // pitch of its rows: eight neighbouring rows' 16-byte pieces lie in different banks

// acc[i][q] += sum over k in [k_lo, k_hi) of A[8 ty + i][k] B[tx + 16 q][k], four k at a time; rows PA and PB apart.  Four
// products are added up before they join the sum: a chain of 128 ends up twice as far from it as one of 32, and the forms
// in chunks are to be no further from 64 bits than the token-by-token kernel, which adds a column up in shares.  Output of
// 2,048 tokens in the 2-norm, in 1e-7, token by token / in chunks with one chain / with fours (and sixteens in the dots): 16
// heads of decays 1 - 2^-5 .. 2^-11 4.62 / 3.67 / 3.05, 8 heads 2.21 / 2.66 / 1.78; the delta rule with logarithms to -0.01
// 3.31 / 2.99 / 1.97, to -2 0.94 / 2.09 / 0.93.  It costs a fifth multiply-add slot: 16 heads 124 to 133 us, 258 to 269.
template <int Q, int PA, int PB>
__device__ __forceinline__ void multiply_rows(float (&acc)[8][Q], const float* __restrict__ A, const float* __restrict__ B, int k_lo,
                                              int k_hi, int ty, int tx) {
    const float* a0 = A + 8 * ty * PA;
    const float* b0 = B + tx * PB;
#pragma unroll 1
    for (int k = k_lo; k < k_hi; k += 4) {
        float4 a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const float4*>(a0 + i * PA + k);
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const float4 b = *reinterpret_cast<const float4*>(b0 + 16 * q * PB + k);
            float t[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) t[i] = a[i].x * b.x;
#pragma unroll
            for (int i = 0; i < 8; ++i) t[i] += a[i].y * b.y;
#pragma unroll
            for (int i = 0; i < 8; ++i) t[i] += a[i].z * b.z;
#pragma unroll
            for (int i = 0; i < 8; ++i) t[i] += a[i].w * b.w;
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i][q] += t[i];
        }
    }
}

// dst[row][k] = src row `row`, number k0 + k, for `rows` rows (n of them there) and MK numbers (of N): zeros elsewhere.  VEC:
// 16 bytes at a time and asynchronously (rows, pitches and N in multiples of four numbers).
template <bool VEC>
__device__ __forceinline__ void fetch_rows(float* __restrict__ dst, const float* __restrict__ src, size_t ld, int rows, int n,
                                           int k0, int N) {
    if (VEC) {
        for (int e = threadIdx.x; e < rows * (MK / 4); e += MTH) {
            const int i = e / (MK / 4), k = e % (MK / 4) * 4;
            const bool there = i < n && k0 + k < N;
            const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst + i * MP + k);
            const float* p = there ? src + (size_t)i * ld + k0 + k : src;
            const int bytes = there ? 16 : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(p), "r"(bytes));
        }
    } else {
        for (int e = threadIdx.x; e < rows * MK; e += MTH) {
            const int i = e / MK, k = e % MK;
            dst[i * MP + k] = i < n && k0 + k < N ? src[(size_t)i * ld + k0 + k] : 0.f;
        }
    }
}

// acc += A B^T over all N numbers of their rows: A has 64 rows (na there), B 16 Q (nb there); two stages of MK numbers in
// `sm` [2][64 + 16 Q][MP], the next on its way while one is multiplied.  RUN > 0: sums of RUN products are made first and
// then added.
template <int Q, bool VEC, int RUN = 0>
__device__ __forceinline__ void product_of_rows(float (&acc)[8][Q], float* __restrict__ sm, const float* __restrict__ A, size_t lda,
                                                int na, const float* __restrict__ B, size_t ldb, int nb, int N, int ty, int tx) {
    constexpr int STAGE = (64 + 16 * Q) * MP;
    auto fetch = [&](int it) {
        float* st = sm + (it & 1) * STAGE;
        fetch_rows<VEC>(st, A, lda, 64, na, it * MK, N);
        fetch_rows<VEC>(st + 64 * MP, B, ldb, 16 * Q, nb, it * MK, N);
        if (VEC) asm volatile("cp.async.commit_group;\n" ::);
    };
    const int its = (N + MK - 1) / MK;
    fetch(0);
    for (int it = 0; it < its; ++it) {
        if (it + 1 < its) {
            fetch(it + 1);
            if (VEC) asm volatile("cp.async.wait_group 1;\n" ::);
        } else {
            if (VEC) asm volatile("cp.async.wait_group 0;\n" ::);
        }
        __syncthreads();
        const float* st = sm + (it & 1) * STAGE;
        if constexpr (RUN > 0) {
#pragma unroll 1
            for (int k = 0; k < MK; k += RUN) {
                float part[8][Q] = {};
                multiply_rows<Q, MP, MP>(part, st, st + 64 * MP, k, k + RUN, ty, tx);
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int q = 0; q < Q; ++q) acc[i][q] += part[i][q];
            }
        } else {
            multiply_rows<Q, MP, MP>(acc, st, st + 64 * MP, 0, MK, ty, tx);
        }
        __syncthreads();
    }
}

__device__ __forceinline__ float4 four(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 four(const bf16* p) {
    const uint2 x = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
// Numbers k .. k + 3 (of N) of row i (of n): zeros where there are none.
template <bool VEC, typename V>
__device__ __forceinline__ float4 values4(const V* __restrict__ src, size_t ld, int i, int n, int k, int N) {
    if (i >= n || k >= N) return make_float4(0.f, 0.f, 0.f, 0.f);
    const V* p = src + (size_t)i * ld + k;
    if (VEC) return four(p);
    return make_float4(to_f32(p[0]), k + 1 < N ? to_f32(p[1]) : 0.f, k + 2 < N ? to_f32(p[2]) : 0.f, k + 3 < N ? to_f32(p[3]) : 0.f);
}

// sums [chunks, H, M]: each chunk's sum becomes the state before the chunk, and the state after the last one goes into the
// request's slot (M = dv d numbers per head, S transposed).  decays [chunks, H], or with CHANNEL [chunks, H, d]: one per
// row of S.  V numbers per thread (with CHANNEL neighbours in a column of S: d % V == 0).
template <int V, bool CHANNEL>
__global__ void chunk_pass_kernel(float* __restrict__ sums, const float* __restrict__ decays, float* __restrict__ state,
                                  const int* __restrict__ cu, const int* __restrict__ start_pos,
                                  const int* __restrict__ slots, int H, int M, int d, int least) {
    pdl_wait();
    pdl_trigger();
    const int r = blockIdx.y;
    if (cu[r + 1] - cu[r] < least) return;
    const long long e = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (e >= (long long)H * M) return;
    const int h = (int)(e / M);
    int c0 = 0;
    for (int q = 0; q < r; ++q) c0 += chunks_of(cu[q + 1] - cu[q], least);
    const int nc = chunks_of(cu[r + 1] - cu[r], least);
    const int slot = slots[r];
    float S[V];
#pragma unroll
    for (int i = 0; i < V; ++i) S[i] = 0.f;
    float* st = state + (size_t)(slot >= 0 ? slot : 0) * H * M + e;
    if (slot >= 0 && start_pos[r] > 0) {
#pragma unroll
        for (int i = 0; i < V; ++i) S[i] = st[i];
    }
    float* p = sums + (size_t)c0 * H * M + e;
    const float* dec = CHANNEL ? decays + (size_t)c0 * H * d + (size_t)h * d + (e - (long long)h * M) % d
                               : decays + (size_t)c0 * H + h;
    const size_t dec_step = CHANNEL ? (size_t)H * d : (size_t)H;
    const size_t step = (size_t)H * M;
    constexpr int U = 4;                              // chunks in flight
    for (int c = 0; c < nc; c += U) {
        float u[U][V], g[U][V];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            if (c + k < nc) {
#pragma unroll
                for (int i = 0; i < V; ++i) g[k][i] = dec[(c + k) * dec_step + (CHANNEL ? i : 0)];
                if (V == 4) {
                    const float4 q = *reinterpret_cast<const float4*>(p + (c + k) * step);
                    u[k][0] = q.x; u[k][1 % V] = q.y; u[k][2 % V] = q.z; u[k][3 % V] = q.w;
                } else {
                    u[k][0] = p[(c + k) * step];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            if (c + k < nc) {
                if (V == 4) *reinterpret_cast<float4*>(p + (c + k) * step) = make_float4(S[0], S[1 % V], S[2 % V], S[3 % V]);
                else p[(c + k) * step] = S[0];
#pragma unroll
                for (int i = 0; i < V; ++i) S[i] = S[i] * g[k][i] + u[k][i];
            }
        }
    }
    if (slot >= 0) {
#pragma unroll
        for (int i = 0; i < V; ++i) st[i] = S[i];
    }
}
