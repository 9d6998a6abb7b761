// The recurrence of Mamba-2 over portions of prompts, in chunks of 64 tokens side by side instead of token by token:
//
//   S <- g_t S + dt_t B_t x_t^T,  o_t = S^T C_t + D x_t,   g_t = exp(a_t),  a_t = -exp(A_log) dt_t
//
// With c_i = a_1 + .. + a_i inside a chunk of L tokens and S the state before it,
//   o_i   = exp(c_i) S^T C_i + sum_(j <= i) exp(c_i - c_j) dt_j (B_j . C_i) x_j + D x_i
//   S_end = exp(c_L) S + sum_j exp(c_L - c_j) dt_j B_j x_j^T
// so that everything but the pass from chunk to chunk is products.  Three kernels:
//   chunk_states   per (chunk, head): the sum in S_end, and exp(c_L); per (chunk, group): all B_j . C_i
//   chunk_pass     per (request, head, number of S): S before every chunk, and the last one into the request's slot
//   chunk_outputs  per (chunk, head): o
// (the block decomposition of Dao and Gu, "Transformers are SSMs: Generalized Models and Efficient Algorithms Through
// Structured State Space Duality").  The products are 32-bit fused multiply-adds; the exponents' sums are 64-bit, since
// their differences are small beside them where a head forgets fast.
//
// The same recurrence with the logarithm of every token's decay given instead of A_log and dt (then dt holds the weights of
// the new terms only), without D, and with n, the sum of the B's with the same decays and weights, carried as one more
// row of the state ("ones": the column of a value that is always 1), for memories that divide by n . C.  n and n . C are
// sums that the light blocks of the launches work out.
//
// And with one fixed decay per head (retention, lightning attention), its logarithm in 64-bit, and dt 1: 2,048 tokens of 16
// heads of 128 x 128 take 133 us (46 + 22 + 55 for states, pass and outputs with products in one chain, see chunk_scan.cuh) where
// the token-by-token kernel takes 358 alone in a loop and took 651 in a model's step.
//
// What bounds it: 19 us of multiply-adds in the outputs' products, 22 in the states' (128 a cycle and SM); the rest is a
// block's chain of loads, which is why the products' rows come asynchronously, a stage ahead, and lie in shared memory as
// they lie in global memory.  With 4 x 4 results a thread and synchronous loads: 67 + 22 + 83 us.
//
// The step's tokens are packed request by request (cu_seqlens); a request's chunks start at its first token of the step.
#include "chunk_scan.cuh"

#define XP (CH + 4)           // pitch of a chunk's values turned (column by token), and of its weights (token by token)

// Shared memory of chunk_states: values [64][68] and B [64][64 W + 4], or two stages of the dots' rows; of chunk_outputs: two
// stages of C's and S's rows, or weights and values of the chunk.
__host__ __device__ constexpr size_t states_smem(int W) {
    const size_t a = (size_t)(CH * (TILE + 4) + CH * (TILE * W + 4)) * 4, b = (size_t)2 * (64 + 64) * MP * 4;
    return a > b ? a : b;
}
__host__ __device__ constexpr size_t outputs_smem(int W) {
    const size_t a = (size_t)2 * (64 + 64 * W) * MP * 4, b = (size_t)(CH + 64 * W) * XP * 4;
    return a > b ? a : b;
}

// x, B, C: rows x_ld, B_ld, C_ld apart (head h's x at column h dv, group g's B and C at column g N).  sums [chunks, H, dv + ones, N],
// decays [chunks, H], dots [chunks, G, 64, 64] = C_i . B_j at [i][j].  grid: chunks, H (tiles of S, 64 columns by 64 W rows: z)
// and then G (z = 0).  VEC: rows and sizes allow four numbers at a time.
template <int W, bool VEC, typename V>
__global__ void __launch_bounds__(MTH, 4)
chunk_states_kernel(const V* __restrict__ x, int x_ld, const float* __restrict__ B, int B_ld, const float* __restrict__ C,
                    int C_ld, const float* __restrict__ dt, const float* __restrict__ loga, const float* __restrict__ A_log,
                    const double* __restrict__ fixed, const int* __restrict__ cu, int R, int least, float* __restrict__ sums,
                    float* __restrict__ decays, float* __restrict__ dots, int H, int G, int N, int dv, int ntiles, int ones) {
    extern __shared__ __align__(16) float sm[];
    __shared__ double cum[CH];
    __shared__ float sdt[CH];
    pdl_wait();
    pdl_trigger();
    int r, lo, n;
    if (!find_chunk(cu, R, blockIdx.x, least, r, lo, n)) return;
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    if ((int)blockIdx.y >= H) {
        if (blockIdx.z > 0) return;
        const int g = blockIdx.y - H;
        float a1[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) a1[i][j] = 0.f;
        product_of_rows<4, VEC, 16>(a1, sm, C + (size_t)lo * C_ld + (size_t)g * N, C_ld, n, B + (size_t)lo * B_ld + (size_t)g * N,
                                B_ld, n, N, ty, tx);
        float* out = dots + ((size_t)blockIdx.x * G + g) * CH * CH;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q) out[(8 * ty + i) * CH + tx + 16 * q] = a1[i][q];
        if (!ones) return;
        for (int h = g * (H / G); h < (g + 1) * (H / G); ++h) {         // the row of n: every head of the group
            __syncthreads();
            chunk_sums(dt, loga, A_log, fixed, lo, n, H, h, cum, sdt);
            __syncthreads();
            const double last = cum[CH - 1];
            __syncthreads();
            if (threadIdx.x < n) sdt[threadIdx.x] *= expf((float)(last - cum[threadIdx.x]));
            __syncthreads();
            for (int k = threadIdx.x; k < N; k += MTH) {
                float s = 0.f;
#pragma unroll 8
                for (int t = 0; t < n; ++t) s += B[(size_t)(lo + t) * B_ld + (size_t)g * N + k] * sdt[t];
                sums[(((size_t)blockIdx.x * H + h) * (dv + 1) + dv) * N + k] = s;
            }
        }
        return;
    }
    const int h = blockIdx.y, grp = h / (H / G);
    const int j0 = (blockIdx.z / ntiles) * TILE, n0 = (blockIdx.z % ntiles) * TILE * W;      // columns of S, rows of S
    // all of the chunk's rows are requested before its decays are worked out
    float* sA = sm;                                         // [token][column], times what is left of it at the chunk's end
    float* sB = sm + CH * (TILE + 4);                       // [token][row of S]
    constexpr int BP = TILE * W + 4;
    const V* xh = x + (size_t)lo * x_ld + (size_t)h * dv;
    const float* Bh = B + (size_t)lo * B_ld + (size_t)grp * N;
    for (int e = threadIdx.x; e < CH * (TILE * W / 4); e += MTH) {
        const int t = e / (TILE * W / 4), k = e % (TILE * W / 4) * 4;
        if (VEC) {
            const bool there = t < n && n0 + k < N;
            const uint32_t d = (uint32_t)__cvta_generic_to_shared(sB + t * BP + k);
            const float* p = there ? Bh + (size_t)t * B_ld + n0 + k : Bh;
            const int bytes = there ? 16 : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(p), "r"(bytes));
        } else {
            *reinterpret_cast<float4*>(sB + t * BP + k) = values4<VEC>(Bh, B_ld, t, n, n0 + k, N);
        }
    }
    if (VEC) asm volatile("cp.async.commit_group;\n" ::);
    constexpr int PER = CH * (TILE / 4) / MTH;
    float4 xv[PER];
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int e = threadIdx.x + p * MTH;
        xv[p] = values4<VEC>(xh, x_ld, e / (TILE / 4), n, j0 + e % (TILE / 4) * 4, dv);
    }
    chunk_sums(dt, loga, A_log, fixed, lo, n, H, h, cum, sdt);
    __syncthreads();
    const double end = cum[CH - 1];
    if (threadIdx.x == 0 && blockIdx.z == 0) decays[(size_t)blockIdx.x * H + h] = expf((float)end);
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int e = threadIdx.x + p * MTH, t = e / (TILE / 4);
        const float f = sdt[t] * expf((float)(end - cum[t]));                // 0 beyond the chunk's tokens
        *reinterpret_cast<float4*>(sA + t * (TILE + 4) + e % (TILE / 4) * 4) =
            make_float4(xv[p].x * f, xv[p].y * f, xv[p].z * f, xv[p].w * f);
    }
    if (VEC) asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
    float acc[8][4 * W];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4 * W; ++j) acc[i][j] = 0.f;
#pragma unroll 4
    for (int t = 0; t < n; ++t) {
        float a[8], b[4 * W];
        *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(sA + t * (TILE + 4) + 8 * ty);
        *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(sA + t * (TILE + 4) + 8 * ty + 4);
#pragma unroll
        for (int w = 0; w < W; ++w)
            *reinterpret_cast<float4*>(b + 4 * w) = *reinterpret_cast<const float4*>(sB + t * BP + TILE * w + 4 * tx);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4 * W; ++j) acc[i][j] += a[i] * b[j];
    }
    float* out = sums + ((size_t)blockIdx.x * H + h) * (dv + ones) * N;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int j = j0 + 8 * ty + i;
        if (j >= dv) continue;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const int k = n0 + TILE * w + 4 * tx;
            if (VEC) {
                if (k < N) *reinterpret_cast<float4*>(out + (size_t)j * N + k) =
                    make_float4(acc[i][4 * w], acc[i][4 * w + 1], acc[i][4 * w + 2], acc[i][4 * w + 3]);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (k + q < N) out[(size_t)j * N + k + q] = acc[i][4 * w + q];
            }
        }
    }
}

// before [chunks, H, dv + ones, N]: the state before every chunk.  o [T, H, dv + ones].  grid: chunks, H, tiles of 64 W
// columns, and with `ones` a light block for n . C.
template <int W, bool VEC, typename V>
__global__ void __launch_bounds__(MTH, 4)
chunk_outputs_kernel(const V* __restrict__ x, int x_ld, const float* __restrict__ C, int C_ld, const float* __restrict__ dt,
                     const float* __restrict__ loga, const float* __restrict__ A_log, const double* __restrict__ fixed,
                     const float* __restrict__ D, const int* __restrict__ cu, int R, int least, const float* __restrict__ before,
                     const float* __restrict__ dots, float* __restrict__ o, int H, int G, int N, int dv, int ones) {
    extern __shared__ __align__(16) float sm[];
    __shared__ double cum[CH];
    __shared__ float sdt[CH];
    pdl_wait();
    pdl_trigger();
    int r, lo, n;
    if (!find_chunk(cu, R, blockIdx.x, least, r, lo, n)) return;
    const int h = blockIdx.y, grp = h / (H / G), j0 = blockIdx.z * TILE * W;
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    const float* dd = dots + ((size_t)blockIdx.x * G + grp) * CH * CH;
    if (j0 >= dv) {
        chunk_sums(dt, loga, A_log, fixed, lo, n, H, h, cum, sdt);
        __syncthreads();
        // n . C_i: two threads a token (neighbouring lanes) share its sums over the chunk's tokens and over n's numbers
        const float* nb = before + (((size_t)blockIdx.x * H + h) * (dv + 1) + dv) * N;
        const int i = threadIdx.x >> 1, part = threadIdx.x & 1;
        float s = 0.f, b = 0.f;
        if (i < n) {
            const float* c = C + (size_t)(lo + i) * C_ld + (size_t)grp * N;
            for (int j = part; j <= i; j += 2) s += dd[i * CH + j] * sdt[j] * expf((float)(cum[i] - cum[j]));
            for (int k = part; k < N; k += 2) b += nb[k] * c[k];
            s += b * expf((float)cum[i]);
        }
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if (i < n && part == 0) o[((size_t)(lo + i) * H + h) * (dv + 1) + dv] = s;
        return;
    }
    float acc[8][4 * W];                                     // tokens 8 ty + i, columns j0 + tx + 16 q
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int q = 0; q < 4 * W; ++q) acc[i][q] = 0.f;
    // from the state before the chunk
    product_of_rows<4 * W, VEC>(acc, sm, C + (size_t)lo * C_ld + (size_t)grp * N, C_ld, n,
                                before + (((size_t)blockIdx.x * H + h) * (dv + ones) + j0) * N, N, dv - j0, N, ty, tx);
    chunk_sums(dt, loga, A_log, fixed, lo, n, H, h, cum, sdt);
    // within it: token j counts for the tokens from j on only.  The values turned, column by token
    float* sX = sm + CH * XP;
    const V* xh = x + (size_t)lo * x_ld + (size_t)h * dv;
#pragma unroll 4
    for (int e = threadIdx.x; e < CH * (TILE * W / 4); e += MTH) {
        const int t = e % CH, k = e / CH * 4;
        const float4 v = values4<VEC>(xh, x_ld, t, n, j0 + k, dv);
        sX[k * XP + t] = v.x; sX[(k + 1) * XP + t] = v.y; sX[(k + 2) * XP + t] = v.z; sX[(k + 3) * XP + t] = v.w;
    }
    __syncthreads();
#pragma unroll 8
    for (int e = threadIdx.x; e < CH * CH; e += MTH) {
        const int i = e / CH, j = e - i * CH;
        sm[i * XP + j] = j <= i && i < n ? dd[e] * sdt[j] * expf((float)(cum[i] - cum[j])) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float g = expf((float)cum[8 * ty + i]);
#pragma unroll
        for (int q = 0; q < 4 * W; ++q) acc[i][q] *= g;
    }
    __syncthreads();
    multiply_rows<4 * W, XP, XP>(acc, sm, sX, 0, 8 * ty, ty, tx);
    // the thread's own eight tokens: a triangle
    const float skip = D ? D[h] : 0.f;
#pragma unroll
    for (int k = 0; k < 8; k += 4) {
        float4 a[8];
#pragma unroll
        for (int i = k; i < 8; ++i) a[i] = *reinterpret_cast<const float4*>(sm + (8 * ty + i) * XP + 8 * ty + k);
#pragma unroll
        for (int q = 0; q < 4 * W; ++q) {
            const float4 b = *reinterpret_cast<const float4*>(sX + (tx + 16 * q) * XP + 8 * ty + k);
            acc[k][q] += skip * b.x; acc[k + 1][q] += skip * b.y; acc[k + 2][q] += skip * b.z; acc[k + 3][q] += skip * b.w;
#pragma unroll
            for (int i = k; i < 8; ++i) {
                acc[i][q] += a[i].x * b.x;
                if (i >= k + 1) acc[i][q] += a[i].y * b.y;
                if (i >= k + 2) acc[i][q] += a[i].z * b.z;
                if (i >= k + 3) acc[i][q] += a[i].w * b.w;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = 8 * ty + i;
        if (t >= n) continue;
        float* out = o + ((size_t)(lo + t) * H + h) * (dv + ones) + j0 + tx;
#pragma unroll
        for (int q = 0; q < 4 * W; ++q)
            if (j0 + tx + 16 * q < dv) out[16 * q] = acc[i][q];
    }
}

// Four numbers at a time: sizes, pitches and addresses in multiples of four numbers.
template <typename V>
static bool by_fours(const V* x, int x_ld, const float* B, int B_ld, const float* C, int C_ld, int N, int dv) {
    return N % 4 == 0 && dv % 4 == 0 && x_ld % 4 == 0 && B_ld % 4 == 0 && C_ld % 4 == 0 &&
           ((uintptr_t)x & (4 * sizeof(V) - 1)) == 0 && (((uintptr_t)B | (uintptr_t)C) & 15) == 0;
}
template <typename K>
static int allow(K kernel, size_t smem) {
    return smem > 46 * 1024 ? (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) : 0;
}

template <typename V>
static int launch_outputs(const V* x, int x_ld, const float* C, int C_ld, const float* dt, const float* loga, const float* A_log,
                          const double* fixed, const float* D, const int* cu_seqlens, const float* before, const float* dots,
                          float* o, int chunks, int R, int least, int H, int G, int N, int dv, int ones, cudaStream_t s) {
    // 128 columns a block where that leaves three blocks an SM (2,048 tokens, 16 heads: 55 us), else 64: 30 chunks of 8 heads
    // take 52 us with 128
    const int wide = dv > TILE && (long long)chunks * H * ((dv + 2 * TILE - 1) / (2 * TILE)) >= 3 * 148 ? 2 : 1;
    const bool vec = by_fours(x, x_ld, before, 0, C, C_ld, N, dv);
    auto kernel = wide == 2 ? (vec ? chunk_outputs_kernel<2, true, V> : chunk_outputs_kernel<2, false, V>)
                            : (vec ? chunk_outputs_kernel<1, true, V> : chunk_outputs_kernel<1, false, V>);
    const size_t smem = outputs_smem(wide);
    const int e = allow(kernel, smem);
    if (e) return e;
    return rg_launch(kernel, dim3(chunks, H, (dv + TILE * wide - 1) / (TILE * wide) + ones), dim3(MTH), smem, s, 1, x, x_ld, C,
                     C_ld, dt, loga, A_log, fixed, D, cu_seqlens, R, least, before, dots, o, H, G, N, dv, ones);
}

// x [T, H * dv] float or bfloat16, rows x_ld apart; B, C [T, G * N] float, rows B_ld, C_ld apart.  dt [T, H], or null: 1.
// The decays: loga [T, H], or fixed [H] (logarithms, the same for every token), or A_log [H] with dt.  D [H] or null.
// state [slots, H, dv + ones, N].
// Requests that bring fewer than `least` tokens are left alone, rows of o and state.  chunks: at least the number of chunks of
// the others (T / 64 + R, rounded down, is enough).  Scratch of the caller: sums [chunks, H, dv + ones, N], decays [chunks, H],
// dots [chunks, G, 64, 64].
template <typename V>
static int chunk_scan(const V* x, int x_ld, const float* B, int B_ld, const float* C, int C_ld, const float* dt,
                      const float* loga, const float* A_log, const double* fixed, const float* D, float* state,
                      const int* cu_seqlens, const int* start_pos, const int* slots, float* sums, float* decays, float* dots,
                      float* o, int chunks, int R, int least, int H, int G, int N, int dv, int ones, cudaStream_t s) {
    const int wide = N > TILE ? 2 : 1;
    const int jt = (dv + TILE - 1) / TILE, nt = (N + TILE * wide - 1) / (TILE * wide);
    if (jt * nt > 65535) return RG_ERR_UNSUPPORTED;
    dim3 g1(chunks, H + G, jt * nt);
    const bool four_each = by_fours(x, x_ld, B, B_ld, C, C_ld, N, dv) && ((uintptr_t)sums & 15) == 0;
    auto states = wide == 2 ? (four_each ? chunk_states_kernel<2, true, V> : chunk_states_kernel<2, false, V>)
                            : (four_each ? chunk_states_kernel<1, true, V> : chunk_states_kernel<1, false, V>);
    const size_t smem = states_smem(wide);
    int e = allow(states, smem);
    if (e) return e;
    e = rg_launch(states, g1, dim3(MTH), smem, s, 1, x, x_ld, B, B_ld, C, C_ld, dt, loga, A_log, fixed, cu_seqlens, R, least, sums,
                  decays, dots, H, G, N, dv, nt, ones);
    if (e) return e;
    const int M = (dv + ones) * N;
    const bool vec = M % 4 == 0 && ((uintptr_t)state & 15) == 0;
    const long long work = vec ? (long long)H * M / 4 : (long long)H * M;
    dim3 g2((unsigned)((work + 255) / 256), R);
    e = vec ? rg_launch(chunk_pass_kernel<4, false>, g2, dim3(256), 0, s, 1, sums, (const float*)decays, state, cu_seqlens, start_pos, slots, H, M, N, least)
            : rg_launch(chunk_pass_kernel<1, false>, g2, dim3(256), 0, s, 1, sums, (const float*)decays, state, cu_seqlens, start_pos, slots, H, M, N, least);
    if (e) return e;
    return launch_outputs(x, x_ld, C, C_ld, dt, loga, A_log, fixed, D, cu_seqlens, (const float*)sums, (const float*)dots, o, chunks,
                          R, least, H, G, N, dv, ones, s);
}

extern "C" int rg_ssd_chunk_scan(const void* x, int x_dtype, int x_ld, const float* B, int B_ld, const float* C, int C_ld,
                                 const float* dt, const float* loga, const float* A_log, const double* fixed, const float* D,
                                 float* state, const int* cu_seqlens, const int* start_pos, const int* slots, float* sums,
                                 float* decays, float* dots, float* o, int chunks, int R, int least, int H, int G, int N,
                                 int dv, int ones, void* stream) {
    if (chunks <= 0 || R <= 0) return 0;
    if ((!loga && !fixed && !(A_log && dt)) || ones < 0 || ones > 1) return RG_ERR_UNSUPPORTED;
    if (H < 1 || G < 1 || H % G || N < 1 || dv < 1 || H + G > 65535 || R > 65535) return RG_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    if (x_dtype == RG_DTYPE_F32)
        return chunk_scan((const float*)x, x_ld, B, B_ld, C, C_ld, dt, loga, A_log, fixed, D, state, cu_seqlens, start_pos, slots,
                          sums, decays, dots, o, chunks, R, least, H, G, N, dv, ones, s);
    if (x_dtype == RG_DTYPE_BF16)
        return chunk_scan((const bf16*)x, x_ld, B, B_ld, C, C_ld, dt, loga, A_log, fixed, D, state, cu_seqlens, start_pos, slots,
                          sums, decays, dots, o, chunks, R, least, H, G, N, dv, ones, s);
    return RG_ERR_UNSUPPORTED;
}

// The last of the three kernels alone, for a recurrence whose states and dots come from elsewhere (delta_chunk.cu): x float
// [T, H * dv], loga [T, H], before [chunks, H, dv, N].
extern "C" int rg_chunk_outputs(const float* x, int x_ld, const float* C, int C_ld, const float* loga, const int* cu_seqlens,
                                const float* before, const float* dots, float* o, int chunks, int R, int least, int H, int G,
                                int N, int dv, void* stream) {
    if (chunks <= 0 || R <= 0) return 0;
    if (H < 1 || G < 1 || H % G || N < 1 || dv < 1 || H > 65535 || (dv + TILE - 1) / TILE > 65535) return RG_ERR_UNSUPPORTED;
    return launch_outputs(x, x_ld, C, C_ld, (const float*)nullptr, loga, (const float*)nullptr, (const double*)nullptr,
                          (const float*)nullptr, cu_seqlens, before, dots, o, chunks, R, least, H, G, N, dv, 0, (cudaStream_t)stream);
}
