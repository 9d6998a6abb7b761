// The gated delta rule over portions of prompts in chunks of 64 tokens, instead of token by token:
//
//   S <- g_t S,  u_t = beta_t (v_t - S^T k_t),  S <- S + k_t u_t^T,  o_t = S^T q_t,   g_t = exp(a_t)
//
// With c_i = a_1 + .. + a_i inside a chunk and S0 the state before it, the u of a chunk solve a triangular system,
//   (I + A) U = beta V - (beta exp(c) K) S0,   A_ij = beta_i exp(c_i - c_j) k_i . k_j  for j < i,
// so that U = X - W S0 with X = (I + A)^-1 (beta V) and W = (I + A)^-1 (beta exp(c) K), which need no state, and
//   S1 = exp(c_L) S0 + sum_j exp(c_L - c_j) k_j u_j^T,
//   o_i = exp(c_i) S0^T q_i + sum_(j <= i) exp(c_i - c_j) (k_j . q_i) u_j
// (the block form of Yang et al., "Parallelizing Linear Transformers with the Delta Rule over Sequence Length").
//   delta_solve    per (chunk, head): (I + A)^-1 by substitution in blocks, X and W; per (chunk, query/key head): all k_j . q_i
//   delta_states   per (request, head, 16 columns of S): chunk after chunk, U, the state before every chunk, and the last
//                  one into the request's slot
// and chunk_outputs (ssd_chunk.cu) with U in the place of the values.  Everything is 32-bit fused multiply-adds; the
// exponents' sums are 64-bit.
//
// What bounds it: the 32-bit multiply-adds (128 a cycle and SM, packed or not), and in delta_states the chain from chunk to
// chunk, 2 x 64 x d of them per column and chunk.  16 columns a block fill 128 of 148 SMs at 16 heads of 128 columns;
// narrower blocks fetch the same W and K more often.  A chunk's 2,048 cycles of multiply-adds stand beside its copies, sums
// across lanes and three barriers: sixteen warps (eighths of k, quarters of the tokens) overlap those better than eight, 119 us
// against 141 behind delta_solve at 16 heads of 128 x 128, where d is also a compile-time number, 93 against 135 at 64 x 64, where
// it is not.
// Measured (2,048 tokens, 16 heads of 128 x 128 on 8, under ncu): 70 us the systems, 122 the states, 65 the outputs, their products
// in fours (chunk_scan.cuh).  The token-by-token kernel (state_mixers.cu) takes 473 alone in a loop and took 908 in a model's
// step.  Requests that bring fewer than 256 tokens stay on that one (ops.py, DELTA_CHUNK_MIN_TOKENS).
#include "chunk_scan.cuh"
#include <type_traits>

#define DC_CB 16              // columns of S per block of delta_states
#define DC_TH 512             // threads of delta_states
#define DC_SP 24              // pitch of S and U in shared memory: eight neighbouring k lie in different banks
#define DC_WP 72              // pitch of W's rows (k) in shared memory: four neighbouring k lie in different banks
#define DC_MAX_D 128

// q, k: rows q_ld, k_ld apart, head h of the H reads head h / (H / Hqk).  beta, loga [T, H].  x_out [T, H, dv] = X;
// w_out [chunks, H, d, 64] = W transposed; factors [chunks, H, 64] = exp(c_L - c_i) (1 beyond the chunk's tokens), decays
// [chunks, H] = exp(c_L); dots [chunks, Hqk, 64, 64] = q_i . k_j at [i][j].  grid: chunks, H (systems) and then Hqk (dots).
// The inverse T of I + A is made once per system, in blocks of 16: the diagonal blocks by substitution (64 threads, one column
// each), then row of blocks by row of blocks T_rc = -T_rr sum_k A_rk T_kc; X and W are products with it.  (Substituting
// all dv + d right-hand sides, one a thread with 64 unknowns in registers, was 2,600 instructions that ran once: 85 us for
// 528 systems of 2,048 tokens, 58 now.)
#define DS_TP (CH + 4)        // pitch of T transposed
#define DS_CP (128 + 4)       // pitch of 128 columns of the right-hand sides

constexpr size_t ds_smem() {
    const size_t a = (size_t)2 * (64 + 64) * MP * 4, b = (size_t)(CH * DS_TP + CH * DS_CP) * 4;
    return a > b ? a : b;
}

template <bool VEC, typename V>
__global__ void __launch_bounds__(MTH, 4)
delta_solve_kernel(const float* __restrict__ q, int q_ld, const float* __restrict__ k, int k_ld, const V* __restrict__ v,
                   int v_ld, const float* __restrict__ beta, const float* __restrict__ loga, const int* __restrict__ cu,
                   int R, int least, float* __restrict__ x_out, float* __restrict__ w_out, float* __restrict__ factors,
                   float* __restrict__ decays, float* __restrict__ dots, int H, int Hqk, int d, int dv) {
    extern __shared__ __align__(16) float sm[];
    __shared__ double cum[CH];
    __shared__ float sbeta[CH], grown[CH];
    pdl_wait();
    pdl_trigger();
    int r, lo, n;
    if (!find_chunk(cu, R, blockIdx.x, least, r, lo, n)) return;
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    const bool system = (int)blockIdx.y < H;
    const int h = blockIdx.y, hq = system ? h / (H / Hqk) : h - H;
    const float* kh = k + (size_t)lo * k_ld + (size_t)hq * d;
    {
        // k_i . k_j, or q_i . k_j: i = 8 ty .., j = tx + 16 q
        float acc[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
        if (system) product_of_rows<4, true, 16>(acc, sm, kh, k_ld, n, kh, k_ld, n, d, ty, tx);
        else product_of_rows<4, VEC, 16>(acc, sm, q + (size_t)lo * q_ld + (size_t)hq * d, q_ld, n, kh, k_ld, n, d, ty, tx);
        if (!system) {
            float* out = dots + ((size_t)blockIdx.x * Hqk + hq) * CH * CH;
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) out[(8 * ty + i) * CH + tx + 16 * j] = acc[i][j];
            return;
        }
        chunk_sums(nullptr, loga, nullptr, nullptr, lo, n, H, h, cum, grown);
        if (threadIdx.x >= 64) {
            const int i = threadIdx.x - 64;
            sbeta[i] = i < n ? beta[(size_t)(lo + i) * H + h] : 0.f;
        }
        __syncthreads();
        // A as it lies: sm[i][j], zero for j >= i and beyond the chunk's tokens (whose beta is 0)
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int i = 8 * ty + a, j = tx + 16 * b;
                sm[i * DS_TP + j] = j < i && i < n ? sbeta[i] * expf((float)(cum[i] - cum[j])) * acc[a][b] : 0.f;
            }
    }
    float* sA = sm;                                      // A, then T transposed
    float* sT = sm + CH * DS_TP;                         // T, [i][j]; then the right-hand sides
    if (threadIdx.x < CH) {
        const size_t at = (size_t)blockIdx.x * H + h;
        const double end = cum[CH - 1];
        grown[threadIdx.x] = expf((float)cum[threadIdx.x]);
        factors[at * CH + threadIdx.x] = expf((float)(end - cum[threadIdx.x]));
        if (threadIdx.x == 0) decays[at] = expf((float)end);
    }
    for (int e = threadIdx.x; e < CH * DS_TP; e += MTH) sT[e] = 0.f;
    __syncthreads();
    if (threadIdx.x < CH) {
        // column c of the diagonal block b
        const int b0 = threadIdx.x & 48, c = threadIdx.x & 15;
        float y[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float t = i == c ? 1.f : 0.f;
#pragma unroll
            for (int j = 0; j < i; ++j) t -= sA[(b0 + i) * DS_TP + b0 + j] * y[j];
            y[i] = t;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) sT[(b0 + i) * DS_TP + b0 + c] = y[i];
    }
    __syncthreads();
    for (int br = 1; br < 4; ++br) {
        // P_c = sum_(k = c .. br - 1) A_(br, k) T_(k, c) for all c < br: rows 16 br + i, columns 0 .. 16 br - 1, two columns a thread
        // at a time; then T_(br, c) = -T_(br, br) P_c
        const int cols = 16 * br, i = threadIdx.x >> 3, c0 = threadIdx.x & 7;       // 16 rows x 8 threads
        float p[6];
#pragma unroll
        for (int m = 0; m < 6; ++m) {
            p[m] = 0.f;
            const int c = c0 + 8 * m;
            if (c < cols)
                for (int k2 = c & 48; k2 < cols; ++k2) p[m] += sA[(cols + i) * DS_TP + k2] * sT[k2 * DS_TP + c];
        }
        __syncthreads();
        // P takes A's place in this row of blocks (its columns left of the diagonal block are not needed again)
#pragma unroll
        for (int m = 0; m < 6; ++m)
            if (c0 + 8 * m < cols) sA[(cols + i) * DS_TP + c0 + 8 * m] = p[m];
        __syncthreads();
#pragma unroll
        for (int m = 0; m < 6; ++m) {
            const int c = c0 + 8 * m;
            if (c < cols) {
                float t = 0.f;
                for (int j = 0; j <= i; ++j) t -= sT[(cols + i) * DS_TP + cols + j] * sA[(cols + j) * DS_TP + c];
                sT[(cols + i) * DS_TP + c] = t;
            }
        }
        __syncthreads();
    }
    // T transposed and times beta of its columns: sA[j][i]
    for (int e = threadIdx.x; e < CH * CH; e += MTH) {
        const int j = e / CH, i = e % CH;
        sA[j * DS_TP + i] = sT[i * DS_TP + j] * sbeta[j];
    }
    // X = T (beta V) and W = T (beta exp(c) K), 128 columns at a time
    const int vt = (dv + 127) / 128, kt = (d + 127) / 128;
    for (int t = 0; t < vt + kt; ++t) {
        const bool values = t < vt;
        const int col0 = (values ? t : t - vt) * 128, N = values ? dv : d;
        __syncthreads();
#pragma unroll 4
        for (int e = threadIdx.x; e < CH * 32; e += MTH) {
            const int j = e / 32, c = e % 32 * 4;
            float4 x;
            if (values) {
                x = values4<VEC>(v + (size_t)lo * v_ld + (size_t)h * dv, v_ld, j, n, col0 + c, N);
            } else {
                x = values4<true>(kh, k_ld, j, n, col0 + c, N);
                const float g = grown[j];
                x.x *= g; x.y *= g; x.z *= g; x.w *= g;
            }
            *reinterpret_cast<float4*>(sT + j * DS_CP + c) = x;
        }
        __syncthreads();
        float acc[8][8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
        // T is lower triangular: the thread's own eight tokens are a triangle (a later token's infinities stay out of it)
        auto step = [&](int j, auto from) {
            float a[8], b[8];
            *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(sA + j * DS_TP + 8 * ty);
            *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(sA + j * DS_TP + 8 * ty + 4);
            *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(sT + j * DS_CP + 4 * tx);
            *reinterpret_cast<float4*>(b + 4) = *reinterpret_cast<const float4*>(sT + j * DS_CP + 64 + 4 * tx);
#pragma unroll
            for (int i = decltype(from)::value; i < 8; ++i)
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[i][c] += a[i] * b[c];
        };
#pragma unroll 2
        for (int j = 0; j < 8 * ty; ++j) step(j, std::integral_constant<int, 0>{});
        step(8 * ty, std::integral_constant<int, 0>{});
        step(8 * ty + 1, std::integral_constant<int, 1>{});
        step(8 * ty + 2, std::integral_constant<int, 2>{});
        step(8 * ty + 3, std::integral_constant<int, 3>{});
        step(8 * ty + 4, std::integral_constant<int, 4>{});
        step(8 * ty + 5, std::integral_constant<int, 5>{});
        step(8 * ty + 6, std::integral_constant<int, 6>{});
        step(8 * ty + 7, std::integral_constant<int, 7>{});
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int c = col0 + 64 * half + 4 * tx;
            if (c >= N) continue;                          // N is a multiple of 4
            if (values) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (8 * ty + i < n)
                        *reinterpret_cast<float4*>(x_out + ((size_t)(lo + 8 * ty + i) * H + h) * dv + c) =
                            make_float4(acc[i][4 * half], acc[i][4 * half + 1], acc[i][4 * half + 2], acc[i][4 * half + 3]);
            } else {
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    float* dst = w_out + (((size_t)blockIdx.x * H + h) * d + c + m) * CH + 8 * ty;
                    *reinterpret_cast<float4*>(dst) = make_float4(acc[0][4 * half + m], acc[1][4 * half + m], acc[2][4 * half + m], acc[3][4 * half + m]);
                    *reinterpret_cast<float4*>(dst + 4) = make_float4(acc[4][4 * half + m], acc[5][4 * half + m], acc[6][4 * half + m], acc[7][4 * half + m]);
                }
            }
        }
    }
}

// 16 bytes from global to shared memory, zeros where there are none
__device__ __forceinline__ void dc_copy16(float* dst, const float* src, bool there) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = there ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(a), "l"(src), "r"(n));
}

// u [T, H, dv]: X on entry, U on return.  before [chunks, H, dv, d]: the state before every chunk.  d % 4 == 0, d <= 128,
// dv % 4 == 0, rows of k 16-byte aligned.  grid: requests, H, groups of DC_CB columns; a chunk's W, K, X and factors are
// fetched (cp.async) while the chunk before it is worked on.  D: d, or 0.
template <int D>
__global__ void __launch_bounds__(DC_TH)
delta_states_kernel(const float* __restrict__ k, int k_ld, const float* __restrict__ w, const float* __restrict__ factors,
                    const float* __restrict__ decays, float* __restrict__ u, float* __restrict__ before,
                    float* __restrict__ state, const int* __restrict__ cu, const int* __restrict__ start_pos,
                    const int* __restrict__ slots, int least, int H, int Hqk, int d_arg, int dv) {
    extern __shared__ __align__(16) float sm[];
    const int d = D ? D : d_arg;
    const int KP = d + 16;                              // pitch of K's rows: two neighbouring tokens lie 16 banks apart
    const int stage_floats = d * DC_WP + CH * KP + CH * DC_CB + CH;
    float* sS = sm + 2 * stage_floats;                  // [d][DC_SP], S
    float* sU = sS + d * DC_SP;                         // [64][DC_SP], exp(c_L - c_i) u_i
    pdl_wait();
    pdl_trigger();
    const int r = blockIdx.x, h = blockIdx.y, j0 = blockIdx.z * DC_CB, hq = h / (H / Hqk);
    const int first = cu[r], last = cu[r + 1];
    const int nc = chunks_of(last - first, least);
    if (nc < 1) return;
    int c0 = 0;
    for (int x = 0; x < r; ++x) c0 += chunks_of(cu[x + 1] - cu[x], least);
    const int cols = min(DC_CB, dv - j0);               // a multiple of 4
    const int d4 = d / 4;
    auto issue = [&](int c) {
        float* st = sm + (c & 1) * stage_floats;
        const int lo = first + c * CH, n = min(CH, last - lo);
        const size_t at = (size_t)(c0 + c) * H + h;
        for (int e = threadIdx.x; e < d * (CH / 4); e += DC_TH) {
            const int kk = e / (CH / 4), i = e % (CH / 4) * 4;
            dc_copy16(st + kk * DC_WP + i, w + (at * d + kk) * CH + i, true);
        }
        st += d * DC_WP;
        for (int e = threadIdx.x; e < CH * d4; e += DC_TH) {
            const int i = e / d4, kk = (e - i * d4) * 4;
            dc_copy16(st + i * KP + kk, k + (size_t)(lo + min(i, n - 1)) * k_ld + (size_t)hq * d + kk, i < n);
        }
        st += CH * KP;
        for (int e = threadIdx.x; e < CH * (DC_CB / 4); e += DC_TH) {
            const int i = e / (DC_CB / 4), j = e % (DC_CB / 4) * 4;
            const bool there = i < n && j < cols;
            dc_copy16(st + i * DC_CB + j, u + ((size_t)(lo + min(i, n - 1)) * H + h) * dv + j0 + (j < cols ? j : 0), there);
        }
        if (threadIdx.x < CH / 4) dc_copy16(st + CH * DC_CB + 4 * threadIdx.x, factors + at * CH + 4 * threadIdx.x, true);
        asm volatile("cp.async.commit_group;\n" ::);
    };
    issue(0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // S: thread (k tile kt, column tile jt, quarter ih of the tokens, interleaved) keeps rows 4 kt .. + 3 of column 4 jt + ih
    const int ih = lane >> 3, jt = (warp & 1) * 2 + (lane & 1), kt = (warp >> 1) * 4 + ((lane >> 1) & 3);
    const bool owner = kt < d4;
    const int slot = slots[r], column = 4 * jt + ih;
    float S[4];
    {
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (owner && column < cols && slot >= 0 && start_pos[r] > 0)
            x = *reinterpret_cast<const float4*>(state + (((size_t)slot * H + h) * dv + j0 + column) * d + 4 * kt);
        S[0] = x.x; S[1] = x.y; S[2] = x.z; S[3] = x.w;
    }
    // the products W S0: thread (token tile it, column tile ju, eighth kq of the k, interleaved)
    const int kq = lane >> 2, ju = (warp & 1) * 2 + (lane & 1), it = (warp >> 1) * 2 + ((lane >> 1) & 1);
    for (int c = 0; c < nc; ++c) {
        const int lo = first + c * CH, n = min(CH, last - lo);
        if (c + 1 < nc) issue(c + 1);
        const float g = decays[(size_t)(c0 + c) * H + h];
        if (owner) {
#pragma unroll
            for (int a = 0; a < 4; ++a) sS[(4 * kt + a) * DC_SP + column] = S[a];
            if (column < cols)
                *reinterpret_cast<float4*>(before + (((size_t)(c0 + c) * H + h) * dv + j0 + column) * d + 4 * kt) =
                    make_float4(S[0], S[1], S[2], S[3]);
        }
        if (c + 1 < nc) asm volatile("cp.async.wait_group 1;\n" ::);
        else asm volatile("cp.async.wait_group 0;\n" ::);
        __syncthreads();
        const float* sW = sm + (c & 1) * stage_floats;
        const float* sK = sW + d * DC_WP;
        const float* sX = sK + CH * KP;
        const float* sF = sX + CH * DC_CB;
        {
            float acc[4][4];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) acc[a][b] = 0.f;
#pragma unroll 8
            for (int kk = kq; kk < d; kk += 8) {
                const float4 wv = *reinterpret_cast<const float4*>(sW + kk * DC_WP + 4 * it);
                const float4 sv = *reinterpret_cast<const float4*>(sS + kk * DC_SP + 4 * ju);
                acc[0][0] += wv.x * sv.x; acc[0][1] += wv.x * sv.y; acc[0][2] += wv.x * sv.z; acc[0][3] += wv.x * sv.w;
                acc[1][0] += wv.y * sv.x; acc[1][1] += wv.y * sv.y; acc[1][2] += wv.y * sv.z; acc[1][3] += wv.y * sv.w;
                acc[2][0] += wv.z * sv.x; acc[2][1] += wv.z * sv.y; acc[2][2] += wv.z * sv.z; acc[2][3] += wv.z * sv.w;
                acc[3][0] += wv.w * sv.x; acc[3][1] += wv.w * sv.y; acc[3][2] += wv.w * sv.z; acc[3][3] += wv.w * sv.w;
            }
            // the eighths' sums: lane kq ends up with token 4 it + kq / 2, its first or second two columns
            float half[2][4], one[4], two[2];
            const bool up4 = kq & 4, up2 = kq & 2, up1 = kq & 1;
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const float give = up4 ? acc[a][b] : acc[a + 2][b], keep = up4 ? acc[a + 2][b] : acc[a][b];
                    half[a][b] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
                }
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const float give = up2 ? half[0][b] : half[1][b], keep = up2 ? half[1][b] : half[0][b];
                one[b] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
            }
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const float give = up1 ? one[b] : one[b + 2], keep = up1 ? one[b + 2] : one[b];
                two[b] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
            }
            const int i = 4 * it + (kq >> 1), j = 4 * ju + 2 * (kq & 1);
            const float2 xv = *reinterpret_cast<const float2*>(sX + i * DC_CB + j);
            const float2 uv = make_float2(xv.x - two[0], xv.y - two[1]);
            const float f = sF[i];
            if (i < n && j < cols) *reinterpret_cast<float2*>(u + ((size_t)(lo + i) * H + h) * dv + j0 + j) = uv;
            *reinterpret_cast<float2*>(sU + i * DC_SP + j) = i < n ? make_float2(f * uv.x, f * uv.y) : make_float2(0.f, 0.f);
        }
        __syncthreads();
        {
            float acc[4][4];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) acc[a][b] = 0.f;
            if (owner) {
#pragma unroll 8
                for (int i = ih; i < n; i += 4) {
                    const float4 kv = *reinterpret_cast<const float4*>(sK + i * KP + 4 * kt);
                    const float4 uv = *reinterpret_cast<const float4*>(sU + i * DC_SP + 4 * jt);
                    acc[0][0] += kv.x * uv.x; acc[0][1] += kv.x * uv.y; acc[0][2] += kv.x * uv.z; acc[0][3] += kv.x * uv.w;
                    acc[1][0] += kv.y * uv.x; acc[1][1] += kv.y * uv.y; acc[1][2] += kv.y * uv.z; acc[1][3] += kv.y * uv.w;
                    acc[2][0] += kv.z * uv.x; acc[2][1] += kv.z * uv.y; acc[2][2] += kv.z * uv.z; acc[2][3] += kv.z * uv.w;
                    acc[3][0] += kv.w * uv.x; acc[3][1] += kv.w * uv.y; acc[3][2] += kv.w * uv.z; acc[3][3] += kv.w * uv.w;
                }
            }
            // the quarters' sums: each keeps its column
            const bool up2 = ih & 2, up1 = ih & 1;
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                float pair[2];
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const float give = up2 ? acc[a][b] : acc[a][b + 2], keep = up2 ? acc[a][b + 2] : acc[a][b];
                    pair[b] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
                }
                const float give = up1 ? pair[0] : pair[1], keep = up1 ? pair[1] : pair[0];
                S[a] = g * S[a] + (keep + __shfl_xor_sync(0xffffffffu, give, 8));
            }
        }
        __syncthreads();                                // the stage and S may be overwritten
    }
    if (owner && slot >= 0 && column < cols)
        *reinterpret_cast<float4*>(state + (((size_t)slot * H + h) * dv + j0 + column) * d + 4 * kt) = make_float4(S[0], S[1], S[2], S[3]);
}

// q, k [T, Hqk * d] float rows q_ld, k_ld apart; v [T, H * dv] float or bfloat16, rows v_ld apart; beta, loga [T, H];
// state [slots, H, dv, d].  chunks, least: as ssd_chunk.cu's.  Results and scratch of the caller: u [T, H, dv],
// before [chunks, H, dv, d], dots [chunks, Hqk, 64, 64]; w [chunks, H, d, 64], factors [chunks, H, 64], decays [chunks, H].
// Takes d and dv in multiples of 4, d up to 128, rows of k and the state on 16-byte boundaries.
extern "C" int rg_delta_chunk(const float* q, int q_ld, const float* k, int k_ld, const void* v, int v_dtype, int v_ld,
                              const float* beta, const float* loga, float* state, const int* cu_seqlens, const int* start_pos,
                              const int* slots, float* u, float* before, float* dots, float* w, float* factors, float* decays,
                              int chunks, int R, int least, int H, int Hqk, int d, int dv, void* stream) {
    if (chunks <= 0 || R <= 0) return 0;
    if (H < 1 || Hqk < 1 || H % Hqk || d < 4 || d % 4 || d > DC_MAX_D || dv < 4 || dv % 4 || H + Hqk > 65535 || k_ld % 4 ||
        ((uintptr_t)k & 15) || ((uintptr_t)state & 15) || ((uintptr_t)u & 15) || ((uintptr_t)before & 15))
        return RG_ERR_UNSUPPORTED;
    const int groups = (dv + DC_CB - 1) / DC_CB;
    if (groups > 65535) return RG_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    dim3 g1(chunks, H + Hqk);
    int e;
    const bool q4 = q_ld % 4 == 0 && ((uintptr_t)q & 15) == 0 && v_ld % 4 == 0;
#define DC_SOLVE(VEC_, V_) { \
        const cudaError_t ce = cudaFuncSetAttribute(delta_solve_kernel<VEC_, V_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ds_smem()); \
        if (ce != cudaSuccess) return (int)ce; \
        e = rg_launch(delta_solve_kernel<VEC_, V_>, g1, dim3(MTH), ds_smem(), s, 1, q, q_ld, k, k_ld, (const V_*)v, v_ld, beta, loga, \
                      cu_seqlens, R, least, u, w, factors, decays, dots, H, Hqk, d, dv); }
    if (v_dtype == RG_DTYPE_F32) {
        if (q4 && ((uintptr_t)v & 15) == 0) DC_SOLVE(true, float) else DC_SOLVE(false, float)
    } else if (v_dtype == RG_DTYPE_BF16) {
        if (q4 && ((uintptr_t)v & 7) == 0) DC_SOLVE(true, bf16) else DC_SOLVE(false, bf16)
    } else {
        return RG_ERR_UNSUPPORTED;
    }
#undef DC_SOLVE
    if (e) return e;
    const size_t smem = ((size_t)2 * (d * DC_WP + CH * (d + 16) + CH * DC_CB + CH) + (d + CH) * DC_SP) * sizeof(float);
    auto states = d == 128 ? delta_states_kernel<128> : delta_states_kernel<0>;
    cudaError_t ce = cudaFuncSetAttribute(states, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (ce != cudaSuccess) return (int)ce;
    return rg_launch(states, dim3(R, H, groups), dim3(DC_TH), smem, s, 1, k, k_ld, (const float*)w, (const float*)factors,
                     (const float*)decays, u, before, state, cu_seqlens, start_pos, slots, least, H, Hqk, d, dv);
}
