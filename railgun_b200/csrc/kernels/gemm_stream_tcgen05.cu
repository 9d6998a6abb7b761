// Weight-streaming matrix product for steps of 17 to 256 rows on the 5th-generation tensor cores:
// y[M, N] = x[M, K] W[N, K]^T with the operands swapped, so that 128 rows of W fill the M side of tcgen05.mma
// and the step's tokens (in steps of 16) its N side: D[128 weight rows, tokens] accumulates in tensor memory while W
// streams through a ring of TMA stages once (twice where the tokens go in two parts, dispatch_ts).  At these sizes the product is bound by reading W, and a
// product with few rows of W (q|k|v, O, down) has too few 128-row tiles to occupy the GPU, so K is split over the
// CTAs of a thread-block cluster: every CTA accumulates its K range of the cluster's tile, leaves the partial sums
// in its shared memory (over the stages, which are done with by then), and the cluster's CTAs add them, each for its
// share of the tokens, reading the others' through distributed shared memory in rank order: one fixed order, no
// atomics: with a given number of splits a token's result does not depend on the other tokens, and the number that the
// launcher picks is one for all steps of up to 64 tokens and one for all above.  Products with many tiles (gate|up, the head) run unsplit
// and persistent: a CTA takes tile after tile with two accumulators in tensor memory, so that a tile's epilogue
// overlaps the next tile's loads.
//
// Roles as in gemm_tcgen05.cu: warps 0-3 epilogue (one lane of tensor memory = one row of W each), warp 4 the TMA
// producer, warp 5 issues the MMAs and owns the tensor memory; above 64 tokens warps 8-11 are a second epilogue group and of
// unsplit products above 128 warps 12-15 a third, since an epilogue is a chain that one warp per scheduler walks at a quarter of
// its rate.  Epilogues: plain (bfloat16 or 32-bit out) and
// SiLU-mul over interleaved gate|up rows (crates/vllm-models/src/llama/architecture.rs:81-85).  The reference runs
// these products through cuBLAS (crates/vllm-models/src/llama/attention.rs:94-96,133).
//
// Every wait on an mbarrier is bounded (tcgen05.cuh): a waiter that gives up records where in *err, every role
// stops, the CTA waits for copies in flight, frees its tensor memory and returns; the host reads *err and raises.
#include "tcgen05.cuh"

#define TS_ROWS 128               // rows of W per tile (the MMA's M)
#define TS_MAX_TOK 256            // tokens per tile, at most: a kernel is made for 64, 128 or 256; boxes and the MMA's N are of those that are there, in steps of 16 (zeros from TMA behind them)
#define TS_BK 64
#define TS_MAX_SPLITS 8
#define TS_EPI_NONE 0
#define TS_EPI_SILU_MUL 1
#define TS_EPI_RESIDUAL 2         // out (32-bit) += product; also the next norm's input and sums of squares
#define TS_EPI_ROPE_CACHE 3       // the q|k|v projection: rotate q and k, write q out and k, v into the paged cache
#define TS_PRO_PLAIN 0
#define TS_PRO_SCALED 1           // x is a residual row times the norm's weight; 1 / rms is applied to the sums

// RMSNorm around the product without a kernel of its own, as in gemm_skinny.cuh: y = W (w . r) / rms(r) is linear
// in 1 / rms, so the producer of the residual r leaves bf16(r * norm weight) and partial sums of squares, and the
// product that reads them multiplies its 32-bit sums by 1 / rms.
//   TS_EPI_RESIDUAL:  r = out[m, n] += product;  scaled_out[m, n] = bf16(r * norm_w[n]);
//                     ss_out[tile, m] = sum over the tile's 128 columns of r^2.
//   TS_PRO_SCALED:    every sum is multiplied by rsqrt(sum_p ss_in[p, m] / K + eps) before the epilogue.
// TS_EPI_ROPE_CACHE: N = (nh + 2 nkv) d, d % 16 == 0, the rows of every q and k head in the order that puts rotation
// pair i at (16 (i / 8) + i % 8, + 8) (rope_cache.cu's paired8 layout, as gemm_skinny.cuh's fused projection): rows
// (r, r + 8) of a group of 16 are a pair, rotated in 32-bit by the angles of the token's position (table
// [max_pos, d] = cos | sin); q goes to out, k and v to the token's slot of the cache [pages, 2, nkv, page_size, d].
struct StreamFusion {
    const float* norm_w;
    bf16* scaled_out;             // [M, N], rows ldo apart like out
    float* ss_out;                // [tiles, ss_ld]
    const float* ss_in;           // [ss_in_blocks, ss_ld]
    int ss_in_blocks;
    int ss_ld;
    float eps;
    const float* rope_table;      // TS_EPI_ROPE_CACHE from here
    const int* positions;
    const int* slots;             // nullptr: nothing is written to the cache
    bf16* kv_cache;
    int nh, nkv, d, page_size, max_pos;
    int* pos_err;                 // set to 1 when a position is outside the table (never read outside it)
};

__device__ __forceinline__ float4 ts_ld_remote4(uint32_t addr) {
    float4 v;
    // (volatile: not before the cluster's barrier; no clobber, so that several are in flight between stores)
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}

// A tile's sums -> the output, for the tokens m_lo .. m_hi - 1, by 128 threads.  A thread keeps its rows of W: four
// consecutive ones (plain, residual: a token's 128 rows are one warp's), or four and their partners eight rows on (gate and
// up, rotation pairs), and goes from token to token.  What it reads from global memory for the next four tokens (residual;
// angles, cache slots) is requested ahead: for the first four before the tile's product is there, else every token would
// wait for HBM or L2 once.  (The residual product of 64 rows by 2,048 x 8,192 unsplit, where one CTA writes a tile's 64
// tokens: 48.2 us before, 41.1 after; in eight splits 13.4 and 12.6.)  AHEAD tokens at a time: four, but one of eight
// splits and two of fewer up to 64 rows, where a thread has one to eight and what counts is how much code runs once (see
// `FEW`).
template <int EPI, int AHEAD>
struct TileEpilogue {
    static constexpr bool PAIRS = EPI == TS_EPI_SILU_MUL || EPI == TS_EPI_ROPE_CACHE;
    static constexpr int STEP = PAIRS ? 8 : 4;                               // from a thread's token to its next
    int row, m_off;                                                          // first row of W within the tile; place of the first token
    float4 resid[EPI == TS_EPI_RESIDUAL ? AHEAD : 1];
    float4 cosv[EPI == TS_EPI_ROPE_CACHE ? AHEAD : 1], sinv[EPI == TS_EPI_ROPE_CACHE ? AHEAD : 1];
    int slot[EPI == TS_EPI_ROPE_CACHE ? AHEAD : 1];

    __device__ __forceinline__ explicit TileEpilogue(int tid) {
        if (PAIRS) {
            const int q = tid & 15;                                          // rows 16 t .. + 7 and their partners + 8
            row = (q >> 1) * 16 + (q & 1) * 4;
            m_off = tid >> 4;
        } else {
            row = (tid & 31) * 4;
            m_off = tid >> 5;
        }
    }
    // four consecutive numbers of the output at n, in one piece where `vec`
    template <typename T>
    static __device__ __forceinline__ void put4(T* o, const float (&v)[4], bool vec, int room) {
        if (vec && room >= 4) {
            if constexpr (sizeof(T) == 4) {
                *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
                const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
                *reinterpret_cast<uint2*>(o) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i < room) o[i] = from_f32<T>(v[i]);
        }
    }
    // requests what the tokens m, m + STEP, .. (AHEAD of them) need
    template <typename OUT>
    __device__ __forceinline__ void fetch(int m, int m_hi, int n0, int N, const OUT* out, int ldo, bool vec, const StreamFusion& fu) {
        if constexpr (EPI == TS_EPI_RESIDUAL) {
            const int n = n0 + row;
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                const float* o = reinterpret_cast<const float*>(out) + (size_t)(m + u * STEP) * ldo + n;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (m + u * STEP < m_hi) {
                    if (vec && n + 4 <= N) {
                        v = *reinterpret_cast<const float4*>(o);
                    } else {
                        if (n < N) v.x = o[0];
                        if (n + 1 < N) v.y = o[1];
                        if (n + 2 < N) v.z = o[2];
                        if (n + 3 < N) v.w = o[3];
                    }
                }
                resid[u] = v;
            }
        }
        if constexpr (EPI == TS_EPI_ROPE_CACHE) {
            const int f = n0 + row, head = f / fu.d, e = f - head * fu.d, half = fu.d >> 1;
            const int i0 = ((e >> 4) << 3) + (e & 7);                        // the first pair's number = its angle's index
            int pos[AHEAD];
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                const bool there = m + u * STEP < m_hi && f + 8 < N;
                pos[u] = there && head < fu.nh + fu.nkv ? fu.positions[m + u * STEP] : 0;
                slot[u] = there && head >= fu.nh && fu.slots ? fu.slots[m + u * STEP] : -1;
            }
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                if (pos[u] < 0 || pos[u] >= fu.max_pos) {
                    if (fu.pos_err) atomicExch(fu.pos_err, 1);
                    pos[u] = 0;
                }
                if (m + u * STEP < m_hi && f + 8 < N && head < fu.nh + fu.nkv) {
                    cosv[u] = __ldg(reinterpret_cast<const float4*>(fu.rope_table + (size_t)pos[u] * fu.d + i0));
                    sinv[u] = __ldg(reinterpret_cast<const float4*>(fu.rope_table + (size_t)pos[u] * fu.d + half + i0));
                }
            }
        }
    }
    // load4(r, i): partial sums i .. i + 3 of CTA r's [token][row] array; they are added in rank order, and all are requested
    // before the first is used.  inv: 1 / rms per token (TS_PRO_SCALED).
    template <bool SPLIT, int FEW, int PRO, typename OUT, typename Load>
    __device__ __forceinline__ void write(Load load4, int splits, OUT* __restrict__ out, int ldo, int N, int n0, int tile,
                                          int m_lo, int m_hi, bool vec, const float* inv, const StreamFusion& fu) {
        // AHEAD tokens' sums at row `at` of the tile.  A few tokens a thread (FEW): all CTAs' partial sums of one token in
        // flight at a time; else three CTAs' of all four tokens (two at a time took o's eight splits of 64 rows from 6.8 to
        // 10.1 us).  FEW is the number of splits, so that nothing is skipped at run time: this code runs once in a block,
        // and twice as much of it for up to eight of them and four tokens cost a layer's products of 64 rows 2 to 6 %
        // (in a chain, 1B / 3B / 8B-sized: 46.8 / 66.0 / 107.7 us, now 45.4 / 62.5 / 102.8).
        auto sums = [&](float4 (&v)[AHEAD], int mb, int at) {
            auto place = [&](int u) { return min(mb + u * STEP, m_hi - 1) * TS_ROWS + at; };
            auto add = [](float4& a, const float4& b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; };
            if constexpr (!SPLIT || FEW > 0) {
                constexpr int MAXS = SPLIT ? FEW : 1;
#pragma unroll
                for (int u = 0; u < AHEAD; ++u) {
                    if (mb + u * STEP >= m_hi) break;
                    float4 p[MAXS];
#pragma unroll
                    for (int r = 0; r < MAXS; ++r) p[r] = load4(r, place(u));
                    v[u] = p[0];
#pragma unroll
                    for (int r = 1; r < MAXS; ++r) add(v[u], p[r]);
                }
            } else {
#pragma unroll
                for (int u = 0; u < AHEAD; ++u) v[u] = load4(0, place(u));
                for (int r0 = 1; r0 < splits; r0 += 3) {
                    float4 p[3][AHEAD];
#pragma unroll
                    for (int r = 0; r < 3; ++r)
#pragma unroll
                        for (int u = 0; u < AHEAD; ++u)
                            if (r0 + r < splits) p[r][u] = load4(r0 + r, place(u));
#pragma unroll
                    for (int r = 0; r < 3; ++r)
#pragma unroll
                        for (int u = 0; u < AHEAD; ++u)
                            if (r0 + r < splits) add(v[u], p[r][u]);
                }
            }
        };
        float norm[4] = {0.f, 0.f, 0.f, 0.f};
        if constexpr (EPI == TS_EPI_RESIDUAL) {
            if (fu.scaled_out)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (n0 + row + i < N) norm[i] = __ldg(fu.norm_w + n0 + row + i);
        }
        for (int mb = m_lo + m_off; mb - m_off < m_hi; mb += AHEAD * STEP) {
            const TileEpilogue now = *this;
            fetch(mb + AHEAD * STEP, m_hi, n0, N, out, ldo, vec, fu);
            float4 s0[AHEAD], s1[PAIRS ? AHEAD : 1];
            sums(s0, mb, row);
            if constexpr (PAIRS) sums(s1, mb, row + 8);
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                const int m = mb + u * STEP;
                if (m >= m_hi) break;                                        // the same for a whole warp, but for PAIRS
                const float sc = PRO == TS_PRO_SCALED ? inv[m] : 1.f;
                float a[4] = {s0[u].x * sc, s0[u].y * sc, s0[u].z * sc, s0[u].w * sc};
                if constexpr (PAIRS) {
                    const float b[4] = {s1[u].x * sc, s1[u].y * sc, s1[u].z * sc, s1[u].w * sc};
                    if constexpr (EPI == TS_EPI_SILU_MUL) {
                        float y[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) y[i] = a[i] / (1.f + expf(-a[i])) * b[i];
                        put4(out + (size_t)m * ldo + ((n0 + (row & ~15)) >> 1) + (row & 7), y, vec, N - (n0 + row + 8));
                    } else {
                        const int f = n0 + row;                              // output feature of the first pair's first element
                        if (f + 8 >= N) continue;
                        const int head = f / fu.d, e = f - head * fu.d;      // e: storage index inside the head (a multiple of 4)
                        float y0[4], y1[4];
                        if (head < fu.nh + fu.nkv) {
                            const float c[4] = {now.cosv[u].x, now.cosv[u].y, now.cosv[u].z, now.cosv[u].w};
                            const float sn[4] = {now.sinv[u].x, now.sinv[u].y, now.sinv[u].z, now.sinv[u].w};
#pragma unroll
                            for (int i = 0; i < 4; ++i) { y0[i] = a[i] * c[i] - b[i] * sn[i]; y1[i] = b[i] * c[i] + a[i] * sn[i]; }
                        } else {
#pragma unroll
                            for (int i = 0; i < 4; ++i) { y0[i] = a[i]; y1[i] = b[i]; }
                        }
                        bf16* dst = nullptr;
                        if (head < fu.nh) {
                            dst = reinterpret_cast<bf16*>(out) + (size_t)m * ldo + f;
                        } else if (now.slot[u] >= 0) {
                            const int kind = head < fu.nh + fu.nkv ? 0 : 1, kvh = head - fu.nh - kind * fu.nkv;
                            const int page = now.slot[u] / fu.page_size, off = now.slot[u] - page * fu.page_size;
                            dst = fu.kv_cache + ((((size_t)page * 2 + kind) * fu.nkv + kvh) * fu.page_size + off) * fu.d + e;
                        }
                        if (dst) {                                           // d % 16 == 0: the cache's places are 8-byte aligned
                            put4(dst, y0, vec, 4);
                            put4(dst + 8, y1, vec, 4);
                        }
                    }
                } else if constexpr (EPI == TS_EPI_RESIDUAL) {
                    const int n = n0 + row;
                    const float r[4] = {now.resid[u].x, now.resid[u].y, now.resid[u].z, now.resid[u].w};
                    float ssq = 0.f, y[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        a[i] = n + i < N ? r[i] + a[i] : 0.f;
                        ssq += a[i] * a[i];
                        y[i] = a[i] * norm[i];
                    }
                    put4(reinterpret_cast<float*>(out) + (size_t)m * ldo + n, a, vec, N - n);
                    if (fu.scaled_out) put4(fu.scaled_out + (size_t)m * ldo + n, y, vec, N - n);
                    ssq = warp_sum(ssq);
                    if ((threadIdx.x & 31) == 0) fu.ss_out[(size_t)tile * fu.ss_ld + m] = ssq;
                } else {
                    put4(out + (size_t)m * ldo + n0 + row, a, vec, N - (n0 + row));
                }
            }
        }
    }
};

// The 128 threads of an epilogue group.
__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory"); }

// Stages.  Eight splits of up to 64 tokens leave room for a second CTA on the SM (four stages of 24 KB): a cluster of eight
// large CTAs starts late, and the next kernel's can fetch its weights while this one's still run (a step of 64 rows of a
// 1B-sized model: 966 us, 1,177 with six; 17 rows by 2,048 x 16,384: 17.1 us, 26.5 with eight).  Two and four splits take
// six: 17 rows of 8B-sized o 10.9 us with four, 10.2 with six, a step of 17 rows of six 3B-sized layers 522 and 516.  Where
// a CTA's share of K is long (SPLIT 2) they take eight.
// Split products' partial sums take the stages' place.  few: the number of splits of up to 64 tokens.
__host__ __device__ constexpr int ts_groups(int split, int tok) { return tok > 128 && !split ? 3 : tok > 64 ? 2 : 1; }
__host__ __device__ constexpr int ts_threads(int split, int tok) { return tok > 64 ? 128 + 128 * ts_groups(split, tok) : 192; }
__host__ __device__ constexpr int ts_chunk(int tok) { return tok > 128 ? 32 : 64; }       // tokens an unsplit tile's epilogue takes at a time
__host__ __device__ constexpr int ts_stages(int split, int tok, int few) {
    return tok == 64 ? (!split && few == 1 ? 3 : split == 2 ? 8 : few == 8 ? 4 : 6) : tok == 128 ? (split ? 6 : 4) : (split ? 4 : 3);
}
__host__ __device__ constexpr size_t ts_smem(int split, int tok, int few) {
    return (size_t)ts_stages(split, tok, few) * (TS_ROWS + tok) * TS_BK * 2 + (split ? 0 : ts_groups(split, tok) * ts_chunk(tok) * TS_ROWS * 4) +
           8 * (2 * ts_stages(split, tok, few) + 4) + 1024;
}

// Rows of x in a box, and the MMA's N: what lies behind a part's tokens is neither fetched nor multiplied (175 tokens on 256
// columns: a third of the x traffic and of the MMAs' time).
__host__ __device__ __forceinline__ int ts_box(int tokens) { return (tokens + 15) & ~15; }

// FEW: the number of splits, or 0 where it is known at run time only; of unsplit products 0, or 1: two CTAs fit an SM.
template <int SPLIT, int FEW, int TOK, int EPI, int PRO, typename OUT>
__global__ void __launch_bounds__(ts_threads(SPLIT, TOK))
tc_stream_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                 OUT* __restrict__ out, int ldo, int M, int N, int K, int splits, int* err, StreamFusion fu) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ float inv_rms[TOK];
    constexpr int STAGES = ts_stages(SPLIT, TOK, FEW), GROUPS = ts_groups(SPLIT, TOK), TS_CHUNK = ts_chunk(TOK);
    constexpr uint32_t W_BYTES = TS_ROWS * TS_BK * 2, X_BYTES = TOK * TS_BK * 2, STAGE_BYTES = W_BYTES + X_BYTES;
    // blockIdx.y: one of gridDim.y parts of the tokens; everything below is about that part alone
    const int per_part = (M + (int)gridDim.y - 1) / (int)gridDim.y, part_lo = (int)blockIdx.y * per_part;
    M = min(per_part, M - part_lo);
    if (gridDim.y > 1) {
        out += (size_t)part_lo * ldo;
        if (EPI == TS_EPI_RESIDUAL) {
            if (fu.scaled_out) fu.scaled_out += (size_t)part_lo * ldo;
            fu.ss_out += part_lo;
        }
        if (EPI == TS_EPI_ROPE_CACHE) {
            fu.positions += part_lo;
            if (fu.slots) fu.slots += part_lo;
        }
        if (PRO == TS_PRO_SCALED) fu.ss_in += part_lo;
    }
    // the part's tokens in whole groups of 16, as the x boxes hold them (ts_box) and the MMA takes them
    const int n_mma = ts_box(per_part);
    const uint32_t stage_tx = W_BYTES + (uint32_t)n_mma * TS_BK * 2;
    static_assert(!SPLIT || (uint32_t)TOK * TS_ROWS * 4 <= STAGES * STAGE_BYTES, "the partial sums take the stages' place");
    const uint32_t base = (smem_addr(smem_raw) + 1023u) & ~1023u;          // swizzled tiles need 1024-byte alignment
    unsigned char* base_ptr = smem_raw + (base - smem_addr(smem_raw));
    // [TOK][TS_ROWS] over the stages, or [TS_CHUNK][TS_ROWS] per epilogue group behind them
    float* part = reinterpret_cast<float*>(base_ptr + (SPLIT ? 0 : STAGES * STAGE_BYTES));
    const uint32_t bars = base + STAGES * STAGE_BYTES + (SPLIT ? 0 : GROUPS * TS_CHUNK * TS_ROWS * 4);
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
    auto acc_full = [&](int b) { return bars + 8u * (2 * STAGES + b); };
    auto acc_empty = [&](int b) { return bars + 8u * (2 * STAGES + 2 + b); };
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = SPLIT ? (int)cluster_ctarank() : 0;
    const int n_tiles = (N + TS_ROWS - 1) / TS_ROWS;
    const int KT_all = (K + TS_BK - 1) / TS_BK;
    const int kt_lo = KT_all * rank / splits, kt_hi = KT_all * (rank + 1) / splits;       // this CTA's K range, in boxes
    const int KT = kt_hi - kt_lo;
    // split products: one tile per cluster; unsplit ones: tile after tile
    const int first_tile = SPLIT ? (int)(blockIdx.x / splits) : (int)blockIdx.x;
    const int tile_step = SPLIT ? n_tiles : (int)gridDim.x;
    constexpr uint32_t TMEM_COLS = SPLIT ? TOK : 2 * TOK;
    // The tokens that this thread's epilogue group writes: of a split tile the group's part of the CTA's share; of an unsplit one
    // every GROUPS-th chunk, from its own on.
    const int group = threadIdx.x < 128 ? 0 : ((int)threadIdx.x >> 7) - 1;
    const int cta_lo = M * rank / splits, cta_hi = M * (rank + 1) / splits;
    const int m_lo = SPLIT ? cta_lo + (cta_hi - cta_lo) * group / GROUPS : group * TS_CHUNK;
    const int m_hi = SPLIT ? cta_lo + (cta_hi - cta_lo) * (group + 1) / GROUPS : min(M, (group + 1) * TS_CHUNK);
    // four numbers of the output at a time
    const bool vec = ldo % 4 == 0 && ((uintptr_t)out & (4 * sizeof(OUT) - 1)) == 0 && (((uintptr_t)fu.scaled_out | (uintptr_t)fu.kv_cache) & 7) == 0;
    TileEpilogue<EPI, FEW == 8 ? 1 : (FEW > 1 ? 2 : 4)> epilogue((int)threadIdx.x & 127);

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 4 * GROUPS); }
        fence_barrier_init();
    }
    if (warp == 5) tmem_alloc(&tmem_base_slot, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;

    if (warp == 4 && lane == 0) {
        // ---- producer: W does not depend on the kernel before this one, x does: the first stages' W boxes are
        // requested before the wait, their x boxes after it (both count on the stage's barrier)
        int it = 0;
        bool ok = true, waited = false;
        int early = 0;
        if (first_tile < n_tiles) {
            for (; early < KT && early < STAGES; ++early) {
                mbar_expect_tx(full_bar(early), stage_tx);
                tma_load_2d(base + early * STAGE_BYTES, &map_w, full_bar(early), (kt_lo + early) * TS_BK, first_tile * TS_ROWS);
            }
        }
        pdl_wait();
        pdl_trigger();
        waited = true;
        for (int e = 0; e < early; ++e)
            tma_load_2d(base + e * STAGE_BYTES + W_BYTES, &map_x, full_bar(e), (kt_lo + e) * TS_BK, part_lo);
        for (int t = first_tile; t < n_tiles && ok; t += tile_step) {
            for (int kt = 0; kt < KT; ++kt, ++it) {
                if (it < early) continue;                                    // requested above
                const int s = it % STAGES, r = it / STAGES;
                if (r > 0 && !mbar_wait(empty_bar(s), (r & 1) ^ 1, err, 1, &abort_flag)) { ok = false; break; }
                mbar_expect_tx(full_bar(s), stage_tx);
                const uint32_t sa = base + s * STAGE_BYTES;
                tma_load_2d(sa, &map_w, full_bar(s), (kt_lo + kt) * TS_BK, t * TS_ROWS);
                tma_load_2d(sa + W_BYTES, &map_x, full_bar(s), (kt_lo + kt) * TS_BK, part_lo);
            }
        }
        (void)waited;
    } else {
        pdl_wait();
        pdl_trigger();
    }
    if (warp == 5 && lane == 0) {
        // ---- MMA issue: D[128 x n_mma] (+)= W[128 x 16] x[n_mma x 16]^T, four K steps per stage
        const uint32_t idesc = make_idesc(TS_ROWS, n_mma, false);
        int it = 0, local = 0;
        bool ok = true;
        for (int t = first_tile; t < n_tiles && ok; t += tile_step, ++local) {
            const int b = local & 1, u = local >> 1;
            if (u > 0 && !mbar_wait(acc_empty(b), (u & 1) ^ 1, err, 4, &abort_flag)) { ok = false; break; }
            tc_fence_after();
            const uint32_t tmem_d = tmem_base + (uint32_t)(b * TOK);
            for (int kt = 0; kt < KT; ++kt, ++it) {
                const int s = it % STAGES, r = it / STAGES;
                if (!mbar_wait(full_bar(s), r & 1, err, 2, &abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint32_t sa = base + s * STAGE_BYTES;
                const uint64_t adesc = desc_k_major(sa), bdesc = desc_k_major(sa + W_BYTES);
#pragma unroll
                for (int k = 0; k < TS_BK / 16; ++k)
                    tc_mma(tmem_d, adesc + 2u * k, bdesc + 2u * k, idesc, (kt > 0 || k > 0) ? 1u : 0u);
                tc_commit(empty_bar(s));
            }
            if (ok) tc_commit(acc_full(b));
        }
    } else if (warp < 4 || warp >= 8) {
        // ---- epilogue, first half: this warp's 32 rows of the accumulator into shared memory, token-major, so
        // that what follows reads and writes along rows of W
        int local = 0;
        bool ok = true;
        if (PRO == TS_PRO_SCALED) {
            // 1 / rms of every token from the producer's partial sums of squares, added in their order (every group all of
            // them: the same numbers, and no group waits for another)
            for (int m = threadIdx.x & 127; m < M; m += 128) {
                float ssq = 0.f;
#pragma unroll 8
                for (int p = 0; p < fu.ss_in_blocks; ++p) ssq += fu.ss_in[(size_t)p * fu.ss_ld + m];
                inv_rms[m] = rsqrtf(ssq / (float)K + fu.eps);
            }
        }
        for (int t = first_tile; t < n_tiles && ok; t += tile_step, ++local) {
            const int b = local & 1, u = local >> 1;
            epilogue.fetch(m_lo + epilogue.m_off, m_hi, t * TS_ROWS, N, out, ldo, vec, fu);
            if (!mbar_wait(acc_full(b), u & 1, err, 3, &abort_flag)) { ok = false; break; }
            tc_fence_after();
            const uint32_t tmem_d = tmem_base + (uint32_t)(b * TOK) + ((uint32_t)((warp & 3) * 32) << 16);
            const int row_of = (warp & 3) * 32 + lane;
            if (SPLIT) {
                // this group's share of the tokens (the stages' copies have landed and been multiplied)
#pragma unroll
                for (int c = 0; c < (TOK + 32 * GROUPS - 1) / (32 * GROUPS); ++c) {
                    const int t0 = (c * GROUPS + group) * 32;
                    if (t0 >= M) break;
                    uint32_t v[32];
                    tc_ld32(tmem_d + (uint32_t)t0, v);
#pragma unroll
                    for (int i = 0; i < 32; ++i) part[(t0 + i) * TS_ROWS + row_of] = __uint_as_float(v[i]);
                }
            } else {
                float* mine = part + group * TS_CHUNK * TS_ROWS;
                for (int m0 = group * TS_CHUNK; m0 < M; m0 += GROUPS * TS_CHUNK) {
                    // what was there has been written out
                    if (local > 0 || m0 >= GROUPS * TS_CHUNK) group_sync(group);
#pragma unroll
                    for (int c = 0; c < TS_CHUNK / 32; ++c) {
                        uint32_t v[32];
                        tc_ld32(tmem_d + (uint32_t)(m0 + c * 32), v);
#pragma unroll
                        for (int i = 0; i < 32; ++i) mine[(c * 32 + i) * TS_ROWS + row_of] = __uint_as_float(v[i]);
                    }
                    // ---- second half, unsplit: the group's warps write the chunk out
                    group_sync(group);
                    const int m1 = min(M, m0 + TS_CHUNK);
                    if (m0 >= GROUPS * TS_CHUNK) epilogue.fetch(m0 + epilogue.m_off, m1, t * TS_ROWS, N, out, ldo, vec, fu);
                    auto load4 = [&](int, int i) { return *reinterpret_cast<const float4*>(mine + i - m0 * TS_ROWS); };
                    epilogue.template write<false, 0, PRO>(load4, 1, out, ldo, N, t * TS_ROWS, t, m0, m1, vec, inv_rms, fu);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty(b));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (SPLIT) {
        // ---- second half, split over the cluster: CTA `rank` adds the partial sums of its share of the tokens
        cluster_sync_all();                                                 // every CTA's partial sums are in its shared memory
        if (first_tile < n_tiles && !abort_flag) {
            const int n0 = first_tile * TS_ROWS;
            const uint32_t mine = smem_addr(part);
            auto load4 = [&](int r, int i) { return ts_ld_remote4(mapa_shared(mine, (uint32_t)r) + (uint32_t)i * 4u); };
            if (warp < 4 || warp >= 8)
                epilogue.template write<true, FEW, PRO>(load4, splits, out, ldo, N, n0, first_tile, m_lo, m_hi, vec, inv_rms, fu);
        }
        cluster_sync_all();                                                 // nobody leaves while its partial sums are being read
    }
    if (abort_flag) {                                                       // give copies in flight time to land
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 5) {
        tc_fence_after();
        tmem_free(tmem_base, TMEM_COLS);
    }
}

static int ts_num_sms() {
    static int num_sms = 0;
    if (num_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || num_sms <= 0)
            num_sms = 148;
    }
    return num_sms;
}

template <int SPLIT, int FEW, int TOK, int EPI, int PRO, typename OUT>
static int launch_ts(const CUtensorMap& mw, const CUtensorMap& mx, OUT* out, int ldo, int M, int N, int K, int splits, int parts,
                     int* err, const StreamFusion& fu, cudaStream_t s) {
    constexpr size_t smem = ts_smem(SPLIT, TOK, FEW);
    static_assert(smem <= 227 * 1024, "shared memory of a block");
    auto kernel = tc_stream_kernel<SPLIT, FEW, TOK, EPI, PRO, OUT>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const int n_tiles = (N + TS_ROWS - 1) / TS_ROWS;
    const int sms = ts_num_sms();
    const int at_once = !SPLIT && FEW == 1 ? 2 * sms : sms;
    const unsigned grid = SPLIT ? (unsigned)(n_tiles * splits) : (unsigned)(n_tiles < at_once ? n_tiles : at_once);
    return rg_launch(kernel, dim3(grid, (unsigned)parts), dim3(ts_threads(SPLIT, TOK)), smem, s, splits, mw, mx, out, ldo, M, N, K, splits, err, fu);
}

static int ts_pick_splits(int splits, int N, int K, int M) {
    const int n_tiles = (N + TS_ROWS - 1) / TS_ROWS, kt = (K + TS_BK - 1) / TS_BK;
    if (splits == 0) {
        // As many CTAs per tile as keep the whole product in one wave of one CTA per SM, with at least two boxes of K each.
        // 64 rows by 2,048 x 2,048 / 2,048 x 8,192: 7.8 / 15.5 us with 4, 6.8 / 12.6 with 8; a second CTA per SM from one
        // product (16 splits' worth) only delays the product behind it (a 64-row step 1,281 against 1,333 us).
        splits = 1;
        // Above 64 rows a CTA fills an SM, and clusters of eight such start slowly (180 rows by 2,048 x 2,048: 11.5 us in
        // four splits, 23.9 in eight).
        const int most = M <= 64 ? TS_MAX_SPLITS : 4;
        while (splits < most && n_tiles * splits * 2 <= ts_num_sms() && kt >= splits * 4) splits *= 2;
    }
    if ((splits != 1 && splits != 2 && splits != 4 && splits != 8) || kt < splits) return -1;
    return splits;
}

template <int TOK, int EPI, int PRO, typename OUT>
static int dispatch_ts_tok(const void* x, int ldx, const CUtensorMap& mw, OUT* out, int ldo, int M, int N, int K, int splits,
                           int parts, int* err, const StreamFusion& fu, cudaStream_t s) {
    CUtensorMap mx;
    const int e = rg_make_map(&mx, x, M, K, ldx, ts_box((M + parts - 1) / parts));
    if (e) return e;
    if constexpr (TOK == 64) {
        // Many boxes of K a CTA: more copies in flight.  down with six / eight stages: 32 boxes (17 rows by 3,072 x 8,192) 14.16
        // / 14.18 us, 56 boxes (17 rows by 4,096 x 14,336) 24.8 / 24.3, 64 rows of it 26.8 / 26.2.
        const bool many = (K + TS_BK - 1) / TS_BK > 32 * splits;
#define TS_SPLITS(S_) (many ? launch_ts<2, S_, TOK, EPI, PRO, OUT>(mw, mx, out, ldo, M, N, K, S_, parts, err, fu, s) \
                            : launch_ts<1, S_, TOK, EPI, PRO, OUT>(mw, mx, out, ldo, M, N, K, S_, parts, err, fu, s))
        if (splits == 8) return launch_ts<1, 8, TOK, EPI, PRO, OUT>(mw, mx, out, ldo, M, N, K, 8, parts, err, fu, s);
        if (splits > 1) return splits == 2 ? TS_SPLITS(2) : TS_SPLITS(4);
#undef TS_SPLITS
        // More tiles than SMs, but not more than twice as many: all of them at once, two CTAs an SM with three stages each, where a
        // second round would leave half of the GPU idle (64 rows by 4,096 x 28,672, 224 tiles: 48.8 to 46.0 us, 17 rows 46.3 to 44.1)
        const int n_tiles = (N + TS_ROWS - 1) / TS_ROWS;
        if (n_tiles > ts_num_sms() && n_tiles <= 2 * ts_num_sms())
            return launch_ts<0, 1, TOK, EPI, PRO, OUT>(mw, mx, out, ldo, M, N, K, 1, parts, err, fu, s);
    }
    if constexpr (TOK > 64) {
        if (splits > 1) return launch_ts<1, 0, TOK, EPI, PRO, OUT>(mw, mx, out, ldo, M, N, K, splits, parts, err, fu, s);
    }
    return launch_ts<0, 0, TOK, EPI, PRO, OUT>(mw, mx, out, ldo, M, N, K, 1, parts, err, fu, s);
}

template <int EPI, int PRO, typename OUT>
static int dispatch_ts(const void* x, int ldx, const void* W, OUT* out, int ldo, int M, int N, int K, int splits,
                       int* err, const StreamFusion& fu, cudaStream_t s) {
    CUtensorMap mw;
    const int e = rg_make_map(&mw, W, N, K, K, TS_ROWS);
    if (e) return e;
    // Above 64 tokens a split product whose CTAs are fewer than half of the SMs takes the tokens in two parts: W crosses L2 twice,
    // but what a CTA fetches and writes is halved (175 rows by 2,048 x 2,048 11.1 to 10.3 us, by 8,192 x 2,048 19.9 to 17.7).
    const int n_tiles = (N + TS_ROWS - 1) / TS_ROWS;
    const int parts = M > 64 && splits > 1 && n_tiles * splits * 2 <= ts_num_sms() ? 2 : 1, per_part = (M + parts - 1) / parts;
    return per_part <= 64 ? dispatch_ts_tok<64, EPI, PRO, OUT>(x, ldx, mw, out, ldo, M, N, K, splits, parts, err, fu, s)
         : per_part <= 128 ? dispatch_ts_tok<128, EPI, PRO, OUT>(x, ldx, mw, out, ldo, M, N, K, splits, parts, err, fu, s)
                           : dispatch_ts_tok<256, EPI, PRO, OUT>(x, ldx, mw, out, ldo, M, N, K, splits, parts, err, fu, s);
}

static bool ts_operands_ok(const void* x, int ldx, const void* W, int M, int K) {
    return M <= TS_MAX_TOK && K > 0 && K % 8 == 0 && ldx % 8 == 0 && !((uintptr_t)x & 15) && !((uintptr_t)W & 15);
}

// y = x W^T for 1 <= M <= 256 rows of x (bfloat16, rows ldx elements apart), W [N, K] bfloat16 contiguous.
// out_dtype: RG_DTYPE_BF16 or RG_DTYPE_F32; epilogue 0 plain (out [M, N]) or 1 SiLU-mul over interleaved gate|up
// rows (out [M, N / 2], bfloat16).  splits: 1, 2, 4 or 8 CTAs share a tile's K (K >= 64 x splits); 0 picks.
// ss_in (may be null): x holds residual rows times a norm's weight and ss_in [ss_in_blocks, ss_ld] their partial
// sums of squares; the sums are multiplied by 1 / rms (eps inside the root).  err: device int, non-zero afterwards
// if a wait gave up.
extern "C" int rg_tc_stream_gemm(const void* x, int ldx, const void* W, void* out, int ldo, int out_dtype, int epilogue,
                                 int M, int N, int K, int splits, const float* ss_in, int ss_in_blocks, int ss_ld,
                                 float eps, int* err, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (!ts_operands_ok(x, ldx, W, M, K)) return RG_ERR_UNSUPPORTED;
    if (epilogue == TS_EPI_SILU_MUL && (N % 16 || out_dtype != RG_DTYPE_BF16)) return RG_ERR_UNSUPPORTED;
    if (ss_in && (ss_in_blocks < 1 || ss_ld < M)) return RG_ERR_UNSUPPORTED;
    splits = ts_pick_splits(splits, N, K, M);
    if (splits < 0) return RG_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    StreamFusion fu = {};
    fu.ss_in = ss_in; fu.ss_in_blocks = ss_in_blocks; fu.ss_ld = ss_ld; fu.eps = eps;
#define RG_TS(EPI_, OUT_) (ss_in ? dispatch_ts<EPI_, TS_PRO_SCALED, OUT_>(x, ldx, W, (OUT_*)out, ldo, M, N, K, splits, err, fu, s) \
                                 : dispatch_ts<EPI_, TS_PRO_PLAIN, OUT_>(x, ldx, W, (OUT_*)out, ldo, M, N, K, splits, err, fu, s))
    if (epilogue == TS_EPI_SILU_MUL) return RG_TS(TS_EPI_SILU_MUL, bf16);
    if (epilogue != TS_EPI_NONE) return RG_ERR_UNSUPPORTED;
    if (out_dtype == RG_DTYPE_BF16) return RG_TS(TS_EPI_NONE, bf16);
    if (out_dtype == RG_DTYPE_F32) return RG_TS(TS_EPI_NONE, float);
#undef RG_TS
    return RG_ERR_UNSUPPORTED;
}

// The q|k|v projection of M tokens with the rotary encoding and the cache write in the product's epilogue:
// out [M, N] (bfloat16) receives the rotated q heads (its k and v columns are not written), k (rotated) and v go to
// kv_cache at slots (null: no write).  W's q and k rows are in the paired8 order.  ss_in as in rg_tc_stream_gemm.
extern "C" int rg_tc_stream_gemm_rope_cache(const void* x, int ldx, const void* W, void* out, int ldo, int M, int N, int K,
                                            int splits, const float* ss_in, int ss_in_blocks, int ss_ld, float eps,
                                            const float* rope_table, const int* positions, const int* slots,
                                            void* kv_cache, int nh, int nkv, int d, int page_size, int max_pos,
                                            int* pos_err, int* err, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (!ts_operands_ok(x, ldx, W, M, K) || d < 16 || d % 16 || nkv < 1 || nh < nkv || N != (nh + 2 * nkv) * d ||
        !rope_table || !positions || max_pos < 1 || (slots && (!kv_cache || page_size < 1)) ||
        (ss_in && (ss_in_blocks < 1 || ss_ld < M)))
        return RG_ERR_UNSUPPORTED;
    splits = ts_pick_splits(splits, N, K, M);
    if (splits < 0) return RG_ERR_UNSUPPORTED;
    StreamFusion fu = {};
    fu.ss_in = ss_in; fu.ss_in_blocks = ss_in_blocks; fu.ss_ld = ss_ld; fu.eps = eps;
    fu.rope_table = rope_table; fu.positions = positions; fu.slots = slots; fu.kv_cache = (bf16*)kv_cache;
    fu.nh = nh; fu.nkv = nkv; fu.d = d; fu.page_size = page_size; fu.max_pos = max_pos; fu.pos_err = pos_err;
    cudaStream_t s = (cudaStream_t)stream;
    return ss_in ? dispatch_ts<TS_EPI_ROPE_CACHE, TS_PRO_SCALED, bf16>(x, ldx, W, (bf16*)out, ldo, M, N, K, splits, err, fu, s)
                 : dispatch_ts<TS_EPI_ROPE_CACHE, TS_PRO_PLAIN, bf16>(x, ldx, W, (bf16*)out, ldo, M, N, K, splits, err, fu, s);
}

// resid [M, N] (32-bit, rows ldr apart) += x W^T, and the next RMSNorm prepared: scaled_out [M, N] (bfloat16, rows
// ldr apart) = bf16(resid * norm_w), ss_out [tiles of 128 columns, ss_ld >= M] = sums of squares of the new residual
// over each tile's columns.  *tiles_out receives the number of tiles.
extern "C" int rg_tc_stream_gemm_residual(const void* x, int ldx, const void* W, float* resid, int ldr,
                                          const float* norm_w, void* scaled_out, float* ss_out, int ss_ld, int M, int N,
                                          int K, int splits, int* tiles_out, int* err, void* stream) {
    if (tiles_out) *tiles_out = (N + TS_ROWS - 1) / TS_ROWS;
    if (M <= 0 || N <= 0) return 0;
    if (!ts_operands_ok(x, ldx, W, M, K) || ss_ld < M || !ss_out || !norm_w) return RG_ERR_UNSUPPORTED;
    splits = ts_pick_splits(splits, N, K, M);
    if (splits < 0) return RG_ERR_UNSUPPORTED;
    StreamFusion fu = {};
    fu.norm_w = norm_w; fu.scaled_out = (bf16*)scaled_out; fu.ss_out = ss_out; fu.ss_ld = ss_ld;
    return dispatch_ts<TS_EPI_RESIDUAL, TS_PRO_PLAIN, float>(x, ldx, W, resid, ldr, M, N, K, splits, err, fu,
                                                             (cudaStream_t)stream);
}
