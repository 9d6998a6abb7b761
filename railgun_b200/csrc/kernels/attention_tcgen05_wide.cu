// Flash attention for portions of prompts on the 5th-generation tensor cores (bfloat16, head size 128).
//
// One CTA per SM takes 128 consecutive positions of one request and up to two heads that read the same key/value head
// (a "group" each: its own queries, softmax threads, accumulator and issuing warp), so a K/V tile is fetched once for
// both.  K and V come in stages of 128 keys (rings of three and two, TMA through the block table, one box per page and
// half of the head, 128-byte swizzle).  Per group and stage:
//   S = Q K^T            tcgen05.mma, M 128 x N 128 keys x K 128, into 128 TMEM columns
//   softmax              128 threads, one query row each, 64 keys at a time as in attention_tcgen05.cu: one pass with a
//                        reference maximum that is raised only when the 64 weights sum to more than 2^8
//   O += P V             tcgen05.mma, M 128 x N 128 x K 64 per half stage and twice: P is the sum of two bfloat16 numbers, in
//                        TMEM over the columns of the scores it was made from; O in 128 TMEM columns
// Two groups use all 512 columns.  A group's chain (scores, exponentials, product) is serial but for the product of a
// stage's first 64 keys, which runs under the second 64 keys' exponentials; the other group's exponentials run under
// its products and the other way round.
//
// What bounds it: per 64 keys and row tile the exponentials take 512 cycles of an SM's 16 lanes, the products 780 of its
// tensor core (N 128 is the narrowest shape at full rate: 65 cycles for 16 of K, N 64 takes 49), on different units.
// Measured (32 heads on 8, this kernel against attention_mma.cu's): 68 against 209 us for a prompt of 2,048 tokens (505
// against 164 TFLOP/s of the QK and PV that are needed), 154 against 631 us for 2,048 tokens behind 2,048, 680 against
// 2,989 us for 8,192 (808 TFLOP/s); 16 heads on 2, a window of 512: 36 against 71 us.  Shared memory (64 KB of queries,
// 160 KB of stages) and tensor memory allow one block per SM.
//
// Why two numbers a weight: under a reference that is the row's maximum the largest weight is 1, which bfloat16 holds; under
// one that is seldom raised it is any number up to 2^8 and loses 2^-9 like the others.  In the 2-norm against 64 bits
// (2,048 tokens, queries times 0.3 / 1 / 3): one number 2.07e-3 / 2.07e-3 / 2.14e-3, attention_mma.cu 2.07e-3 / 2.02e-3 /
// 1.76e-3, two numbers 1.56e-3 / 1.61e-3 / 1.65e-3, which is the rounding of the output.  The second product costs 4 to 12 %
// (2,048 tokens 61 to 68 us, 8,192 651 to 680); raising the reference for every new maximum would read and write O in
// nearly every pass, since one row of a warp's 32 has one.
//
// P is stored only once the 64 weights' sum is known to be small enough, because the scores under it are needed again
// otherwise.  Masks, sink, gate and the formulas are those of attention_mma.cu's prefill kernel (without pooled
// entries).  Every mbarrier wait is bounded and reports through *err (see gemm_tcgen05.cu).
#include "packed_f32.cuh"
#include "tcgen05.cuh"
#include <type_traits>

#define FW_BM 128                  // query rows of a group
#define FW_BN 64                   // keys per softmax pass
#define FW_D 128
#define FW_STAGE 128               // keys per K or V stage
#define FW_K_STAGES 3
#define FW_V_STAGES 2
#define FW_LOW 0x1p-17f             // see `consume`
#define FW_THREADS 352             // warps 0-3, 4-7: softmax of group 0, 1; 8: TMA; 9, 10: MMA issue of group 0, 1

// tiles: [NT][3] = first token row, rows (<= 128), request.  q_map: rows of queries, head h at column h * 128; kv_map:
// the cache as rows of 128, [pages * 2 * nkv * page_size, 128], box = min(page, 64) rows x 64 columns.
__global__ void __launch_bounds__(FW_THREADS, 1)
fa_wide_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap kv_map, bf16* __restrict__ out,
               int out_ld, const int* __restrict__ block_table, int max_blocks, const int* __restrict__ tiles,
               const int* __restrict__ positions, int nh, int nkv, int page_size, int window, int keep_first,
               float scale_log2, const float* __restrict__ sink, const bf16* __restrict__ gate, int gate_ld, float out_scale,
               int* err) {
    extern __shared__ unsigned char smem_raw[];
    constexpr uint32_t Q_BYTES = FW_BM * FW_D * 2, STAGE_BYTES = FW_STAGE * FW_D * 2;          // two halves of 64 columns each
    constexpr uint32_t Q_HALF = Q_BYTES / 2, KV_HALF = STAGE_BYTES / 2, SUB = FW_BN * 128;      // SUB: 64 keys of one half
    const uint32_t base = (smem_addr(smem_raw) + 1023u) & ~1023u;
    const uint32_t sQ = base, sK0 = sQ + 2 * Q_BYTES, sV0 = sK0 + FW_K_STAGES * STAGE_BYTES;
    const uint32_t bars = sV0 + FW_V_STAGES * STAGE_BYTES;
    const uint32_t q_full = bars, k_full0 = bars + 8, k_empty0 = k_full0 + 8 * FW_K_STAGES, v_full0 = k_empty0 + 8 * FW_K_STAGES,
                   v_empty0 = v_full0 + 8 * FW_V_STAGES, s_full0 = v_empty0 + 8 * FW_V_STAGES;   // s_full per group
    const uint32_t p_full0 = s_full0 + 16, p_free0 = p_full0 + 32;                              // per group and half stage
    static_assert(8 + 16 * (FW_K_STAGES + FW_V_STAGES) + 16 + 64 <= 256, "the barriers have 256 bytes");
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = nh / nkv, pairs = (group + 1) / 2, per_tile = nkv * pairs;
    // later tiles of a prompt attend more keys: every head's last tile starts first (blocks are handed out in order)
    const int tile = gridDim.x / per_tile - 1 - blockIdx.x / per_tile, part = blockIdx.x % per_tile;
    const int kvh = part / pairs, h0 = kvh * group + 2 * (part % pairs);
    const int n_groups = min(2, group - 2 * (part % pairs));
    const int row0 = tiles[tile * 3 + 0], nrows = tiles[tile * 3 + 1], r = tiles[tile * 3 + 2];
    const int* bt = block_table + (size_t)r * max_blocks;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        mbar_init(q_full, 1);
        for (int s = 0; s < FW_K_STAGES; ++s) { mbar_init(k_full0 + 8 * s, 1); mbar_init(k_empty0 + 8 * s, n_groups); }
        for (int s = 0; s < FW_V_STAGES; ++s) { mbar_init(v_full0 + 8 * s, 1); mbar_init(v_empty0 + 8 * s, n_groups); }
        for (int g = 0; g < 2; ++g) mbar_init(s_full0 + 8 * g, 1);
        for (int b = 0; b < 4; ++b) { mbar_init(p_full0 + 8 * b, FW_BM); mbar_init(p_free0 + 8 * b, 1); }
        fence_barrier_init();
    }
    if (warp == 9) tmem_alloc(&tmem_base_slot, 512u);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // group g: scores and weights in columns [256 g, 256 g + 128), O in [256 g + 128, 256 g + 256)
    const uint32_t tmem = tmem_base_slot;
    // Tiles, positions and block tables were written before the step's first kernel started: they are read before the
    // wait for the kernel before this one; only what moves q, K, V or the output comes after it.
    const int p0 = positions[row0];
    const int hi = p0 + nrows - 1;
    const int lo = first_seen(p0, window), lo_last = first_seen(hi, window);
    // Passes over 64 keys: those that hold kept first tokens and end before the window, then the window's own.
    const int kt0 = lo / FW_BN, n_keep = window > 0 ? min((keep_first + FW_BN - 1) / FW_BN, kt0) : 0;
    const int n_kt = n_keep + hi / FW_BN - kt0 + 1, n_st = (n_kt + 1) / 2;
    auto first_key = [&](int j) -> int { return (j < n_keep ? j : kt0 + j - n_keep) * FW_BN; };

    if (warp == 8) {
        // ---- producer.  64 keys are 64 / rows_per_box boxes (a page, or 64 rows of a larger page) for each half of the
        // head; lane l fetches the page id of box l % boxes one pass ahead and issues that box of half l / boxes.
        const int rows_per_box = min(page_size, FW_BN), boxes = FW_BN / rows_per_box;           // 2 boxes <= 16 lanes
        const int box = lane % boxes, half = lane / boxes;
        const bool mine = half < 2;
        auto page_of = [&](int j) -> int {                                   // beyond the context: any page (masked)
            return mine && j < n_kt ? bt[min((first_key(j) + box * rows_per_box) / page_size, max_blocks - 1)] : 0;
        };
        int page_next[2] = {page_of(0), page_of(1)};
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&q_map)) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&kv_map)) : "memory");
        }
        pdl_wait();
        pdl_trigger();
        if (lane == 0) {
            mbar_expect_tx(q_full, (uint32_t)n_groups * Q_BYTES);
            for (int g = 0; g < n_groups; ++g)
                for (int x = 0; x < 2; ++x)
                    tma_load_2d(sQ + g * Q_BYTES + x * Q_HALF, &q_map, q_full, (h0 + g) * FW_D + 64 * x, row0);
        }
        bool ok = true;
        for (int J = 0; J < n_st && ok; ++J) {
            const int subs = min(2, n_kt - 2 * J);                            // a last half stage may be absent
            int page[2], in_page[2];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                page[t] = page_next[t];
                in_page[t] = (first_key(2 * J + t) + box * rows_per_box) % page_size;
                page_next[t] = page_of(2 * J + 2 + t);
            }
#pragma unroll
            for (int kv = 0; kv < 2; ++kv) {
                const int n_stages = kv ? FW_V_STAGES : FW_K_STAGES, s = J % n_stages, u = J / n_stages;
                const uint32_t full = (kv ? v_full0 : k_full0) + 8 * s, empty = (kv ? v_empty0 : k_empty0) + 8 * s;
                const uint32_t dst = (kv ? sV0 : sK0) + s * STAGE_BYTES + half * KV_HALF + box * rows_per_box * 128;
                if (u > 0) ok = mbar_wait_all(empty, (u & 1) ^ 1, err, 11 + kv, &abort_flag);
                if (!ok) break;
                if (lane == 0) mbar_expect_tx(full, (uint32_t)subs * 2u * SUB);
                __syncwarp();
                if (mine)
                    for (int t = 0; t < subs; ++t)
                        tma_load_2d(dst + t * SUB, &kv_map, full, 64 * half, ((page[t] * 2 + kv) * nkv + kvh) * page_size + in_page[t]);
            }
        }
    } else if (warp == 9 || warp == 10) {
        pdl_wait();
        // ---- MMA issue of one group.  The whole warp walks the loop and waits; one elected lane issues.
        const int g = warp - 9;
        const uint32_t tmem_s = tmem + 256u * g, tmem_o = tmem_s + 128u;
        constexpr uint32_t idesc_s = make_idesc(FW_BM, FW_STAGE, false), idesc_o = make_idesc(FW_BM, FW_D, true);
        const bool issuer = elect_one();
        auto issue_s = [&](int J) {                                           // K(J) is there
            const int s = J % FW_K_STAGES;
            if (issuer) {
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const uint64_t qd = desc_k_major(sQ + g * Q_BYTES + x * Q_HALF), kd = desc_k_major(sK0 + s * STAGE_BYTES + x * KV_HALF);
#pragma unroll
                    for (int k = 0; k < 4; ++k) tc_mma(tmem_s, qd + 2u * k, kd + 2u * k, idesc_s, x + k > 0 ? 1u : 0u);
                }
                tc_commit(s_full0 + 8 * g);
                tc_commit(k_empty0 + 8 * s);
            }
            __syncwarp();
        };
        bool ok = g < n_groups;
        if (ok) ok = mbar_wait_all(q_full, 0, err, 21, &abort_flag);
        if (ok) ok = mbar_wait_all(k_full0, 0, err, 22, &abort_flag);
        if (ok) { tc_fence_after(); issue_s(0); }
        for (int j = 0; j < n_kt && ok; ++j) {
            const int J = j >> 1, half = j & 1, s = J % FW_V_STAGES;
            if (half == 0) ok = mbar_wait_all(v_full0 + 8 * s, (J / FW_V_STAGES) & 1, err, 24, &abort_flag);
            if (ok && j == n_kt - 1) {
                // The rows of V behind the tile's last key are some other request's, or what an earlier one left: their
                // weights are 0, and 0 times an infinity is a NaN, so zeros take their place.  Both groups' warps may
                // write the same zeros.
                const int over0 = hi + 1 - first_key(j);
                for (int i = lane; i < (FW_BN - over0) * 16; i += 32) {
                    const int key = over0 + (i >> 4);                        // 8 pieces of 16 bytes in each half of a row
                    asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};"
                                 ::"r"(sV0 + s * STAGE_BYTES + half * SUB + ((i >> 3) & 1) * KV_HALF + key * 128 + (i & 7) * 16), "r"(0) : "memory");
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");    // before the product reads them
                __syncwarp();
            }
            const bool next = (half == 1 || j == n_kt - 1) && J + 1 < n_st;
            if (ok && next) ok = mbar_wait_all(k_full0 + 8 * ((J + 1) % FW_K_STAGES), ((J + 1) / FW_K_STAGES) & 1, err, 22, &abort_flag);
            if (ok) ok = mbar_wait_all(p_full0 + 16 * g + 8 * half, J & 1, err, 23, &abort_flag);
            if (!ok) break;
            tc_fence_after();
            if (issuer) {
#pragma unroll
                for (int k = 0; k < FW_BN / 16; ++k) {                       // 16 keys: 16 rows of V, 8 cells of P's halves each
                    const uint64_t vd = desc_mn_major(sV0 + s * STAGE_BYTES + half * SUB + (uint32_t)k * 2048u, KV_HALF);
                    const uint32_t pc = tmem_s + (uint32_t)(half * FW_BN + k * 8);
                    tc_mma_a_tmem(tmem_o, pc, vd, idesc_o, (j > 0 || k > 0) ? 1u : 0u);
                    tc_mma_a_tmem(tmem_o, pc + FW_BN / 2, vd, idesc_o, 1u);
                }
                tc_commit(p_free0 + 16 * g + 8 * half);
                if (half == 1 || j == n_kt - 1) tc_commit(v_empty0 + 8 * s);
            }
            __syncwarp();
            // S(J + 1) over the scores and weights of this stage: the tensor core takes it up after the product that reads them
            if (next) issue_s(J + 1);
        }
    } else if (warp / 4 < n_groups) {
        pdl_wait();
        // ---- softmax and output: thread = query row
        const int g = warp >> 2, row = threadIdx.x & 127, h = h0 + g;
        const int prow = p0 + row, seen0 = first_seen(prow, window);
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t tmem_sg = tmem + 256u * g + lane_off, tmem_o = tmem_sg + 128u;
        const uint32_t p_full = p_full0 + 16 * g, p_free = p_free0 + 16 * g;
        float m_ref = -INFINITY, l_run = 0.f;                                 // reference maximum (log2 domain), row sum
        bool ok = true;
        for (int j = 0; j < n_kt && ok; ++j) {
            const int J = j >> 1, half = j & 1, key_base = first_key(j);
            const uint32_t tmem_s = tmem_sg + (uint32_t)(half * FW_BN);
            if (half == 0) {
                ok = mbar_wait_all(s_full0 + 8 * g, J & 1, err, 31, &abort_flag);
                if (!ok) break;
                tc_fence_after();
            }
            // Passes whose keys every row of the CTA sees take the short path; the others mask by absolute position.
            const bool edge = key_base + FW_BN - 1 > p0 || (key_base < lo_last && key_base + FW_BN > (window > 0 ? keep_first : 0));
            const int k_hi = prow - key_base, k_lo = seen0 - key_base, k_keep = window > 0 ? keep_first - key_base : 0;
            auto sees = [&](int col) -> bool { return col <= k_hi && (col >= k_lo || col < k_keep); };
            uint32_t pk[FW_BN / 2], lo[FW_BN / 2];
            // One pass: p = 2^(s scale - reference), as two bfloat16 numbers each into pk and lo; returns the row sum.
            auto exp_pass = [&](auto edge_c, float ms) -> float {
                constexpr bool EDGE = decltype(edge_c)::value;
                uint64_t rs2[4] = {0ull, 0ull, 0ull, 0ull};
                const uint64_t scale2 = pack2(scale_log2, scale_log2), nms2 = pack2(-ms, -ms);
                uint32_t v[2][32];
                tc_ld32_nowait(tmem_s, v[0]);
                tc_ld32_nowait(tmem_s + 32u, v[1]);
                tc_ld_wait();
                // groups of 16 columns, consumers one group behind the exponentials (see attention_tcgen05.cu)
                float p[2][16];
                auto exps = [&](int c) {
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        const int col = c * 16 + i;
                        float s0 = __uint_as_float(v[col >> 5][col & 31]), s1 = __uint_as_float(v[col >> 5][(col & 31) + 1]);
                        if (EDGE) {
                            if (!sees(col)) s0 = -INFINITY;
                            if (!sees(col + 1)) s1 = -INFINITY;
                        }
                        float t0, t1;
                        unpack2(fma2(pack2(s0, s1), scale2, nms2), t0, t1);
                        p[c & 1][i] = ex2_in_order(t0);
                        p[c & 1][i + 1] = ex2_in_order(t1);
                    }
                };
                // p = high + low: its upper 16 bits, and the rest rounded.  FW_LOW p is added to the rest, so that it is 0
                // only where p is (an infinity in a row of V that is seen stays one); the division at the end takes it out.
                const uint64_t one2 = pack2(1.f + FW_LOW, 1.f + FW_LOW);
                auto consume = [&](int c) {
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        const float p0 = p[c & 1][i], p1 = p[c & 1][i + 1];
                        const uint32_t b0 = __float_as_uint(p0), b1 = __float_as_uint(p1);
                        rs2[(i >> 1) & 3] = add2_in_order(rs2[(i >> 1) & 3], pack2(p0, p1));
                        pk[c * 8 + (i >> 1)] = __byte_perm(b0, b1, 0x7632);
                        float l0, l1;
                        unpack2(fma2(pack2(p0, p1), one2, pack2(__uint_as_float((b0 & 0xffff0000u) | 0x80000000u),
                                                                __uint_as_float((b1 & 0xffff0000u) | 0x80000000u))), l0, l1);
                        lo[c * 8 + (i >> 1)] = bf16x2_in_order(l0, l1);
                    }
                };
                exps(0);
                exps(1);
                consume(0);
                exps(2);
                consume(1);
                exps(3);
                consume(2);
                consume(3);
                float a, b;
                unpack2(add2(add2(rs2[0], rs2[1]), add2(rs2[2], rs2[3])), a, b);
                return a + b;
            };
            auto pass = [&](float ms) -> float {
                return edge ? exp_pass(std::true_type{}, ms) : exp_pass(std::false_type{}, ms);
            };
            bool redo = j == 0;
            float row_sum = 0.f;
            if (!redo) {
                row_sum = pass(m_ref == -INFINITY ? 0.f : m_ref);
                // also catches inf, NaN and a row that has seen no key so far and so has no reference; the lanes behind
                // the tile's rows hold some other request's queries and have no say in how this one's are rounded
                redo = __any_sync(0xffffffffu, row < nrows && (!(row_sum <= 256.f) || m_ref == -INFINITY));
            }
            if (redo) {
                // the row's maximum on the raw scores (scale > 0, so the maximum commutes with it)
                float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    uint32_t v[32];
                    tc_ld32(tmem_s + 32u * c, v);
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (!edge || sees(32 * c + i)) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(v[i]));
                }
                const float m_new = fmaxf(m_ref, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale_log2);
                if (j > 0) {
                    // rescale this warp's rows of O and the row sums: O must be complete through pass j - 1 (the product
                    // of pass j waits for this pass's P, so nothing else writes O meanwhile)
                    ok = mbar_wait_all(p_free + 8 * ((j - 1) & 1), ((j - 1) >> 1) & 1, err, 33, &abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    const float alpha = ex2(m_ref - (m_new == -INFINITY ? 0.f : m_new));
#pragma unroll
                    for (int c = 0; c < FW_D / 32; ++c) {
                        uint32_t o[32];
                        tc_ld32(tmem_o + (uint32_t)(c * 32), o);
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        tc_st32(tmem_o + (uint32_t)(c * 32), o);
                    }
                    tc_st_wait();
                    l_run *= alpha;
                }
                m_ref = m_new;
                row_sum = pass(m_ref == -INFINITY ? 0.f : m_ref);
            }
            l_run += row_sum;
            tc_st32(tmem_s, pk);
            tc_st32(tmem_s + FW_BN / 2, lo);
            tc_st_wait();
            tc_fence_before();
            mbar_arrive(p_full + 8 * half);                                   // this row's scores have been read, its weights written
        }
        if (ok) ok = mbar_wait_all(p_free + 8 * ((n_kt - 1) & 1), ((n_kt - 1) >> 1) & 1, err, 34, &abort_flag);
        if (ok) {
            tc_fence_after();
            float f = out_scale;
            if (sink) {                                                       // one more term of the denominator
                const float sk = sink[h] * 1.4426950408889634f, m = fmaxf(m_ref, sk), a = exp2f(m_ref - m);
                l_run = l_run * a + exp2f(sk - m);
                f *= a;
            }
            if (gate && row < nrows) f *= 1.f / (1.f + __expf(-__bfloat162float(gate[(size_t)(row0 + row) * gate_ld + h])));
            const float inv = l_run > 0.f ? f / (l_run * (1.f + FW_LOW)) : 0.f;
            bf16* dst = out + (size_t)(row0 + row) * out_ld + h * FW_D;
#pragma unroll
            for (int c = 0; c < FW_D / 32; ++c) {
                uint32_t o[32];
                tc_ld32(tmem_o + (uint32_t)(c * 32), o);                      // every lane takes part in the load
                if (row < nrows) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint4 w4;
                        uint32_t* w = reinterpret_cast<uint32_t*>(&w4);
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            __nv_bfloat162 hh = __floats2bfloat162_rn(__uint_as_float(o[i + 2 * t]) * inv, __uint_as_float(o[i + 2 * t + 1]) * inv);
                            w[t] = *reinterpret_cast<uint32_t*>(&hh);
                        }
                        *reinterpret_cast<uint4*>(dst + c * 32 + i) = w4;
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (abort_flag) {                                                         // give copies in flight time to land
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 9) {
        tc_fence_after();
        tmem_free(tmem, 512u);
    }
}

static const size_t FW_SMEM_BYTES =
    (size_t)2 * FW_BM * FW_D * 2 + (size_t)(FW_K_STAGES + FW_V_STAGES) * FW_STAGE * FW_D * 2 + 256 + 1024;

// q [n_rows_total, q_stride] (head h at column h * 128); out rows out_ld apart (nh * 128 numbers each);
// kv_cache [num_pages, 2, nkv, page_size, 128]; tiles [n_tiles][3] with at most 128 rows each; window, keep_first, sink,
// gate and out_scale as in attention_mma.cu.  Takes head size 128 and pages of 8, 16, 32, 64 and 128 tokens.
extern "C" int rg_prefill_attention_wide(const void* q, int q_stride, int n_rows_total, void* out, int out_ld,
                                         const void* kv_cache, int num_pages, const int* block_table, int max_blocks,
                                         const int* tiles, int n_tiles, const int* positions, int nh, int nkv, int d,
                                         int page_size, int window, int keep_first, float scale, const float* sink,
                                         const void* gate, int gate_ld, float out_scale, int* err, void* stream) {
    if (n_tiles <= 0) return 0;
    if (d != FW_D || nkv < 1 || nh < nkv || nh % nkv || page_size < 8 || page_size > 128 || 128 % page_size || q_stride % 8 ||
        out_ld % 8 || out_ld < nh * FW_D || keep_first < 0 || ((uintptr_t)q & 15) || ((uintptr_t)kv_cache & 15) ||
        ((uintptr_t)out & 15) || (long long)num_pages * 2 * nkv * page_size > 0x7fffffffll)
        return RG_ERR_UNSUPPORTED;
    const long long blocks = (long long)n_tiles * nkv * ((nh / nkv + 1) / 2);
    if (blocks > 0x7fffffffll) return RG_ERR_UNSUPPORTED;
    CUtensorMap qm, kvm;
    int e = rg_make_map(&qm, q, (unsigned long long)n_rows_total, (unsigned long long)nh * FW_D, (unsigned long long)q_stride, FW_BM);
    if (e) return e;
    e = rg_make_map(&kvm, kv_cache, (unsigned long long)num_pages * 2ull * nkv * page_size, FW_D, FW_D,
                    page_size < FW_BN ? page_size : FW_BN);
    if (e) return e;
    static unsigned long long smem_allowed = 0;                              // one bit per device: set once, not per call
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev > 63) dev = 63;
    if (dev == 63 || !(smem_allowed >> dev & 1ull)) {
        cudaError_t ce = cudaFuncSetAttribute(fa_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FW_SMEM_BYTES);
        if (ce != cudaSuccess) return (int)ce;
        smem_allowed |= 1ull << dev;
    }
    return rg_launch(fa_wide_kernel, dim3((unsigned)blocks), dim3(FW_THREADS), FW_SMEM_BYTES, (cudaStream_t)stream, 1, qm, kvm,
                     (bf16*)out, out_ld, block_table, max_blocks, tiles, positions, nh, nkv, page_size, window, keep_first,
                     scale * 1.4426950408889634f, sink, (const bf16*)gate, gate_ld, out_scale, err);
}
