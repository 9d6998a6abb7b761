// The experts' products of prompts on CTA pairs of the 5th-generation tensor cores, operands swapped: for every tile of up to 256
// places of one expert, 256 rows of the expert's matrix fill the M side of tcgen05.mma (cta_group::2: 128 rows a CTA) and the
// tile's places its N side, in steps of 32, so that an expert with 270 places costs 256 + 32 columns and not three tiles of
// 128 rows.  D[256 rows of W, places] accumulates in tensor memory, two tiles in turn, so that a tile's epilogue overlaps the
// next tile's products.
//
// What bounds it: every byte of the experts' matrices once from HBM (32 experts of 4,096 x 2,048: 537 MB, 82 us) beside as much time
// of the tensor cores (8,192 places: 84 us), and what crosses L2 -> SM, which this form cuts: a pair's tile of 256 x 256 fetches
// 1,024 bytes of operands per number of k for 65,536 results where one CTA's tile of 128 x 256 fetched 768 for 32,768.  Gate and up rows meet in the
// epilogue: the tensor map walks the matrix [gate rows; up rows] in blocks of 8 gate and the 8 matching up rows, so that lanes
// l and l + 8 of a warp hold a pair, and the activation is applied to 32-bit sums and written once.  2,048 tokens with four choices
// each among 32 experts: gathered rows by 4,096 x 2,048 with the activation 222 us as tiles of 128 x 256 a CTA with a kernel behind
// them, 203 here; by 2,048 x 2,048 101 and 91.
//
// Roles, barriers and bounded waits as in gemm_tcgen05.cu's pair kernel.  No multicast: each CTA fetches what it holds.
#include "tcgen05.cuh"

#define GP_THREADS 192            // warps 0-3: epilogue; warp 4: TMA producer; warp 5: MMA issue and TMEM owner
#define GP_ROWS 128               // rows of W per CTA
#define GP_BK 64
#define GP_PLACES 256             // places per tile, at most
#define GP_BOX 32                 // places per box: a CTA holds half of a tile's places, in one to four boxes
#define GP_STAGES 6
#define GP_W_BYTES (GP_ROWS * GP_BK * 2)
#define GP_STAGE_BYTES (GP_W_BYTES + (GP_PLACES / 2) * GP_BK * 2)
#define GP_SMEM (GP_STAGES * GP_STAGE_BYTES + 8 * (2 * GP_STAGES + 4) + 1024)

// tiles [max_tiles][3] = (expert, or -1 from the first unused entry on; first place; places <= 256).  GATED: out [places, F], F =
// half of W's rows per expert; else out [places, rows].  w_tiles: tiles of 256 rows of W per expert.
template <bool GATED>
__global__ void __launch_bounds__(GP_THREADS)
tc_grouped_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, bf16* __restrict__ out,
                  int ldo, int n_out, int K, const int* __restrict__ tiles, int max_tiles, int w_tiles, int act, float limit, int* err) {
    extern __shared__ unsigned char smem_raw[];
    const uint32_t base = (smem_addr(smem_raw) + 1023u) & ~1023u;
    const uint32_t bars = base + GP_STAGES * GP_STAGE_BYTES;
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (GP_STAGES + s); };
    auto acc_full = [&](int b) { return bars + 8u * (2 * GP_STAGES + b); };
    auto acc_empty = [&](int b) { return bars + 8u * (2 * GP_STAGES + 2 + b); };
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int KT = (K + GP_BK - 1) / GP_BK;
    const int total = max_tiles * w_tiles;                                  // rows of W fastest: a tile's places stay in L2
    constexpr uint32_t TMEM_COLS = 2 * GP_PLACES;
    // half of a tile's places, which a CTA holds: the pair's N in steps of 32
    auto half_of = [](int places) { return ((places + 31) & ~31) >> 1; };

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < GP_STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 8); }
        fence_barrier_init();
    }
    if (warp == 5) tmem_alloc_pair(&tmem_base_slot, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                                     // both CTAs' barriers exist before either is used
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    pdl_wait();                                                             // the places and their tiles are earlier kernels' work
    pdl_trigger();

    if (warp == 4 && lane == 0) {
        int it = 0;
        bool ok = true;
        for (int t = pair; t < total && ok; t += n_pairs) {
            const int* tl = tiles + 3 * (t / w_tiles);
            const int e = tl[0], wt = t % w_tiles;
            if (e < 0) break;                                               // every role ends at the same entry
            const int half = half_of(tl[2]), boxes = (half + GP_BOX - 1) / GP_BOX, first = tl[1] + (int)rank * half;
            const uint32_t tx = 2u * (GP_W_BYTES + (uint32_t)boxes * GP_BOX * GP_BK * 2);
            for (int kt = 0; kt < KT; ++kt, ++it) {
                const int s = it % GP_STAGES, r = it / GP_STAGES;
                if (r > 0 && !mbar_wait(empty_bar(s), (r & 1) ^ 1, err, 1, &abort_flag)) { ok = false; break; }
                if (rank == 0) mbar_expect_tx(full_bar(s), tx);
                const uint32_t sa = base + s * GP_STAGE_BYTES, full0 = mapa_shared(full_bar(s), 0);
                if (GATED) tma_load_5d_pair(sa, &map_w, full0, kt * GP_BK, 0, 0, wt * 16 + (int)rank * 8, e);
                else tma_load_3d_pair(sa, &map_w, full0, kt * GP_BK, wt * 2 * GP_ROWS + (int)rank * GP_ROWS, e);
                for (int j = 0; j < boxes; ++j)
                    tma_load_2d_pair(sa + GP_W_BYTES + j * (GP_BOX * GP_BK * 2), &map_x, full0, kt * GP_BK, first + j * GP_BOX);
            }
        }
    } else if (warp == 5 && lane == 0 && rank == 0) {
        // ---- MMA issue for the pair: D[256 x 2 half] (+)= W[256 x 16] places[2 half x 16]^T
        int it = 0, local = 0;
        bool ok = true;
        for (int t = pair; t < total && ok; t += n_pairs, ++local) {
            const int* tl = tiles + 3 * (t / w_tiles);
            if (tl[0] < 0) break;
            const uint32_t idesc = make_idesc(2 * GP_ROWS, 2 * half_of(tl[2]), false);
            const int b = local & 1, u = local >> 1;
            if (u > 0 && !mbar_wait(acc_empty(b), (u & 1) ^ 1, err, 4, &abort_flag)) { ok = false; break; }
            tc_fence_after();
            const uint32_t tmem_d = tmem_base + (uint32_t)(b * GP_PLACES);
            for (int kt = 0; kt < KT; ++kt, ++it) {
                const int s = it % GP_STAGES, r = it / GP_STAGES;
                if (!mbar_wait(full_bar(s), r & 1, err, 2, &abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint32_t sa = base + s * GP_STAGE_BYTES;
                const uint64_t adesc = desc_k_major(sa), bdesc = desc_k_major(sa + GP_W_BYTES);
#pragma unroll
                for (int k = 0; k < GP_BK / 16; ++k)
                    tc_mma_pair(tmem_d, adesc + 2u * k, bdesc + 2u * k, idesc, (kt > 0 || k > 0) ? 1u : 0u);
                tc_commit_pair(empty_bar(s), 3);
            }
            if (ok) tc_commit_pair(acc_full(b), 3);
        }
    } else if (warp < 4) {
        // ---- epilogue (both CTAs): a lane is a row of W, a column a place
        int local = 0;
        bool ok = true;
        for (int t = pair; t < total && ok; t += n_pairs, ++local) {
            const int* tl = tiles + 3 * (t / w_tiles);
            if (tl[0] < 0) break;
            const int first = tl[1], places = tl[2], wt = t % w_tiles;
            const int b = local & 1, u = local >> 1;
            if (!mbar_wait(acc_full(b), u & 1, err, 3, &abort_flag)) { ok = false; break; }
            tc_fence_after();
            const int row = warp * 32 + lane;                               // within the CTA's 128
            const int n = GATED ? wt * GP_ROWS + (int)rank * (GP_ROWS / 2) + (row >> 4) * 8 + (row & 7)
                                : (wt * 2 + (int)rank) * GP_ROWS + row;
            const uint32_t tmem_d = tmem_base + (uint32_t)(b * GP_PLACES) + ((uint32_t)(warp * 32) << 16);
            bf16* o = out + (size_t)first * ldo + n;
#pragma unroll 1
            for (int c0 = 0; c0 < places; c0 += 32) {
                uint32_t v[32];
                tc_ld32(tmem_d + (uint32_t)c0, v);
                if (GATED) {
                    // lanes l (gate) and l + 8 (up) hold a pair: the first takes the chunk's places 0 .. 15, the second 16 .. 31
                    const bool up = (lane & 8) != 0;
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float give = __uint_as_float(up ? v[j] : v[j + 16]);
                        const float got = __shfl_xor_sync(0xffffffffu, give, 8);
                        const float g = up ? got : __uint_as_float(v[j]), uu = up ? __uint_as_float(v[j + 16]) : got;
                        const int place = c0 + j + (up ? 16 : 0);
                        if (place < places && n < n_out) o[(size_t)place * ldo] = __float2bfloat16_rn(gated_act(g, uu, act, limit));
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (c0 + j < places && n < n_out) o[(size_t)(c0 + j) * ldo] = __float2bfloat16_rn(__uint_as_float(v[j]));
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (rank == 0) mbar_arrive(acc_empty(b));
                else mbar_arrive_cluster(mapa_shared(acc_empty(b), 0));
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (abort_flag) {                                                       // give copies in flight time to land
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
        __syncthreads();
    }
    cluster_sync_all();                                                     // the other CTA's MMAs and arrivals are done with this one
    if (warp == 5) {
        tc_fence_after();
        tmem_free_pair(tmem_base, TMEM_COLS);
    }
}

static int gp_num_sms() {
    static int num_sms = 0;
    if (num_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || num_sms <= 0)
            num_sms = 148;
    }
    return num_sms;
}

// x [P, K] bfloat16: rows in group order, lda apart; W [groups, rows, K], `gated`: rows = gate rows, then as many up rows, and out
// [P, rows / 2] = act(gate) * up (act, limit: gated_act in common.cuh); else out [P, rows].  tiles as above, of at most 256 places.
// K % 8 == 0, lda % 8 == 0, 16-byte aligned x and W; gated: rows % 16 == 0.  Rows of out that belong to no tile are not written.
extern "C" int rg_tc_gemm_grouped(const void* x, int lda, int P, const void* W, int groups, int rows, int K, int gated, int act,
                                  float limit, void* out, int ldo, const int* tiles, int max_tiles, int* err, void* stream) {
    if (P <= 0 || rows <= 0 || max_tiles <= 0) return 0;
    if (K <= 0 || K % 8 || lda % 8 || ((uintptr_t)x & 15) || ((uintptr_t)W & 15) || groups < 1 || (gated && rows % 16))
        return RG_ERR_UNSUPPORTED;
    RgEncodeTiledFn fn = rg_encode_fn();
    if (!fn) return RG_ERR_UNSUPPORTED;
    CUtensorMap mx, mw;
    int e = rg_make_map(&mx, x, P, K, lda, GP_BOX);
    if (e) return e;
    const cuuint64_t k = K, F = rows / 2, row_bytes = (cuuint64_t)K * 2;
    CUresult r;
    if (gated) {
        // k, 8 rows, gate or up, blocks of 8 rows, experts: a box is 8 blocks of (8 gate rows, 8 up rows)
        const cuuint64_t dims[5] = {k, 8, 2, F / 8, (cuuint64_t)groups};
        const cuuint64_t strides[4] = {row_bytes, F * row_bytes, 8 * row_bytes, 2 * F * row_bytes};
        const cuuint32_t box[5] = {GP_BK, 8, 2, GP_ROWS / 16, 1}, estr[5] = {1, 1, 1, 1, 1};
        r = fn(&mw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(W), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    } else {
        const cuuint64_t dims[3] = {k, (cuuint64_t)rows, (cuuint64_t)groups};
        const cuuint64_t strides[2] = {row_bytes, (cuuint64_t)rows * row_bytes};
        const cuuint32_t box[3] = {GP_BK, GP_ROWS, 1}, estr[3] = {1, 1, 1};
        r = fn(&mw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(W), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    if (r != CUDA_SUCCESS) return 20000 + (int)r;
    const int w_tiles = (rows + 2 * GP_ROWS - 1) / (2 * GP_ROWS), n_out = gated ? rows / 2 : rows;
    const long long total = (long long)max_tiles * w_tiles;
    if (total > 0x7fffffffll) return RG_ERR_UNSUPPORTED;
    const int pairs = total < gp_num_sms() / 2 ? (int)total : gp_num_sms() / 2;
    auto kernel = gated ? tc_grouped_kernel<true> : tc_grouped_kernel<false>;
    cudaError_t ce = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GP_SMEM);
    if (ce != cudaSuccess) return (int)ce;
    return rg_launch(kernel, dim3(2 * pairs), dim3(GP_THREADS), (size_t)GP_SMEM, (cudaStream_t)stream, 2, mw, mx, (bf16*)out, ldo, n_out, K,
                     tiles, max_tiles, w_tiles, act, limit, err);
}
