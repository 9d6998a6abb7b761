// Token embedding: residual[t, :] = table[ids[t], :] * scale, written in 32-bit
// (crates/vllm-models/src/llama/architecture.rs:150 does the gather through the
// tensor library, without a factor: scale 1).
#include "common.cuh"

template <typename W>
__global__ void embed_kernel(const int* __restrict__ ids, const W* __restrict__ table,
                             float* __restrict__ out, int H, int V, float scale) {
    pdl_wait();
    pdl_trigger();
    const int t = blockIdx.x;
    const int id = ids[t];
    float* o = out + (size_t)t * H;
    if (id < 0 || id >= V) {                 // the host validates ids; never read outside the table
        for (int i = threadIdx.x; i < H; i += blockDim.x) o[i] = 0.f;
        return;
    }
    const W* row = table + (size_t)id * H;
    for (int i = threadIdx.x; i < H; i += blockDim.x) o[i] = to_f32(row[i]) * scale;
}

// The same for bfloat16 rows that start on 8-byte boundaries, four numbers a load.  What bounds it at a few tokens is the chain
// id -> row (two trips to memory), so a thread has all of its row's loads under way at once; at many, their bytes.  Rows of
// 2,048, one after another from a warm L2: 2.4 us for one token with single numbers, 1.4 with four; 5.5 and 3.9 for 2,048.
#define EMBED_AT_ONCE 4
__global__ void embed_vec4_kernel(const int* __restrict__ ids, const bf16* __restrict__ table, float* __restrict__ out, int H, int V,
                                  float scale) {
    pdl_wait();
    pdl_trigger();
    const int t = blockIdx.x, quads = H >> 2;
    const int id = ids[t];
    const bool there = id >= 0 && id < V;                  // the host validates ids; never read outside the table
    const uint2* row = (const uint2*)(table + (size_t)(there ? id : 0) * H);
    float4* o = (float4*)(out + (size_t)t * H);
    for (int i0 = threadIdx.x; i0 < quads; i0 += EMBED_AT_ONCE * blockDim.x) {
        uint2 v[EMBED_AT_ONCE];
#pragma unroll
        for (int j = 0; j < EMBED_AT_ONCE; ++j)
            if (there && i0 + j * blockDim.x < quads) v[j] = row[i0 + j * blockDim.x];
#pragma unroll
        for (int j = 0; j < EMBED_AT_ONCE; ++j) {
            if (i0 + j * blockDim.x >= quads) break;
            o[i0 + j * blockDim.x] = there ? make_float4(__uint_as_float(v[j].x << 16) * scale, __uint_as_float(v[j].x & 0xffff0000u) * scale,
                                                         __uint_as_float(v[j].y << 16) * scale, __uint_as_float(v[j].y & 0xffff0000u) * scale)
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
}

extern "C" int rg_embedding(const int* ids, const void* table, int table_dtype, float* out,
                            int T, int H, int V, float scale, void* stream) {
    if (T <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    const int threads = H >= 1024 ? 256 : 128;
    if (table_dtype == RG_DTYPE_BF16 && H % 4 == 0 && ((uintptr_t)table & 7u) == 0 && ((uintptr_t)out & 15u) == 0)
        return rg_launch(embed_vec4_kernel, dim3(T), dim3(threads), 0, s, 1, ids, (const bf16*)table, out, H, V, scale);
    if (table_dtype == RG_DTYPE_BF16)
        return rg_launch(embed_kernel<bf16>, dim3(T), dim3(threads), 0, s, 1, ids, (const bf16*)table, out, H, V, scale);
    if (table_dtype == RG_DTYPE_F32)
        return rg_launch(embed_kernel<float>, dim3(T), dim3(threads), 0, s, 1, ids, (const float*)table, out, H, V, scale);
    return RG_ERR_UNSUPPORTED;
}
