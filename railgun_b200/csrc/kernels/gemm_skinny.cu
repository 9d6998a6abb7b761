// The plain entry point of the weight-streaming decode product (gemm_skinny.cuh has the kernel).
#include "gemm_skinny.cuh"

// out_dtype: RG_DTYPE_BF16 or RG_DTYPE_F32.  epilogue: 0 plain (out [M, N]); 1 SiLU-mul over interleaved gate|up rows
// (out [M, N / 2]).  Refuses M > 64, K % 8 != 0 and, for the SiLU-mul epilogue, N % 16 != 0.
// bias (plain epilogue): [N] bfloat16 or null.  group_rows > 0 (plain epilogue): W holds groups of that many rows (a multiple
// of 32 that divides N), group i of which multiplies x + i group_x and goes to out + i group_out, [M, group_rows] there.
extern "C" int rg_skinny_gemm(const void* W, const void* x, int ldx, void* out, int ldo, int out_dtype, int epilogue,
                              int M, int N, int K, const void* bias, int group_rows, long long group_x, long long group_out,
                              void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (M > 64 || K % 8 || K <= 0 || ldx % 8) return RG_ERR_UNSUPPORTED;
    if (group_rows < 0 || (group_rows > 0 && (group_rows % 32 || N % group_rows || group_x % 8 || group_x < 0 || group_out < 0)))
        return RG_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    const bf16* w = (const bf16*)W;
    const bf16* xx = (const bf16*)x;
    SkinnyFusion fu = {};
    if (epilogue == EPI_SILU_MUL) {
        if (N % 16 || out_dtype != RG_DTYPE_BF16 || bias || group_rows) return RG_ERR_UNSUPPORTED;
        return dispatch_skinny<EPI_SILU_MUL, PRO_PLAIN, bf16>(w, xx, ldx, (bf16*)out, ldo, M, N, K, fu, nullptr, s);
    }
    if (epilogue != EPI_NONE) return RG_ERR_UNSUPPORTED;
    fu.bias = (const bf16*)bias;
    fu.group_rows = group_rows;
    fu.group_x = (size_t)group_x;
    fu.group_out = (size_t)group_out;
    if (out_dtype == RG_DTYPE_BF16) return dispatch_skinny<EPI_NONE, PRO_PLAIN, bf16>(w, xx, ldx, (bf16*)out, ldo, M, N, K, fu, nullptr, s);
    if (out_dtype == RG_DTYPE_F32) return dispatch_skinny<EPI_NONE, PRO_PLAIN, float>(w, xx, ldx, (float*)out, ldo, M, N, K, fu, nullptr, s);
    return RG_ERR_UNSUPPORTED;
}
