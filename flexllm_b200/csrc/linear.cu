// C-ABI entry points of the W8A8 linear layers: shape checks, choice between the weight-streaming
// GEMV and the tcgen05 GEMM.
#include "common.cuh"

namespace flexllm {
int gemv_i8(const int8_t* a, const float* s_tok, const int8_t* w, const float* s_ch, int M, int N, int K,
            int32_t* acc, float* y, const float* residual, cudaStream_t st);
int gemm_i8_prefill(const int8_t* a, const float* s_tok, const int8_t* w, const float* s_ch, int M, int N, int K,
                    int32_t* acc, float* y, cudaStream_t st, const float* residual);
int gemm_i8_decode(const int8_t* a, const float* s_tok, const int8_t* w, const float* s_ch, int M, int N, int K,
                   int32_t* acc, float* y, cudaStream_t st, const float* residual);
}  // namespace flexllm

using namespace flexllm;

static int check_linear(const int8_t* a, const float* s_tok, const int8_t* w, const float* s_ch, int M, int N, int K,
                        int32_t* acc, float* y) {
    FLEXLLM_REQUIRE(a && w && (acc || y) && M >= 0 && N > 0 && K > 0);
    FLEXLLM_REQUIRE(!y || (s_tok && s_ch));
    FLEXLLM_REQUIRE((K % 16) == 0 && (N % 8) == 0);
    FLEXLLM_REQUIRE(aligned(a, 16) && aligned(w, 16) && (!acc || aligned(acc, 16)) && (!y || aligned(y, 16)) &&
                    (!s_ch || aligned(s_ch, 16)));
    return FLEXLLM_OK;
}

static int linear_prefill(const int8_t* a, const float* s_tok, const int8_t* w, const float* s_ch, int M, int N, int K,
                          int32_t* acc, float* y, const float* residual, void* stream) {
    int rc = check_linear(a, s_tok, w, s_ch, M, N, K, acc, y);
    if (rc != FLEXLLM_OK) return rc;
    FLEXLLM_REQUIRE(!residual || (y && aligned(residual, 16)));
    if (M == 0) return FLEXLLM_OK;
    return gemm_i8_prefill(a, s_tok, w, s_ch, M, N, K, acc, y, (cudaStream_t)stream, residual);
}

static int linear_decode(const int8_t* a, const float* s_tok, const int8_t* w, const float* s_ch, int M, int N, int K,
                         int32_t* acc, float* y, const float* residual, void* stream) {
    int rc = check_linear(a, s_tok, w, s_ch, M, N, K, acc, y);
    if (rc != FLEXLLM_OK) return rc;
    FLEXLLM_REQUIRE(!residual || y);
    if (M == 0) return FLEXLLM_OK;
    if (M > 64) return FLEXLLM_ENOTSUP;
    cudaStream_t st = (cudaStream_t)stream;
    // Up to eight tokens: the GEMV, whose dot products bind it from three tokens on, or the tensor-core form, which costs a few microseconds whatever
    // the tokens (us, GEMV / tensor cores: 3072x2048 4.2 / 6.9 for 3 tokens, 5.5 / 7.0 for 8; 4096x4096 8.9 / 8.9, 9.6 / 8.9; 16384x2048 10.6 / 10.9,
    // 14.7 / 11.0; 2048x8192 10.4 / 10.3, 13.5 / 10.4; 128256x2048 50 / 46, 81 / 47; 2 tokens 44.6 / 45.8 there). Behind other kernels of a chain
    // it has its weights early: MLP block of 3 tokens 22.4 / 17.9, of 8 32.4 / 18.7, of 2 17.5 / 17.9.
    const bool large = (long)N * K >= 12L << 20;
    if (M <= (large ? (in_chain() ? 2 : 3) : 8)) return gemv_i8(a, s_tok, w, s_ch, M, N, K, acc, y, residual, st);
    return gemm_i8_decode(a, s_tok, w, s_ch, M, N, K, acc, y, st, residual);
}

extern "C" int flexllm_linear_prefill_i8(const int8_t* a, const float* s_tok, const int8_t* w, const float* s_ch,
                                         int M, int N, int K, int32_t* acc, float* y, void* stream) {
    return linear_prefill(a, s_tok, w, s_ch, M, N, K, acc, y, nullptr, stream);
}
extern "C" int flexllm_linear_prefill_i8_residual(const int8_t* a, const float* s_tok, const int8_t* w, const float* s_ch,
                                                  int M, int N, int K, const float* residual, float* y, void* stream) {
    FLEXLLM_REQUIRE(residual);
    return linear_prefill(a, s_tok, w, s_ch, M, N, K, nullptr, y, residual, stream);
}
extern "C" int flexllm_linear_decode_i8(const int8_t* a, const float* s_tok, const int8_t* w, const float* s_ch,
                                        int M, int N, int K, int32_t* acc, float* y, void* stream) {
    return linear_decode(a, s_tok, w, s_ch, M, N, K, acc, y, nullptr, stream);
}
extern "C" int flexllm_linear_decode_i8_residual(const int8_t* a, const float* s_tok, const int8_t* w, const float* s_ch,
                                                 int M, int N, int K, const float* residual, float* y, void* stream) {
    FLEXLLM_REQUIRE(residual);
    return linear_decode(a, s_tok, w, s_ch, M, N, K, nullptr, y, residual, stream);
}

// ---- decode MLP block as one call -----------------------------------------------------------------------------------
namespace flexllm {
int swiglu_fht_quant_strided(const float* g, const float* u, long ld, int M, float scale, int8_t* q, float* s, cudaStream_t st);
static size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }
}  // namespace flexllm
extern "C" int flexllm_rmsnorm_quant(const float* x, const float* gamma, int M, int D, float eps, int order, float* y, int8_t* q,
                                     float* s, void* stream);

extern "C" size_t flexllm_mlp_block_workspace(int M, int D, int F) {
    if (M <= 0 || D <= 0 || F <= 0) return 0;
    return up256((size_t)M * D) + 2 * up256((size_t)M * 4) + up256((size_t)M * 2 * F * 4) + up256((size_t)M * F) + 256;
}

// RMSNorm + quant -> fused gate|up projection -> SiLU(gate) * up, FHT-8192, quant -> down projection + residual: the four
// launches follow one another with programmatic dependent launch, so each kernel's launch and, for the products, first weight
// loads overlap the tail of the one before.
extern "C" int flexllm_mlp_block_decode(const float* x, const float* gamma, const int8_t* w_gu, const float* s_gu, const int8_t* w_d,
                                        const float* s_d, int M, int D, int F, float eps, int order, float fht_scale, float* y,
                                        void* workspace, size_t workspace_bytes, void* stream) {
    FLEXLLM_REQUIRE(x && gamma && w_gu && s_gu && w_d && s_d && y && M >= 0 && D > 0);
    if (F != 8192) return FLEXLLM_ENOTSUP;
    if (M == 0) return FLEXLLM_OK;
    if (M > 64) return FLEXLLM_ENOTSUP;
    FLEXLLM_REQUIRE(workspace && workspace_bytes >= flexllm_mlp_block_workspace(M, D, F));
    uint8_t* w = (uint8_t*)(((uintptr_t)workspace + 255) & ~(uintptr_t)255);
    int8_t* xq = (int8_t*)w; w += up256((size_t)M * D);
    float* xs = (float*)w; w += up256((size_t)M * 4);
    float* hs = (float*)w; w += up256((size_t)M * 4);
    float* gu = (float*)w; w += up256((size_t)M * 2 * F * 4);
    int8_t* hq = (int8_t*)w;
    cudaStream_t st = (cudaStream_t)stream;
    // The products ask for their weights without waiting, and a caller's kernel may have written those just before: the first
    // kernel therefore lets the others start only when everything before it in the stream has completed.
    struct PdlScope { LaunchMode before; PdlScope() : before(g_pdl) { if (programmatic_launches()) g_pdl = kChain; } ~PdlScope() { g_pdl = before; } } pdl;
    TRY_RC(flexllm_rmsnorm_quant(x, gamma, M, D, eps, order, nullptr, xq, xs, st));
    TRY_RC(linear_decode(xq, xs, w_gu, s_gu, M, 2 * F, D, nullptr, gu, nullptr, st));
    TRY_RC(swiglu_fht_quant_strided(gu, gu + F, 2L * F, M, fht_scale, hq, hs, st));
    return linear_decode(hq, hs, w_d, s_d, M, D, F, nullptr, y, x, st);
}
