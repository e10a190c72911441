// int8 x int8 -> int32 linear layer on the 5th-generation tensor cores (tcgen05, kind::i8).
//
//   acc[m][n] = sum_k a[m][k] * w[n][k]                    exact
//   y[m][n]   = ((float)acc * s_tok[m]) * s_ch[n]          fused epilogue
//
// One persistent CTA per SM, warp-specialised:
//   warp 0      TMA producer: 128-byte-swizzled K-major tiles of both operands, STAGES-deep ring
//   warp 1      MMA issuer (one thread): 4 x (128 x BN x 32) UMMAs per 128-byte K block into one of
//               two TMEM accumulators; also owns TMEM allocation
//   warps 2..5  epilogue: tcgen05.ld the finished accumulator (one TMEM lane = one output row per
//               thread), dequantise, store; runs while the MMA warp fills the other accumulator
//
// The "A side" is the UMMA M operand (128 rows per tile), the "B side" the N operand (BN rows).
//   prefill : A = activations [M][K], B = weights [N][K]            out[rowA][rowB]
//   decode  : A = weights [N][K],     B = activations [M<=64][K]     out[rowB][rowA]   (SWAP)
// so that a handful of tokens still fills the 128-row dimension of the tensor core with weight
// rows and the weight matrix is streamed exactly once. With split-K (decode) the splits of a tile form a thread-block
// cluster of up to four: each CTA leaves its int32 partial tile in shared memory and the cluster's CTAs add them, a share of
// the tokens each, over distributed shared memory. (Adding into a buffer in global memory, with the last arriver reading it back, took
// 26 us for 64 tokens of 2048 x 8192.) The allocation-free entry point keeps the form that adds into a zeroed buffer.
//
// Replaces pref_Linear_Layer_i4xi4 / dec_Linear_Layer_i4xi4 + the dequant layers
// (Modules/Linear_Layer.h:293-341, :862-923; Modules/quant.h:115-164, :434-524) at 8-bit precision.
#include <atomic>
#include <cstdlib>
#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "fht_core.cuh"
#include "tc_common.cuh"

namespace flexllm {

using namespace tc;

// ------------------------------------------------------------------ tensor-map encoding (host)
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    });
    return fn;
}

int make_tmap_2d_u8_box(CUtensorMap* out, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_bytes,
                        uint32_t box_rows, int swizzle_bytes) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return FLEXLLM_ECUDA;
    if (!aligned(base, 16) || (row_bytes % 16) != 0 || box_rows == 0 || box_rows > 256) return FLEXLLM_EINVAL;
    if ((swizzle_bytes != 64 && swizzle_bytes != 128) || box_bytes == 0 || box_bytes > (uint32_t)swizzle_bytes || (box_bytes % 16) != 0)
        return FLEXLLM_EINVAL;
    cuuint64_t dims[2] = {row_bytes, rows};
    cuuint64_t strides[1] = {row_bytes};
    cuuint32_t box[2] = {box_bytes, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE,
                    swizzle_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { g_last_cuda_error = (int)r; return FLEXLLM_ECUDA; }
    return FLEXLLM_OK;
}

int make_tmap_3d_u8(CUtensorMap* out, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows, uint32_t kch) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return FLEXLLM_ECUDA;
    if (!aligned(base, 16) || (row_bytes % 128) != 0 || box_rows == 0 || box_rows > 256 || kch == 0 || kch > 8) return FLEXLLM_EINVAL;
    cuuint64_t dims[3] = {128, rows, row_bytes / 128};
    cuuint64_t strides[2] = {row_bytes, 128};
    cuuint32_t box[3] = {128, box_rows, kch};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { g_last_cuda_error = (int)r; return FLEXLLM_ECUDA; }
    return FLEXLLM_OK;
}

int make_tmap_rows3_u8(CUtensorMap* out, const void* base, uint64_t outer, uint64_t mid, uint64_t row_bytes, uint32_t box_outer,
                       uint32_t box_mid) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return FLEXLLM_ECUDA;
    if (!aligned(base, 16) || (row_bytes % 16) != 0 || box_outer == 0 || box_mid == 0 || box_outer > 256 || box_mid > 256) return FLEXLLM_EINVAL;
    cuuint64_t dims[3] = {row_bytes, mid, outer};
    cuuint64_t strides[2] = {row_bytes, row_bytes * mid};
    cuuint32_t box[3] = {128, box_mid, box_outer};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { g_last_cuda_error = (int)r; return FLEXLLM_ECUDA; }
    return FLEXLLM_OK;
}

int make_tmap_2d_u8(CUtensorMap* out, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows) {
    return make_tmap_2d_u8_box(out, base, rows, row_bytes, 128, box_rows, 128);
}

// ------------------------------------------------------------------ kernel
struct GemmArgs {
    int rowsA, rowsB, K;     // A side (128-row tiles), B side (BN-row tiles), reduction length
    int tilesA, tilesB, ksplit;
    int ldo;                 // leading dimension of the outputs
    int32_t* acc;            // optional int32 output (required when ksplit > 1 without a cluster: added atomically)
    float* y;                // optional fp32 output (ignored in that case)
    const float* sA;         // per-row scale of the A side
    const float* sB;         // per-row scale of the B side
    int* error_flag;         // set to 1 if a device-side wait ran out
    // fused epilogue extras
    const float* residual;   // optional: y = residual + dequant (same layout as y)
    int ahead;               // decode orientation: the kernels in front may still run when this one starts (programmatic launch)
    int cluster;             // split-K: the splits of a tile are a thread-block cluster (else they add into acc)
};

// KCH = 128-byte K chunks per pipeline stage (1 for prefill; > 1 for the weight-streaming decode
// orientation, where fetching KCH*128 contiguous bytes per weight row keeps HBM pages open).
template <int BN, int KCH = 1> struct GemmCfg {
    static constexpr int A_TILE = 128 * 128;
    static constexpr int B_TILE = BN * 128;
    static constexpr int A_BYTES = KCH * A_TILE;
    static constexpr int B_BYTES = KCH * B_TILE;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int STAGES_MAX = (200 * 1024) / STAGE_BYTES;
    static constexpr int STAGES = KCH > 1 ? (STAGES_MAX > 8 ? 8 : STAGES_MAX)
                                          : (BN == 256 ? 4 : BN == 128 ? 6 : BN == 64 ? 8 : BN == 32 ? 8 : 10);
    static constexpr int TMEM_COLS = 2 * BN < 32 ? 32 : 2 * BN;
    // prefill orientation: per-warp staging (32 rows x 32 fp32, plus the tile's column scales) that turns the accumulator rows a thread
    // owns into row-contiguous 128-byte global stores
    static constexpr int STG_WARP_FLOATS = 32 * 32 + 256;      // one 32 x 32 chunk + the tile's column scales
    static constexpr int STG_BYTES = BN >= 32 ? 4 * STG_WARP_FLOATS * 4 : 0;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/ + STG_BYTES;
};

// ---- epilogue of the prefill orientation, one warp, rows row0 .. row0 + 31, columns col0 .. col0 + BN - 1 ----
// Before the accumulator is waited for: column scales of the tile into shared memory, and the residual rows into L2.
template <int BN> __device__ __forceinline__ void staged_prefetch(const GemmArgs& args, float* stg, int row0, int col0, int lane) {
    float* sbw = stg + 1024;
    if (args.sB)
        for (int i = lane; i < BN; i += 32) sbw[i] = col0 + i < args.rowsB ? args.sB[col0 + i] : 0.0f;
    if (args.residual) {
        for (int i = lane; i < 32 * (BN / 32); i += 32) {
            const int rr = i / (BN / 32), seg = i - rr * (BN / 32);
            const int row = row0 + rr, col = col0 + seg * 32;
            if (row < args.rowsA && col < args.rowsB)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(args.residual + (long)row * args.ldo + col));
        }
    }
}
// Lane = token row of the tile. 32 columns at a time are dequantised into this warp's staging buffer (16-byte granules
// XOR-swizzled by the row), then written out with every warp instruction covering 4 rows x 128 contiguous bytes (the direct
// form stores 32 rows x 16 bytes per instruction and was bound by the store path).
template <int BN>
__device__ __forceinline__ void staged_store(const GemmArgs& args, float* stg, const uint32_t tsrc, const int row0, const int col0, const float sa,
                                             const int lane) {
    const float* sbw = stg + 1024;
    const int rowA = row0 + lane;
    const bool rowA_ok = rowA < args.rowsA;
    __syncwarp();
    // the TMEM load of chunk c + 1 is in flight while chunk c is processed
    constexpr int NCH = BN / 32;
    auto process = [&](const uint32_t (&v)[32], const int c) {
        const int colB0 = col0 + c * 32;
        if (args.acc && rowA_ok) {
            const long o = (long)rowA * args.ldo + colB0;
#pragma unroll
            for (int j = 0; j < 32; j += 4)
                if (colB0 + j < args.rowsB)
                    *reinterpret_cast<int4*>(args.acc + o + j) = make_int4((int)v[j], (int)v[j + 1], (int)v[j + 2], (int)v[j + 3]);
        }
        if (args.y) {
            float* buf = stg;
            const int g = lane & 7;
            // this lane's share of the residual for the write-out below, requested first
            float4 rs[8];
            if (args.residual) {
#pragma unroll
                for (int it = 0; it < 8; it++) {
                    const int row = row0 + it * 4 + (lane >> 3), col = colB0 + 4 * g;
                    rs[it] = (row < args.rowsA && col < args.rowsB) ? *reinterpret_cast<const float4*>(args.residual + (long)row * args.ldo + col)
                                                                    : make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
#pragma unroll
            for (int gg = 0; gg < 8; gg++) {
                const float4 sb = *reinterpret_cast<const float4*>(sbw + c * 32 + 4 * gg);
                float4 r;
                r.x = ((float)(int)v[4 * gg] * sa) * sb.x;
                r.y = ((float)(int)v[4 * gg + 1] * sa) * sb.y;
                r.z = ((float)(int)v[4 * gg + 2] * sa) * sb.z;
                r.w = ((float)(int)v[4 * gg + 3] * sa) * sb.w;
                *reinterpret_cast<float4*>(buf + lane * 32 + ((gg ^ (lane & 7)) << 2)) = r;
            }
            __syncwarp();
#pragma unroll
            for (int it = 0; it < 8; it++) {
                const int rr = it * 4 + (lane >> 3);
                const int row = row0 + rr, col = colB0 + 4 * g;
                if (row < args.rowsA && col < args.rowsB) {
                    float4 r = *reinterpret_cast<const float4*>(buf + rr * 32 + ((g ^ (rr & 7)) << 2));
                    if (args.residual) { r.x = rs[it].x + r.x; r.y = rs[it].y + r.y; r.z = rs[it].z + r.z; r.w = rs[it].w + r.w; }
                    *reinterpret_cast<float4*>(args.y + (long)row * args.ldo + col) = r;
                }
            }
            __syncwarp();      // the staging buffer is reused by the next chunk
        }
    };
    uint32_t va[32], vb[32];
    tmem_ld_32x32(tsrc, va);
#pragma unroll 1
    for (int c = 0; c < NCH; c += 2) {
        tmem_ld_wait();
        if (c + 1 < NCH) tmem_ld_32x32(tsrc + (c + 1) * 32, vb);
        process(va, c);
        if (c + 1 < NCH) {
            tmem_ld_wait();
            if (c + 2 < NCH) tmem_ld_32x32(tsrc + (c + 2) * 32, va);
            process(vb, c + 1);
        }
    }
}

// The same for the fused gate | up product of the feed-forward block: columns 0..127 of the tile are gate channels f0 .. f0 + 127, columns 128..255
// the up channels of the same numbers, and what is stored is silu(gate) * up (each operation rounded as in the kernels that do it apart) after
// the first four stages of the 8192-point transform that follows, index bits 1..4 (Modules/FHT.h:31-53): a lane has 32 channels of its row at a time.
__device__ __forceinline__ void staged_store_swiglu(const GemmArgs& args, float* stg, const uint32_t tsrc, const int row0, const int f0, const float sa,
                                                    const int lane, const int c0) {
    const float* sbw = stg + 1024;                             // scales of the warp's 64 gate and 64 up channels
    const bool row_ok = row0 + lane < args.rowsA;
    const ExpTable tab = exp_table_lane();
    __syncwarp();
#pragma unroll 1
    for (int c = c0; c < c0 + 2; c++) {
        float h[32];
#pragma unroll
        for (int half = 0; half < 2; half++) {
            uint32_t vg[16], vu[16];
            tmem_ld_32x16(tsrc + c * 32 + half * 16, vg);
            tmem_ld_32x16(tsrc + 128 + c * 32 + half * 16, vu);
            tmem_ld_wait();
            const f32x2 sa2 = pack2(sa, sa);
#pragma unroll
            for (int j0 = 0; j0 < 16; j0 += 8) {
                float g[8], u[8], o[8];
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    const int col = (c - c0) * 32 + half * 16 + j0 + j;
                    const float2 sg = *reinterpret_cast<const float2*>(sbw + col), su = *reinterpret_cast<const float2*>(sbw + 64 + col);
                    unpack2(mul2(mul2(pack2((float)(int)vg[j0 + j], (float)(int)vg[j0 + j + 1]), sa2), pack2(sg.x, sg.y)), g[j], g[j + 1]);
                    unpack2(mul2(mul2(pack2((float)(int)vu[j0 + j], (float)(int)vu[j0 + j + 1]), sa2), pack2(su.x, su.y)), u[j], u[j + 1]);
                }
#pragma unroll
                for (int j = 0; j < 8; j++) if (!row_ok) g[j] = 1.0f;             // rows past the last keep the warp on the short form
                silu_mul_warp(g, u, o, tab);
#pragma unroll
                for (int j = 0; j < 8; j++) h[half * 16 + j0 + j] = o[j];
            }
        }
        reg_butterfly<1>(h); reg_butterfly<2>(h); reg_butterfly<3>(h); reg_butterfly<4>(h);
#pragma unroll
        for (int gg = 0; gg < 8; gg++)
            *reinterpret_cast<float4*>(stg + lane * 32 + ((gg ^ (lane & 7)) << 2)) = make_float4(h[4 * gg], h[4 * gg + 1], h[4 * gg + 2], h[4 * gg + 3]);
        __syncwarp();
        const int g = lane & 7;
#pragma unroll
        for (int it = 0; it < 8; it++) {
            const int rr = it * 4 + (lane >> 3), row = row0 + rr;
            if (row < args.rowsA)
                *reinterpret_cast<float4*>(args.y + (long)row * args.ldo + f0 + c * 32 + 4 * g) = *reinterpret_cast<const float4*>(stg + rr * 32 + ((g ^ (rr & 7)) << 2));
        }
        __syncwarp();          // the staging buffer is reused by the next chunk
    }
}

template <int BN, bool SWAP, int KCH = 1>
__global__ void __launch_bounds__(192, 1) gemm_i8_tcgen05_kernel(const __grid_constant__ CUtensorMap tmapA,
                                                                 const __grid_constant__ CUtensorMap tmapB,
                                                                 const GemmArgs args) {
    using Cfg = GemmCfg<BN, KCH>;
    constexpr int STAGES = Cfg::STAGES;
    extern __shared__ uint8_t smem_raw[];
    // 1024-byte aligned operand ring, then barriers
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t ring = (raw + 1023u) & ~1023u;
    uint8_t* ring_ptr = smem_raw + (ring - raw);
    uint64_t* bars = reinterpret_cast<uint64_t*>(ring_ptr + STAGES * Cfg::STAGE_BYTES);
    // bars: full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2]; then tmem base word, abort flag
    const uint32_t bar_full = smem_u32(bars);
    const uint32_t bar_empty = bar_full + 8 * STAGES;
    const uint32_t bar_tfull = bar_empty + 8 * STAGES;
    const uint32_t bar_tempty = bar_tfull + 16;
    uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_base_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int num_kb = ((args.K + 127) >> 7) / KCH;      // pipeline steps of KCH chunks (K % (128*KCH) == 0 when KCH > 1)
    const int total_tiles = args.tilesA * args.tilesB * args.ksplit;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) { mbar_init(bar_full + 8 * s, 1); mbar_init(bar_empty + 8 * s, 1); }
        for (int s = 0; s < 2; s++) { mbar_init(bar_tfull + 8 * s, 1); mbar_init(bar_tempty + 8 * s, 4); }
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_base_slot), Cfg::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_base_slot;
    pdl_launch();
    if (!SWAP || warp != 0) pdl_wait();          // (the decode form's producer asks for weights first)

    // decode form, split K: CTA r of the cluster adds up tokens r, r + ksplit, ... of the tile, TB at a time; the first ones' residuals and scales now
    constexpr int TB = 8;
    const int r = blockIdx.x % args.ksplit, cl_row = (int)(blockIdx.x / args.ksplit) * 128 + (warp & 3) * 32 + lane;
    const bool cl_mine = SWAP && args.cluster && warp >= 2 && cl_row < args.rowsA;
    float cl_rs[TB], cl_sb[TB], cl_sa = 0.0f;
    auto cl_fetch = [&](int i0) {
#pragma unroll
        for (int i = 0; i < TB; i++) {
            const int tok = r + (i0 + i) * args.ksplit;
            cl_rs[i] = tok < args.rowsB && args.residual ? args.residual[(long)tok * args.ldo + cl_row] : 0.0f;
            cl_sb[i] = tok < args.rowsB && args.sB ? args.sB[tok] : 0.0f;
        }
    };
    if (cl_mine) {
        cl_sa = args.sA ? args.sA[cl_row] : 0.0f;
        cl_fetch(0);
    }

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (lane == 0) {
            tma_prefetch_desc(&tmapA);
            tma_prefetch_desc(&tmapB);
            auto load_a = [&](int st, int ta, int kb) {
                const uint32_t dst = ring + st * Cfg::STAGE_BYTES;
                if (KCH == 1) tma_load_2d(dst, &tmapA, bar_full + 8 * st, kb * 128, ta * 128);
                else tma_load_3d(dst, &tmapA, bar_full + 8 * st, 0, ta * 128, kb * KCH);
            };
            // decode form: the A side are weights, which no earlier kernel writes. The ring is filled with the first tile's
            // while the kernels before this one still run. (Where none do, weights and activations stage by stage: 64 tokens x 16384 12.3 us, 13.3
            // with the weights first.)
            int ahead = 0;
            if (SWAP) {
                if (args.ahead && (int)blockIdx.x < total_tiles) {
                    const int split = blockIdx.x % args.ksplit, ta = blockIdx.x / (args.ksplit * args.tilesB);
                    const int kb0 = (int)((long)split * num_kb / args.ksplit), kb1 = (int)((long)(split + 1) * num_kb / args.ksplit);
                    for (; ahead < STAGES && kb0 + ahead < kb1; ahead++) {
                        mbar_expect_tx(bar_full + 8 * ahead, Cfg::STAGE_BYTES);
                        load_a(ahead, ta, kb0 + ahead);
                    }
                }
                pdl_wait();
            }
            int stage = 0; uint32_t phase = 0;
            bool ok = true;
            for (int t = blockIdx.x; ok && t < total_tiles; t += gridDim.x) {
                const int split = t % args.ksplit;
                const int tb = (t / args.ksplit) % args.tilesB;
                const int ta = t / (args.ksplit * args.tilesB);
                const int kb0 = (int)((long)split * num_kb / args.ksplit);
                const int kb1 = (int)((long)(split + 1) * num_kb / args.ksplit);
                for (int kb = kb0; kb < kb1; kb++) {
                    const uint32_t full = bar_full + 8 * stage;
                    if (ahead > 0) ahead--;
                    else {
                        if (!mbar_wait(bar_empty + 8 * stage, phase ^ 1u, abort_flag)) { ok = false; break; }
                        mbar_expect_tx(full, Cfg::STAGE_BYTES);
                        load_a(stage, ta, kb);
                    }
                    const uint32_t dstB = ring + stage * Cfg::STAGE_BYTES + Cfg::A_BYTES;
                    if (KCH == 1) tma_load_2d(dstB, &tmapB, full, kb * 128, tb * BN);
                    else tma_load_3d(dstB, &tmapB, full, 0, tb * BN, kb * KCH);
                    if (++stage == STAGES) { stage = 0; phase ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (lane == 0) {
            constexpr uint32_t idesc = umma_idesc_i8(128, BN, 1, 1);
            int stage = 0; uint32_t phase = 0;
            int it = 0;
            bool ok = true;
            for (int t = blockIdx.x; ok && t < total_tiles; t += gridDim.x, it++) {
                const int split = t % args.ksplit;
                const int kb0 = (int)((long)split * num_kb / args.ksplit);
                const int kb1 = (int)((long)(split + 1) * num_kb / args.ksplit);
                const int as = it & 1;
                const uint32_t aphase = (it >> 1) & 1;
                if (!mbar_wait(bar_tempty + 8 * as, aphase ^ 1u, abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint32_t tmem_d = tmem_base + as * BN;
                for (int kb = kb0; kb < kb1; kb++) {
                    if (!mbar_wait(bar_full + 8 * stage, phase, abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t sa = ring + stage * Cfg::STAGE_BYTES;
#pragma unroll
                    for (int c = 0; c < KCH; c++) {
                        const uint64_t adesc = umma_desc_k_sw128(sa + c * Cfg::A_TILE);
                        const uint64_t bdesc = umma_desc_k_sw128(sa + Cfg::A_BYTES + c * Cfg::B_TILE);
#pragma unroll
                        for (int k = 0; k < 4; k++)   // 32 int8 = 32 bytes = 2 descriptor address units per step
                            umma_i8(tmem_d, adesc + 2 * k, bdesc + 2 * k, idesc, (kb > kb0 || c > 0 || k > 0) ? 1u : 0u);
                    }
                    umma_commit(bar_empty + 8 * stage);   // slot is free once these MMAs have read it
                    if (++stage == STAGES) { stage = 0; phase ^= 1u; }
                }
                if (ok) umma_commit(bar_tfull + 8 * as);
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue (warps 2..5)
        const int q = warp & 3;                 // TMEM lane quarter this warp may read
        int it = 0;
        bool ok = true;
        for (int t = blockIdx.x; ok && t < total_tiles; t += gridDim.x, it++) {
            const int tb = (t / args.ksplit) % args.tilesB;
            const int ta = t / (args.ksplit * args.tilesB);
            const int as = it & 1;
            const uint32_t aphase = (it >> 1) & 1;
            // everything the epilogue needs besides the accumulator is fetched BEFORE the wait, so its
            // global-memory latency hides behind the main loop
            const int rowA = ta * 128 + q * 32 + lane;
            const bool rowA_ok = rowA < args.rowsA;
            const float sa = (rowA_ok && args.sA) ? args.sA[rowA] : 0.0f;
            float sbv[SWAP ? BN : 1], rsv[SWAP ? BN : 1];
            if (SWAP && args.sB && !args.cluster) {
#pragma unroll
                for (int j = 0; j < BN; j++) { const int tok = tb * BN + j; sbv[j] = tok < args.rowsB ? args.sB[tok] : 0.0f; }
            }
            if (SWAP && !args.cluster) {
                const float* rp = args.residual + (long)tb * BN * args.ldo + rowA;
#pragma unroll
                for (int j = 0; j < BN; j++) rsv[j] = args.residual && rowA_ok && tb * BN + j < args.rowsB ? rp[(long)j * args.ldo] : 0.0f;
            }
            float* stg = reinterpret_cast<float*>(ring_ptr + STAGES * Cfg::STAGE_BYTES + 256) + q * Cfg::STG_WARP_FLOATS;
            if constexpr (!SWAP && BN >= 32) staged_prefetch<BN>(args, stg, ta * 128 + q * 32, tb * BN, lane);
            // lane 0 polls; the verdict is broadcast so that the warp stays converged for the
            // warp-collective TMEM loads below
            int got = (lane == 0) ? (mbar_wait(bar_tfull + 8 * as, aphase, abort_flag) ? 1 : 0) : 1;
            got = __shfl_sync(0xffffffffu, got, 0);
            if (!got) { ok = false; break; }
            tc_fence_after();
            if constexpr (!SWAP && BN >= 32) {
                staged_store<BN>(args, stg, tmem_base + ((uint32_t)(q * 32) << 16) + as * BN, ta * 128 + q * 32, tb * BN, sa, lane);
            } else {
        #pragma unroll (SWAP ? BN / 16 : 1)
            for (int c = 0; c < BN / 16; c++) {
                uint32_t v[16];
                tmem_ld_32x16(tmem_base + ((uint32_t)(q * 32) << 16) + as * BN + c * 16, v);
                tmem_ld_wait();
                const int colB0 = tb * BN + c * 16;
                if (!SWAP) {
                    // out[rowA][colB0 + j]: token = rowA, channel = colB
                    if (rowA_ok) {
                        const long o = (long)rowA * args.ldo + colB0;
#pragma unroll
                        for (int j = 0; j < 16; j += 4) {
                            if (colB0 + j < args.rowsB) {
                                if (args.acc) {
                                    *reinterpret_cast<int4*>(args.acc + o + j) =
                                        make_int4((int)v[j], (int)v[j + 1], (int)v[j + 2], (int)v[j + 3]);
                                }
                                if (args.y) {
                                    const float4 sb = *reinterpret_cast<const float4*>(args.sB + colB0 + j);
                                    float4 r;
                                    r.x = ((float)(int)v[j] * sa) * sb.x;
                                    r.y = ((float)(int)v[j + 1] * sa) * sb.y;
                                    r.z = ((float)(int)v[j + 2] * sa) * sb.z;
                                    r.w = ((float)(int)v[j + 3] * sa) * sb.w;
                                    if (args.residual) {
                                        const float4 rs = *reinterpret_cast<const float4*>(args.residual + o + j);
                                        r.x = rs.x + r.x; r.y = rs.y + r.y; r.z = rs.z + r.z; r.w = rs.w + r.w;
                                    }
                                    *reinterpret_cast<float4*>(args.y + o + j) = r;
                                }
                            }
                        }
                    }
                } else {
                    // out[colB0 + j][rowA]: token = colB, channel = rowA; a warp store covers 32 channels
                    if (args.cluster) {
                        int* part = reinterpret_cast<int*>(ring_ptr);        // the MMAs have finished reading the ring
#pragma unroll
                        for (int j = 0; j < 16; j++) part[(c * 16 + j) * 128 + q * 32 + lane] = (int)v[j];
                        continue;
                    }
                    const long o = (long)colB0 * args.ldo + rowA;
                    const int n = rowA_ok ? args.rowsB - colB0 : 0;       // tokens of this chunk
                    if (args.ksplit > 1) {
#pragma unroll
                        for (int j = 0; j < 16; j++) if (j < n) atomicAdd(args.acc + o + (long)j * args.ldo, (int)v[j]);
                        continue;
                    }
                    if (args.acc) {
                        int32_t* ap = args.acc + o;
#pragma unroll
                        for (int j = 0; j < 16; j++) if (j < n) ap[(long)j * args.ldo] = (int)v[j];
                    }
                    if (args.y) {
                        float* yp = args.y + o;
#pragma unroll
                        for (int j = 0; j < 16; j++) {
                            float r = ((float)(int)v[j] * sbv[SWAP ? c * 16 + j : 0]) * sa;
                            if (args.residual) r = rsv[SWAP ? c * 16 + j : 0] + r;
                            if (j < n) yp[(long)j * args.ldo] = r;
                        }
                    }
                }
            }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_tempty + 8 * as);
        }
    }

    if (SWAP && args.cluster) {
        // one tile per CTA, the same for the CTAs of a cluster. All loads of TB tokens in flight together (one token after another was a chain of round trips to the other SMs and to
        // L2: 64 tokens of 2048 x 8192 14.1 -> 12.3 us)
        tc_fence_before();
        const int q = warp & 3;
        cluster_sync();
        if (cl_mine && !*abort_flag) {
            uint32_t from[4];
#pragma unroll
            for (int k = 0; k < 4; k++) from[k] = cluster_addr(ring + (uint32_t)(q * 32 + lane) * 4u, k < args.ksplit ? k : 0);
            for (int i0 = 0; r + i0 * args.ksplit < args.rowsB; i0 += TB) {
                if (i0) cl_fetch(i0);
                int p[TB][4];
#pragma unroll
                for (int i = 0; i < TB; i++) {
                    const int tok = r + (i0 + i) * args.ksplit;
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        p[i][k] = k < args.ksplit && tok < args.rowsB ? __float_as_int(ld_cluster_f32(from[k] + (uint32_t)tok * 512u)) : 0;
                }
#pragma unroll
                for (int i = 0; i < TB; i++) {
                    const int tok = r + (i0 + i) * args.ksplit;
                    if (tok >= args.rowsB) continue;
                    const long o = (long)tok * args.ldo + cl_row;
                    const int t = (p[i][0] + p[i][1]) + (p[i][2] + p[i][3]);
                    if (args.acc) args.acc[o] = t;
                    if (args.y) {
                        float v = ((float)t * cl_sb[i]) * cl_sa;
                        if (args.residual) v = cl_rs[i] + v;
                        args.y[o] = v;
                    }
                }
            }
        }
        cluster_sync();                      // nobody leaves while its partial tile may still be read
    }

    // ---------------------------------------------------------------- tear-down
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        // a wait ran out: give copies still in flight time to land before shared memory is released
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) { __nanosleep(1000); }
        if (threadIdx.x == 0 && args.error_flag) atomicOr(args.error_flag, 1);
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
    }
}

// ------------------------------------------------------------------ prefill form on CTA pairs
// The same product with 256 x 256 tiles on two SMs (cta_group::2): each CTA brings in 128 rows of either side, so that per step of
// 128 bytes of K it writes and reads 32 KB of shared memory where the single-CTA form, with 128 + 256 rows, moves 48 KB. Shared memory
// (TMA writes and operand reads, 128 bytes a clock) is what bounds that form, together with its epilogue. Roles as
// there, in both CTAs, but only the first CTA's warp 1 issues MMAs; its barriers count both CTAs' bytes and readers.
// W8A8 prompt of 32 x 1024 tokens, products of 16 layers included: 78.8 -> 75.3 ms.
constexpr int GP_STAGES_MAX = 6, GP_TILE = 128 * 128, GP_STAGE_BYTES = 2 * GP_TILE, GP_BN = 256;
// SWIGLU: eight epilogue warps, two to a quarter of the tile's rows with half of the columns each (32768 rows of 16384 x 2048: 1343 us with four,
// whose arithmetic took longer than the product, 1240 with eight), and a shorter ring to make room for their staging.
template <bool SWIGLU> struct GpCfg {
    static constexpr int STAGES = SWIGLU ? 5 : GP_STAGES_MAX, EPI_WARPS = SWIGLU ? 8 : 4, THREADS = 64 + 32 * EPI_WARPS;
    static constexpr int STG_FLOATS = SWIGLU ? 1024 + 128 : GemmCfg<GP_BN>::STG_WARP_FLOATS;
    static constexpr int SMEM = STAGES * GP_STAGE_BYTES + 1024 + 256 + EPI_WARPS * STG_FLOATS * 4;
};
template <bool SWIGLU>
__global__ void __launch_bounds__(GpCfg<SWIGLU>::THREADS, 1) gemm_i8_pair_kernel(const __grid_constant__ CUtensorMap tmapA, const __grid_constant__ CUtensorMap tmapB,
                                                              const GemmArgs args) {
    constexpr int GP_STAGES = GpCfg<SWIGLU>::STAGES, EPI_WARPS = GpCfg<SWIGLU>::EPI_WARPS;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t ring = (raw + 1023u) & ~1023u;
    uint8_t* ring_ptr = smem_raw + (ring - raw);
    uint64_t* bars = reinterpret_cast<uint64_t*>(ring_ptr + GP_STAGES * GP_STAGE_BYTES);
    const uint32_t bar_full = smem_u32(bars);                    // first CTA: bytes of both CTAs
    const uint32_t bar_empty = bar_full + 8 * GP_STAGES;         // both CTAs, each for its own producer
    const uint32_t bar_tfull = bar_empty + 8 * GP_STAGES;        // both CTAs
    const uint32_t bar_tempty = bar_tfull + 16;                  // first CTA: the epilogue warps of both
    uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(bars + 2 * GP_STAGES + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_base_slot + 1);
    float* stg_all = reinterpret_cast<float*>(ring_ptr + GP_STAGES * GP_STAGE_BYTES + 256);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int num_kb = (args.K + 127) >> 7;
    const int total_tiles = args.tilesA * args.tilesB;           // tilesA: 256-row tiles

    if (threadIdx.x == 0) {
        for (int s = 0; s < GP_STAGES; s++) { mbar_init(bar_full + 8 * s, 1); mbar_init(bar_empty + 8 * s, 1); }
        for (int s = 0; s < 2; s++) { mbar_init(bar_tfull + 8 * s, 1); mbar_init(bar_tempty + 8 * s, 2 * EPI_WARPS); }
        *abort_flag = 0;
        fence_barrier_init();
    }
    __syncthreads();
    if (warp == 1) {
        tmem_alloc_pair(smem_u32(tmem_base_slot), 2 * GP_BN);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                              // the other CTA's barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_base_slot;
    pdl_sync();                                                  // with this CTA's columns taken: a kernel that starts early cannot take them

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer, one per CTA
        if (lane == 0) {
            tma_prefetch_desc(&tmapA);
            tma_prefetch_desc(&tmapB);
            int stage = 0; uint32_t phase = 0;
            bool ok = true;
            for (int t = pair; ok && t < total_tiles; t += pairs) {
                const int rowA = (t / args.tilesB) * 256 + rank * 128, rowB = SWIGLU ? (t % args.tilesB) * 128 + rank * (args.rowsB >> 1) : (t % args.tilesB) * GP_BN + rank * 128;
                for (int kb = 0; kb < num_kb; kb++) {
                    if (!mbar_wait(bar_empty + 8 * stage, phase ^ 1u, abort_flag)) { ok = false; break; }
                    const uint32_t full = bar_full + 8 * stage, full0 = cluster_addr(full, 0);
                    if (rank == 0) mbar_expect_tx(full, 2 * GP_STAGE_BYTES);
                    const uint32_t dst = ring + stage * GP_STAGE_BYTES;
                    tma_load_2d_pair(dst, &tmapA, full0, kb * 128, rowA);
                    tma_load_2d_pair(dst + GP_TILE, &tmapB, full0, kb * 128, rowB);
                    if (++stage == GP_STAGES) { stage = 0; phase ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer, first CTA
        if (lane == 0 && rank == 0) {
            constexpr uint32_t idesc = umma_idesc_i8(256, GP_BN, 1, 1);
            int stage = 0; uint32_t phase = 0;
            int it = 0;
            bool ok = true;
            for (int t = pair; ok && t < total_tiles; t += pairs, it++) {
                const int as = it & 1;
                if (!mbar_wait(bar_tempty + 8 * as, (uint32_t)((it >> 1) & 1) ^ 1u, abort_flag)) { ok = false; break; }
                tc_fence_after();
                for (int kb = 0; kb < num_kb; kb++) {
                    if (!mbar_wait(bar_full + 8 * stage, phase, abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t sa = ring + stage * GP_STAGE_BYTES;
                    const uint64_t adesc = umma_desc_k_sw128(sa), bdesc = umma_desc_k_sw128(sa + GP_TILE);
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        umma_i8_pair(tmem_base + as * GP_BN, adesc + 2 * k, bdesc + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    umma_commit_pair(bar_empty + 8 * stage);
                    if (++stage == GP_STAGES) { stage = 0; phase ^= 1u; }
                }
                if (ok) umma_commit_pair(bar_tfull + 8 * as);
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue (warps 2.. of both CTAs)
        const int q = warp & 3, half = (warp - 2) >> 2;          // TMEM lanes 32 q ..; SWIGLU: columns 64 half ..
        float* stg = stg_all + (warp - 2) * GpCfg<SWIGLU>::STG_FLOATS;
        int it = 0;
        for (int t = pair; t < total_tiles; t += pairs, it++) {
            const int row0 = (t / args.tilesB) * 256 + rank * 128 + q * 32, col0 = (t % args.tilesB) * GP_BN;
            const int as = it & 1;
            const float sa = (row0 + lane < args.rowsA && args.sA) ? args.sA[row0 + lane] : 0.0f;
            if (SWIGLU) {
                for (int i = lane; i < 64; i += 32) {
                    stg[1024 + i] = args.sB[col0 / 2 + half * 64 + i];
                    stg[1024 + 64 + i] = args.sB[(args.rowsB >> 1) + col0 / 2 + half * 64 + i];
                }
            } else {
                staged_prefetch<GP_BN>(args, stg, row0, col0, lane);
            }
            int got = (lane == 0) ? (mbar_wait(bar_tfull + 8 * as, (uint32_t)((it >> 1) & 1), abort_flag) ? 1 : 0) : 1;
            got = __shfl_sync(0xffffffffu, got, 0);
            if (!got) break;
            tc_fence_after();
            const uint32_t tsrc = tmem_base + ((uint32_t)(q * 32) << 16) + as * GP_BN;
            if (SWIGLU) staged_store_swiglu(args, stg, tsrc, row0, col0 / 2, sa, lane, half * 2);
            else staged_store<GP_BN>(args, stg, tsrc, row0, col0, sa, lane);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(cluster_addr(bar_tempty + 8 * as, 0));
        }
    }

    // ---------------------------------------------------------------- tear-down
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        // a wait ran out: give copies still in flight time to land before shared memory is released
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) { __nanosleep(1000); }
        if (threadIdx.x == 0 && args.error_flag) atomicOr(args.error_flag, 1);
        __syncthreads();
    }
    cluster_sync();                                              // both CTAs are done with each other's memory
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 2 * GP_BN);
    }
}

// ------------------------------------------------------------------ host launcher
struct TmapKey {
    const void* base; uint64_t rows, row_bytes; uint32_t box_rows, kch;   // kch 0: 2-D map
    bool operator==(const TmapKey& o) const {
        return base == o.base && rows == o.rows && row_bytes == o.row_bytes && box_rows == o.box_rows && kch == o.kch;
    }
};
struct TmapKeyHash {
    size_t operator()(const TmapKey& k) const {
        size_t h = std::hash<const void*>()(k.base);
        h ^= std::hash<uint64_t>()(k.rows * 1000003ull + k.row_bytes * 31ull + k.box_rows + 977ull * k.kch) + 0x9e3779b97f4a7c15ull + (h << 6) + (h >> 2);
        return h;
    }
};
// Encoding a tensor map costs a few microseconds of host time; the same weights and activation
// buffers come back every layer call, so maps are cached by (pointer, shape, box).
static int cached_tmap(CUtensorMap* out, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows, uint32_t kch = 0) {
    static std::mutex mu;
    static std::unordered_map<TmapKey, CUtensorMap, TmapKeyHash> cache;
    TmapKey key{base, rows, row_bytes, box_rows, kch};
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find(key);
    if (it != cache.end()) { *out = it->second; return FLEXLLM_OK; }
    int st = kch ? make_tmap_3d_u8(out, base, rows, row_bytes, box_rows, kch) : make_tmap_2d_u8(out, base, rows, row_bytes, box_rows);
    if (st != FLEXLLM_OK) return st;
    if (cache.size() > 4096) cache.clear();
    cache.emplace(key, *out);
    return FLEXLLM_OK;
}

int cached_tmap_u8(CUtensorMap* out, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows, uint32_t kch) {
    return cached_tmap(out, base, rows, row_bytes, box_rows, kch);
}

// One error word per device: bit 0 is raised by any kernel of the library whose bounded device-side wait ran
// out, bit 1 by a kernel that found (and clamped) a token id or context length in device memory out of range. It lives in the library's device image (no allocation needed to reach it); its device address
// is looked up once per device. Process-wide: a time-out raised by a launch from one host thread is
// seen by a status check from any other.
static __device__ int g_error_flag;
struct DevFlag { std::once_flag once; int* p = nullptr; };
static DevFlag g_dev_flag[kMaxDevices];

int* device_error_flag() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    DevFlag& f = g_dev_flag[dev];
    std::call_once(f.once, [&] {
        int* p = nullptr;
        if (cudaGetSymbolAddress((void**)&p, g_error_flag) == cudaSuccess) f.p = p;
    });
    return f.p;
}

static int sm_count() {
    static int n[kMaxDevices] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= kMaxDevices) return 148;
    if (!n[dev]) cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev);
    return n[dev] > 0 ? n[dev] : 148;
}

template <int BN, bool SWAP, int KCH = 1>
static int launch_gemm(const int8_t* A, int rowsA, const int8_t* B, int rowsB, int K, int ksplit, int ldo,
                       int32_t* acc, float* y, const float* sA, const float* sB, cudaStream_t st,
                       const float* residual = nullptr) {
    using Cfg = GemmCfg<BN, KCH>;
    CUtensorMap ta, tb;
    int rc = cached_tmap(&ta, A, (uint64_t)rowsA, (uint64_t)K, 128, KCH > 1 ? KCH : 0);
    if (rc != FLEXLLM_OK) return rc;
    rc = cached_tmap(&tb, B, (uint64_t)rowsB, (uint64_t)K, BN, KCH > 1 ? KCH : 0);
    if (rc != FLEXLLM_OK) return rc;
    GemmArgs g;
    g.rowsA = rowsA; g.rowsB = rowsB; g.K = K;
    g.tilesA = (rowsA + 127) / 128; g.tilesB = (rowsB + BN - 1) / BN; g.ksplit = ksplit;
    g.ldo = ldo; g.acc = acc; g.y = y; g.sA = sA; g.sB = sB; g.error_flag = device_error_flag();
    g.residual = residual; g.cluster = SWAP && ksplit > 1; g.ahead = may_read_ahead();
    auto kern = gemm_i8_tcgen05_kernel<BN, SWAP, KCH>;
    // the attribute belongs to (function, device): once per device, not once per process
    static std::atomic<bool> attr_set[kMaxDevices];
    const int dev = current_device();
    if (dev < 0) return FLEXLLM_ECUDA;
    if (!attr_set[dev].load(std::memory_order_acquire)) {
        FLEXLLM_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
        attr_set[dev].store(true, std::memory_order_release);
    }
    const int total = g.tilesA * g.tilesB * g.ksplit;
    if (g.cluster) {                       // one tile per CTA (tilesB is 1)
        launch_cluster(kern, dim3(total), dim3(192), ksplit, (size_t)Cfg::SMEM_BYTES, st, ta, tb, g);
        return launch_status();
    }
    const int grid = total < sm_count() ? total : sm_count();
    launch_k(kern, dim3(grid), dim3(192), (size_t)Cfg::SMEM_BYTES, st, ta, tb, g);
    return launch_status();
}

// SWIGLU: w holds N / 2 gate and N / 2 up rows, y is [M][N / 2].
template <bool SWIGLU = false>
static int launch_gemm_pair(const int8_t* a, const float* s_tok, const int8_t* w, const float* s_ch, int M, int N, int K, int32_t* acc, float* y,
                            cudaStream_t st, const float* residual) {
    CUtensorMap ta, tb;
    int rc = cached_tmap(&ta, a, (uint64_t)M, (uint64_t)K, 128);
    if (rc != FLEXLLM_OK) return rc;
    rc = cached_tmap(&tb, w, (uint64_t)N, (uint64_t)K, 128);
    if (rc != FLEXLLM_OK) return rc;
    GemmArgs g;
    g.rowsA = M; g.rowsB = N; g.K = K;
    g.tilesA = (M + 255) / 256; g.tilesB = (N + GP_BN - 1) / GP_BN; g.ksplit = 1;
    g.ldo = SWIGLU ? N / 2 : N; g.acc = acc; g.y = y; g.sA = s_tok; g.sB = s_ch; g.error_flag = device_error_flag();
    g.residual = residual; g.cluster = 0; g.ahead = 0;
    auto kern = gemm_i8_pair_kernel<SWIGLU>;
    static std::atomic<bool> attr_set[kMaxDevices];
    const int dev = current_device();
    if (dev < 0) return FLEXLLM_ECUDA;
    if (!attr_set[dev].load(std::memory_order_acquire)) {
        FLEXLLM_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GpCfg<SWIGLU>::SMEM));
        attr_set[dev].store(true, std::memory_order_release);
    }
    const int tiles = g.tilesA * g.tilesB, pairs = sm_count() / 2;
    launch_cluster(kern, dim3(2 * (tiles < pairs ? tiles : pairs)), dim3(GpCfg<SWIGLU>::THREADS), 2, (size_t)GpCfg<SWIGLU>::SMEM, st, ta, tb, g);
    return launch_status();
}

// Prefill orientation: activations on the 128-row side. residual (optional): y = residual + dequant.
// The tile is the one with the shortest time by a count of shared-memory traffic: per step of 128 bytes of K a CTA moves (128 + BN)
// rows (the pair form 256 for twice the output), plus a fixed part; times the rounds of tiles that the SMs go through. (With 256
// columns whenever there are that many, a product of 128 x 2048 x 2048 ran on 8 SMs for 15 us.)
struct TileCosts { long c256, c128, c64, c32; bool pair; };
static TileCosts tile_costs(int M, int N) {
    const int sms = sm_count();
    auto cost = [&](int rows, int cols, int units, int step) {
        const long tiles = (long)((M + rows - 1) / rows) * ((N + cols - 1) / cols);
        return (tiles + units - 1) / units * step;
    };
    TileCosts c = {cost(128, 256, sms, 128 + 256 + 32), cost(128, 128, sms, 128 + 128 + 32), cost(128, 64, sms, 128 + 64 + 32),
                   cost(128, 32, sms, 128 + 32 + 32), false};
    const long cpair = cost(256, 256, sms / 2, 256 + 48);
    c.pair = N > 128 && M > 128 && cpair <= c.c256 && cpair <= c.c128 && cpair <= c.c64 && cpair <= c.c32;
    return c;
}
int gemm_i8_prefill(const int8_t* a, const float* s_tok, const int8_t* w, const float* s_ch, int M, int N, int K,
                    int32_t* acc, float* y, cudaStream_t st, const float* residual) {
    const SetUpEarly early;
    const TileCosts t = tile_costs(M, N);
    const long c256 = t.c256, c128 = t.c128, c64 = t.c64, c32 = t.c32;
    if (t.pair) return launch_gemm_pair(a, s_tok, w, s_ch, M, N, K, acc, y, st, residual);
    if (N > 128 && c256 <= c128 && c256 <= c64 && c256 <= c32) return launch_gemm<256, false>(a, M, w, N, K, 1, N, acc, y, s_tok, s_ch, st, residual);
    if (N > 64 && c128 <= c64 && c128 <= c32) return launch_gemm<128, false>(a, M, w, N, K, 1, N, acc, y, s_tok, s_ch, st, residual);
    if (N > 32 && c64 <= c32) return launch_gemm<64, false>(a, M, w, N, K, 1, N, acc, y, s_tok, s_ch, st, residual);
    if (N > 16) return launch_gemm<32, false>(a, M, w, N, K, 1, N, acc, y, s_tok, s_ch, st, residual);
    return launch_gemm<16, false>(a, M, w, N, K, 1, N, acc, y, s_tok, s_ch, st, residual);
}

// The fused gate | up product (w: F gate rows, then F up rows) with silu(gate) * up and the transform's index bits 1..4 in its epilogue: h [M][F],
// for fht8192_rest. It writes half of what the plain product writes and the transform then reads, and the transform loses its first passes. 32768
// rows, 8192 channels: product 1006 + SiLU, transform and quantiser 692 us apart, 1240 + 254 us this way (2 x 1.07 GB less through memory);
// a prompt of 32 x 1024 tokens 74.9 -> 71.4 ms, 32 x 256 15.8 -> 15.0, 1 x 256 2.58 -> 2.48. Taken where the product runs on CTA pairs
// anyway (more than 128 rows); elsewhere FLEXLLM_ENOTSUP and nothing is launched.
int gemm_i8_prefill_swiglu(const int8_t* a, const float* s_tok, const int8_t* w, const float* s_ch, int M, int F, int K, float* h, cudaStream_t st) {
    if (F % 128 != 0 || !tile_costs(M, 2 * F).pair) return FLEXLLM_ENOTSUP;
    const SetUpEarly early;
    return launch_gemm_pair<true>(a, s_tok, w, s_ch, M, 2 * F, K, nullptr, h, st, nullptr);
}

// Decode orientation: weights on the 128-row side, M <= 64 tokens on the N side. K is split over clusters of up to four CTAs as
// long as the tiles leave half the SMs idle and every split keeps two 128-byte blocks. (64 tokens of 2048 x 8192: 23.5 / 19.8 /
// 14.0 / 18.3 us with clusters of 1 / 2 / 4 / 8, of 2048 x 2048: 13.3 / 14.4 / 10.4 / 15.4 us: larger clusters start and meet later. Those were taken
// with an epilogue that loaded value by value; with its loads in flight together the clusters of four take 12 and 8 us.)
int gemm_i8_decode(const int8_t* a, const float* s_tok, const int8_t* w, const float* s_ch, int M, int N, int K,
                   int32_t* acc, float* y, cudaStream_t st, const float* residual) {
    if (M > 64) return FLEXLLM_ENOTSUP;
    const int tiles = (N + 127) / 128, kb = (K + 127) / 128;
    int ksplit = 1;
    while (ksplit < 4 && tiles * ksplit * 2 <= sm_count() && kb >= 4 * ksplit) ksplit *= 2;
    // chunks of K per pipeline stage: KCH*128 contiguous bytes per weight row and TMA request, two steps per split
    int kch = 1;
    if (K % 512 == 0 && kb / 4 >= 2 * ksplit) kch = 4;
    else if (K % 256 == 0 && kb / 2 >= 2 * ksplit) kch = 2;
#define FLEXLLM_DEC(BN_, KCH_) \
    return launch_gemm<BN_, true, KCH_>(w, N, a, M, K, ksplit, N, acc, y, s_ch, s_tok, st, residual)
    if (M > 32) { if (kch == 4) FLEXLLM_DEC(64, 4); if (kch == 2) FLEXLLM_DEC(64, 2); FLEXLLM_DEC(64, 1); }
    if (M > 16) { if (kch == 4) FLEXLLM_DEC(32, 4); if (kch == 2) FLEXLLM_DEC(32, 2); FLEXLLM_DEC(32, 1); }
    if (kch == 4) FLEXLLM_DEC(16, 4);
    if (kch == 2) FLEXLLM_DEC(16, 2);
    FLEXLLM_DEC(16, 1);
#undef FLEXLLM_DEC
}

// Reads and clears the current device's error word (synchronises the device: the copy is ordered
// behind all work queued so far).
int gemm_check_error_flag() {
    int* f = device_error_flag();
    if (!f) return FLEXLLM_ECUDA;
    int h = 0;
    FLEXLLM_CHECK_CUDA(cudaMemcpy(&h, f, sizeof(int), cudaMemcpyDeviceToHost));
    if (h) {
        FLEXLLM_CHECK_CUDA(cudaMemset(f, 0, sizeof(int)));
        return (h & 1) ? FLEXLLM_ETIMEDOUT : FLEXLLM_EDEVDATA;      // bit 0: a wait ran out; bit 1: an index in device memory was clamped
    }
    return FLEXLLM_OK;
}

int gemm_sm_count() { return sm_count(); }

// ------------------------------------------------------------------ allocation-free decode linear
// Built-in scratch for the split-K partial sums of flexllm_linear_decode_i8_noalloc: a fixed array in
// the library's device image, so the entry point never has to ask the driver for memory. Every GPU
// that loads the library carries these 4 MiB until the process exits.
constexpr long kNoAllocMaxElems = 64L * 16384L;   // tokens x output channels, int32 each
static __device__ __align__(256) int32_t g_noalloc_scratch[kNoAllocMaxElems];

struct NoAllocDev { std::once_flag once; int32_t* scratch = nullptr; int* flag = nullptr; int rc = FLEXLLM_ECUDA; };
static NoAllocDev g_noalloc_dev[kMaxDevices];

template <int BN>
static int launch_gemm_noalloc(const int8_t* w, int N, const int8_t* a, int M, int K, int ksplit, int32_t* acc, int* flag,
                               cudaStream_t st) {
    using Cfg = GemmCfg<BN>;
    CUtensorMap ta, tb;   // encoded on the stack: no cache, nothing retained
    int rc = make_tmap_2d_u8(&ta, w, (uint64_t)N, (uint64_t)K, 128);
    if (rc != FLEXLLM_OK) return rc;
    rc = make_tmap_2d_u8(&tb, a, (uint64_t)M, (uint64_t)K, BN);
    if (rc != FLEXLLM_OK) return rc;
    GemmArgs g;
    g.rowsA = N; g.rowsB = M; g.K = K;
    g.tilesA = (N + 127) / 128; g.tilesB = 1; g.ksplit = ksplit;
    g.ldo = N; g.acc = acc; g.y = nullptr; g.sA = nullptr; g.sB = nullptr; g.error_flag = flag;
    g.residual = nullptr; g.cluster = 0; g.ahead = 0;
    auto kern = gemm_i8_tcgen05_kernel<BN, true>;
    static std::atomic<bool> attr_set[kMaxDevices];
    const int dev = current_device();
    if (dev < 0) return FLEXLLM_ECUDA;
    if (!attr_set[dev].load(std::memory_order_acquire)) {
        FLEXLLM_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
        attr_set[dev].store(true, std::memory_order_release);
    }
    const int total = g.tilesA * g.ksplit;
    const int grid = total < sm_count() ? total : sm_count();
    kern<<<grid, 192, Cfg::SMEM_BYTES, st>>>(ta, tb, g);
    return launch_status();
}

}  // namespace flexllm

using namespace flexllm;

// See include/flexllm_b200.h.
extern "C" int flexllm_device_status(void) { return gemm_check_error_flag(); }

// See include/flexllm_b200.h: the prefill GEMM with nothing to store (the epilogue warps still drain TMEM).
extern "C" int flexllm_gemm_i8_mainloop_probe(const int8_t* a, const int8_t* w, int M, int N, int K, void* stream) {
    FLEXLLM_REQUIRE(a && w && M > 0 && N > 128 && K > 0 && (K % 16) == 0 && aligned(a, 16) && aligned(w, 16));
    return launch_gemm<256, false>(a, M, w, N, K, 1, N, nullptr, nullptr, nullptr, nullptr, (cudaStream_t)stream);
}

// See include/flexllm_b200.h. The first call on a device resolves the device addresses of the
// built-in arrays (cudaGetSymbolAddress: the array's name is only a host-side handle, not a device
// pointer); make that first call outside any stream capture.
extern "C" int flexllm_linear_decode_i8_noalloc(const int8_t* a, const float* s_tok, const int8_t* w, const float* s_ch,
                                                int M, int N, int K, float* y, void* stream) {
    FLEXLLM_REQUIRE(M >= 0 && N > 0 && K > 0 && (K % 16) == 0 && (N % 8) == 0);
    if (M == 0) return FLEXLLM_OK;
    FLEXLLM_REQUIRE(a && s_tok && w && s_ch && y);
    FLEXLLM_REQUIRE(aligned(a, 16) && aligned(w, 16) && aligned(y, 16) && aligned(s_ch, 16));
    if (M > 64) return FLEXLLM_ENOTSUP;
    if ((long)M * N > kNoAllocMaxElems) return FLEXLLM_ETOOBIG;   // larger than the built-in scratch
    const int dev = current_device();
    if (dev < 0) return FLEXLLM_ECUDA;
    NoAllocDev& d = g_noalloc_dev[dev];
    // set-up, once per device, with that device current: the array's name is only a host-side handle,
    // the kernel needs the address cudaGetSymbolAddress returns. The error word is the library's
    // per-device one, so a time-out in this path is reported by flexllm_device_status() like any other.
    std::call_once(d.once, [&] {
        d.rc = cuda_status(cudaGetSymbolAddress((void**)&d.scratch, g_noalloc_scratch));
        if (d.rc == FLEXLLM_OK) { d.flag = device_error_flag(); if (!d.flag) d.rc = FLEXLLM_ECUDA; }
    });
    if (d.rc != FLEXLLM_OK) return d.rc;
    cudaStream_t st = (cudaStream_t)stream;
    // split-K as in the allocating entry point: enough CTAs to pull the weights at full HBM rate
    const int tiles = (N + 127) / 128, num_kb = (K + 127) / 128;
    int ks = sm_count() / tiles;
    if (ks > num_kb / 2) ks = num_kb / 2;
    if (ks < 1) ks = 1;
    // the array keeps whatever the previous call left in it: the partial sums must start from zero
    FLEXLLM_CHECK_CUDA(cudaMemsetAsync(d.scratch, 0, (size_t)M * N * sizeof(int32_t), st));
    int rc;
    if (M > 32) rc = launch_gemm_noalloc<64>(w, N, a, M, K, ks, d.scratch, d.flag, st);
    else if (M > 16) rc = launch_gemm_noalloc<32>(w, N, a, M, K, ks, d.scratch, d.flag, st);
    else rc = launch_gemm_noalloc<16>(w, N, a, M, K, ks, d.scratch, d.flag, st);
    if (rc != FLEXLLM_OK) return rc;
    return flexllm_dequant(d.scratch, s_tok, s_ch, M, N, y, stream);
}
