// Walsh-Hadamard transforms of the SpinQuant online rotations.
//
// The reference computes the transform with an Omega network (Modules/FHT.h:31-53). Its fp32
// result is bit-identical to in-place butterflies (lo,hi) <- (lo+hi, lo-hi) applied on index
// bits in the order 1, 2, ..., log2(N)-1, 0; every kernel here keeps exactly that stage order.
//
//  * fht8192_kernel  : R4, the 8192-point transform on the down_proj input. One CTA per token, the row in
//                      shared memory between three register passes of 1+6+6 stages. Optionally fused
//                      with silu(gate)*up on the way in and with the per-token int8 quantiser on the way out.
//  * fht8192_cluster_kernel: the fused form for few rows, a cluster of eight CTAs per token.
//  * fht_generic     : any power of two <= 8192, one stage per barrier (API completeness).
//  * qk_prepare      : R3, the 64-point transform on Q/K heads, in registers with warp shuffles,
//                      fused with dequant, RoPE and the per-head int8 quantiser.
#include "common.cuh"
#include "fht_core.cuh"
#include "tc_common.cuh"

namespace flexllm {
using namespace tc;

// FUSED: 0 = y = FHT(x)/scale (fp32 out); 1 = h = silu(g)*u, FHT, /scale, per-token int8 quant;
// 2 = like 1 without the silu, input gathered from `win.g` ranks as x[g][rows][N/g], int8 output only
// for the column window [win.col0, win.col0 + win.cols) written compactly (tensor-parallel down_proj).
struct FhtWindow { int g; long rows; int col0, cols; };

// One CTA of 128 threads per row, 64 elements a thread. Bound by issue slots and by shared-memory bandwidth (128 bytes a
// clock), so the row passes through shared memory twice and not three times: index bit 1 is done on the float4 as it comes
// from memory, bits 2..7 with 64 values in registers, bits 8..12 and then 0 likewise. Element i lives at i + 4 * (i >> 8): the
// lanes of a warp, which hold two low bits and three of the bits from 8 up in the second pass, then use different banks.
// Four CTAs an SM. 32768 rows: 1058 us with three exchanges, full divisions and exponentials on 256 threads; 695 us now (2.4 GB
// in and out: 370 us).
__device__ __forceinline__ int fht_at(int i) { return i + 4 * (i >> 8); }
template <int FUSED>
__global__ void __launch_bounds__(128, 4) fht8192_kernel(const float* __restrict__ x, const float* __restrict__ u, long ld_in,
                                                         float scale, float* __restrict__ y, int8_t* __restrict__ q,
                                                         float* __restrict__ s, float* __restrict__ act, FhtWindow win) {
    constexpr int N = 8192;
    __shared__ __align__(16) float buf[N + 4 * (N / 256)];
    __shared__ float red[4], red_nan[4];
    pdl_sync();
    const int tid = threadIdx.x;
    const long row = blockIdx.x;
    const float4* xr = reinterpret_cast<const float4*>(x + row * ld_in);   // ld_in: input row stride in floats
    const float4* ur = FUSED == 1 ? reinterpret_cast<const float4*>(u + row * ld_in) : nullptr;
    const ExpTable tab = exp_table_lane();
    auto load = [&](int c) {                                               // vector c of the row
        if (FUSED == 2) {
            const int segw = N / win.g, e = c * 4, seg = e / segw;
            return *reinterpret_cast<const float4*>(x + ((long)seg * win.rows + row) * segw + (e - seg * segw));
        }
        return xr[c];
    };
    // four batches of 16 elements; the next batch's loads are issued before this one's arithmetic
    float4 gv[4], uv[4];
#pragma unroll
    for (int i = 0; i < 4; i++) { gv[i] = load(i * 128 + tid); if (FUSED == 1) uv[i] = ur[i * 128 + tid]; }
#pragma unroll
    for (int b = 0; b < 4; b++) {
        float4 gn[4], un[4];
        if (b < 3) {
#pragma unroll
            for (int i = 0; i < 4; i++) { gn[i] = load(((b + 1) * 4 + i) * 128 + tid); if (FUSED == 1) un[i] = ur[((b + 1) * 4 + i) * 128 + tid]; }
        }
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
            float v[8] = {gv[i].x, gv[i].y, gv[i].z, gv[i].w, gv[i + 1].x, gv[i + 1].y, gv[i + 1].z, gv[i + 1].w};
            if (FUSED == 1) {
                const float w[8] = {uv[i].x, uv[i].y, uv[i].z, uv[i].w, uv[i + 1].x, uv[i + 1].y, uv[i + 1].z, uv[i + 1].w};
                float o[8];
                silu_mul_warp(v, w, o, tab);
#pragma unroll
                for (int j = 0; j < 8; j++) v[j] = o[j];
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int c = (b * 4 + i + h) * 128 + tid;
                if (FUSED == 1 && act) reinterpret_cast<float4*>(act + row * N)[c] = make_float4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
                // index bit 1
                *reinterpret_cast<float4*>(buf + fht_at(c * 4)) =
                    make_float4(v[4 * h] + v[4 * h + 2], v[4 * h + 1] + v[4 * h + 3], v[4 * h] - v[4 * h + 2], v[4 * h + 1] - v[4 * h + 3]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) { gv[i] = gn[i]; if (FUSED == 1) uv[i] = un[i]; }
    }
    __syncthreads();
    float r[64];
    {   // index bits 2..7
        float* at = buf + fht_at((tid & 3) | ((tid >> 2) << 8));
#pragma unroll
        for (int v = 0; v < 64; v++) r[v] = at[v * 4];
        reg_butterfly<0>(r); reg_butterfly<1>(r); reg_butterfly<2>(r); reg_butterfly<3>(r); reg_butterfly<4>(r); reg_butterfly<5>(r);
#pragma unroll
        for (int v = 0; v < 64; v++) at[v * 4] = r[v];
    }
    __syncthreads();
    {   // index bits 8..12, then 0: register v holds index bit 0 in its bit 0, bits 8..12 in its bits 1..5
#pragma unroll
        for (int h = 0; h < 32; h++) {
            const float2 t = *reinterpret_cast<const float2*>(buf + tid * 2 + h * (256 + 4));
            r[2 * h] = t.x; r[2 * h + 1] = t.y;
        }
        reg_butterfly<1>(r); reg_butterfly<2>(r); reg_butterfly<3>(r); reg_butterfly<4>(r); reg_butterfly<5>(r); reg_butterfly<0>(r);
    }
    if (FUSED == 0) {
        div_rn_array(r, div_by(scale));
#pragma unroll
        for (int h = 0; h < 32; h++) *reinterpret_cast<float2*>(y + row * N + h * 256 + tid * 2) = make_float2(r[2 * h], r[2 * h + 1]);
        return;
    }
    // the quantiser's scale is the largest magnitude / 127; division by `scale` keeps the order, so one division of the largest does
    float mx = 0.0f, mn = 0.0f;                                            // mn: NaN when a value is
#pragma unroll
    for (int v = 0; v < 64; v += 2) { mx = max3(mx, fabsf(r[v]), fabsf(r[v + 1])); mn = max3_nan(mn, fabsf(r[v]), fabsf(r[v + 1])); }
    mx = warp_max(mx);
    const bool bad = __any_sync(0xffffffffu, !(mn <= mx));
    if ((tid & 31) == 0) { red[tid >> 5] = mx; red_nan[tid >> 5] = bad ? 1.0f : 0.0f; }
    __syncthreads();
    mx = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
    const bool ok = fht_q8_in_range(mx, scale) && (red_nan[0] + red_nan[1]) + (red_nan[2] + red_nan[3]) == 0.0f;
    const float sc = fht_row_scale(mx, scale);
    if (tid == 0) s[row] = sc;
#pragma unroll
    for (int h0 = 0; h0 < 32; h0 += 4) {
        float t[8];
        uint32_t b[8];
#pragma unroll
        for (int i = 0; i < 8; i++) t[i] = r[2 * h0 + i];
        q8_short(t, 1.0f / (scale * sc), ok, b, [&](float v) { return fht_q8_exact(v, scale, sc); });
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint16_t two = (uint16_t)__byte_perm(b[2 * i], b[2 * i + 1], 0x0040);
            const int idx = (h0 + i) * 256 + tid * 2;
            if (FUSED == 2) {
                if (idx >= win.col0 && idx < win.col0 + win.cols) *reinterpret_cast<uint16_t*>(q + row * win.cols + (idx - win.col0)) = two;
            } else {
                *reinterpret_cast<uint16_t*>(q + row * N + idx) = two;
            }
        }
    }
}

// The rest of the fused form behind a product that has done silu(gate) * up and index bits 1..4 itself (gemm_i8_prefill_swiglu): bits 5..10 with the
// values as they come from memory (a lane's values 32 apart, so that a warp reads 128 bytes at a time), bits 11, 12 and 0 after the only exchange
// through shared memory, then the quantiser. Bound by memory: 254 us for 32768 rows (1.34 GB, 205 us at the copy rate). Element i lives at i with its 16-byte granule exchanged by index bits 5 and 6: both sides of the
// exchange touch every bank once.
__device__ __forceinline__ int fht_rest_at(int i) { return i ^ (((i >> 5) & 3) << 2); }
__global__ void __launch_bounds__(128, 4) fht8192_rest_kernel(const float* __restrict__ x, float scale, int8_t* __restrict__ q, float* __restrict__ s) {
    constexpr int N = 8192;
    __shared__ __align__(16) float buf[N];
    __shared__ float red[4], red_nan[4];
    pdl_sync();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long row = blockIdx.x;
    float r[64];
    {
        const float* xr = x + row * N + warp * 2048 + lane;
#pragma unroll
        for (int v = 0; v < 64; v++) r[v] = xr[v * 32];
        reg_butterfly<0>(r); reg_butterfly<1>(r); reg_butterfly<2>(r); reg_butterfly<3>(r); reg_butterfly<4>(r); reg_butterfly<5>(r);
#pragma unroll
        for (int v = 0; v < 64; v++) buf[fht_rest_at(warp * 2048 + v * 32 + lane)] = r[v];
    }
    __syncthreads();
    // register bits 0..3: index bits 0..3, bits 4 and 5: index bits 11 and 12; index bits 4..10 are the thread's
#pragma unroll
    for (int h = 0; h < 4; h++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const float4 t = *reinterpret_cast<const float4*>(buf + fht_rest_at(h * 2048 + tid * 16 + c * 4));
            r[h * 16 + c * 4] = t.x; r[h * 16 + c * 4 + 1] = t.y; r[h * 16 + c * 4 + 2] = t.z; r[h * 16 + c * 4 + 3] = t.w;
        }
    reg_butterfly<4>(r); reg_butterfly<5>(r); reg_butterfly<0>(r);
    float mx = 0.0f, mn = 0.0f;                                            // mn: NaN when a value is
#pragma unroll
    for (int v = 0; v < 64; v += 2) { mx = max3(mx, fabsf(r[v]), fabsf(r[v + 1])); mn = max3_nan(mn, fabsf(r[v]), fabsf(r[v + 1])); }
    mx = warp_max(mx);
    const bool bad = __any_sync(0xffffffffu, !(mn <= mx));
    if (lane == 0) { red[warp] = mx; red_nan[warp] = bad ? 1.0f : 0.0f; }
    __syncthreads();
    mx = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
    const bool ok = fht_q8_in_range(mx, scale) && (red_nan[0] + red_nan[1]) + (red_nan[2] + red_nan[3]) == 0.0f;
    const float sc = fht_row_scale(mx, scale);
    if (tid == 0) s[row] = sc;
#pragma unroll
    for (int h = 0; h < 4; h++) {
        uint32_t o[4];
#pragma unroll
        for (int c = 0; c < 4; c += 2) {
            float t[8];
            uint32_t b[8];
#pragma unroll
            for (int i = 0; i < 8; i++) t[i] = r[h * 16 + c * 4 + i];
            q8_short(t, 1.0f / (scale * sc), ok, b, [&](float v) { return fht_q8_exact(v, scale, sc); });
#pragma unroll
            for (int i = 0; i < 2; i++)
                o[c + i] = __byte_perm(__byte_perm(b[4 * i], b[4 * i + 1], 0x0040), __byte_perm(b[4 * i + 2], b[4 * i + 3], 0x0040), 0x5410);
        }
        *reinterpret_cast<uint4*>(q + row * N + h * 2048 + tid * 16) = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// The same for few rows (decoding): a cluster of eight CTAs per row, 1024 elements a CTA, eight a thread, so that SiLU's
// arithmetic and the loads, which one SM does one after another, are spread over eight. Index bits 1 and 9 are a thread's
// own, 2..6 the lane's (shuffles), 7 and 8 the warp's: bit 1 in registers, 2..6 by shuffle, 7..9 after an exchange through
// shared memory, 10..12 after one between the CTAs, bit 0 by shuffle.
constexpr int FHT_CL = 8;
__global__ void __launch_bounds__(128) fht8192_cluster_kernel(const float* __restrict__ g, const float* __restrict__ u, long ld_in, float scale,
                                                              int8_t* __restrict__ q, float* __restrict__ s, float* __restrict__ act) {
    constexpr int N = 8192, L = N / FHT_CL;
    __shared__ __align__(16) float buf[L], out[L];
    __shared__ float peer_mx[FHT_CL], red[4];
    __shared__ int peer_bad[FHT_CL];
    pdl_sync();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long row = blockIdx.x / FHT_CL;
    const int part = blockIdx.x % FHT_CL;
    const float4* gr = reinterpret_cast<const float4*>(g + row * ld_in + part * L);
    const float4* ur = reinterpret_cast<const float4*>(u + row * ld_in + part * L);
    const float4 g0 = gr[tid], g1 = gr[128 + tid], u0 = ur[tid], u1 = ur[128 + tid];
    const ExpTable tab = exp_table_lane();
    const float gg[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w}, uu[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
    float r[8];
    silu_mul_warp(gg, uu, r, tab);
    if (act) {
        float4* ao = reinterpret_cast<float4*>(act + row * N + part * L);
        ao[tid] = make_float4(r[0], r[1], r[2], r[3]);
        ao[128 + tid] = make_float4(r[4], r[5], r[6], r[7]);
    }
    reg_butterfly<1>(r);                                                   // index bit 1
    auto lane_stage = [&](int bit) {
        const bool up = lane & (1 << bit);
#pragma unroll
        for (int v = 0; v < 8; v++) {
            const float p = __shfl_xor_sync(0xffffffffu, r[v], 1 << bit);
            r[v] = up ? p - r[v] : r[v] + p;
        }
    };
#pragma unroll
    for (int bit = 0; bit < 5; bit++) lane_stage(bit);                     // index bits 2..6
    reinterpret_cast<float4*>(buf)[tid] = make_float4(r[0], r[1], r[2], r[3]);
    reinterpret_cast<float4*>(buf)[128 + tid] = make_float4(r[4], r[5], r[6], r[7]);
    __syncthreads();
#pragma unroll
    for (int v = 0; v < 8; v++) r[v] = buf[v * 128 + tid];                 // register bits: index bits 7, 8, 9
    reg_butterfly<0>(r); reg_butterfly<1>(r); reg_butterfly<2>(r);
#pragma unroll
    for (int v = 0; v < 8; v++) out[v * 128 + tid] = r[v];
    cluster_sync();
    // thread tid takes index bits 0..6 = tid, 7..9 = part; register bits: index bits 10, 11, 12
    const uint32_t mine = smem_u32(out + part * 128 + tid);
#pragma unroll
    for (int v = 0; v < 8; v++) r[v] = ld_cluster_f32(cluster_addr(mine, v));
    reg_butterfly<0>(r); reg_butterfly<1>(r); reg_butterfly<2>(r);
    lane_stage(0);                                                         // index bit 0
    float mx = 0.0f, mn = 0.0f;
#pragma unroll
    for (int v = 0; v < 8; v += 2) { mx = max3(mx, fabsf(r[v]), fabsf(r[v + 1])); mn = max3_nan(mn, fabsf(r[v]), fabsf(r[v + 1])); }
    mx = warp_max(mx);
    if (lane == 0) red[warp] = mx;
    const int bad = __syncthreads_or(!(mn <= mx));                         // a NaN anywhere in this CTA
    if (tid < FHT_CL) {
        const float m = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
        const uint32_t am = cluster_addr(smem_u32(peer_mx + part), tid), ab = cluster_addr(smem_u32(peer_bad + part), tid);
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(am), "f"(m) : "memory");
        asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(ab), "r"(bad) : "memory");
    }
    cluster_sync();
    int any_bad = 0;
    mx = 0.0f;
#pragma unroll
    for (int v = 0; v < FHT_CL; v++) { mx = fmaxf(mx, peer_mx[v]); any_bad |= peer_bad[v]; }
    const float sc = fht_row_scale(mx, scale);
    if (part == 0 && tid == 0) s[row] = sc;
    uint32_t b[8];
    q8_short(r, 1.0f / (scale * sc), fht_q8_in_range(mx, scale) && !any_bad, b, [&](float v) { return fht_q8_exact(v, scale, sc); });
#pragma unroll
    for (int v = 0; v < 8; v++) q[row * N + v * L + part * 128 + tid] = (int8_t)b[v];
}
// Rows up to which the cluster form is taken: 1 / 64 / 128 / 142 / 143 / 148 / 296 rows take it 3.5 / 6.0 / 7.5 / 8.3 / 9.3 / 9.8 / 15.0 us, the
// other form 6.8 / 8.1 / 8.5 / 9.1 / 9.1 / 9.2 / 10.7 us (launches of a graph, inputs from memory; with 143 clusters a second wave begins). One
// CTA of 256 threads per row, in three exchanges, took 7.7 us for 1 row, 9.5 us for 64, 10 us for 148.
constexpr int FHT_CLUSTER_ROWS = 142;

static int swiglu_fht_quant(const float* g, const float* u, long ld, int M, float scale, int8_t* q, float* s, float* act, cudaStream_t st) {
    if (M == 0) return FLEXLLM_OK;
    if (M <= FHT_CLUSTER_ROWS)
        launch_cluster(fht8192_cluster_kernel, dim3(M * FHT_CL), dim3(128), FHT_CL, 0, st, g, u, ld, scale, q, s, act);
    else
        launch_k(fht8192_kernel<1>, dim3(M), dim3(128), 0, st, g, u, ld, scale, (float*)nullptr, q, s, act, FhtWindow{1, 0, 0, 0});
    return launch_status();
}

__global__ void __launch_bounds__(256) fht_generic_kernel(const float* __restrict__ x, int N, float scale,
                                                          float* __restrict__ y) {
    extern __shared__ float sb[];
    const long row = blockIdx.x;
    for (int i = threadIdx.x; i < N; i += blockDim.x) sb[i] = x[row * N + i];
    __syncthreads();
    auto stage = [&](int h) {
        for (int p = threadIdx.x; p < N / 2; p += blockDim.x) {
            int i = (p / h) * 2 * h + (p % h);
            float a = sb[i], b = sb[i + h];
            sb[i] = a + b;
            sb[i + h] = a - b;
        }
        __syncthreads();
    };
    for (int h = 2; h < N; h <<= 1) stage(h);
    stage(1);
    for (int i = threadIdx.x; i < N; i += blockDim.x) y[row * N + i] = sb[i] / scale;
}

// One warp per (token, head): lane L holds elements L and L+32 of the 64-wide head.
__global__ void __launch_bounds__(256) qk_prepare_kernel(const int8_t* __restrict__ q, const float* __restrict__ s,
                                                         const int32_t* __restrict__ pos, const float* __restrict__ cos_t,
                                                         const float* __restrict__ sin_t, long T, int H,
                                                         int8_t* __restrict__ q_out, float* __restrict__ s_out) {
    const long w = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= T * H) return;
    const long t = w / H;
    const int p = pos[t];
    const float sc_in = s[w];
    const float x0 = (float)q[w * 64 + lane] * sc_in;
    const float x1 = (float)q[w * 64 + 32 + lane] * sc_in;
    const float c = cos_t[(long)p * 32 + lane], sn = sin_t[(long)p * 32 + lane];
    float a = x0 * c - x1 * sn;   // element lane
    float b = x0 * sn + x1 * c;   // element lane + 32
    auto lane_stage = [&](int bit) {
        float pa = __shfl_xor_sync(0xffffffffu, a, 1 << bit);
        float pb = __shfl_xor_sync(0xffffffffu, b, 1 << bit);
        if (lane & (1 << bit)) { a = pa - a; b = pb - b; }
        else { a = a + pa; b = b + pb; }
    };
    lane_stage(1); lane_stage(2); lane_stage(3); lane_stage(4);
    { float lo = a, hi = b; a = lo + hi; b = lo - hi; }   // index bit 5
    lane_stage(0);
    a = a / 8.0f;
    b = b / 8.0f;
    float mx = warp_max(fmaxf(a, b)), mn = warp_min(fminf(a, b));
    const float sc = sym_scale_from(mx, mn);
    if (lane == 0) s_out[w] = sc;
    q_out[w * 64 + lane] = quant_s8(a, sc);
    q_out[w * 64 + 32 + lane] = quant_s8(b, sc);
}

// gate and up halves of one fused projection output: rows of `ld` floats, gate at g, up at u
int fht8192_rest(const float* h, int M, float scale, int8_t* q, float* s, cudaStream_t st) {
    if (M == 0) return FLEXLLM_OK;
    launch_k(fht8192_rest_kernel, dim3(M), dim3(128), 0, st, h, scale, q, s);
    return launch_status();
}
int swiglu_fht_quant_strided(const float* g, const float* u, long ld, int M, float scale, int8_t* q, float* s, cudaStream_t st) {
    return swiglu_fht_quant(g, u, ld, M, scale, q, s, nullptr, st);
}

// h gathered from g ranks as [g][M][8192/g] -> FHT-8192/scale -> per-token int8 (scale from the whole
// row), this rank's columns [r*8192/g, (r+1)*8192/g) written compactly.
int fht_quant_gathered(const float* h, int M, int g, int r, float scale, int8_t* q, float* s, cudaStream_t st) {
    if (M == 0) return FLEXLLM_OK;
    const int W = 8192 / g;
    launch_k(fht8192_kernel<2>, dim3(M), dim3(128), 0, st, h, (const float*)nullptr, 0L, scale, (float*)nullptr, q, s, (float*)nullptr,
             FhtWindow{g, (long)M, r * W, W});
    return launch_status();
}

// The same input layout, whole rows out: h [g][M][8192/g] -> FHT-8192/scale -> per-token int8 [M][8192].
int fht_quant_gathered_rows(const float* h, int M, int g, float scale, int8_t* q, float* s, cudaStream_t st) {
    if (M == 0) return FLEXLLM_OK;
    launch_k(fht8192_kernel<2>, dim3(M), dim3(128), 0, st, h, (const float*)nullptr, 0L, scale, (float*)nullptr, q, s, (float*)nullptr,
             FhtWindow{g, (long)M, 0, 8192});
    return launch_status();
}

}  // namespace flexllm

using namespace flexllm;

extern "C" int flexllm_fht(const float* x, long rows, int N, float scale, float* y, void* stream) {
    FLEXLLM_REQUIRE(x && y && rows >= 0 && N >= 2 && N <= 8192 && (N & (N - 1)) == 0);
    if (rows == 0) return FLEXLLM_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (N == 8192 && aligned(x, 16) && aligned(y, 16)) {
        fht8192_kernel<0><<<(unsigned)rows, 128, 0, st>>>(x, nullptr, N, scale, y, nullptr, nullptr, nullptr, FhtWindow{1, 0, 0, 0});
    } else {
        int threads = N / 2 < 256 ? (N / 2 < 32 ? 32 : N / 2) : 256;
        fht_generic_kernel<<<(unsigned)rows, threads, N * sizeof(float), st>>>(x, N, scale, y);
    }
    return launch_status();
}

extern "C" int flexllm_swiglu_fht_quant(const float* g, const float* u, int M, int N, float scale, int8_t* q,
                                        float* s, float* act, void* stream) {
    FLEXLLM_REQUIRE(g && u && q && s && M >= 0);
    if (N != 8192) return FLEXLLM_ENOTSUP;
    FLEXLLM_REQUIRE(aligned(g, 16) && aligned(u, 16) && aligned(q, 8) && (!act || aligned(act, 16)));
    return swiglu_fht_quant(g, u, N, M, scale, q, s, act, (cudaStream_t)stream);
}

extern "C" int flexllm_qk_prepare(const int8_t* q, const float* s, const int32_t* pos, const float* cos_t,
                                  const float* sin_t, long T, int H, int8_t* q_out, float* s_out, void* stream) {
    FLEXLLM_REQUIRE(q && s && pos && cos_t && sin_t && q_out && s_out && T >= 0 && H > 0);
    if (T == 0) return FLEXLLM_OK;
    const long warps = T * H;
    qk_prepare_kernel<<<(unsigned)((warps + 7) / 8), 256, 0, (cudaStream_t)stream>>>(q, s, pos, cos_t, sin_t, T, H, q_out, s_out);
    return launch_status();
}
