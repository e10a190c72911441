// Row-wise and elementwise operators of the quantized Llama path: per-token quantisation, dequant,
// static quantisation, RMSNorm(+quant), SiLU, gate, residual, RoPE, softmax, greedy argmax.
// All are HBM-bound: one pass over the data with 128-bit accesses where the layout allows.
#include <stdlib.h>

#include <atomic>
#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "tc_common.cuh"

namespace flexllm {

thread_local int g_last_cuda_error = 0;
thread_local LaunchMode g_pdl = kWhole;
bool programmatic_launches() {
    static const bool on = [] { const char* e = getenv("FLEXLLM_PDL"); return e ? atoi(e) != 0 : true; }();
    return on;
}
std::atomic<unsigned long long> g_launch_count{0};

int raise_shared_limit(const void* kern, size_t bytes) {
    static std::mutex lock;
    static std::unordered_map<const void*, size_t> limits[kMaxDevices];
    const int dev = current_device();
    if (dev < 0) return FLEXLLM_ECUDA;
    std::lock_guard<std::mutex> hold(lock);
    auto it = limits[dev].find(kern);
    if (it == limits[dev].end()) {
        int most = 0;
        cudaFuncAttributes fa;
        FLEXLLM_CHECK_CUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        FLEXLLM_CHECK_CUDA(cudaFuncGetAttributes(&fa, kern));
        most -= (int)fa.sharedSizeBytes;
        FLEXLLM_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        it = limits[dev].emplace(kern, (size_t)most).first;
    }
    return bytes <= it->second ? FLEXLLM_OK : cuda_status(cudaErrorInvalidValue);
}

// ---------------------------------------------------------------------------------------------
// Per-token symmetric int8 quantisation (Modules/quant.h:6-112, symmetric branch).
// One CTA per row; the row stays in registers between the max/min pass and the rounding pass.
// ---------------------------------------------------------------------------------------------
template <int VPT>  // float4 vectors per thread
__global__ void __launch_bounds__(256) quant_per_token_kernel(const float* __restrict__ x, int K,
                                                              int8_t* __restrict__ q, float* __restrict__ s) {
    __shared__ float red[64];
    pdl_sync();
    const long row = blockIdx.x;
    const float4* xr = reinterpret_cast<const float4*>(x + row * K);
    const int nv = K >> 2;
    float4 v[VPT];
    float mx = -1e32f, mn = 1e32f;
#pragma unroll
    for (int i = 0; i < VPT; i++) {
        int c = threadIdx.x + i * 256;
        if (c < nv) {
            v[i] = xr[c];
            mx = fmaxf(mx, fmaxf(fmaxf(v[i].x, v[i].y), fmaxf(v[i].z, v[i].w)));
            mn = fminf(mn, fminf(fminf(v[i].x, v[i].y), fminf(v[i].z, v[i].w)));
        }
    }
    block_max_min(mx, mn, red);
    const float sc = sym_scale_from(mx, mn);
    const DivBy dsc = div_by(sc);       // one reciprocal per row: every element is then quantised without a full division
    if (threadIdx.x == 0) s[row] = sc;
    char4* qr = reinterpret_cast<char4*>(q + row * K);
#pragma unroll
    for (int i = 0; i < VPT; i++) {
        int c = threadIdx.x + i * 256;
        if (c < nv) {
            char4 o;
            o.x = (int8_t)round_half_away_to_int(div_for_rounding(v[i].x, dsc)); o.y = (int8_t)round_half_away_to_int(div_for_rounding(v[i].y, dsc));
            o.z = (int8_t)round_half_away_to_int(div_for_rounding(v[i].z, dsc)); o.w = (int8_t)round_half_away_to_int(div_for_rounding(v[i].w, dsc));
            qr[c] = o;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Asymmetric per-token quantisation (Modules/quant.h:53-81): s = (max - min) / (2^bits - 1) (0 -> 1), zero point
// b = min, q = (unsigned) round((x - b) / s). Same structure as the symmetric kernel above.
// ---------------------------------------------------------------------------------------------
template <int VPT>
__global__ void __launch_bounds__(256) quant_per_token_asym_kernel(const float* __restrict__ x, int K, float base, unsigned mask,
                                                                   uint8_t* __restrict__ q, float* __restrict__ s, float* __restrict__ b) {
    __shared__ float red[64];
    const long row = blockIdx.x;
    const float4* xr = reinterpret_cast<const float4*>(x + row * K);
    const int nv = K >> 2;
    float4 v[VPT];
    float mx = -1e32f, mn = 1e32f;
#pragma unroll
    for (int i = 0; i < VPT; i++) {
        int c = threadIdx.x + i * 256;
        if (c < nv) {
            v[i] = xr[c];
            mx = fmaxf(mx, fmaxf(fmaxf(v[i].x, v[i].y), fmaxf(v[i].z, v[i].w)));
            mn = fminf(mn, fminf(fminf(v[i].x, v[i].y), fminf(v[i].z, v[i].w)));
        }
    }
    block_max_min(mx, mn, red);
    float sc = (mx - mn) / base;
    if (sc == 0.0f) sc = 1.0f;
    if (threadIdx.x == 0) { s[row] = sc; b[row] = mn; }
    uchar4* qr = reinterpret_cast<uchar4*>(q + row * K);
    auto qz = [&](float t) { return (unsigned char)((unsigned)(long long)roundf((t - mn) / sc) & mask); };
#pragma unroll
    for (int i = 0; i < VPT; i++) {
        int c = threadIdx.x + i * 256;
        if (c < nv) qr[c] = make_uchar4(qz(v[i].x), qz(v[i].y), qz(v[i].z), qz(v[i].w));
    }
}

// y = ((float)acc * s_tok[m]) * s_ch[n] + b_tok[m] * wsum[n]     (Modules/quant.h:146-148; every operation rounded on its own)
__global__ void dequant_asym_kernel(const int32_t* __restrict__ acc, const float* __restrict__ s_tok, const float* __restrict__ b_tok,
                                    const float* __restrict__ s_ch, const float* __restrict__ wsum, int M, int N, float* __restrict__ y) {
    const long nv = (long)M * (N >> 2);
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < nv; i += (long)gridDim.x * blockDim.x) {
        const int m = (int)(i / (N >> 2)), c = (int)(i % (N >> 2));
        const int4 a = reinterpret_cast<const int4*>(acc)[i];
        const float4 w = reinterpret_cast<const float4*>(s_ch)[c];
        const float4 z = reinterpret_cast<const float4*>(wsum)[c];
        const float st = s_tok[m], bt = b_tok[m];
        float4 o;
        o.x = ((float)a.x * st) * w.x + bt * z.x; o.y = ((float)a.y * st) * w.y + bt * z.y;
        o.z = ((float)a.z * st) * w.z + bt * z.z; o.w = ((float)a.w * st) * w.w + bt * z.w;
        reinterpret_cast<float4*>(y)[i] = o;
    }
}

// ---------------------------------------------------------------------------------------------
// Dequant (Modules/quant.h:151): y = ((float)acc * s_tok[m]) * s_ch[n]
// ---------------------------------------------------------------------------------------------
__global__ void dequant_kernel(const int32_t* __restrict__ acc, const float* __restrict__ s_tok,
                               const float* __restrict__ s_ch, int M, int N, float* __restrict__ y) {
    const long nv = (long)M * (N >> 2);
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < nv; i += (long)gridDim.x * blockDim.x) {
        int m = (int)(i / (N >> 2)), c = (int)(i % (N >> 2));
        int4 a = reinterpret_cast<const int4*>(acc)[i];
        float4 w = reinterpret_cast<const float4*>(s_ch)[c];
        float st = s_tok[m];
        float4 o;
        o.x = ((float)a.x * st) * w.x; o.y = ((float)a.y * st) * w.y;
        o.z = ((float)a.z * st) * w.z; o.w = ((float)a.w * st) * w.w;
        reinterpret_cast<float4*>(y)[i] = o;
    }
}

// ---------------------------------------------------------------------------------------------
// Static symmetric quantisation (Modules/quant.h:252-295, :166-211)
// ---------------------------------------------------------------------------------------------
__global__ void static_quant_kernel(const float* __restrict__ x, long rows, int n, const float* __restrict__ s,
                                    int s_stride, float f, int is_signed, uint8_t* __restrict__ q) {
    const long total = rows * n;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        long r = i / n;
        float d = f * s[r * s_stride];
        int v = (int)roundf(x[i] / d);
        if (is_signed) v = v > 127 ? 127 : (v < -128 ? -128 : v);
        else v = v > 255 ? 255 : v;
        q[i] = (uint8_t)v;
    }
}

// ---------------------------------------------------------------------------------------------
// RMSNorm (+ optional per-token int8 quant).
// Sum of squares follows the reference order exactly:
//   prefill (LayerNorm.h:82-114): 4 chains j = k mod 4 over the whole row, (p0+p1)+(p2+p3);
//   decode  (LayerNorm.h:263-300): `lanes` contiguous chunks, 4 chains inside each, chunk totals
//                                  added from 0 in chunk order.
// A chain is a strictly sequential fp32 accumulation, so one thread owns it. To keep all 32 lanes
// busy a warp runs 32 chains at once: in the prefill order the 4 chains of 8 different rows, in the
// decode order the (up to) 32 chains of one row. The rows sit on chip between the sum and the output
// pass: each is read from global memory once.
// ---------------------------------------------------------------------------------------------
constexpr int RMS_PIECE = 128;           // floats per row per staging step

// Prefill order: a CTA of 4 warps takes 4 consecutive rows. Each warp brings one into shared memory (coalesced 128-bit loads, all in flight at
// once); warp 0 then runs the 16 chains (4 per row) over them; afterwards every thread normalises and quantises the same columns of all four rows, whose
// gains it has held since the start -- each row is read from global memory once. Row stride D + 4 floats: the chains' reads (row rr, element
// 4k + j) fall into different banks. Requires D % 128 == 0. COLS: groups of four columns a thread.
// Bound by the ordered sums and the phases around them, which six CTAs an SM take turns in: 32768 rows of 2048 98 us (336 MB: 51 us at the copy rate), 32 rows
// 6.7 us. A warp per row in the last phase, eight rows a CTA, waited for the gains at every step: 124 and 8.5 us (rows of 4096: 493 and 15.5 us, now
// 298 and 12.1); eight rows a CTA by columns 102 and 7.0 us; four and two rows by rows 118 and 113 us.
constexpr int RMSP_ROWS = 4;
template <int COLS>
__global__ void __launch_bounds__(RMSP_ROWS * 32) rmsnorm_prefill_kernel(const float* __restrict__ x, const float* __restrict__ gamma,
                                                                         int M, int D, float eps, float* __restrict__ y,
                                                                         int8_t* __restrict__ q, float* __restrict__ s) {
    extern __shared__ __align__(16) float rows_sm[];          // [rows][D + 4], then rinv[rows]
    __shared__ uint32_t amax_sm[RMSP_ROWS][RMSP_ROWS], nan_sm[RMSP_ROWS];      // per warp: the largest magnitude of each row, rows with a NaN
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ld = D + 4, nv = D >> 2;
    const long row0 = (long)blockIdx.x * RMSP_ROWS;
    float* rinv_sm = rows_sm + RMSP_ROWS * ld;
    pdl_wait();            // before the kernels after this one may start: see rmsnorm_decode_kernel
    pdl_launch();
    float4 gm[COLS];                                          // this thread's columns of every row
#pragma unroll
    for (int i = 0; i < COLS; i++) {
        const int c = threadIdx.x + i * RMSP_ROWS * 32;
        gm[i] = c < nv ? reinterpret_cast<const float4*>(gamma)[c] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    {   // warp w brings in row w
        const bool in = row0 + w < M;
        const float4* src = reinterpret_cast<const float4*>(x + (row0 + w) * D);
        float4* dst = reinterpret_cast<float4*>(rows_sm + w * ld);
#pragma unroll 8
        for (int c = lane; c < nv; c += 32) dst[c] = in ? src[c] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    if (w == 0) {
        const int rr = lane >> 2, j = lane & 3;      // chain (row rr, residue j)
        const float* src = rows_sm + min(rr, RMSP_ROWS - 1) * ld + j;
        float ss = 0.0f;
        // blocks of 16 elements, the next block's loads under way while this one is added: a step then costs the
        // addition's latency alone
        constexpr int UB = 16;
        float cur[UB], nxt[UB];
        const int blocks = nv / UB;
        if (blocks > 0) {
#pragma unroll
            for (int i = 0; i < UB; i++) cur[i] = src[4 * i];
        }
#pragma unroll 2
        for (int bk = 0; bk < blocks; bk++) {
            const float* at = src + 4 * UB * (bk + 1 < blocks ? bk + 1 : bk);
#pragma unroll
            for (int i = 0; i < UB; i++) nxt[i] = at[4 * i];
#pragma unroll
            for (int i = 0; i < UB; i++) ss += cur[i] * cur[i];
#pragma unroll
            for (int i = 0; i < UB; i++) cur[i] = nxt[i];
        }
        for (int k = blocks * UB; k < nv; k++) { const float v = src[4 * k]; ss += v * v; }
        // (p0+p1)+(p2+p3) inside each group of four lanes
        const int base = lane & ~3;
        const float p0 = __shfl_sync(0xffffffffu, ss, base), p1 = __shfl_sync(0xffffffffu, ss, base + 1);
        const float p2 = __shfl_sync(0xffffffffu, ss, base + 2), p3 = __shfl_sync(0xffffffffu, ss, base + 3);
        const float tot = (p0 + p1) + (p2 + p3);
        if (j == 0 && rr < RMSP_ROWS) rinv_sm[rr] = 1.0f / sqrtf(tot / (float)D + eps);
    }
    __syncthreads();
    // first pass: every row's largest magnitude (max(|max|, |min|) of the row = max of |.|), fp32 output if asked for; second pass: the same products
    // again (same bits) and the quantiser
    const int rows = (int)(M - row0 < RMSP_ROWS ? M - row0 : RMSP_ROWS);
    auto normed = [&](int rr, int i, float (&o)[4]) {
        const float4 v = reinterpret_cast<const float4*>(rows_sm + rr * ld)[threadIdx.x + i * RMSP_ROWS * 32], g = gm[i];
        const float r = rinv_sm[rr];
        const f32x2 r2 = pack2(r, r);
        unpack2(mul2(mul2(pack2(v.x, v.y), r2), pack2(g.x, g.y)), o[0], o[1]);
        unpack2(mul2(mul2(pack2(v.z, v.w), r2), pack2(g.z, g.w)), o[2], o[3]);
    };
    uint32_t nan_rows = 0;
#pragma unroll
    for (int rr = 0; rr < RMSP_ROWS; rr++) {
        float amax = 0.0f, nan = 0.0f;
#pragma unroll
        for (int i = 0; i < COLS; i++) {
            const int c = threadIdx.x + i * RMSP_ROWS * 32;
            if (c >= nv) continue;
            float o[4];
            normed(rr, i, o);
            if (y && rr < rows) reinterpret_cast<float4*>(y + (row0 + rr) * D)[c] = make_float4(o[0], o[1], o[2], o[3]);
            amax = max3(max3(amax, fabsf(o[0]), fabsf(o[1])), fabsf(o[2]), fabsf(o[3]));
            nan = max3_nan(max3_nan(nan, o[0], o[1]), o[2], o[3]);
        }
        const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));      // not negative, not NaN: ordered as its bits
        if (lane == 0) amax_sm[w][rr] = m;
        nan_rows |= (uint32_t)(nan != nan) << rr;
    }
    if (!q) return;
    nan_rows = __reduce_or_sync(0xffffffffu, nan_rows);
    if (lane == 0) nan_sm[w] = nan_rows;
    __syncthreads();
    // lane rr, rr + RMSP_ROWS, ...: the scale of row rr
    const int mine = lane % RMSP_ROWS;
    uint32_t m = 0, bad = 0;
#pragma unroll
    for (int k = 0; k < RMSP_ROWS; k++) { m = max(m, amax_sm[k][mine]); bad |= nan_sm[k]; }
    const float sc_mine = sym_scale_from(__uint_as_float(m), -__uint_as_float(m)), w8_mine = 1.0f / sc_mine;         // one reciprocal per row
    const uint32_t ok_rows = __ballot_sync(0xffffffffu, !(bad >> mine & 1) && sc_mine >= 0x1p-60f && sc_mine <= 0x1p60f);
    if (w == 0 && lane < rows) s[row0 + lane] = sc_mine;
#pragma unroll
    for (int rr = 0; rr < RMSP_ROWS; rr++) {
        const float sc = __shfl_sync(0xffffffffu, sc_mine, rr), w8 = __shfl_sync(0xffffffffu, w8_mine, rr);
        const bool ok = ok_rows >> rr & 1;
        if (rr >= rows) break;
#pragma unroll
        for (int i = 0; i < COLS; i++) {
            const int c = threadIdx.x + i * RMSP_ROWS * 32;
            if (c >= nv) continue;
            float o[4];
            uint32_t b[4];
            normed(rr, i, o);
            q8_short(o, w8, ok, b, [&](float t) { return q8_exact(t, sc); });
            reinterpret_cast<uint32_t*>(q + (row0 + rr) * D)[c] = __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
        }
    }
}

// Decode order with `lanes` (4 or 8) chunks, Modules/LayerNorm.h:210-370: one CTA per row, so that the loads, the normalised values
// and the quantiser are spread over eight warps and only the ordered sums stay on one: lane = chunk*4 + j sums the squares of the chunk's
// elements k with k mod 4 == j in increasing k; the chunks' totals are added from 0 in chunk order. Latency-bound at a decode step's
// row counts. Rows of 2048, 1 / 592 / 4736 of them: 4.3 / 6.3 / 18.7 us; one warp per row, four rows a CTA, took 8.4 / 8.4 / 24.6 us.
template <int MAXV>
__global__ void __launch_bounds__(256) rmsnorm_decode_kernel(const float* __restrict__ x, const float* __restrict__ gamma, int D, float eps,
                                                                 int lanes, float* __restrict__ y, int8_t* __restrict__ q, float* __restrict__ s) {
    extern __shared__ __align__(16) float rowbuf[];          // D + 4*lanes
    __shared__ float rinv_sm, red[8];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long row = blockIdx.x;
    const int nv = D >> 2, C = D / lanes;
    const float4* gr = reinterpret_cast<const float4*>(gamma);
    float4 v[MAXV], g[MAXV];
    pdl_wait();            // before the kernels after this one may start: they ask for weights at once (see the MLP block)
    pdl_launch();
#pragma unroll
    for (int i = 0; i < MAXV; i++) {
        const int c = tid + i * 256;
        v[i] = g[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < nv) {
            v[i] = reinterpret_cast<const float4*>(x + row * D)[c];
            g[i] = gr[c];
            *reinterpret_cast<float4*>(rowbuf + c * 4 + 4 * (c * 4 / C)) = v[i];      // element e at e + 4*(e / C)
        }
    }
    __syncthreads();
    if (warp == 0) {
        const int chunk = lane >> 2, j = lane & 3;
        float ss = 0.0f;
        if (chunk < lanes) {
            const float* bc = rowbuf + chunk * (C + 4) + j;
            const int n = C >> 2;
#pragma unroll 16
            for (int k = 0; k < n; k++) { const float t = bc[4 * k]; ss += t * t; }
        }
        float tot = 0.0f;
        for (int c = 0; c < lanes; c++) {
            const float p0 = __shfl_sync(0xffffffffu, ss, c * 4 + 0), p1 = __shfl_sync(0xffffffffu, ss, c * 4 + 1);
            const float p2 = __shfl_sync(0xffffffffu, ss, c * 4 + 2), p3 = __shfl_sync(0xffffffffu, ss, c * 4 + 3);
            tot += (p0 + p1) + (p2 + p3);
        }
        if (lane == 0) rinv_sm = 1.0f / sqrtf(tot / (float)D + eps);
    }
    __syncthreads();
    const float r = rinv_sm;
    float o[4 * MAXV], mx = -1.0f, nan = 0.0f;           // mx stays below zero if every value is NaN
#pragma unroll
    for (int i = 0; i < MAXV; i++) {
        const int c = tid + i * 256;
        const bool in = c < nv;
        o[4 * i] = in ? (v[i].x * r) * g[i].x : 0.0f; o[4 * i + 1] = in ? (v[i].y * r) * g[i].y : 0.0f;
        o[4 * i + 2] = in ? (v[i].z * r) * g[i].z : 0.0f; o[4 * i + 3] = in ? (v[i].w * r) * g[i].w : 0.0f;
        if (in && y) reinterpret_cast<float4*>(y + row * D)[c] = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
#pragma unroll
        for (int k = 0; k < 4; k++) { if (in) mx = fmaxf(mx, fabsf(o[4 * i + k])); nan = max3_nan(nan, nan, o[4 * i + k]); }
    }
    if (!q) return;
    mx = warp_max(mx);
    if (lane == 0) red[warp] = mx;
    const int bad = __syncthreads_or(!(nan == nan));
#pragma unroll
    for (int w = 0; w < 8; w++) mx = fmaxf(mx, red[w]);
    if (mx < 0.0f) mx = 1e32f;                            // the reference's starting values
    const float sc = sym_scale_from(mx, -mx);
    if (tid == 0) s[row] = sc;
    uint32_t b[4 * MAXV];
    q8_short(o, 1.0f / sc, !bad && sc >= 0x1p-60f && sc <= 0x1p60f, b, [&](float t) { return q8_exact(t, sc); });
#pragma unroll
    for (int i = 0; i < MAXV; i++) {
        const int c = tid + i * 256;
        if (c < nv)
            reinterpret_cast<uint32_t*>(q + row * D)[c] =
                __byte_perm(__byte_perm(b[4 * i], b[4 * i + 1], 0x0040), __byte_perm(b[4 * i + 2], b[4 * i + 3], 0x0040), 0x5410);
    }
}

// ---------------------------------------------------------------------------------------------
// SiLU / gate / residual (Swish.h:19, Linear_Layer.h:626, Residual_Layer.h:61)
// ---------------------------------------------------------------------------------------------
template <int OP>  // 0 silu, 1 mul, 2 add
__global__ void eltwise_kernel(const float* __restrict__ a, const float* __restrict__ b, long n, float* __restrict__ y) {
    const long nv = n >> 2;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < nv; i += (long)gridDim.x * blockDim.x) {
        float4 u = reinterpret_cast<const float4*>(a)[i];
        float4 o;
        if (OP == 0) { o.x = silu_f(u.x); o.y = silu_f(u.y); o.z = silu_f(u.z); o.w = silu_f(u.w); }
        else {
            float4 v = reinterpret_cast<const float4*>(b)[i];
            if (OP == 1) { o.x = u.x * v.x; o.y = u.y * v.y; o.z = u.z * v.z; o.w = u.w * v.w; }
            else { o.x = u.x + v.x; o.y = u.y + v.y; o.z = u.z + v.z; o.w = u.w + v.w; }
        }
        reinterpret_cast<float4*>(y)[i] = o;
    }
    // tail
    for (long i = (nv << 2) + blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        if (OP == 0) y[i] = silu_f(a[i]);
        else if (OP == 1) y[i] = a[i] * b[i];
        else y[i] = a[i] + b[i];
    }
}

// ---------------------------------------------------------------------------------------------
// RoPE by table (RoPE.h:61-90): one warp per (token, head); lane k holds x[k] and x[k+32].
// ---------------------------------------------------------------------------------------------
__global__ void rope_kernel(const float* __restrict__ x, const int32_t* __restrict__ pos, const float* __restrict__ cos_t,
                            const float* __restrict__ sin_t, long T, int H, float* __restrict__ y) {
    const long w = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= T * H) return;
    const long t = w / H;
    const int p = pos[t];
    const float c = cos_t[(long)p * 32 + lane], sn = sin_t[(long)p * 32 + lane];
    const float x0 = x[w * 64 + lane], x1 = x[w * 64 + 32 + lane];
    y[w * 64 + lane] = x0 * c - x1 * sn;
    y[w * 64 + 32 + lane] = x0 * sn + x1 * c;
}

// ---------------------------------------------------------------------------------------------
// Softmax (Softmax.h:25-161 / :474-634): one warp per row. exp values are written to p first,
// then lanes 0..3 run the four sequential chains k = j mod 4, then every lane scales.
// ---------------------------------------------------------------------------------------------
__global__ void softmax_kernel(const float* __restrict__ x, long rows, int len, const int32_t* __restrict__ valid,
                               float* __restrict__ p) {
    const long row = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= rows) return;
    const float* xr = x + row * len;
    float* pr = p + row * len;
    const int nvld = valid ? valid[row] : len;
    float mx = -1e32f;
    for (int k = lane; k < len; k += 32) {
        float v = k < nvld ? xr[k] : -1e32f;
        mx = v > mx ? v : mx;
    }
    mx = warp_max(mx);
    for (int k = lane; k < len; k += 32) {
        float v = k < nvld ? xr[k] : -1e32f;
        pr[k] = ref_expf(v - mx);
    }
    __syncwarp();
    float ps = 0.0f;
    if (lane < 4) {
#pragma unroll 8
        for (int k = lane; k < len; k += 4) ps += pr[k];
    }
    float p0 = __shfl_sync(0xffffffffu, ps, 0), p1 = __shfl_sync(0xffffffffu, ps, 1);
    float p2 = __shfl_sync(0xffffffffu, ps, 2), p3 = __shfl_sync(0xffffffffu, ps, 3);
    const float r = 1.0f / ((p0 + p1) + (p2 + p3));
    for (int k = lane; k < len; k += 32) pr[k] = pr[k] * r;
}

// ---------------------------------------------------------------------------------------------
// Greedy argmax, ties to the lowest index (Logits.h:13-17 strict '>'). One CTA of 1024 threads per row, or, few long rows, a cluster of eight
// CTAs with an eighth of the row each: one SM takes 12 us for a row of 128256 (it reads 43 GB/s), which a decode step waits for; eight take 4.
// ---------------------------------------------------------------------------------------------
constexpr int ARGMAX_CL = 8;
template <int CL, int NT>
__global__ void __launch_bounds__(NT) argmax_kernel(const float* __restrict__ logits, long V, int32_t* __restrict__ idx) {
    __shared__ float sv[32];
    __shared__ int si[32];
    __shared__ float cv[CL];
    __shared__ int ci[CL];
    if (CL > 1) asm volatile("barrier.cluster.arrive.release;" ::: "memory");      // the first CTA's slots may be written once all have started
    pdl_sync();
    const int part = blockIdx.x % CL;
    const long row = blockIdx.x / CL, v1 = V * (part + 1) / CL;
    const float* l = logits + row * V;
    const float first = l[0];
    GreedyToken g;
    // strided scan in increasing v; eight loads in flight
    long v = V * part / CL + threadIdx.x;
    const bool has_first = v == 0;
    g.begin(v, v1);
    for (; v + 7L * NT < v1; v += 8L * NT) {
        float t[8];
#pragma unroll
        for (int i = 0; i < 8; i++) t[i] = l[v + (long)i * NT];
#pragma unroll
        for (int i = 0; i < 8; i++) g.take(t[i], v + (long)i * NT);
    }
    for (; v < v1; v += NT) g.take(l[v], v);
    if (has_first) g.first_of_row(first);
    g.merge_warp();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (CL > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    if (lane == 0) { sv[w] = g.v; si[w] = g.i; }
    __syncthreads();
    if (w == 0) {
        g = lane < NT / 32 ? GreedyToken(sv[lane], si[lane]) : GreedyToken();
        g.merge_warp();
        if (CL == 1) {
            if (lane == 0) idx[row] = g.i;
        } else if (lane == 0) {
            const uint32_t av = tc::cluster_addr(tc::smem_u32(cv + part), 0), ai = tc::cluster_addr(tc::smem_u32(ci + part), 0);
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(av), "f"(g.v) : "memory");
            asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(ai), "r"(g.i) : "memory");
        }
    }
    if (CL > 1) {
        tc::cluster_sync();
        if (part == 0 && w == 0) {
            g = lane < CL ? GreedyToken(cv[lane % CL], ci[lane % CL]) : GreedyToken();
            g.merge_warp();
            if (lane == 0) idx[row] = g.i;
        }
    }
}

static inline int grid_for(long n, int block, int cap = 148 * 16) {
    long g = (n + block - 1) / block;
    if (g < 1) g = 1;
    return (int)(g > cap ? cap : g);
}

}  // namespace flexllm

using namespace flexllm;

extern "C" int flexllm_version(void) { return 100; }

extern "C" const char* flexllm_status_string(int st) {
    switch (st) {
        case FLEXLLM_OK: return "ok";
        case FLEXLLM_EINVAL: return "invalid argument";
        case FLEXLLM_ECUDA: return "CUDA error";
        case FLEXLLM_ETIMEDOUT: return "device wait timed out";
        case FLEXLLM_ENOTSUP: return "unsupported shape";
        case FLEXLLM_ENOMEM: return "out of memory";
        case FLEXLLM_ETOOBIG: return "problem exceeds a fixed built-in buffer";
        case FLEXLLM_EDEVDATA: return "token id or context length in device memory out of range (clamped)";
        case FLEXLLM_EIO: return "parameter file missing or too short";
        default: return "unknown status";
    }
}

extern "C" int flexllm_last_cuda_error(void) { return g_last_cuda_error; }
extern "C" unsigned long long flexllm_launch_count(void) { return g_launch_count.load(std::memory_order_relaxed); }

extern "C" int flexllm_quant_per_token(const float* x, int M, int K, int8_t* q, float* s, void* stream) {
    FLEXLLM_REQUIRE(M >= 0 && K > 0 && (K % 4) == 0 && K <= 8192);
    if (M == 0) return FLEXLLM_OK;   // empty batch: nothing to do, pointers may be null
    FLEXLLM_REQUIRE(x && q && s);
    FLEXLLM_REQUIRE(aligned(x, 16) && aligned(q, 4));
    cudaStream_t st = (cudaStream_t)stream;
    const int nv = K / 4;
    if (nv <= 256) launch_k(quant_per_token_kernel<1>, dim3(M), dim3(256), 0, st, x, K, q, s);
    else if (nv <= 512) launch_k(quant_per_token_kernel<2>, dim3(M), dim3(256), 0, st, x, K, q, s);
    else if (nv <= 1024) launch_k(quant_per_token_kernel<4>, dim3(M), dim3(256), 0, st, x, K, q, s);
    else launch_k(quant_per_token_kernel<8>, dim3(M), dim3(256), 0, st, x, K, q, s);
    return launch_status();
}

extern "C" int flexllm_quant_per_token_asym(const float* x, int M, int K, int bits, uint8_t* q, float* s, float* b, void* stream) {
    FLEXLLM_REQUIRE(M >= 0 && K > 0 && (K % 4) == 0 && K <= 8192);
    if (bits < 2 || bits > 7) return FLEXLLM_ENOTSUP;
    if (M == 0) return FLEXLLM_OK;
    FLEXLLM_REQUIRE(x && q && s && b && aligned(x, 16) && aligned(q, 4));
    cudaStream_t st = (cudaStream_t)stream;
    const float base = (float)((1 << bits) - 1);
    const unsigned mask = (1u << bits) - 1u;
    const int nv = K / 4;
    if (nv <= 256) quant_per_token_asym_kernel<1><<<M, 256, 0, st>>>(x, K, base, mask, q, s, b);
    else if (nv <= 512) quant_per_token_asym_kernel<2><<<M, 256, 0, st>>>(x, K, base, mask, q, s, b);
    else if (nv <= 1024) quant_per_token_asym_kernel<4><<<M, 256, 0, st>>>(x, K, base, mask, q, s, b);
    else quant_per_token_asym_kernel<8><<<M, 256, 0, st>>>(x, K, base, mask, q, s, b);
    return launch_status();
}

extern "C" int flexllm_dequant_asym(const int32_t* acc, const float* s_tok, const float* b_tok, const float* s_ch, const float* wsum,
                                    int M, int N, float* y, void* stream) {
    FLEXLLM_REQUIRE(acc && s_tok && b_tok && s_ch && wsum && y && M >= 0 && N > 0 && (N % 4) == 0);
    FLEXLLM_REQUIRE(aligned(acc, 16) && aligned(s_ch, 16) && aligned(wsum, 16) && aligned(y, 16));
    if (M == 0) return FLEXLLM_OK;
    dequant_asym_kernel<<<grid_for((long)M * N / 4, 256), 256, 0, (cudaStream_t)stream>>>(acc, s_tok, b_tok, s_ch, wsum, M, N, y);
    return launch_status();
}

// The integer product of the asymmetric layers runs on the int8 GEMMs (activation values of up to 7 bits are non-negative
// int8); the zero point enters in the dequantiser.
extern "C" int flexllm_linear_prefill_asym(const uint8_t* a, const float* s_tok, const float* b_tok, const int8_t* w, const float* s_ch,
                                           const float* wsum, int M, int N, int K, int32_t* acc, float* y, void* stream) {
    FLEXLLM_REQUIRE(acc && y);
    TRY_RC(flexllm_linear_prefill_i8(reinterpret_cast<const int8_t*>(a), nullptr, w, nullptr, M, N, K, acc, nullptr, stream));
    return flexllm_dequant_asym(acc, s_tok, b_tok, s_ch, wsum, M, N, y, stream);
}
extern "C" int flexllm_linear_decode_asym(const uint8_t* a, const float* s_tok, const float* b_tok, const int8_t* w, const float* s_ch,
                                          const float* wsum, int M, int N, int K, int32_t* acc, float* y, void* stream) {
    FLEXLLM_REQUIRE(acc && y);
    TRY_RC(flexllm_linear_decode_i8(reinterpret_cast<const int8_t*>(a), nullptr, w, nullptr, M, N, K, acc, nullptr, stream));
    return flexllm_dequant_asym(acc, s_tok, b_tok, s_ch, wsum, M, N, y, stream);
}

extern "C" int flexllm_dequant(const int32_t* acc, const float* s_tok, const float* s_ch, int M, int N, float* y,
                               void* stream) {
    FLEXLLM_REQUIRE(acc && s_tok && s_ch && y && M >= 0 && N > 0 && (N % 4) == 0);
    FLEXLLM_REQUIRE(aligned(acc, 16) && aligned(s_ch, 16) && aligned(y, 16));
    if (M == 0) return FLEXLLM_OK;
    dequant_kernel<<<grid_for((long)M * N / 4, 256), 256, 0, (cudaStream_t)stream>>>(acc, s_tok, s_ch, M, N, y);
    return launch_status();
}

extern "C" int flexllm_static_quant(const float* x, long rows, int n, const float* s, int s_stride, float f,
                                    int is_signed, uint8_t* q, void* stream) {
    FLEXLLM_REQUIRE(x && s && q && rows >= 0 && n > 0 && (s_stride == 0 || s_stride == 1));
    if (rows == 0) return FLEXLLM_OK;
    static_quant_kernel<<<grid_for(rows * n, 256), 256, 0, (cudaStream_t)stream>>>(x, rows, n, s, s_stride, f, is_signed, q);
    return launch_status();
}

extern "C" int flexllm_rmsnorm_quant(const float* x, const float* gamma, int M, int D, float eps, int order,
                                     float* y, int8_t* q, float* s, void* stream) {
    FLEXLLM_REQUIRE(x && gamma && (y || q) && (!q || s) && M >= 0 && D > 0);
    FLEXLLM_REQUIRE((D % 4) == 0 && D <= 4096 && (order == 0 || order == 4 || order == 8));
    FLEXLLM_REQUIRE(order == 0 || (D % (order * 4)) == 0);
    FLEXLLM_REQUIRE(aligned(x, 16) && aligned(gamma, 16) && (!y || aligned(y, 16)) && (!q || aligned(q, 4)));
    if (M == 0) return FLEXLLM_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (order == 0) {
        if (D % RMS_PIECE != 0) return FLEXLLM_ENOTSUP;
        const int grid = (M + RMSP_ROWS - 1) / RMSP_ROWS;
        const size_t smem = ((size_t)RMSP_ROWS * (D + 4) + RMSP_ROWS) * sizeof(float);
        static std::atomic<int> attr_done[kMaxDevices];
        const int dev = current_device();
        if (dev < 0) return FLEXLLM_ECUDA;
        if (!attr_done[dev].load(std::memory_order_acquire)) {
            for (auto kern : {rmsnorm_prefill_kernel<16 / RMSP_ROWS>, rmsnorm_prefill_kernel<32 / RMSP_ROWS>}) {
                FLEXLLM_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                        (int)(((size_t)RMSP_ROWS * (4096 + 4) + RMSP_ROWS) * sizeof(float))));
                // six 33 KB CTAs per SM need the largest shared-memory carve-out
                FLEXLLM_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
            }
            attr_done[dev].store(1, std::memory_order_release);
        }
        launch_k(D <= 2048 ? rmsnorm_prefill_kernel<16 / RMSP_ROWS> : rmsnorm_prefill_kernel<32 / RMSP_ROWS>, dim3(grid), dim3(RMSP_ROWS * 32), smem, st, x, gamma, M, D, eps, y, q, s);
    } else {
        const size_t smem = (size_t)(D + 4 * order) * sizeof(float);
        launch_k(D <= 2048 ? rmsnorm_decode_kernel<2> : rmsnorm_decode_kernel<4>, dim3(M), dim3(256), smem, st, x, gamma, D, eps, order, y, q, s);
    }
    return launch_status();
}

// See include/flexllm_b200.h: both forms of exp_warp, eight values of every lane, as the kernels call them.
static __global__ void __launch_bounds__(256) exp_probe_kernel(const float* __restrict__ x, long n, int negated, float* __restrict__ y) {
    const ExpTable tab = exp_table_lane();
    const long base = ((long)blockIdx.x * 256 + threadIdx.x) * 8;
    float v[8], e[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        v[i] = base + i < n ? x[base + i] : 0.0f;
        if (!(fabsf(v[i]) <= kExpFastLimit)) v[i] = 0.0f;
    }
    if (negated) exp_warp<true>(v, e, tab);
    else exp_warp<false>(v, e, tab);
#pragma unroll
    for (int i = 0; i < 8; i++)
        if (base + i < n) y[base + i] = e[i];
}

extern "C" int flexllm_exp_probe(const float* x, long n, int negated, float* y, void* stream) {
    FLEXLLM_REQUIRE(x && y && n >= 0 && n <= (1L << 31) && (negated == 0 || negated == 1));
    if (n == 0) return FLEXLLM_OK;
    exp_probe_kernel<<<(unsigned)((n + 2047) / 2048), 256, 0, (cudaStream_t)stream>>>(x, n, negated, y);
    return launch_status();
}

extern "C" int flexllm_swish(const float* g, long n, float* y, void* stream) {
    FLEXLLM_REQUIRE(g && y && n >= 0 && aligned(g, 16) && aligned(y, 16));
    if (n == 0) return FLEXLLM_OK;
    eltwise_kernel<0><<<grid_for((n + 3) / 4, 256), 256, 0, (cudaStream_t)stream>>>(g, nullptr, n, y);
    return launch_status();
}
extern "C" int flexllm_gate(const float* a, const float* b, long n, float* y, void* stream) {
    FLEXLLM_REQUIRE(a && b && y && n >= 0 && aligned(a, 16) && aligned(b, 16) && aligned(y, 16));
    if (n == 0) return FLEXLLM_OK;
    eltwise_kernel<1><<<grid_for((n + 3) / 4, 256), 256, 0, (cudaStream_t)stream>>>(a, b, n, y);
    return launch_status();
}
extern "C" int flexllm_residual(const float* a, const float* b, long n, float* y, void* stream) {
    FLEXLLM_REQUIRE(a && b && y && n >= 0 && aligned(a, 16) && aligned(b, 16) && aligned(y, 16));
    if (n == 0) return FLEXLLM_OK;
    eltwise_kernel<2><<<grid_for((n + 3) / 4, 256), 256, 0, (cudaStream_t)stream>>>(a, b, n, y);
    return launch_status();
}

extern "C" int flexllm_rope(const float* x, const int32_t* pos, const float* cos_t, const float* sin_t, long T,
                            int H, float* y, void* stream) {
    FLEXLLM_REQUIRE(x && pos && cos_t && sin_t && y && T >= 0 && H > 0);
    if (T == 0) return FLEXLLM_OK;
    const long warps = T * H;
    rope_kernel<<<(unsigned)((warps + 7) / 8), 256, 0, (cudaStream_t)stream>>>(x, pos, cos_t, sin_t, T, H, y);
    return launch_status();
}

extern "C" int flexllm_softmax(const float* x, long rows, int len, const int32_t* valid, float* p, void* stream) {
    FLEXLLM_REQUIRE(x && p && rows >= 0 && len > 0);
    if (rows == 0) return FLEXLLM_OK;
    softmax_kernel<<<(unsigned)((rows + 3) / 4), 128, 0, (cudaStream_t)stream>>>(x, rows, len, valid, p);
    return launch_status();
}

extern "C" int flexllm_logits_argmax(const float* logits, int B, long V, int32_t* idx, void* stream) {
    FLEXLLM_REQUIRE(logits && idx && B >= 0 && V > 0);
    if (B == 0) return FLEXLLM_OK;
    // clusters while all of them run at once, and where an eighth is more than a few loads a thread
    if (B <= 64 && V >= 8192)
        launch_cluster(argmax_kernel<ARGMAX_CL, 256>, dim3(B * ARGMAX_CL), dim3(256), ARGMAX_CL, 0, (cudaStream_t)stream, logits, V, idx);
    else
        launch_k(argmax_kernel<1, 1024>, dim3(B), dim3(1024), 0, (cudaStream_t)stream, logits, V, idx);
    return launch_status();
}
