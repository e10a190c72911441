// Decode attention over a paged int8 KV cache (one new token per sequence, GQA).
//
// Cache layout, per layer (pool of `n_pages` pages of PAGE = 64 tokens, any page order):
//   K   [n_pages][HKV][PAGE][64] s8    one 64-byte row per token
//   Ks  [n_pages][HKV][PAGE]     f32   per-token-per-head scale
//   V^T [n_pages][HKV][64][PAGE] s8    transposed inside the page: for each of the 64 dims the
//                                       page's 64 tokens are contiguous, so P.V runs as dp4a over keys
//   Vs  [n_pages][HKV][PAGE]     f32
// (the reference keeps K token-major and V dimension-major for the same reason: Modules/MHA.h:85-90,
// :311-316; its caches are contiguous, Modules/MHA.h:447-559, :741-851 -- paging is new here.)
//
// One step for B sequences on one layer = the oracle's composition (decode graph order,
// SpinQuant_Llama_32_1B/MHA_i8xi8.h:1072-1111):
//   1. append : q,k -> dequant, RoPE(ctx), FHT-64/8, per-head int8 quant; k,v written at slot ctx
//   2. scores : x[h][j] = (((float)(q.k_j) * qs) * ks_j) * 0.125 for j <= ctx, per-split row max
//   3. softmax: row max, e = exp(x - max) (kept in place of x), the four ordered partial sums over
//               j mod 4, r = 1 / ((p0+p1)+(p2+p3))        -- one thread per chain, sequential adds
//   4. pv     : U_j = min(round(((e_j * r) * vs_j) / a_s), 255); O[d] += U_j * v_j[d] in int32,
//               partial sums of key ranges combined with integer atomics (exact, order-free)
//   5. out    : (float)O * a_s
// HBM-bound on the K and V pages (read once each); scores cost 2 x 4 bytes per (head, key).
#include <new>

#include "common.cuh"
#include "attention_decode.cuh"

namespace flexllm {

int* device_error_flag();
int gemm_sm_count();

static inline KvLayer kv_layer(const flexllm_kv_cache* c, int layer) {
    KvLayer l;
    l.k = c->k + (size_t)layer * c->page_bytes;
    l.v = c->v + (size_t)layer * c->page_bytes;
    l.ks = c->ks + (size_t)layer * (c->scale_bytes / 4);
    l.vs = c->vs + (size_t)layer * (c->scale_bytes / 4);
    return l;
}

// ---- 1. append ---------------------------------------------------------------------------------
// One warp per (sequence, head). Heads [0,HQ) are query heads, [HQ, HQ+HKV) key heads,
// [HQ+HKV, HQ+2*HKV) value heads.
// With IN_F32 the inputs are one fp32 row [ (HQ+2*HKV)*64 ] per sequence (q heads, k heads, v heads,
// the output of the fused q/k/v projection); value heads are then quantised per head here.
template <bool IN_F32>
__global__ void __launch_bounds__(256) dec_append_kernel(const int8_t* __restrict__ q, const float* __restrict__ qs,
                                                         const int8_t* __restrict__ k, const float* __restrict__ ks,
                                                         const int8_t* __restrict__ v, const float* __restrict__ vs,
                                                         const float* __restrict__ qkv_f32,
                                                         const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                                         KvLayer cache, const int32_t* __restrict__ page_table, int max_pages,
                                                         const int32_t* __restrict__ ctx, int B, int HQ, int HKV,
                                                         int8_t* __restrict__ q2, float* __restrict__ qs2, int max_pos,
                                                         int* error_flag) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int heads = HQ + 2 * HKV;
    if (w >= B * heads) return;
    const int b = w / heads, h = w % heads;
    const int pos = dec_guarded_pos(ctx, b, max_pos, error_flag);
    const long pg = page_table[(long)b * max_pages + pos / PAGE];
    const int slot = pos % PAGE;
    if (h >= HQ + HKV) {   // value head: into the transposed page
        const int hv = h - HQ - HKV;
        int8_t* dst = cache.v + (pg * HKV + hv) * (long)(64 * PAGE);
        if (IN_F32) {
            const float* src = qkv_f32 + (long)b * heads * 64 + (long)h * 64;
            const float a = src[lane], bb = src[lane + 32];
            const float mx = warp_max(fmaxf(a, bb)), mn = warp_min(fminf(a, bb));
            const float sc = sym_scale_from(mx, mn);
            dst[(long)lane * PAGE + slot] = quant_s8(a, sc);
            dst[(long)(lane + 32) * PAGE + slot] = quant_s8(bb, sc);
            if (lane == 0) cache.vs[(pg * HKV + hv) * PAGE + slot] = sc;
        } else {
            const int8_t* src = v + ((long)b * HKV + hv) * 64;
            dst[(long)lane * PAGE + slot] = src[lane];
            dst[(long)(lane + 32) * PAGE + slot] = src[lane + 32];
            if (lane == 0) cache.vs[(pg * HKV + hv) * PAGE + slot] = vs[(long)b * HKV + hv];
        }
        return;
    }
    const bool is_q = h < HQ;
    const int hh = is_q ? h : h - HQ;
    float x0, x1;
    if (IN_F32) {
        const float* src = qkv_f32 + (long)b * heads * 64 + (long)h * 64;
        x0 = src[lane]; x1 = src[lane + 32];
    } else {
        const int8_t* src = is_q ? q + ((long)b * HQ + hh) * 64 : k + ((long)b * HKV + hh) * 64;
        const float sc_in = is_q ? qs[(long)b * HQ + hh] : ks[(long)b * HKV + hh];
        x0 = (float)src[lane] * sc_in;
        x1 = (float)src[lane + 32] * sc_in;
    }
    const float c = cos_t[(long)pos * 32 + lane], sn = sin_t[(long)pos * 32 + lane];
    float a = x0 * c - x1 * sn;
    float bb = x0 * sn + x1 * c;
    auto lane_stage = [&](int bit) {
        float pa = __shfl_xor_sync(0xffffffffu, a, 1 << bit);
        float pb = __shfl_xor_sync(0xffffffffu, bb, 1 << bit);
        if (lane & (1 << bit)) { a = pa - a; bb = pb - bb; }
        else { a = a + pa; bb = bb + pb; }
    };
    lane_stage(1); lane_stage(2); lane_stage(3); lane_stage(4);
    { float lo = a, hi = bb; a = lo + hi; bb = lo - hi; }
    lane_stage(0);
    a = a / 8.0f;
    bb = bb / 8.0f;
    const float mx = warp_max(fmaxf(a, bb)), mn = warp_min(fminf(a, bb));
    const float sc = sym_scale_from(mx, mn);
    int8_t* dst;
    if (is_q) {
        dst = q2 + ((long)b * HQ + hh) * 64;
        if (lane == 0) qs2[(long)b * HQ + hh] = sc;
    } else {
        dst = cache.k + ((pg * HKV + hh) * PAGE + slot) * 64L;
        if (lane == 0) cache.ks[(pg * HKV + hh) * PAGE + slot] = sc;
    }
    dst[lane] = quant_s8(a, sc);
    dst[lane + 32] = quant_s8(bb, sc);
}

// Append only: the int8 K and V heads of one new token per sequence (already rotated / quantised by the caller) go to
// slot ctx[b] of the sequence's current page. One warp per (sequence, K or V head).
__global__ void __launch_bounds__(256) kv_append_kernel(const int8_t* __restrict__ k, const float* __restrict__ ks,
                                                        const int8_t* __restrict__ v, const float* __restrict__ vs, KvLayer cache,
                                                        const int32_t* __restrict__ page_table, int max_pages,
                                                        const int32_t* __restrict__ ctx, int B, int HKV, int max_pos, int* error_flag) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= B * 2 * HKV) return;
    const int b = w / (2 * HKV), h = w % (2 * HKV);
    const int pos = dec_guarded_pos(ctx, b, max_pos, error_flag);
    const long pg = page_table[(long)b * max_pages + pos / PAGE];
    const int slot = pos % PAGE;
    if (h < HKV) {
        const int8_t* src = k + ((long)b * HKV + h) * 64;
        int8_t* dst = cache.k + ((pg * HKV + h) * PAGE + slot) * 64L;
        dst[lane] = src[lane]; dst[lane + 32] = src[lane + 32];
        if (lane == 0) cache.ks[(pg * HKV + h) * PAGE + slot] = ks[(long)b * HKV + h];
    } else {
        const int hv = h - HKV;
        const int8_t* src = v + ((long)b * HKV + hv) * 64;
        int8_t* dst = cache.v + (pg * HKV + hv) * (long)(64 * PAGE);
        dst[(long)lane * PAGE + slot] = src[lane];
        dst[(long)(lane + 32) * PAGE + slot] = src[lane + 32];
        if (lane == 0) cache.vs[(pg * HKV + hv) * PAGE + slot] = vs[(long)b * HKV + hv];
    }
}

// ---- 2. scores ---------------------------------------------------------------------------------
// grid (splits, HKV, B), 256 threads: one key per thread per iteration (4 pages at a time),
// the G = HQ/HKV query heads of the group against each key.
template <int G>
__global__ void __launch_bounds__(256) dec_scores_kernel(const int8_t* __restrict__ q2, const float* __restrict__ qs2,
                                                         KvLayer cache, const int32_t* __restrict__ page_table, int max_pages,
                                                         const int32_t* __restrict__ ctx, int HQ, int HKV, int ctx_stride,
                                                         int nsplit, float* __restrict__ scores, float* __restrict__ smax, int max_pos) {
    const int split = blockIdx.x, hkv = blockIdx.y, b = blockIdx.z;
    const int nk = dec_guarded_pos(ctx, b, max_pos, nullptr) + 1;
    const int k_begin = split * KEYS_PER_CTA;
    __shared__ int qsm[G][16];
    __shared__ float red[G][8];
    if (threadIdx.x < G * 16) {
        const int g = threadIdx.x / 16, i = threadIdx.x % 16;
        qsm[g][i] = reinterpret_cast<const int*>(q2 + ((long)b * HQ + hkv * G + g) * 64)[i];
    }
    __syncthreads();
    float qsc[G];
    float mx[G];
#pragma unroll
    for (int g = 0; g < G; g++) { qsc[g] = qs2[(long)b * HQ + hkv * G + g]; mx[g] = -1e32f; }
    if (k_begin < nk) {
        const int k_end = min(nk, k_begin + KEYS_PER_CTA);
        for (int key = k_begin + threadIdx.x; key < k_end; key += 256) {
            const long pg = page_table[(long)b * max_pages + key / PAGE];
            const long row = (pg * HKV + hkv) * PAGE + (key % PAGE);
            const int4* kp = reinterpret_cast<const int4*>(cache.k + row * 64);
            const int4 k0 = kp[0], k1 = kp[1], k2 = kp[2], k3 = kp[3];
            const float ksc = cache.ks[row];
#pragma unroll
            for (int g = 0; g < G; g++) {
                int acc = 0;
                acc = __dp4a(qsm[g][0], k0.x, acc); acc = __dp4a(qsm[g][1], k0.y, acc);
                acc = __dp4a(qsm[g][2], k0.z, acc); acc = __dp4a(qsm[g][3], k0.w, acc);
                acc = __dp4a(qsm[g][4], k1.x, acc); acc = __dp4a(qsm[g][5], k1.y, acc);
                acc = __dp4a(qsm[g][6], k1.z, acc); acc = __dp4a(qsm[g][7], k1.w, acc);
                acc = __dp4a(qsm[g][8], k2.x, acc); acc = __dp4a(qsm[g][9], k2.y, acc);
                acc = __dp4a(qsm[g][10], k2.z, acc); acc = __dp4a(qsm[g][11], k2.w, acc);
                acc = __dp4a(qsm[g][12], k3.x, acc); acc = __dp4a(qsm[g][13], k3.y, acc);
                acc = __dp4a(qsm[g][14], k3.z, acc); acc = __dp4a(qsm[g][15], k3.w, acc);
                const float x = (((float)acc * qsc[g]) * ksc) * 0.125f;
                scores[((long)b * HQ + hkv * G + g) * ctx_stride + key] = x;
                mx[g] = x > mx[g] ? x : mx[g];
            }
        }
    }
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int g = 0; g < G; g++) {
        const float m = warp_max(mx[g]);
        if (lane == 0) red[g][w] = m;
    }
    __syncthreads();
    if (threadIdx.x < G) {
        float m = red[threadIdx.x][0];
        for (int i = 1; i < 8; i++) m = fmaxf(m, red[threadIdx.x][i]);
        smax[((long)b * HQ + hkv * G + threadIdx.x) * nsplit + split] = m;
    }
}

// ---- 3. softmax statistics ---------------------------------------------------------------------
// One CTA (128 threads) per (sequence, query head) row. e = exp(x - max) replaces x; the four
// chains k mod 4 are summed by four threads in increasing k (Softmax.h:514-553), staged through
// shared memory in chunks.
__global__ void __launch_bounds__(128) dec_softmax_kernel(const int32_t* __restrict__ ctx, int HQ, int ctx_stride, int nsplit,
                                                          float* __restrict__ scores, const float* __restrict__ smax,
                                                          float* __restrict__ rinv, int max_pos) {
    constexpr int CH = 2048;
    __shared__ float e_sm[CH];
    __shared__ float part[4];
    const int row = blockIdx.x;
    const int b = row / HQ;
    const int nk = dec_guarded_pos(ctx, b, max_pos, nullptr) + 1;
    float* x = scores + (long)row * ctx_stride;
    float mx = -1e32f;
    const int used = (nk + KEYS_PER_CTA - 1) / KEYS_PER_CTA;
    for (int i = 0; i < used; i++) mx = fmaxf(mx, smax[(long)row * nsplit + i]);
    float ps = 0.0f;
    for (int c0 = 0; c0 < nk; c0 += CH) {
        const int n = min(CH, nk - c0);
        for (int i = threadIdx.x; i < n; i += 128) {
            const float e = ref_expf(x[c0 + i] - mx);
            e_sm[i] = e;
            x[c0 + i] = e;
        }
        __syncthreads();
        if (threadIdx.x < 4) {
#pragma unroll 8
            for (int i = threadIdx.x; i < n; i += 4) ps += e_sm[i];   // c0 is a multiple of 4
        }
        __syncthreads();
    }
    if (threadIdx.x < 4) part[threadIdx.x] = ps;
    __syncthreads();
    if (threadIdx.x == 0) rinv[row] = 1.0f / ((part[0] + part[1]) + (part[2] + part[3]));
}

// ---- 4. P.V ------------------------------------------------------------------------------------
// grid (splits, HKV, B), 256 threads = G(4) heads x 64. Per page: thread (g, key) quantises its
// probability to u8 into shared memory; then thread (g, d) runs 16 dp4a over the page's 64 keys
// against row d of the transposed V page.
template <int G>
__global__ void __launch_bounds__(64 * G) dec_pv_kernel(KvLayer cache, const int32_t* __restrict__ page_table, int max_pages,
                                                        const int32_t* __restrict__ ctx, int HQ, int HKV, int ctx_stride,
                                                        const float* __restrict__ scores, const float* __restrict__ rinv,
                                                        const float* __restrict__ a_s, int32_t* __restrict__ oacc, int max_pos) {
    const int split = blockIdx.x, hkv = blockIdx.y, b = blockIdx.z;
    const int nk = dec_guarded_pos(ctx, b, max_pos, nullptr) + 1;
    const int k_begin = split * KEYS_PER_CTA;
    if (k_begin >= nk) return;
    const int k_end = min(nk, k_begin + KEYS_PER_CTA);
    __shared__ __align__(16) uint8_t u_sm[G][PAGE];
    const int g = threadIdx.x / 64, t = threadIdx.x % 64;
    const int hq = hkv * G + g;
    const float r = rinv[(long)b * HQ + hq];
    const float as = a_s[hq];
    const float* e = scores + ((long)b * HQ + hq) * ctx_stride;
    int acc = 0;
    for (int p0 = k_begin; p0 < k_end; p0 += PAGE) {
        const long pg = page_table[(long)b * max_pages + p0 / PAGE];
        const long prow = (pg * HKV + hkv) * PAGE;
        const int key = p0 + t;
        uint8_t u = 0;
        if (key < k_end) {
            const float p = e[key] * r;
            const float tt = (p * cache.vs[prow + t]) / as;
            int q = round_half_away_to_int(tt);
            q = q > 255 ? 255 : q;
            u = (uint8_t)q;
        }
        // this thread's V^T row for the page (issued before the barrier to overlap the latency)
        const int4* vp = reinterpret_cast<const int4*>(cache.v + (prow * 64) + (long)t * PAGE);
        const int4 v0 = vp[0], v1 = vp[1], v2 = vp[2], v3 = vp[3];
        __syncthreads();   // previous page's u_sm fully consumed
        u_sm[g][t] = u;
        __syncthreads();
        const int4* up = reinterpret_cast<const int4*>(u_sm[g]);
        const int4 u0 = up[0], u1 = up[1], u2 = up[2], u3 = up[3];
        // u is unsigned, v signed: mixed-sign dp4a
        acc = dp4a_u8s8((unsigned)u0.x, v0.x, acc); acc = dp4a_u8s8((unsigned)u0.y, v0.y, acc);
        acc = dp4a_u8s8((unsigned)u0.z, v0.z, acc); acc = dp4a_u8s8((unsigned)u0.w, v0.w, acc);
        acc = dp4a_u8s8((unsigned)u1.x, v1.x, acc); acc = dp4a_u8s8((unsigned)u1.y, v1.y, acc);
        acc = dp4a_u8s8((unsigned)u1.z, v1.z, acc); acc = dp4a_u8s8((unsigned)u1.w, v1.w, acc);
        acc = dp4a_u8s8((unsigned)u2.x, v2.x, acc); acc = dp4a_u8s8((unsigned)u2.y, v2.y, acc);
        acc = dp4a_u8s8((unsigned)u2.z, v2.z, acc); acc = dp4a_u8s8((unsigned)u2.w, v2.w, acc);
        acc = dp4a_u8s8((unsigned)u3.x, v3.x, acc); acc = dp4a_u8s8((unsigned)u3.y, v3.y, acc);
        acc = dp4a_u8s8((unsigned)u3.z, v3.z, acc); acc = dp4a_u8s8((unsigned)u3.w, v3.w, acc);
    }
    atomicAdd(oacc + ((long)b * HQ + hq) * 64 + t, acc);
}

// ---- fused single-kernel path (body in attention_decode.cuh): short contexts ------------------------------------------------------
// Grid (4 / G HKV, B): a CTA per (sequence, KV head) with the four query heads of the group, or two CTAs with two heads each, which halves
// a CTA's chain of phases for a second reading of the pages from L2. Two CTAs share an SM.
template <bool IN_F32, int NT, int G>
__global__ void __launch_bounds__(NT, 2) dec_attn_fused_kernel(const int8_t* __restrict__ q, const float* __restrict__ qs,
                                                             const int8_t* __restrict__ k, const float* __restrict__ ks,
                                                             const int8_t* __restrict__ v, const float* __restrict__ vs,
                                                             const float* __restrict__ qkv_f32, const float* __restrict__ cos_t,
                                                             const float* __restrict__ sin_t, const float* __restrict__ a_s,
                                                             KvLayer cache, const int32_t* __restrict__ page_table, int max_pages,
                                                             const int32_t* __restrict__ ctx, int HQ, int HKV, int cs,
                                                             float* __restrict__ out, int32_t* __restrict__ oacc, int max_pos,
                                                             int* error_flag) {
    extern __shared__ __align__(16) uint8_t dsm[];
    __shared__ DecAttnSmem sm;
    pdl_sync();
    DecAttnIn in;
    in.q = q; in.qs = qs; in.k = k; in.ks = ks; in.v = v; in.vs = vs; in.qkv_f32 = qkv_f32;
    in.qkv_acc = nullptr; in.tok_scale = nullptr; in.ch_scale = nullptr; in.n_slabs = 0; in.slab_stride = 0;
    in.max_pos = max_pos; in.error_flag = error_flag;
    dec_attn_fused_body<IN_F32 ? 1 : 0, NT, G>(in, cos_t, sin_t, a_s, cache, page_table, max_pages, ctx, HQ, HKV, cs, out, oacc,
                                               (int)blockIdx.x / (4 / G), (int)blockIdx.y, dsm, sm, (int)threadIdx.x, 0, (int)blockIdx.x % (4 / G));
}

template <int G>
static int launch_dec_fused(bool in_f32, const int8_t* q, const float* qs, const int8_t* k, const float* ks, const int8_t* v, const float* vs,
                            const float* qkv_f32, const float* cos_t, const float* sin_t, const float* a_s, const KvLayer& L, const int32_t* page_table,
                            int max_pages, const int32_t* ctx, int B, int HQ, int HKV, int cs, float* out, int32_t* oacc, int max_ctx, int* err,
                            cudaStream_t st) {
    const size_t smem = dec_attn_smem_bytes<G>(cs);
    auto kern = in_f32 ? dec_attn_fused_kernel<true, 512, G> : dec_attn_fused_kernel<false, 512, G>;
    TRY_RC(allow_shared(kern, smem));
    launch_k(kern, dim3(4 / G * HKV, B), dim3(512), smem, st, q, qs, k, ks, v, vs, qkv_f32, cos_t, sin_t, a_s, L, page_table, max_pages, ctx,
             HQ, HKV, cs, out, oacc, max_ctx, err);
    return launch_status(1);
}

// ---- the same step by a cluster of four CTAs per (sequence, KV head) ------------------------------------------------------------------
// Grid (4 HKV, B). CTA r takes the r-th quarter of the item's pages for the two products, so every page is read by one SM only, and the softmax of
// the group's query head r over all keys, so the ordered sums run for the four heads at once. Scores go straight into the shared memory of the
// CTA of their head, the 8-bit probabilities from there to the CTA that has the key's page; three cluster barriers in all. Both
// products are warp-level integer MMAs whose inner index is permuted the same way on both sides, so that a lane's 16 consecutive
// bytes of a row are its four operand words. A CTA needs 5 bytes per key, so four share an SM (64 registers a thread): while one waits for its
// pages, its peers or the ordered sums, the others have work.
// Bound by that chain of phases (64 x 8100 keys, one generation of CTAs: 46 us, of which the scores 11, ordered sums 8, P.V 5) and by memory:
// 64 sequences of 512 to 8192 keys (47 us at the copy rate), calls one after another: 99 to 116 us by the draw of the lengths, 122 to 146 with every
// page read by two SMs.
constexpr int DEC_FUSED_KEYS = 10240;      // most keys of the forms with an item per CTA
constexpr int DEC_CL = 4, DEC_CL_NT = 256, DEC_CL_PAGES = 512;       // CTAs of a cluster (one per query head), threads, most pages of a sequence
struct DecClusterSmem {
    __align__(16) int8_t q_sm[4][64];
    __align__(16) int8_t new_k[64];
    float q_scale[4], new_ks, wmax[32], rinv;
    int pv[4][64], tot[64];
    int pt[DEC_CL_PAGES];
    int b;
};
// dynamic shared memory: one score row over all pages, then four rows of 8-bit probabilities over a CTA's pages
__host__ __device__ constexpr int dec_cluster_own(int pages) { return (pages + DEC_CL - 1) / DEC_CL; }
constexpr size_t dec_cluster_smem_bytes(int pages) { return (size_t)pages * PAGE * 4 + (size_t)DEC_CL * dec_cluster_own(pages) * PAGE; }

__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cluster_u32(uint32_t addr, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

template <bool IN_F32>
__global__ void __launch_bounds__(DEC_CL_NT, 4) dec_attn_cluster_kernel(const DecAttnIn in, const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                                                        const float* __restrict__ a_s, KvLayer cache,
                                                                        const int32_t* __restrict__ page_table, int max_pages,
                                                                        const int32_t* __restrict__ ctx, int HQ, int HKV, int pages, int rank_b,
                                                                        float* __restrict__ out, int32_t* __restrict__ oacc) {
    constexpr int NW = DEC_CL_NT / 32, CL = DEC_CL;
    extern __shared__ __align__(16) uint8_t dsm[];
    __shared__ DecClusterSmem sm;
    float* row = reinterpret_cast<float*>(dsm);                      // [pages * PAGE]: scores, then exponentials, of head r
    uint8_t* u_sm = dsm + (size_t)pages * PAGE * 4;                  // [4][own * PAGE]
    const int ur = dec_cluster_own(pages) * PAGE;                    // row length of u_sm
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, gi = lane >> 2, ti = lane & 3;
    const int r = blockIdx.x % CL, hkv = blockIdx.x / CL;
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");    // the peers may write here once all have arrived (waited for below)
    sm.pv[tid >> 6][tid & 63] = 0;
    if (tid < 64) sm.tot[tid] = 0;
    pdl_sync();
    int b = blockIdx.y;
    if (rank_b) {
        // grid row y takes the sequence with the y-th largest context (equal ones in order): the last clusters to start are the shortest
        const int B = gridDim.y;
        int* len = reinterpret_cast<int*>(u_sm);                     // (no peer writes here before the second cluster barrier)
        for (int t = tid; t < B; t += DEC_CL_NT) len[t] = ctx[t];
        __syncthreads();
        for (int t0 = 0; t0 < B; t0 += DEC_CL_NT / 4) {              // four lanes count for one sequence
            const int t = t0 + (tid >> 2), mine = t < B ? len[t] : 0;
            int rank = 0;
#pragma unroll 4
            for (int u = ti; u < B; u += 4) rank += len[u] > mine || (len[u] == mine && u < t);
            rank += __shfl_xor_sync(0xffffffffu, rank, 1);
            rank += __shfl_xor_sync(0xffffffffu, rank, 2);
            if (t < B && rank == (int)blockIdx.y) sm.b = t;
        }
        __syncthreads();
        b = sm.b;
    }
    const int heads = HQ + 2 * HKV;
    const int pos = dec_guarded_pos(ctx, b, in.max_pos, in.error_flag);
    const int nk = pos + 1, np_all = (nk + PAGE - 1) / PAGE;
    auto first_page = [&](int c) { return np_all * c / CL; };        // of CTA c
    const int p0 = first_page(r), np = first_page(r + 1) - p0;       // this CTA's pages (none in short contexts)
    const bool has_new = r == CL - 1;                                // the new token is in the last page
    for (int p = tid; p < np_all; p += DEC_CL_NT) sm.pt[p] = page_table[(long)b * max_pages + p];
    // ---- A. prepare: warps 0..3 the query heads (every CTA), warp 4 the key head and warp 5 the value head (the CTA that has the new token)
    if (w < 4 || (w < 6 && has_new)) {
        const int h = w < 4 ? hkv * 4 + w : (w == 4 ? HQ + hkv : HQ + HKV + hkv);
        float a, bb;
        int8_t c0 = 0, c1 = 0;
        float sc_in = 0.0f;
        if (IN_F32) {
            const float* src = in.qkv_f32 + (long)b * heads * 64 + (long)h * 64;
            a = src[lane]; bb = src[lane + 32];
        } else {
            const int8_t* src = w < 4 ? in.q + ((long)b * HQ + hkv * 4 + w) * 64 : (w == 4 ? in.k : in.v) + ((long)b * HKV + hkv) * 64;
            sc_in = w < 4 ? in.qs[(long)b * HQ + hkv * 4 + w] : (w == 4 ? in.ks : in.vs)[(long)b * HKV + hkv];
            c0 = src[lane]; c1 = src[lane + 32];
            a = (float)c0 * sc_in; bb = (float)c1 * sc_in;
        }
        const int slot = pos % PAGE;
        const long pg = w >= 4 ? page_table[(long)b * max_pages + pos / PAGE] : 0;
        float s2 = sc_in;
        int8_t qa = c0, qb = c1;                                     // an int8 value head is copied
        if (IN_F32 || w < 5) {
            if (w < 5) {
                const float c = cos_t[(long)pos * 32 + lane], sn = sin_t[(long)pos * 32 + lane];
                const float x0 = a, x1 = bb;
                a = x0 * c - x1 * sn;
                bb = x0 * sn + x1 * c;
                auto lane_stage = [&](int bit) {
                    float pa = __shfl_xor_sync(0xffffffffu, a, 1 << bit);
                    float pb = __shfl_xor_sync(0xffffffffu, bb, 1 << bit);
                    if (lane & (1 << bit)) { a = pa - a; bb = pb - bb; }
                    else { a = a + pa; bb = bb + pb; }
                };
                lane_stage(1); lane_stage(2); lane_stage(3); lane_stage(4);
                { float lo = a, hi = bb; a = lo + hi; bb = lo - hi; }
                lane_stage(0);
                a = a / 8.0f;
                bb = bb / 8.0f;
            }
            const float mx = warp_max(fmaxf(a, bb)), mn = warp_min(fminf(a, bb));
            s2 = sym_scale_from(mx, mn);
            qa = quant_s8(a, s2); qb = quant_s8(bb, s2);
        }
        if (w < 4) {
            sm.q_sm[w][lane] = qa; sm.q_sm[w][lane + 32] = qb;
            if (lane == 0) sm.q_scale[w] = s2;
        } else if (w == 4) {                                         // into the cache, and beside it for this step's product
            int8_t* dst = cache.k + ((pg * HKV + hkv) * PAGE + slot) * 64L;
            dst[lane] = qa; dst[lane + 32] = qb;
            sm.new_k[lane] = qa; sm.new_k[lane + 32] = qb;
            if (lane == 0) { cache.ks[(pg * HKV + hkv) * PAGE + slot] = s2; sm.new_ks = s2; }
        } else {
            int8_t* dst = cache.v + (pg * HKV + hkv) * (long)(64 * PAGE);
            dst[(long)lane * PAGE + slot] = qa;
            dst[(long)(lane + 32) * PAGE + slot] = qb;
            if (lane == 0) cache.vs[(pg * HKV + hkv) * PAGE + slot] = s2;
        }
    }
    __syncthreads();
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");      // every peer has started
    // ---- B. scores: a warp takes a page at a time; A = 16 key rows, B = the four query heads (columns 4..7 zero). Lanes with ti = 2, 3 take over
    //         the sums of key rows 8..15 from lanes ti - 2: every lane then has one key of two heads.
    {
        int bq[4];
#pragma unroll
        for (int i = 0; i < 4; i++) bq[i] = gi < 4 ? *reinterpret_cast<const int*>(&sm.q_sm[gi & 3][ti * 16 + i * 4]) : 0;
        const int h0 = (ti & 1) * 2, kl = gi + 8 * (ti >> 1);
        const float qs0 = sm.q_scale[h0], qs1 = sm.q_scale[h0 + 1];
        const uint32_t row0 = tc::cluster_addr(tc::smem_u32(row), h0), row1 = tc::cluster_addr(tc::smem_u32(row), h0 + 1);
        float mx0 = -1e32f, mx1 = -1e32f;
        for (int p = w; p < np; p += NW) {
            const long base = (long)sm.pt[p0 + p] * HKV + hkv;
            const int8_t* rows = cache.k + base * (long)(64 * PAGE) + gi * 64 + ti * 16;
            int4 k4[8];
            float ks[4];
#pragma unroll
            for (int i = 0; i < 8; i++) k4[i] = *reinterpret_cast<const int4*>(rows + i * 512);
#pragma unroll
            for (int i = 0; i < 4; i++) ks[i] = cache.ks[base * PAGE + i * 16 + kl];
            // the page of V is asked into L2 meanwhile, with its scales
            asm volatile("prefetch.global.L2 [%0];" ::"l"(cache.v + base * (long)(64 * PAGE) + lane * 128));
            if (lane < 2) asm volatile("prefetch.global.L2 [%0];" ::"l"(cache.vs + base * PAGE + lane * 32));
            if (has_new && p == np - 1) {                            // the new token's row, which the loads may or may not have seen
                const int slot = pos % PAGE;
#pragma unroll
                for (int i = 0; i < 8; i++) if (i * 8 + gi == slot) k4[i] = *reinterpret_cast<const int4*>(sm.new_k + ti * 16);
#pragma unroll
                for (int i = 0; i < 4; i++) if (i * 16 + kl == slot) ks[i] = sm.new_ks;
            }
            const int key0 = (p0 + p) * PAGE + kl;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                int d[4] = {0, 0, 0, 0};
                const int a0[4] = {k4[2 * i].x, k4[2 * i + 1].x, k4[2 * i].y, k4[2 * i + 1].y}, b0[2] = {bq[0], bq[1]};
                const int a1[4] = {k4[2 * i].z, k4[2 * i + 1].z, k4[2 * i].w, k4[2 * i + 1].w}, b1[2] = {bq[2], bq[3]};
                mma_s8s8(d, a0, b0);
                mma_s8s8(d, a1, b1);
                const int o2 = __shfl_sync(0xffffffffu, d[2], lane & ~2), o3 = __shfl_sync(0xffffffffu, d[3], lane & ~2);
                const float x0 = (((float)(ti < 2 ? d[0] : o2) * qs0) * ks[i]) * 0.125f, x1 = (((float)(ti < 2 ? d[1] : o3) * qs1) * ks[i]) * 0.125f;
                const int key = key0 + i * 16;
                st_cluster_f32(row0 + key * 4, x0);
                st_cluster_f32(row1 + key * 4, x1);
                if (key < nk) { mx0 = x0 > mx0 ? x0 : mx0; mx1 = x1 > mx1 ? x1 : mx1; }
            }
        }
        // maximum over the lanes with the same ti & 1 (xor 2, 4, 8, 16)
#pragma unroll
        for (int o = 2; o < 32; o <<= 1) {
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
        }
        // lanes 0 and 2 hold heads 0 and 1, lanes 1 and 3 heads 2 and 3
        if (lane < 4) st_cluster_f32(tc::cluster_addr(tc::smem_u32(&sm.wmax[r * NW + w]), ((lane & 1) << 1) | (lane >> 1)), lane >> 1 ? mx1 : mx0);
    }
    const ExpTable tab = exp_table_lane();
    tc::cluster_sync();
    // ---- D. e = exp(x - max) in place, zero beyond the last key: eight values at a time
    const int npk = np_all * PAGE;
    {
        const float m = warp_max(sm.wmax[lane]) + 0.0f;              // a zero without a sign: max - x is then never -0 (exp_warp)
        for (int k0 = w * 256; k0 < npk; k0 += DEC_CL_NT * 8) {      // a warp takes 256 keys, a lane eight of them
            float u[8], e[8], far = 0.0f;
            float4* at[2];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int key = k0 + i * 128 + lane * 4;
                at[i] = reinterpret_cast<float4*>(row + key);
                const float4 x = key < npk ? *at[i] : make_float4(m, m, m, m);
                u[4 * i] = key < nk ? m - x.x : 0.0f; u[4 * i + 1] = key + 1 < nk ? m - x.y : 0.0f;
                u[4 * i + 2] = key + 2 < nk ? m - x.z : 0.0f; u[4 * i + 3] = key + 3 < nk ? m - x.w : 0.0f;
                far = max3_nan(max3_nan(far, u[4 * i], u[4 * i + 1]), u[4 * i + 2], u[4 * i + 3]);
            }
            if (__all_sync(0xffffffffu, far <= kExpFastLimit)) exp_warp<true>(u, e, tab);
            else {
#pragma unroll
                for (int i = 0; i < 8; i++) e[i] = ref_expf(-u[i]);
            }
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int key = k0 + i * 128 + lane * 4;
                if (key < npk) *at[i] = make_float4(key < nk ? e[4 * i] : 0.0f, key + 1 < nk ? e[4 * i + 1] : 0.0f, key + 2 < nk ? e[4 * i + 2] : 0.0f,
                                                    key + 3 < nk ? e[4 * i + 3] : 0.0f);
            }
        }
    }
    __syncthreads();
    // ---- E. the four ordered chains of the head, key = j mod 4 (Softmax.h:514-553): one lane per chain, the 16 terms of a page at a time, the next page's
    //         loads under way while this one is added: a step costs the addition's latency. (The zeros of the last page change nothing.)
    //         Meanwhile the other warps, which quantise, fetch their keys' V scales.
    constexpr int FV = 8, F_KEYS = (DEC_CL_NT - 32) * 4;             // vectors of four scales held by a thread, keys of one pass over its warps
    float4 vs4[FV];
    auto v_scales = [&](int k) { return *reinterpret_cast<const float4*>(cache.vs + ((long)sm.pt[k / PAGE] * HKV + hkv) * PAGE + k % PAGE); };
    if (w == 0) {
        float ps = 0.0f, c0[16], c1[16];
        auto load = [&](float (&c)[16], int p) {
#pragma unroll
            for (int t = 0; t < 16; t++) c[t] = row[p * PAGE + 4 * t + ti];
        };
        auto add = [&](const float (&c)[16]) {
#pragma unroll
            for (int t = 0; t < 16; t++) ps += c[t];
        };
        load(c0, 0);
        int p = 0;
        for (; p + 2 < np_all; p += 2) { load(c1, p + 1); add(c0); load(c0, p + 2); add(c1); }
        if (p + 1 < np_all) { load(c1, p + 1); add(c0); add(c1); }
        else add(c0);
        const float q0 = __shfl_sync(0xffffffffu, ps, 0), q1 = __shfl_sync(0xffffffffu, ps, 1);
        const float q2 = __shfl_sync(0xffffffffu, ps, 2), q3 = __shfl_sync(0xffffffffu, ps, 3);
        if (lane == 0) sm.rinv = 1.0f / ((q0 + q1) + (q2 + q3));
    } else {
#pragma unroll
        for (int i = 0; i < FV; i++) {
            const int k = i * F_KEYS + (tid - 32) * 4;
            if (k < npk) vs4[i] = v_scales(k);
        }
    }
    __syncthreads();
    // ---- F. probabilities to u8 (zero beyond the last key), four keys a thread, into the CTA that has their page
    if (w > 0) {
        const float rinv = sm.rinv, as = a_s[hkv * 4 + r];
        bool ok;
        const float c = dec_u8_factor(rinv, as, ok);
        const uint32_t u_at = tc::smem_u32(u_sm) + r * ur;
        const int f1 = first_page(1), f2 = first_page(2), f3 = first_page(3);
        auto quantise = [&](int k, const float4& s4) {
            const int p = k / PAGE, own = (p >= f1) + (p >= f2) + (p >= f3), fp = own == 0 ? 0 : own == 1 ? f1 : own == 2 ? f2 : f3;
            const float4 e4 = *reinterpret_cast<const float4*>(row + k);
            const float e[4] = {e4.x, e4.y, e4.z, e4.w}, vs[4] = {s4.x, s4.y, s4.z, s4.w};
            uint32_t v = 0;
#pragma unroll
            for (int i = 0; i < 4; i++) v |= (k + i < nk ? dec_u8(e[i], c, ok, rinv, vs[i], as) : 0u) << (8 * i);
            st_cluster_u32(tc::cluster_addr(u_at + (p - fp) * PAGE + k % PAGE, own), v);
        };
#pragma unroll
        for (int i = 0; i < FV; i++) {
            const int k = i * F_KEYS + (tid - 32) * 4;
            if (k < npk) quantise(k, vs4[i]);
        }
        for (int k = FV * F_KEYS + (tid - 32) * 4; k < npk; k += F_KEYS) quantise(k, v_scales(k));
    }
    tc::cluster_sync();
    // ---- G. P.V, a page per warp at a time: A = 16 dims x keys of the V^T page, B = keys x the four heads
    {
        int acc[4][4] = {};
        for (int p = w; p < np; p += NW) {
            const long base = (long)sm.pt[p0 + p] * HKV + hkv;
            const int8_t* rows = cache.v + base * (long)(64 * PAGE) + gi * PAGE + ti * 16;
            int4 v4[8];
#pragma unroll
            for (int i = 0; i < 8; i++) v4[i] = *reinterpret_cast<const int4*>(rows + i * 8 * PAGE);
            const int4 u4 = gi < 4 ? *reinterpret_cast<const int4*>(u_sm + gi * ur + p * PAGE + ti * 16) : make_int4(0, 0, 0, 0);
            const int b0[2] = {u4.x, u4.y}, b1[2] = {u4.z, u4.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int a0[4] = {v4[2 * i].x, v4[2 * i + 1].x, v4[2 * i].y, v4[2 * i + 1].y};
                const int a1[4] = {v4[2 * i].z, v4[2 * i + 1].z, v4[2 * i].w, v4[2 * i + 1].w};
                mma_s8u8(acc[i], a0, b0);
                mma_s8u8(acc[i], a1, b1);
            }
        }
        if (ti < 2 && w < np) {
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) atomicAdd(&sm.pv[2 * ti + (j & 1)][i * 16 + gi + (j >> 1) * 8], acc[i][j]);
        }
    }
    __syncthreads();
    if (np > 0)                                                      // whole numbers: exact in any order
        asm volatile("red.relaxed.cluster.shared::cluster.add.s32 [%0], %1;"
                     ::"r"(tc::cluster_addr(tc::smem_u32(&sm.tot[tid & 63]), tid >> 6)), "r"(sm.pv[tid >> 6][tid & 63]) : "memory");
    tc::cluster_sync();
    if (tid < 64) {
        const int hq = hkv * 4 + r, tot = sm.tot[tid];
        const long o = ((long)b * HQ + hq) * 64 + tid;
        out[o] = (float)tot * a_s[hq];
        if (oacc) oacc[o] = tot;
    }
}

static int launch_dec_cluster(bool in_f32, const DecAttnIn& in, const float* cos_t, const float* sin_t, const float* a_s, const KvLayer& L,
                              const int32_t* page_table, int max_pages, const int32_t* ctx, int B, int HQ, int HKV, int pages, bool rank, float* out,
                              int32_t* oacc, cudaStream_t st) {
    const size_t smem = dec_cluster_smem_bytes(pages);
    auto kern = in_f32 ? dec_attn_cluster_kernel<true> : dec_attn_cluster_kernel<false>;
    TRY_RC(allow_shared(kern, smem));
    launch_cluster(kern, dim3(DEC_CL * HKV, B), dim3(DEC_CL_NT), DEC_CL, smem, st, in, cos_t, sin_t, a_s, L, page_table, max_pages, ctx, HQ, HKV,
                   pages, rank ? 1 : 0, out, oacc);
    return launch_status(1);
}

// ---- 5. out ------------------------------------------------------------------------------------
__global__ void dec_out_kernel(const int32_t* __restrict__ oacc, const float* __restrict__ a_s, int B, int HQ,
                               float* __restrict__ out, int32_t* __restrict__ oacc_out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B * HQ * 64) return;
    const int hq = (i / 64) % HQ;
    const int v = oacc[i];
    out[i] = (float)v * a_s[hq];
    if (oacc_out) oacc_out[i] = v;
}

}  // namespace flexllm

using namespace flexllm;

static size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

extern "C" int flexllm_kv_cache_create(flexllm_kv_cache** out, int layers, int n_pages, int hkv, int page) {
    FLEXLLM_REQUIRE(out && layers > 0 && n_pages > 0 && hkv > 0);
    if (page != PAGE) return FLEXLLM_ENOTSUP;
    flexllm_kv_cache* c = new (std::nothrow) flexllm_kv_cache();
    if (!c) return FLEXLLM_ENOMEM;
    c->layers = layers; c->n_pages = n_pages; c->hkv = hkv; c->page = page; c->elem_bytes = 1; c->k_bytes = c->v_bytes = 0;
    c->page_bytes = (size_t)n_pages * hkv * PAGE * 64;
    c->scale_bytes = (size_t)n_pages * hkv * PAGE * sizeof(float);
    c->k = c->v = nullptr; c->ks = c->vs = nullptr;
    cudaError_t e = cudaMalloc(&c->k, c->page_bytes * layers);
    if (e == cudaSuccess) e = cudaMalloc(&c->v, c->page_bytes * layers);
    if (e == cudaSuccess) e = cudaMalloc(&c->ks, c->scale_bytes * layers);
    if (e == cudaSuccess) e = cudaMalloc(&c->vs, c->scale_bytes * layers);
    if (e != cudaSuccess) {
        flexllm_kv_cache_destroy(c);
        g_last_cuda_error = (int)e;
        return e == cudaErrorMemoryAllocation ? FLEXLLM_ENOMEM : FLEXLLM_ECUDA;
    }
    *out = c;
    return flexllm_kv_cache_reset(c, nullptr);
}

// Floating-point flavour: one pool pair per layer, each with its own shape (256-byte aligned inside two allocations).
extern "C" int flexllm_kv_cache_create_float(flexllm_kv_cache** out, int layers, int n_pages, const flexllm_kv_shape* shapes, int page,
                                             int elem_bytes) {
    FLEXLLM_REQUIRE(out && layers >= 0 && n_pages > 0 && (shapes || layers == 0) && (elem_bytes == 2 || elem_bytes == 4));
    if (page != PAGE) return FLEXLLM_ENOTSUP;
    for (int l = 0; l < layers; l++) FLEXLLM_REQUIRE(shapes[l].hkv > 0 && shapes[l].kdim > 0 && shapes[l].vdim > 0);
    flexllm_kv_cache* c = new (std::nothrow) flexllm_kv_cache();
    if (!c) return FLEXLLM_ENOMEM;
    c->layers = layers; c->n_pages = n_pages; c->hkv = 0; c->page = page; c->elem_bytes = elem_bytes;
    c->page_bytes = c->scale_bytes = 0;
    c->k = c->v = nullptr; c->ks = c->vs = nullptr;
    c->shape.assign(shapes, shapes + layers);
    size_t nk = 0, nv = 0;
    for (int l = 0; l < layers; l++) {
        c->k_off.push_back(nk); c->v_off.push_back(nv);
        nk += align_up((size_t)n_pages * shapes[l].hkv * PAGE * shapes[l].kdim * elem_bytes, 256);
        nv += align_up((size_t)n_pages * shapes[l].hkv * PAGE * shapes[l].vdim * elem_bytes, 256);
    }
    c->k_bytes = nk; c->v_bytes = nv;
    cudaError_t e = cudaMalloc(&c->k, nk ? nk : 256);
    if (e == cudaSuccess) e = cudaMalloc(&c->v, nv ? nv : 256);
    if (e != cudaSuccess) {
        flexllm_kv_cache_destroy(c);
        g_last_cuda_error = (int)e;
        return e == cudaErrorMemoryAllocation ? FLEXLLM_ENOMEM : FLEXLLM_ECUDA;
    }
    *out = c;
    return flexllm_kv_cache_reset(c, nullptr);
}

int flexllm::kv_cache_add_states(flexllm_kv_cache* c, int slots, const std::vector<size_t>& slot_bytes) {
    FLEXLLM_REQUIRE(c && !c->states && c->elem_bytes != 1 && slots > 0);
    size_t n = 0;
    for (size_t b : slot_bytes) {
        c->s_off.push_back(n); c->s_slot.push_back(b);
        n += align_up(b * slots, 256);
    }
    c->states_bytes = n;
    if (n == 0) return FLEXLLM_OK;
    const cudaError_t e = cudaMalloc(&c->states, n);
    if (e != cudaSuccess) { g_last_cuda_error = (int)e; return e == cudaErrorMemoryAllocation ? FLEXLLM_ENOMEM : FLEXLLM_ECUDA; }
    return cuda_status(cudaMemset(c->states, 0, n));
}

extern "C" int flexllm_kv_cache_destroy(flexllm_kv_cache* c) {
    if (!c) return FLEXLLM_OK;
    cudaFree(c->k); cudaFree(c->v); cudaFree(c->ks); cudaFree(c->vs); cudaFree(c->states);
    delete c;
    return FLEXLLM_OK;
}

extern "C" int flexllm_kv_cache_reset(flexllm_kv_cache* c, void* stream) {
    FLEXLLM_REQUIRE(c);
    cudaStream_t st = (cudaStream_t)stream;
    if (c->elem_bytes != 1) {
        FLEXLLM_CHECK_CUDA(cudaMemsetAsync(c->k, 0, c->k_bytes, st));
        FLEXLLM_CHECK_CUDA(cudaMemsetAsync(c->v, 0, c->v_bytes, st));
        if (c->states) FLEXLLM_CHECK_CUDA(cudaMemsetAsync(c->states, 0, c->states_bytes, st));
        return FLEXLLM_OK;
    }
    FLEXLLM_CHECK_CUDA(cudaMemsetAsync(c->k, 0, c->page_bytes * c->layers, st));
    FLEXLLM_CHECK_CUDA(cudaMemsetAsync(c->v, 0, c->page_bytes * c->layers, st));
    FLEXLLM_CHECK_CUDA(cudaMemsetAsync(c->ks, 0, c->scale_bytes * c->layers, st));
    FLEXLLM_CHECK_CUDA(cudaMemsetAsync(c->vs, 0, c->scale_bytes * c->layers, st));
    return FLEXLLM_OK;
}

extern "C" int flexllm_kv_cache_pools(flexllm_kv_cache* c, int layer, int8_t** k, float** ks, int8_t** v, float** vs) {
    FLEXLLM_REQUIRE(c && layer >= 0 && layer < c->layers);
    if (c->elem_bytes != 1) {
        if (k) *k = c->k + c->k_off[layer];
        if (ks) *ks = nullptr;
        if (v) *v = c->v + c->v_off[layer];
        if (vs) *vs = nullptr;
        return FLEXLLM_OK;
    }
    KvLayer l = kv_layer(c, layer);
    if (k) *k = l.k;
    if (ks) *ks = l.ks;
    if (v) *v = l.v;
    if (vs) *vs = l.vs;
    return FLEXLLM_OK;
}

extern "C" size_t flexllm_mha_decode_workspace(int B, int HQ, int max_ctx) {
    if (B <= 0 || HQ <= 0 || max_ctx < 0) return 0;
    const size_t ctx_stride = align_up((size_t)max_ctx + 1, 64);
    const size_t nsplit = (ctx_stride + KEYS_PER_CTA - 1) / KEYS_PER_CTA;
    size_t n = 0;
    n += align_up((size_t)B * HQ * 64, 256);                 // q2
    n += align_up((size_t)B * HQ * 4, 256);                  // qs2
    n += align_up((size_t)B * HQ * ctx_stride * 4, 256);     // scores / e
    n += align_up((size_t)B * HQ * nsplit * 4, 256);         // per-split max
    n += align_up((size_t)B * HQ * 4, 256);                  // 1 / sum
    n += align_up((size_t)B * HQ * 64 * 4, 256);             // int32 accumulators
    return n + 256;
}

namespace flexllm {
// Shared body of the int8 and fp32 front ends (qkv_f32 != nullptr selects the latter).
int mha_decode_run(flexllm_kv_cache* c, int layer, const int8_t* q, const float* qs, const int8_t* k, const float* ks,
                   const int8_t* v, const float* vs, const float* qkv_f32, const float* cos_t, const float* sin_t,
                   const float* a_s, const int32_t* page_table, int max_pages, const int32_t* ctx, int max_ctx, int B, int HQ,
                   float* out, int32_t* oacc, void* workspace, cudaStream_t st);

}  // namespace flexllm

// The cache managers' append on its own (dec_K_cache_manager_template / dec_V_cache_manager_template,
// Modules/MHA.h:484-513, :773-801): store the new token's K and V heads at position ctx[b], nothing else.
extern "C" int flexllm_kv_append(flexllm_kv_cache* c, int layer, const int8_t* k, const float* ks, const int8_t* v, const float* vs,
                                 const int32_t* page_table, int max_pages, const int32_t* ctx, int max_ctx, int B, void* stream) {
    FLEXLLM_REQUIRE(c && c->elem_bytes == 1 && layer >= 0 && layer < c->layers && B >= 0 && max_ctx >= 0 && max_pages > 0);
    if (B == 0) return FLEXLLM_OK;
    FLEXLLM_REQUIRE(k && ks && v && vs && page_table && ctx);
    FLEXLLM_REQUIRE((long)max_pages * PAGE > max_ctx);
    const int warps = B * 2 * c->hkv;
    kv_append_kernel<<<(warps + 7) / 8, 256, 0, (cudaStream_t)stream>>>(k, ks, v, vs, kv_layer(c, layer), page_table, max_pages, ctx, B, c->hkv,
                                                                         max_ctx, device_error_flag());
    return launch_status();
}

extern "C" int flexllm_mha_i8xi8_decode(flexllm_kv_cache* c, int layer, const int8_t* q, const float* qs,
                                        const int8_t* k, const float* ks, const int8_t* v, const float* vs,
                                        const float* cos_t, const float* sin_t, const float* a_s,
                                        const int32_t* page_table, int max_pages, const int32_t* ctx, int max_ctx,
                                        int B, int HQ, float* out, int32_t* oacc, void* workspace,
                                        size_t workspace_bytes, void* stream) {
    FLEXLLM_REQUIRE(c && c->elem_bytes == 1 && layer >= 0 && layer < c->layers && B >= 0 && HQ > 0 && max_ctx >= 0 && max_pages > 0);
    if (B == 0) return FLEXLLM_OK;
    FLEXLLM_REQUIRE(q && qs && k && ks && v && vs && cos_t && sin_t && a_s && page_table && ctx && out && workspace);
    FLEXLLM_REQUIRE(HQ % c->hkv == 0);
    if (HQ / c->hkv != 4) return FLEXLLM_ENOTSUP;
    FLEXLLM_REQUIRE((long)max_pages * PAGE > max_ctx);
    FLEXLLM_REQUIRE(workspace_bytes >= flexllm_mha_decode_workspace(B, HQ, max_ctx));
    return mha_decode_run(c, layer, q, qs, k, ks, v, vs, nullptr, cos_t, sin_t, a_s, page_table, max_pages, ctx, max_ctx, B,
                          HQ, out, oacc, workspace, (cudaStream_t)stream);
}

int flexllm::mha_decode_run(flexllm_kv_cache* c, int layer, const int8_t* q, const float* qs, const int8_t* k, const float* ks,
                            const int8_t* v, const float* vs, const float* qkv_f32, const float* cos_t, const float* sin_t,
                            const float* a_s, const int32_t* page_table, int max_pages, const int32_t* ctx, int max_ctx, int B,
                            int HQ, float* out, int32_t* oacc, void* workspace, cudaStream_t st) {
    const int HKV = c->hkv;
    const int ctx_stride = (int)align_up((size_t)max_ctx + 1, 64);
    const int nsplit = (ctx_stride + KEYS_PER_CTA - 1) / KEYS_PER_CTA;
    uint8_t* w = (uint8_t*)align_up((size_t)workspace, 256);
    int8_t* q2 = (int8_t*)w; w += align_up((size_t)B * HQ * 64, 256);
    float* qs2 = (float*)w; w += align_up((size_t)B * HQ * 4, 256);
    float* scores = (float*)w; w += align_up((size_t)B * HQ * ctx_stride * 4, 256);
    float* smax = (float*)w; w += align_up((size_t)B * HQ * nsplit * 4, 256);
    float* rinv = (float*)w; w += align_up((size_t)B * HQ * 4, 256);
    int32_t* acc = (int32_t*)w;
    KvLayer L = kv_layer(c, layer);
    int* err = device_error_flag();     // raised (and the length clamped) when a ctx[] entry lies beyond max_ctx

    // Three forms. us, 8 KV heads: one or two CTAs per (sequence, head) / a cluster of four: 1 x 400 keys 8.0 / 8.2, 1 x 513 9.0 / 7.9,
    // 1 x 2000 13.3 / 9.6; 16 x 400 9.4 / 10.3, 16 x 513 11.6 / 10.6, 16 x 8100 66.6 / 43.2; 18 x 2000 20.3 / 21.7; 32 x 1400 22.8 / 25.5,
    // 32 x 1700 27.6 / 27.2, 32 x 8100 132 / 93.5; 64 x 300 19.2 / 33.3, 64 x 1700 57.7 / 56.1, 64 x 4096 120 / 102, 64 x 8100 245 / 170, 64 of 512 to
    // 8192 (five draws of the lengths) 122 to 146 / 99 to 116. So clusters from 513 keys where they all run at once (25 for every 24 SMs do
    // not: their CTAs share a part of the chip), from 1665 where they follow one another, and where the second wave would be nearly empty not at all.
    // Kernel per phase / cluster, the only choices for contexts above DEC_FUSED_KEYS: 1 x 10500 65 / 25, 16 x 32000 449 / 346, 64 x 14000 535 / 335.
    // at_once counts four CTAs an SM, which their shared memory allows up to about 10600 keys. Beyond that they may follow one another also
    // where it holds; they then run in the order of the sequences and not by length.
    const int sms = gemm_sm_count(), items = B * HKV;
    const bool at_once = items * 25 <= sms * 24;
    if (max_ctx > (at_once ? 512 : 1664) && ctx_stride <= DEC_CL_PAGES * PAGE && (at_once || items > sms || ctx_stride > DEC_FUSED_KEYS)) {
        DecAttnIn in = {};
        in.q = q; in.qs = qs; in.k = k; in.ks = ks; in.v = v; in.vs = vs; in.qkv_f32 = qkv_f32; in.max_pos = max_ctx; in.error_flag = err;
        return launch_dec_cluster(qkv_f32 != nullptr, in, cos_t, sin_t, a_s, L, page_table, max_pages, ctx, B, HQ, HKV, ctx_stride / PAGE,
                                  !at_once && B <= dec_cluster_own(ctx_stride / PAGE) * PAGE, out, oacc, st);
    }
    if (ctx_stride <= DEC_FUSED_KEYS) {
        // Four heads to a CTA, or two where the CTAs are few: every SM at most one, or at most two and long contexts.
        const auto launch = 2 * items <= sms || (items <= sms && max_ctx > 1536) ? launch_dec_fused<2> : launch_dec_fused<4>;
        return launch(qkv_f32 != nullptr, q, qs, k, ks, v, vs, qkv_f32, cos_t, sin_t, a_s, L, page_table, max_pages, ctx, B, HQ, HKV, ctx_stride, out, oacc,
                      max_ctx, err, st);
    }
    const int warps = B * (HQ + 2 * HKV);
    if (qkv_f32)
        dec_append_kernel<true><<<(warps + 7) / 8, 256, 0, st>>>(q, qs, k, ks, v, vs, qkv_f32, cos_t, sin_t, L, page_table,
                                                                 max_pages, ctx, B, HQ, HKV, q2, qs2, max_ctx, err);
    else
        dec_append_kernel<false><<<(warps + 7) / 8, 256, 0, st>>>(q, qs, k, ks, v, vs, nullptr, cos_t, sin_t, L, page_table,
                                                                  max_pages, ctx, B, HQ, HKV, q2, qs2, max_ctx, err);
    dim3 grid(nsplit, HKV, B);
    dec_scores_kernel<4><<<grid, 256, 0, st>>>(q2, qs2, L, page_table, max_pages, ctx, HQ, HKV, ctx_stride, nsplit, scores, smax, max_ctx);
    dec_softmax_kernel<<<B * HQ, 128, 0, st>>>(ctx, HQ, ctx_stride, nsplit, scores, smax, rinv, max_ctx);
    FLEXLLM_CHECK_CUDA(cudaMemsetAsync(acc, 0, (size_t)B * HQ * 64 * 4, st));
    dec_pv_kernel<4><<<grid, 256, 0, st>>>(L, page_table, max_pages, ctx, HQ, HKV, ctx_stride, scores, rinv, a_s, acc, max_ctx);
    dec_out_kernel<<<(B * HQ * 64 + 255) / 256, 256, 0, st>>>(acc, a_s, B, HQ, out, oacc);
    return launch_status(5);
}
