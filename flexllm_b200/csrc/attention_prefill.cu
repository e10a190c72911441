// Prefill GQA attention, int8 x int8, on tcgen05 tensor cores.
//
// Semantics (bit-for-bit the composition the CPU oracle states; reference operators:
// Modules/MHA.h:189-243 Q.K^T, :246-273 mask, Modules/Softmax.h:25-161, Modules/quant.h:252-295
// unsigned static quant of P, Modules/MHA.h:339-389 P.V, Modules/quant.h:297-326 dequant):
//
//   S[q][k]  = sum_d Q[q][d] K[k][d]                       s8 x s8 -> s32   (tensor cores)
//   x[q][k]  = (((float)S * qs[q]) * ks[k]) * 0.125         k <= q only
//   P        = softmax(x): max, e = exp(x - max), four interleaved partial sums over k mod 4 in
//              increasing k, (p0+p1)+(p2+p3), r = 1/total, P = e * r
//   U[q][k]  = min(round((P * vs[k]) / a_s), 255)           u8
//   O[q][d]  = sum_k U[q][k] V[k][d]                        u8 x s8 -> s32   (tensor cores)
//   out      = (float)O * a_s
//
// The reference quantises the FINAL normalised P and accumulates a whole row of P.V in one int32, so a rescaling online
// softmax cannot reproduce it. The kernel therefore sweeps the keys three times; the scores are recomputed on the tensor
// cores each time, which are idle otherwise, and nothing is parked in memory between the sweeps:
//   sweep 0: Q.K^T tile -> row max
//   sweep 1: Q.K^T tile again -> e = exp(x - max) to the last bit, ordered partial sums
//   sweep 2: Q.K^T tile again -> U from the hardware exponential with a proven error bound; a value so close to a rounding
//            boundary that the bound does not decide it is worked out again as the reference does (about one in 30000 at U = 1)
//            -> U (u8, 64-byte-swizzled shared memory) -> O += U.V
// One thread owns one query row (TMEM lane), so every per-row fp32 chain runs in the reference's order. One CTA = 128
// queries of one (batch, query head) against 64-key tiles; 4 softmax warps + TMA warp + MMA warp; TMEM: S (64 columns) +
// O (64 columns) = 128 columns, so four CTAs share an SM and their 16 softmax warps hide each other's latencies. S is
// released as soon as its last columns are in registers: the next tile's product runs under this tile's arithmetic.
//
// Bound: instruction issue of the softmax warps (59 % of the issue slots busy; double precision and the special-function
// pipe 15 % each, DRAM idle). 4 prompts of 1024 tokens, 32 / 8 heads: 513 us with the exponentials of sweep 1 parked in a
// scratch (568 MB written and read back through L2), separate fp32 operations and full divisions; 230 us now (252 us with one
// test per four values in sweep 2 and the rare forms inline, 243 us with barrier waits that polled).
#include <cstdlib>

#include "attention_decode.cuh"     // layout of the paged KV cache
#include "common.cuh"
#include "tc_common.cuh"

namespace flexllm {
using namespace tc;

// ------------------------------------------------------------------ pre-pass
// Eight lanes share one 64-wide head: lane l of the eight holds elements 4l..4l+3 (lo) and 32+4l..32+4l+3 (hi), so that a
// rotation pair, and index bits 0, 1 and 5 of the transform, are one lane's own and bits 2, 3, 4 take one shuffle a value.
// (A whole warp per head, two elements a lane, spent most of its instructions on shuffles and on the divisions of the
// quantiser: 32768 tokens of 32 + 2 x 8 heads took 269 us, 4 x 1024 tokens of 32 + 8 heads 46 us.)
// RoPE, then the 64-point transform in the reference's stage order (index bits 1, 2, 3, 4, 5, 0), / 8
__device__ __forceinline__ void head8_rotate_fht(float (&x)[8], const float4 c, const float4 s, const int l8) {
    const float cc[4] = {c.x, c.y, c.z, c.w}, ss[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float x0 = x[i], x1 = x[4 + i];
        x[i] = x0 * cc[i] - x1 * ss[i];
        x[4 + i] = x0 * ss[i] + x1 * cc[i];
    }
    auto pair = [&](int i, int j) { const float a = x[i], b = x[j]; x[i] = a + b; x[j] = a - b; };
    pair(0, 2); pair(1, 3); pair(4, 6); pair(5, 7);                    // index bit 1
#pragma unroll
    for (int bit = 0; bit < 3; bit++) {                                // index bits 2, 3, 4
        const bool up = l8 & (1 << bit);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float p = __shfl_xor_sync(0xffffffffu, x[i], 1 << bit);
            x[i] = up ? p - x[i] : x[i] + p;
        }
    }
    pair(0, 4); pair(1, 5); pair(2, 6); pair(3, 7);                    // index bit 5
    pair(0, 1); pair(2, 3); pair(4, 5); pair(6, 7);                    // index bit 0
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] = x[i] / 8.0f;
}
// symmetric int8 of the head: returns the scale, the lane's eight values as two groups of four bytes
__device__ __forceinline__ float head8_quant(const float (&x)[8], uint32_t& lo, uint32_t& hi) {
    float amax = fabsf(x[0]), nan = amax;
#pragma unroll
    for (int i = 1; i < 8; i++) { amax = fmaxf(amax, fabsf(x[i])); nan = max3_nan(nan, nan, x[i]); }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float sc = sym_scale_from(amax, -amax);
    uint32_t q[8];
    q8_short(x, 1.0f / sc, sc >= 0x1p-60f && sc <= 0x1p60f && nan == nan, q, [&](float v) { return q8_exact(v, sc); });
    lo = __byte_perm(__byte_perm(q[0], q[1], 0x0040), __byte_perm(q[2], q[3], 0x0040), 0x5410);
    hi = __byte_perm(__byte_perm(q[4], q[5], 0x0040), __byte_perm(q[6], q[7], 0x0040), 0x5410);
    return sc;
}

// 32 tokens of one value head: V [B][S][HKV][64] -> V^T [B][HKV][64][S] (keys contiguous, the K-major operand of P.V) and
// vs [B][S][HKV] -> [B][HKV][S]. S is a multiple of 16, v 4-byte aligned.
__device__ __forceinline__ void v_transpose_tile(const int8_t* __restrict__ v, const float* __restrict__ vs, int S, int HKV, int h,
                                                 int8_t* __restrict__ vT, float* __restrict__ vsT) {
    __shared__ int8_t tile[32][64 + 4];
    const int b = blockIdx.z, s0 = blockIdx.y * 32, tid = threadIdx.x;
    for (int i = tid; i < 32 * 16; i += 256) {
        const int r = i >> 4, c4 = i & 15;                             // token, group of 4 dims
        if (s0 + r < S) *reinterpret_cast<int*>(&tile[r][c4 * 4]) = *reinterpret_cast<const int*>(v + (((long)b * S + s0 + r) * HKV + h) * 64 + c4 * 4);
    }
    if (tid < 32 && s0 + tid < S) vsT[((long)b * HKV + h) * S + s0 + tid] = vs[((long)b * S + s0 + tid) * HKV + h];
    __syncthreads();
    for (int i = tid; i < 64 * 8; i += 256) {
        const int d = i >> 3, r = (i & 7) * 4;                         // dim, group of 4 tokens
        if (s0 + r < S)
            *reinterpret_cast<char4*>(vT + (((long)b * HKV + h) * 64 + d) * S + s0 + r) = make_char4(tile[r][d], tile[r + 1][d], tile[r + 2][d], tile[r + 3][d]);
    }
}

// Q and K of the stand-alone operator (and, in the last HKV columns of the grid, V): dequant -> RoPE -> FHT-64/8 -> per-head int8 quant (same arithmetic as
// qk_prepare_kernel), written head-major [B][H][S][64] with scales [B][H][S] so that one head's rows are contiguous.
// VEC: q and k are 4-byte and the tables 16-byte aligned (else the same values are fetched one by one).
// Grid (head, 32 tokens, sequence), so that nothing has to be divided to find a thread's head and token: with a flat index the four 64-bit
// divisions were most of the kernel (4 x 1024 tokens, 32 + 8 heads: 21.0 us and 5.3 us for V apart -> 19.7 us for both).
template <bool VEC>
__global__ void __launch_bounds__(256) attn_qk_prepare_kernel(const int8_t* __restrict__ q, const float* __restrict__ qs,
                                                              const int8_t* __restrict__ k, const float* __restrict__ ks,
                                                              const float* __restrict__ cos_t, const float* __restrict__ sin_t, int B, int S,
                                                              int HQ, int HKV, int8_t* __restrict__ q_out, float* __restrict__ qs_out,
                                                              int8_t* __restrict__ k_out, float* __restrict__ ks_out, const int8_t* __restrict__ v,
                                                              const float* __restrict__ vs, int8_t* __restrict__ vT, float* __restrict__ vsT) {
    if ((int)blockIdx.x >= HQ + HKV) { v_transpose_tile(v, vs, S, HKV, (int)blockIdx.x - HQ - HKV, vT, vsT); return; }
    const int l8 = threadIdx.x & 7, b = blockIdx.z, t_mine = blockIdx.y * 32 + (threadIdx.x >> 3);
    const bool live = t_mine < S;
    const int t = live ? t_mine : S - 1;                               // the shuffles below take whole warps
    const bool is_q = (int)blockIdx.x < HQ;
    const int H = is_q ? HQ : HKV, h = is_q ? blockIdx.x : blockIdx.x - HQ;
    const long i = ((long)b * S + t) * H + h;
    const float sc_in = (is_q ? qs : ks)[i];
    const int8_t* src = (is_q ? q : k) + i * 64;
    auto four = [&](const int8_t* p) { return VEC ? *reinterpret_cast<const char4*>(p) : make_char4(p[0], p[1], p[2], p[3]); };
    auto table = [&](const float* p) { return VEC ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]); };
    const char4 a = four(src + 4 * l8), c = four(src + 32 + 4 * l8);
    float x[8] = {(float)a.x * sc_in, (float)a.y * sc_in, (float)a.z * sc_in, (float)a.w * sc_in,
                  (float)c.x * sc_in, (float)c.y * sc_in, (float)c.z * sc_in, (float)c.w * sc_in};
    head8_rotate_fht(x, table(cos_t + (long)t * 32 + 4 * l8), table(sin_t + (long)t * 32 + 4 * l8), l8);
    uint32_t lo, hi;
    const float sc = head8_quant(x, lo, hi);
    if (!live) return;
    const long o = ((long)b * H + h) * S + t;
    if (l8 == 0) (is_q ? qs_out : ks_out)[o] = sc;
    uint32_t* dst = reinterpret_cast<uint32_t*>((is_q ? q_out : k_out) + o * 64);
    dst[l8] = lo;
    dst[8 + l8] = hi;
}

// ------------------------------------------------------------------ main kernel
struct AttnArgs {
    int B, HQ, HKV;
    int Sq;             // queries per sequence in this call (positions q_off .. q_off + Sq - 1)
    int q_off;          // position of the first query, a multiple of 128; the keys are positions 0 .. q_off + Sq - 1
    int Sk;             // contiguous K/V: rows per (batch, KV head) of the K, V^T and scale buffers
    const float* qs;    // [B][HQ][Sq]
    const float* ks;    // contiguous: [B][HKV][Sk]; paged: the cache's K scale pool [page][HKV][64]
    const float* vs;    // likewise
    const int32_t* page_table; int max_pages;   // non-null: K / V^T tiles are pages of the KV cache (one 64-key tile = one page)
    const float* a_s;   // [HQ]
    float* out;         // [B][Sq][HQ*64]
    int32_t* oacc;      // optional, same shape
    int* error_flag;
};

__device__ __forceinline__ uint64_t umma_desc_k_sw64(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;   // 8 rows of 64 bytes
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;            // SWIZZLE_64B
    return d;
}

// Key tile = 64 keys. TMEM per CTA: S (64 columns) + O (64 columns) = 128 columns, so four CTAs share
// an SM (16 softmax warps per SM hide each other's latencies).
constexpr int ATT_KT = 64;                    // keys per tile
constexpr int ATT_SLOTS = 4;                  // K / V^T tile ring
constexpr int ATT_Q_BYTES = 128 * 64;
constexpr int ATT_TILE_BYTES = 64 * 64;       // one K tile [64 keys][64 B] or one V^T tile [64 dims][64 keys]
constexpr int ATT_P_BYTES = 128 * 64;         // U tile [128 queries][64 keys] u8
constexpr int ATT_SMEM = ATT_Q_BYTES + ATT_SLOTS * ATT_TILE_BYTES + 2 * ATT_P_BYTES + 1024 + 256;
constexpr int ATT_TMEM_COLS = 128;
constexpr int ATT_EXP_GROUP = 8;              // exponentials whose dependency chains interleave

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Sweep 2's decision on one probability (see there): the two sides of 255.25 t as rounded integers in the low bits, t the
// approximate quotient / 255.25.
constexpr float ATT_U8_HI = 255.25f * (1.0f + 0x1p-16f), ATT_U8_LO = 255.25f * (1.0f - 0x1p-16f), ATT_MAGIC = 12582912.0f;
// One value of a group with an undecided one, or of a row or tile outside the range of the bound (fast false): the same
// decision again, and where it does not hold the reference's arithmetic, U = min(round((e * r * vs) / a_s), 255), e = exp(-u).
__device__ __noinline__ static uint32_t attn_u8_resolve(float u, float c_row, float rinv, float vs, float a_s, bool fast) {
    if (fast) {
        const float t = __saturatef(ex2_approx(__fmaf_rn(u, -1.4426950408889634f, c_row)) * vs);
        const uint32_t h = __float_as_uint(__fmaf_rn(t, ATT_U8_HI, ATT_MAGIC));
        if (h == __float_as_uint(__fmaf_rn(t, ATT_U8_LO, ATT_MAGIC))) return h;
    }
    const float p = ref_expf(-u) * rinv;
    const int r = round_half_away_to_int((p * vs) / a_s);
    return (uint32_t)(r > 255 ? 255 : r) & 0xffu;
}
// Four exponentials exp(-u), any u >= 0 or NaN: out of line, for chunks with a key far below the row's maximum
__device__ __noinline__ static float4 attn_exp_any(float4 u) {
    const float x[4] = {-u.x, -u.y, -u.z, -u.w};
    float e[4];
    ref_expf_x4<true>(x, e);
    return make_float4(e[0], e[1], e[2], e[3]);
}

__global__ void __launch_bounds__(192, 4) attn_prefill_kernel(const __grid_constant__ CUtensorMap tmapQ,
                                                              const __grid_constant__ CUtensorMap tmapK,
                                                              const __grid_constant__ CUtensorMap tmapV,
                                                              const AttnArgs args) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* base_ptr = smem_raw + (base - raw);
    const uint32_t sQ = base;
    const uint32_t sT = sQ + ATT_Q_BYTES;                         // tile ring
    const uint32_t sP = sT + ATT_SLOTS * ATT_TILE_BYTES;          // two U tiles
    uint8_t* sP_ptr = base_ptr + ATT_Q_BYTES + ATT_SLOTS * ATT_TILE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sP_ptr + 2 * ATT_P_BYTES);
    // barriers: q_full, t_full[4], t_empty[4], s_full, s_empty, p_full[2], p_empty[2], o_full
    const uint32_t bar_qfull = smem_u32(bars);
    const uint32_t bar_tfull = bar_qfull + 8;
    const uint32_t bar_tempty = bar_tfull + 8 * ATT_SLOTS;
    const uint32_t bar_sfull = bar_tempty + 8 * ATT_SLOTS;
    const uint32_t bar_sempty = bar_sfull + 8;
    const uint32_t bar_pfull = bar_sempty + 8;
    const uint32_t bar_pempty = bar_pfull + 16;
    const uint32_t bar_ofull = bar_pempty + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8 + 2 * ATT_SLOTS);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = args.q_off + args.Sq;                            // keys (positions 0 .. S-1)
    const int n_qt = (args.Sq + 127) >> 7;
    // the heaviest query tiles (most keys) of all heads first, so that the last CTAs to start are the shortest
    const int heads = args.B * args.HQ;
    const int qt_l = n_qt - 1 - (int)(blockIdx.x / heads);         // query tile within the call
    const int qt0 = args.q_off >> 7, qt = qt0 + qt_l;              // ... and within the sequence
    const int hq = (int)(blockIdx.x % heads) % args.HQ;
    const int b = (int)(blockIdx.x % heads) / args.HQ;
    const int hkv = hq / (args.HQ / args.HKV);
    const int n_kt_all = (S + ATT_KT - 1) / ATT_KT;
    const int n_kt = 2 * (qt + 1) < n_kt_all ? 2 * (qt + 1) : n_kt_all;   // causal: 64-key tiles 0 .. 2*qt+1 (those that hold keys)
    const bool paged = args.page_table != nullptr;
    const int32_t* pt = paged ? args.page_table + (long)b * args.max_pages : nullptr;
    if (threadIdx.x == 0) {
        mbar_init(bar_qfull, 1);
        for (int i = 0; i < ATT_SLOTS; i++) { mbar_init(bar_tfull + 8 * i, 1); mbar_init(bar_tempty + 8 * i, 1); }
        mbar_init(bar_sfull, 1); mbar_init(bar_sempty, 4);
        for (int i = 0; i < 2; i++) { mbar_init(bar_pfull + 8 * i, 4); mbar_init(bar_pempty + 8 * i, 1); }
        mbar_init(bar_ofull, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 5) { tmem_alloc(smem_u32(tmem_slot), ATT_TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();                                                    // barriers and TMEM are ready before the kernel in front has finished
    const uint32_t tmem_S = tmem_base, tmem_O = tmem_base + 64;

    if (warp == 4) {
        // ------------------------------------------------------------ TMA producer
        // K tiles of sweeps 0 and 1 in order; then, for sweep 2, K one tile ahead of V^T: K0, K1, V0, K2, V1, ...
        if (lane == 0) {
            tma_prefetch_desc(&tmapQ); tma_prefetch_desc(&tmapK); tma_prefetch_desc(&tmapV);
            mbar_expect_tx(bar_qfull, ATT_Q_BYTES);
            tma_load_2d(sQ, &tmapQ, bar_qfull, 0, ((b * args.HQ + hq) * args.Sq) + qt_l * 128);
            int slot = 0; uint32_t phase = 0;
            auto load = [&](bool is_k, int j) {
                if (!mbar_wait(bar_tempty + 8 * slot, phase ^ 1u, abort_flag)) return false;
                const uint32_t full = bar_tfull + 8 * slot;
                const uint32_t dst = sT + slot * ATT_TILE_BYTES;
                mbar_expect_tx(full, ATT_TILE_BYTES);
                // paged: one tile = one page of the cache: K rows [64 keys][64 B], V^T rows [64 dims][64 keys]
                if (paged) tma_load_2d(dst, is_k ? &tmapK : &tmapV, full, 0, (__ldg(pt + j) * args.HKV + hkv) * 64);
                else if (is_k) tma_load_2d(dst, &tmapK, full, 0, ((b * args.HKV + hkv) * args.Sk) + j * ATT_KT);
                else tma_load_2d(dst, &tmapV, full, j * ATT_KT, (b * args.HKV + hkv) * 64);
                if (++slot == ATT_SLOTS) { slot = 0; phase ^= 1u; }
                return true;
            };
            bool ok = true;
            for (int sweep = 0; ok && sweep < 2; sweep++)
                for (int j = 0; ok && j < n_kt; j++) ok = load(true, j);
            if (ok) ok = load(true, 0);
            for (int j = 0; ok && j < n_kt; j++) {
                if (j + 1 < n_kt) ok = load(true, j + 1);
                if (ok) ok = load(false, j);
            }
        }
    } else if (warp == 5) {
        // ------------------------------------------------------------ MMA issuer
        if (lane == 0) {
            constexpr uint32_t idesc_qk = umma_idesc_i8(128, ATT_KT, 1, 1);
            constexpr uint32_t idesc_pv = umma_idesc_i8(128, 64, 0, 1);   // U unsigned, V signed
            bool ok = mbar_wait(bar_qfull, 0, abort_flag);
            const uint64_t qdesc = umma_desc_k_sw64(sQ);
            int slot = 0; uint32_t tphase = 0;
            int it = 0;                                   // score tiles so far: S is single-buffered, its phase is it & 1
            auto release_tile = [&]() {
                umma_commit(bar_tempty + 8 * slot);
                if (++slot == ATT_SLOTS) { slot = 0; tphase ^= 1u; }
            };
            auto issue_qk = [&]() {                       // S = Q.K^T of the next key tile, once the last scores are read
                if (!mbar_wait(bar_tfull + 8 * slot, tphase, abort_flag)) return false;
                if (!mbar_wait(bar_sempty, (uint32_t)(it & 1) ^ 1u, abort_flag)) return false;
                tc_fence_after();
                const uint64_t kdesc = umma_desc_k_sw64(sT + slot * ATT_TILE_BYTES);
                umma_i8(tmem_S, qdesc, kdesc, idesc_qk, 0u);
                umma_i8(tmem_S, qdesc + 2, kdesc + 2, idesc_qk, 1u);
                umma_commit(bar_sfull);
                release_tile();
                it++;
                return true;
            };
            for (int j = 0; ok && j < 2 * n_kt + 1; j++) ok = issue_qk();      // sweeps 0 and 1, and sweep 2's first tile
            for (int j = 0; ok && j < n_kt; j++) {
                if (j + 1 < n_kt && !issue_qk()) { ok = false; break; }
                // O += U.V of key tile j once the softmax warps have written U
                const int pb = j & 1;
                if (!mbar_wait(bar_tfull + 8 * slot, tphase, abort_flag)) { ok = false; break; }
                if (!mbar_wait(bar_pfull + 8 * pb, (uint32_t)((j >> 1) & 1), abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint64_t pdesc = umma_desc_k_sw64(sP + pb * ATT_P_BYTES);
                const uint64_t vdesc = umma_desc_k_sw64(sT + slot * ATT_TILE_BYTES);
                umma_i8(tmem_O, pdesc, vdesc, idesc_pv, j > 0 ? 1u : 0u);
                umma_i8(tmem_O, pdesc + 2, vdesc + 2, idesc_pv, 1u);
                umma_commit(bar_pempty + 8 * pb);
                release_tile();
            }
            if (ok) umma_commit(bar_ofull);
        }
    } else {
        // ------------------------------------------------------------ softmax warps 0..3
        const int row_in_tile = warp * 32 + lane;
        const int qpos = qt * 128 + row_in_tile;               // position of this thread's query
        const bool q_ok = qpos < S;
        const int qlim = q_ok ? qpos : S - 1;                  // keys 0..qlim are visible to this row (rows beyond S: zeros, not stored)
        const float qscale = q_ok ? args.qs[((long)b * args.HQ + hq) * args.Sq + (qpos - args.q_off)] : 0.0f;
        const f32x2 qscale2 = pack2(qscale, qscale);
        const float* ksp = args.ks + ((long)b * args.HKV + hkv) * args.Sk;      // contiguous layout
        const float* vsp = args.vs + ((long)b * args.HKV + hkv) * args.Sk;
        const float a_s = args.a_s[hq];
        const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
        bool ok = true;
        // waits for score tile number it; false when the wait ran out
        auto scores_ready = [&](int it) {
            int got = (lane == 0) ? (mbar_wait(bar_sfull, (uint32_t)(it & 1), abort_flag) ? 1 : 0) : 1;
            got = __shfl_sync(0xffffffffu, got, 0);
            if (got) tc_fence_after();
            return got != 0;
        };
        auto release_scores = [&]() {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_sempty);
        };
        // (S * qs) * ks of 16 keys starting at kc (chunk c of the tile), two values to a register pair; keys beyond S get scale 0.
        // S is released after the tile's last chunk.
        auto scores16 = [&](const float* kst, int kc, int c, f32x2 (&y)[8]) {
            uint32_t v[16];
            tmem_ld_32x16(tmem_S + lane_addr + c * 16, v);
            float4 ks4[4];
#pragma unroll
            for (int i = 0; i < 4; i++)
                ks4[i] = (kc + 4 * i < S) ? *reinterpret_cast<const float4*>(kst + c * 16 + 4 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
            tmem_ld_wait();
            if (c == ATT_KT / 16 - 1) release_scores();
#pragma unroll
            for (int i = 0; i < 4; i++) {
                y[2 * i] = mul2(mul2(pack2((float)(int)v[4 * i], (float)(int)v[4 * i + 1]), qscale2), pack2(ks4[i].x, ks4[i].y));
                y[2 * i + 1] = mul2(mul2(pack2((float)(int)v[4 * i + 2], (float)(int)v[4 * i + 3]), qscale2), pack2(ks4[i].z, ks4[i].w));
            }
        };
        const int first_masked = 2 * qt;                       // tiles before this one are visible to every row of the CTA

        // ---- sweep 0: the row maximum, tracked WITHOUT the factor 0.125 (scaling by a power of two keeps the order: applied
        // once after the sweep)
        float mx = -1e32f;
        for (int j = 0; ok && j < n_kt; j++) {
            if (!scores_ready(j)) { ok = false; break; }
            const float* kst = paged ? args.ks + ((long)__ldg(pt + j) * args.HKV + hkv) * 64 : ksp + j * ATT_KT;   // this tile's key scales
#pragma unroll 1
            for (int c = 0; c < ATT_KT / 16; c++) {
                const int kc = j * ATT_KT + c * 16;
                f32x2 y[8];
                scores16(kst, kc, c, y);
                float x[16];
#pragma unroll
                for (int i = 0; i < 8; i++) unpack2(y[i], x[2 * i], x[2 * i + 1]);
                if (j >= first_masked) {                       // causal mask (MHA.h:262-267)
#pragma unroll
                    for (int i = 0; i < 16; i++) x[i] = (kc + i <= qlim) ? x[i] : -1e32f;
                }
#pragma unroll
                for (int i = 0; i < 16; i += 2) mx = max3(mx, x[i], x[i + 1]);
            }
        }
        // Rounded up and without a sign if it is zero: max - x below is then never negative and never -0, which exp_warp does not take.
        // (The product is exact unless |max| < 2^-123; there the last bit of a subnormal makes no difference to the exponentials.)
        mx = __fmul_ru(mx, 0.125f) + 0.0f;
        const f32x2 mx2 = pack2(mx, mx), neg8th = pack2(-0.125f, -0.125f);

        // ---- sweep 1: e = exp(-u) with u = max - x, and the four ordered chains (key mod 4 == i mod 4, because a chunk starts at
        // a multiple of 16; adding the exact zeros of masked keys leaves the sums unchanged, as in the reference). max - x is
        // one fused step: x = y / 8 is exact, so a single rounding is left, the subtraction's. (Only for |y| < 2^-123 does y / 8 round in
        // the reference and not here; u can then differ where it is below 2^-100, and its exponential is 1 on both sides.)
        f32x2 s01 = pack2(0.f, 0.f), s23 = s01;
        const ExpTable tab = exp_table_lane();
        for (int j = 0; ok && j < n_kt; j++) {
            if (!scores_ready(n_kt + j)) { ok = false; break; }
            const float* kst = paged ? args.ks + ((long)__ldg(pt + j) * args.HKV + hkv) * 64 : ksp + j * ATT_KT;
            const bool masked = j >= first_masked;
#pragma unroll 1
            for (int c = 0; c < ATT_KT / 16; c++) {
                const int kc = j * ATT_KT + c * 16;
                float u[16], e[16];
                {
                    f32x2 y[8];
                    scores16(kst, kc, c, y);
#pragma unroll
                    for (int i = 0; i < 8; i++) unpack2(fma2(y[i], neg8th, mx2), u[2 * i], u[2 * i + 1]);
                }
                if (masked) {
#pragma unroll
                    for (int i = 0; i < 16; i++) u[i] = (kc + i <= qlim) ? u[i] : 0.0f;
                }
                float far = u[0];                              // NaN when one of them is
#pragma unroll
                for (int i = 1; i < 15; i += 2) far = max3_nan(far, u[i], u[i + 1]);
                far = max3_nan(far, far, u[15]);
                if (__all_sync(0xffffffffu, far <= kExpFastLimit)) {
#pragma unroll
                    for (int i0 = 0; i0 < 16; i0 += ATT_EXP_GROUP) {
                        float uu[ATT_EXP_GROUP], ee[ATT_EXP_GROUP];
#pragma unroll
                        for (int i = 0; i < ATT_EXP_GROUP; i++) uu[i] = u[i0 + i];
                        exp_warp<true>(uu, ee, tab);
#pragma unroll
                        for (int i = 0; i < ATT_EXP_GROUP; i++) e[i0 + i] = ee[i];
                    }
                } else {                                       // a key far below the maximum (or NaN): the general form
                    float near = u[0];
#pragma unroll
                    for (int i = 1; i < 16; i++) near = fminf(near, u[i]);
                    const bool zero = __all_sync(0xffffffffu, near > 104.0f && far == far);     // exp(-104) rounds to 0
#pragma unroll
                    for (int i4 = 0; i4 < 16; i4 += 4) {
                        const float4 ee = zero ? make_float4(0.f, 0.f, 0.f, 0.f) : attn_exp_any(make_float4(u[i4], u[i4 + 1], u[i4 + 2], u[i4 + 3]));
                        e[i4] = ee.x; e[i4 + 1] = ee.y; e[i4 + 2] = ee.z; e[i4 + 3] = ee.w;
                    }
                }
                if (masked) {
#pragma unroll
                    for (int i = 0; i < 16; i++) e[i] = (kc + i <= qlim) ? e[i] : 0.0f;
                }
#pragma unroll
                for (int i = 0; i < 16; i += 4) { s01 = add2(s01, pack2(e[i], e[i + 1])); s23 = add2(s23, pack2(e[i + 2], e[i + 3])); }
            }
        }
        float ps0, ps1, ps2, ps3;
        unpack2(s01, ps0, ps1); unpack2(s23, ps2, ps3);
        const float rinv = 1.0f / ((ps0 + ps1) + (ps2 + ps3));

        // ---- sweep 2: U = min(round((e * r * vs) / a_s), 255) into shared memory.
        // t = e * r * vs / (255.25 a_s) comes from ex2.approx: 2^(c - u log2 e) * vs with c = log2(r / (255.25 a_s)). For u <= 64,
        // -64 <= c <= 32 and 0 <= vs <= 2^40 its relative distance from the reference's quotient is below 5e-6: roundings of
        // the argument and its terms (2^-25 to 2^-24 of magnitudes up to 32, 64 and 92), 2^-22 of ex2.approx, and the
        // reference's own four roundings. (For larger u the quotient is below 2^-11 and the error
        // cannot lift it to a half.) So where 255.25 t (1 + 2^-16) and 255.25 t (1 - 2^-16) round to the same integer, that is U;
        // the saturating product holds t at 1, that is U at 255. Otherwise the reference's arithmetic decides, as it does for
        // scales outside these ranges.
        const float inv_as = 1.0f / a_s;
        const float c_row = log2f((rinv * inv_as) * (1.0f / 255.25f));
        const bool warp_ok = __all_sync(0xffffffffu, c_row >= -64.0f && c_row <= 32.0f);
        const f32x2 c2 = pack2(c_row, c_row), nlog2e = pack2(-1.4426950408889634f, -1.4426950408889634f);
        const f32x2 hi2 = pack2(ATT_U8_HI, ATT_U8_HI), lo2 = pack2(ATT_U8_LO, ATT_U8_LO);
        const f32x2 magic2 = pack2(ATT_MAGIC, ATT_MAGIC);      // 1.5 * 2^23: adding it rounds to an integer, kept in the low bits
        for (int j = 0; ok && j < n_kt; j++) {
            const int pb = j & 1;
            const int k0 = j * ATT_KT;
            const float* kst = paged ? args.ks + ((long)__ldg(pt + j) * args.HKV + hkv) * 64 : ksp + k0;
            const float* vst = paged ? args.vs + ((long)__ldg(pt + j) * args.HKV + hkv) * 64 : vsp + k0;   // this tile's value scales
            const float va = (k0 + lane < S) ? vst[lane] : 0.0f, vb = (k0 + 32 + lane < S) ? vst[32 + lane] : 0.0f;
            const bool fast = __all_sync(0xffffffffu, va >= 0.0f && va <= 0x1p40f && vb >= 0.0f && vb <= 0x1p40f) && warp_ok;
            const bool masked = j >= first_masked;
            int got = (lane == 0) ? (mbar_wait(bar_pempty + 8 * pb, (uint32_t)((j >> 1) & 1) ^ 1u, abort_flag) ? 1 : 0) : 1;
            got = __shfl_sync(0xffffffffu, got, 0);
            if (!got) { ok = false; break; }
            if (!scores_ready(2 * n_kt + j)) { ok = false; break; }
            uint8_t* prow = sP_ptr + pb * ATT_P_BYTES + row_in_tile * 64;
#pragma unroll 1
            for (int c = 0; c < ATT_KT / 16; c++) {            // 16 keys = one 16-byte chunk of the U row
                const int kc = k0 + c * 16;
                f32x2 y[8];
                scores16(kst, kc, c, y);
                uint32_t r[16], open = fast ? 0u : 1u;
                float4 vs4[4];
#pragma unroll
                for (int i4 = 0; i4 < 4; i4++) {
                    vs4[i4] = (kc + 4 * i4 < S) ? *reinterpret_cast<const float4*>(vst + c * 16 + 4 * i4) : make_float4(0.f, 0.f, 0.f, 0.f);
                    const float vv[4] = {vs4[i4].x, vs4[i4].y, vs4[i4].z, vs4[i4].w};
#pragma unroll
                    for (int i = 0; i < 4; i += 2) {
                        float a0, a1, h0, h1, l0, l1;
                        f32x2& yy = y[2 * i4 + (i >> 1)];
                        yy = fma2(yy, neg8th, mx2);            // u = max - x
                        unpack2(fma2(yy, nlog2e, c2), a0, a1);
                        const f32x2 t = pack2(__saturatef(ex2_approx(a0) * vv[i]), __saturatef(ex2_approx(a1) * vv[i + 1]));
                        unpack2(fma2(t, hi2, magic2), h0, h1);
                        unpack2(fma2(t, lo2, magic2), l0, l1);
                        r[4 * i4 + i] = __float_as_uint(h0); r[4 * i4 + i + 1] = __float_as_uint(h1);
                        open |= (__float_as_uint(h0) ^ __float_as_uint(l0)) | (__float_as_uint(h1) ^ __float_as_uint(l1));
                    }
                }
                if (open) {
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        float u0, u1;
                        unpack2(y[i >> 1], u0, u1);
                        const float4 q = vs4[i >> 2];
                        r[i] = attn_u8_resolve(u0, c_row, rinv, (i & 3) ? q.z : q.x, a_s, fast);
                        r[i + 1] = attn_u8_resolve(u1, c_row, rinv, (i & 3) ? q.w : q.y, a_s, fast);
                    }
                }
                if (masked) {
#pragma unroll
                    for (int i = 0; i < 16; i++) r[i] = (kc + i <= qlim) ? r[i] : 0u;
                }
                uint32_t packed[4];
#pragma unroll
                for (int i4 = 0; i4 < 4; i4++)
                    packed[i4] = __byte_perm(__byte_perm(r[4 * i4], r[4 * i4 + 1], 0x0040), __byte_perm(r[4 * i4 + 2], r[4 * i4 + 3], 0x0040), 0x5410);
                // 64-byte rows with 64-byte swizzle: chunk index XOR ((row >> 1) & 3)
                const int chunk = c ^ ((row_in_tile >> 1) & 3);
                *reinterpret_cast<uint4*>(prow + chunk * 16) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
            }
            fence_proxy_async_smem();   // make the U tile visible to the tensor core
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_pfull + 8 * pb);
        }
        // ---- epilogue: O -> out
        if (ok) {
            int got = (lane == 0) ? (mbar_wait(bar_ofull, 0, abort_flag) ? 1 : 0) : 1;
            got = __shfl_sync(0xffffffffu, got, 0);
            if (got) {
                tc_fence_after();
#pragma unroll 1
                for (int c = 0; c < 4; c++) {
                    uint32_t v[16];
                    tmem_ld_32x16(tmem_O + lane_addr + c * 16, v);
                    tmem_ld_wait();
                    if (q_ok) {
                        const long o = (((long)b * args.Sq + (qpos - args.q_off)) * args.HQ + hq) * 64 + c * 16;
#pragma unroll
                        for (int i = 0; i < 16; i += 4) {
                            float4 r;
                            r.x = (float)(int)v[i] * a_s; r.y = (float)(int)v[i + 1] * a_s;
                            r.z = (float)(int)v[i + 2] * a_s; r.w = (float)(int)v[i + 3] * a_s;
                            *reinterpret_cast<float4*>(args.out + o + i) = r;
                            if (args.oacc)
                                *reinterpret_cast<int4*>(args.oacc + o + i) = make_int4((int)v[i], (int)v[i + 1], (int)v[i + 2], (int)v[i + 3]);
                        }
                    }
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) { __nanosleep(1000); }
        if (threadIdx.x == 0 && args.error_flag) atomicOr(args.error_flag, 1);
        __syncthreads();
    }
    if (warp == 5) { tc_fence_after(); tmem_dealloc(tmem_base, ATT_TMEM_COLS); }
}


// ------------------------------------------------------------------ single-sweep variant (not bit-exact)
// The same attention with a flash-style online softmax: ONE sweep over the key tiles, a running row maximum and
// denominator, fast exponentials (ex2.approx), P quantised per key tile to u8 against that tile's largest value scale,
// P.V on the tensor core per tile, and the running output rescaled in fp32 registers. It does NOT reproduce the
// reference's arithmetic (which quantises the final normalised P against a static scale and accumulates a whole row in
// int32): it exists to measure what that exactness costs, is off by default, and is checked to fp32 tolerance only.
//   per tile j:  x = S * (qs * 0.125 * log2 e) * ks[k];  m' = max(m, max_k x);  alpha = 2^(m - m')
//                c_j = 255 / max_k vs[k];  pc = 2^(x - m') * c_j;  U = rint(pc * vs[k]) (<= 255);  l = l * alpha + sum(pc) / c_j
//                O_j = U . V (tensor core, int32);  o = o * alpha + O_j / c_j
//   out = o / l
// TMEM: S and O double-buffered (4 x 64 columns): the MMA warp runs one key tile ahead of the softmax warps.
constexpr int ATO_TMEM_COLS = 256;
constexpr int ATO_SLOTS = 6;
constexpr int ATO_SMEM = ATT_Q_BYTES + ATO_SLOTS * ATT_TILE_BYTES + 2 * ATT_P_BYTES + 1024 + 256;

__device__ __forceinline__ float lg2_approx(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__global__ void __launch_bounds__(192, 2) attn_prefill_online_kernel(const __grid_constant__ CUtensorMap tmapQ,
                                                                     const __grid_constant__ CUtensorMap tmapK,
                                                                     const __grid_constant__ CUtensorMap tmapV,
                                                                     const AttnArgs args) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* base_ptr = smem_raw + (base - raw);
    const uint32_t sQ = base;
    const uint32_t sT = sQ + ATT_Q_BYTES;
    const uint32_t sP = sT + ATO_SLOTS * ATT_TILE_BYTES;
    uint8_t* sP_ptr = base_ptr + ATT_Q_BYTES + ATO_SLOTS * ATT_TILE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sP_ptr + 2 * ATT_P_BYTES);
    // barriers: q_full, t_full[6], t_empty[6], s_full[2], s_empty[2], p_full[2], p_empty[2], o_full[2], o_empty[2]
    const uint32_t bar_qfull = smem_u32(bars);
    const uint32_t bar_tfull = bar_qfull + 8;
    const uint32_t bar_tempty = bar_tfull + 8 * ATO_SLOTS;
    const uint32_t bar_sfull = bar_tempty + 8 * ATO_SLOTS;
    const uint32_t bar_sempty = bar_sfull + 16;
    const uint32_t bar_pfull = bar_sempty + 16;
    const uint32_t bar_pempty = bar_pfull + 16;
    const uint32_t bar_ofull = bar_pempty + 16;
    const uint32_t bar_oempty = bar_ofull + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 1 + 2 * ATO_SLOTS + 12);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = args.q_off + args.Sq;
    const int n_qt = (args.Sq + 127) >> 7;
    const int qt_l = n_qt - 1 - (int)(blockIdx.x % n_qt);
    const int qt0 = args.q_off >> 7, qt = qt0 + qt_l;
    const int hq = (int)((blockIdx.x / n_qt) % args.HQ);
    const int b = (int)(blockIdx.x / ((long)n_qt * args.HQ));
    const int hkv = hq / (args.HQ / args.HKV);
    const int n_kt_all = (S + ATT_KT - 1) / ATT_KT;
    const int n_kt = 2 * (qt + 1) < n_kt_all ? 2 * (qt + 1) : n_kt_all;
    const bool paged = args.page_table != nullptr;
    const int32_t* pt = paged ? args.page_table + (long)b * args.max_pages : nullptr;

    if (threadIdx.x == 0) {
        mbar_init(bar_qfull, 1);
        for (int i = 0; i < ATO_SLOTS; i++) { mbar_init(bar_tfull + 8 * i, 1); mbar_init(bar_tempty + 8 * i, 1); }
        for (int i = 0; i < 2; i++) {
            mbar_init(bar_sfull + 8 * i, 1); mbar_init(bar_sempty + 8 * i, 4);
            mbar_init(bar_pfull + 8 * i, 4); mbar_init(bar_pempty + 8 * i, 1);
            mbar_init(bar_ofull + 8 * i, 1); mbar_init(bar_oempty + 8 * i, 4);
        }
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 5) { tmem_alloc(smem_u32(tmem_slot), ATO_TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 4) {
        // ------------------------------------------------------------ TMA producer: K_0, then K_{j+1}, V_j for every tile j
        if (lane == 0) {
            tma_prefetch_desc(&tmapQ); tma_prefetch_desc(&tmapK); tma_prefetch_desc(&tmapV);
            mbar_expect_tx(bar_qfull, ATT_Q_BYTES);
            tma_load_2d(sQ, &tmapQ, bar_qfull, 0, ((b * args.HQ + hq) * args.Sq) + qt_l * 128);
            int slot = 0; uint32_t phase = 0;
            auto load = [&](bool is_k, int j) {
                if (!mbar_wait(bar_tempty + 8 * slot, phase ^ 1u, abort_flag)) return false;
                const uint32_t full = bar_tfull + 8 * slot;
                const uint32_t dst = sT + slot * ATT_TILE_BYTES;
                mbar_expect_tx(full, ATT_TILE_BYTES);
                if (paged) tma_load_2d(dst, is_k ? &tmapK : &tmapV, full, 0, (__ldg(pt + j) * args.HKV + hkv) * 64);
                else if (is_k) tma_load_2d(dst, &tmapK, full, 0, ((b * args.HKV + hkv) * args.Sk) + j * ATT_KT);
                else tma_load_2d(dst, &tmapV, full, j * ATT_KT, (b * args.HKV + hkv) * 64);
                if (++slot == ATO_SLOTS) { slot = 0; phase ^= 1u; }
                return true;
            };
            bool ok = load(true, 0);
            for (int j = 0; ok && j < n_kt; j++) {
                if (j + 1 < n_kt) ok = load(true, j + 1);
                if (ok) ok = load(false, j);
            }
        }
    } else if (warp == 5) {
        // ------------------------------------------------------------ MMA issuer: Q.K^T one tile ahead of U.V
        if (lane == 0) {
            constexpr uint32_t idesc_qk = umma_idesc_i8(128, ATT_KT, 1, 1);
            constexpr uint32_t idesc_pv = umma_idesc_i8(128, 64, 0, 1);
            bool ok = mbar_wait(bar_qfull, 0, abort_flag);
            const uint64_t qdesc = umma_desc_k_sw64(sQ);
            int slot = 0; uint32_t tphase = 0;
            auto next_tile = [&](uint32_t& sTile) {       // waits for the next ring slot in load order
                if (!mbar_wait(bar_tfull + 8 * slot, tphase, abort_flag)) return false;
                sTile = sT + slot * ATT_TILE_BYTES;
                return true;
            };
            auto release_tile = [&]() {
                umma_commit(bar_tempty + 8 * slot);
                if (++slot == ATO_SLOTS) { slot = 0; tphase ^= 1u; }
            };
            auto issue_qk = [&](int j) {
                uint32_t sTile;
                const int sb = j & 1;
                if (!next_tile(sTile)) return false;
                if (!mbar_wait(bar_sempty + 8 * sb, (uint32_t)((j >> 1) & 1) ^ 1u, abort_flag)) return false;
                tc_fence_after();
                const uint64_t kdesc = umma_desc_k_sw64(sTile);
                umma_i8(tmem_base + sb * 64, qdesc, kdesc, idesc_qk, 0u);
                umma_i8(tmem_base + sb * 64, qdesc + 2, kdesc + 2, idesc_qk, 1u);
                umma_commit(bar_sfull + 8 * sb);
                release_tile();
                return true;
            };
            if (ok) ok = issue_qk(0);
            for (int j = 0; ok && j < n_kt; j++) {
                if (j + 1 < n_kt && !issue_qk(j + 1)) { ok = false; break; }
                const int pb = j & 1;
                uint32_t sTile;
                if (!next_tile(sTile)) { ok = false; break; }
                if (!mbar_wait(bar_pfull + 8 * pb, (uint32_t)((j >> 1) & 1), abort_flag)) { ok = false; break; }
                if (!mbar_wait(bar_oempty + 8 * pb, (uint32_t)((j >> 1) & 1) ^ 1u, abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint64_t pdesc = umma_desc_k_sw64(sP + pb * ATT_P_BYTES);
                const uint64_t vdesc = umma_desc_k_sw64(sTile);
                umma_i8(tmem_base + 128 + pb * 64, pdesc, vdesc, idesc_pv, 0u);
                umma_i8(tmem_base + 128 + pb * 64, pdesc + 2, vdesc + 2, idesc_pv, 1u);
                umma_commit(bar_ofull + 8 * pb);
                umma_commit(bar_pempty + 8 * pb);
                release_tile();
            }
        }
    } else {
        // ------------------------------------------------------------ softmax warps 0..3: one query row per thread
        const int row_in_tile = warp * 32 + lane;
        const int qpos = qt * 128 + row_in_tile;
        const bool q_ok = qpos < S;
        const int qlim = q_ok ? qpos : -1;
        const float qsl = q_ok ? args.qs[((long)b * args.HQ + hq) * args.Sq + (qpos - args.q_off)] * (0.125f * 1.4426950408889634f) : 0.0f;
        const float* ksp = args.ks + ((long)b * args.HKV + hkv) * args.Sk;
        const float* vsp = args.vs + ((long)b * args.HKV + hkv) * args.Sk;
        const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
        float m = -1e30f, l = 0.0f;
        float o[64];
#pragma unroll
        for (int i = 0; i < 64; i++) o[i] = 0.0f;
        float alpha_prev = 1.0f, f_prev = 0.0f;
        bool ok = true;
        auto wait_bar = [&](uint32_t bar, uint32_t parity) {
            int got = (lane == 0) ? (mbar_wait(bar, parity, abort_flag) ? 1 : 0) : 1;
            return __shfl_sync(0xffffffffu, got, 0) != 0;
        };
        auto fold_o = [&](int jj) {        // o = o * alpha + O_jj * f, O_jj from its TMEM buffer
            const int ob = jj & 1;
            if (!wait_bar(bar_ofull + 8 * ob, (uint32_t)((jj >> 1) & 1))) return false;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < 4; c++) {
                uint32_t v[16];
                tmem_ld_32x16(tmem_base + 128 + ob * 64 + lane_addr + c * 16, v);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 16; i++) o[c * 16 + i] = __fmaf_rn(o[c * 16 + i], alpha_prev, (float)(int)v[i] * f_prev);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_oempty + 8 * ob);
            return true;
        };
        for (int j = 0; ok && j < n_kt; j++) {
            const int sb = j & 1;
            const int k0 = j * ATT_KT;
            const float* kst = paged ? args.ks + ((long)__ldg(pt + j) * args.HKV + hkv) * 64 : ksp + k0;
            const float* vst = paged ? args.vs + ((long)__ldg(pt + j) * args.HKV + hkv) * 64 : vsp + k0;
            // this tile's largest value scale (keys beyond the sequence count as 0)
            float vmax = fmaxf(k0 + lane < S ? vst[lane] : 0.0f, k0 + 32 + lane < S ? vst[32 + lane] : 0.0f);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, off));
            vmax = fmaxf(vmax, 1e-30f);
            const float cj = 255.0f / vmax, lcj = lg2_approx(cj), fj = vmax * (1.0f / 255.0f);
            const bool diag = k0 + ATT_KT - 1 > qt * 128;          // tile may hold keys beyond some row's own position
            if (!wait_bar(bar_sfull + 8 * sb, (uint32_t)((j >> 1) & 1))) { ok = false; break; }
            tc_fence_after();
            const uint32_t tS = tmem_base + sb * 64 + lane_addr;
            // pass 1: the tile's row maximum
            float tmax = -1e30f;
#pragma unroll 1
            for (int c = 0; c < 4; c++) {
                uint32_t v[16];
                tmem_ld_32x16(tS + c * 16, v);
                float ksv[16];
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const float4 t = (k0 + c * 16 + i < S) ? *reinterpret_cast<const float4*>(kst + c * 16 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
                    ksv[i] = t.x; ksv[i + 1] = t.y; ksv[i + 2] = t.z; ksv[i + 3] = t.w;
                }
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    float x = ((float)(int)v[i] * qsl) * ksv[i];
                    if (diag) x = (k0 + c * 16 + i <= qlim) ? x : -1e30f;
                    tmax = fmaxf(tmax, x);
                }
            }
            const float m_new = fmaxf(m, tmax);
            const float alpha = ex2_approx(m - m_new);
            const float mref = m_new - lcj;                        // 2^(x - mref) = 2^(x - m_new) * c_j
            if (!wait_bar(bar_pempty + 8 * sb, (uint32_t)((j >> 1) & 1) ^ 1u)) { ok = false; break; }
            // pass 2: pc, its sum, U into shared memory
            uint8_t* prow = sP_ptr + sb * ATT_P_BYTES + row_in_tile * 64;
            float sum = 0.0f;
#pragma unroll 1
            for (int c = 0; c < 4; c++) {
                uint32_t v[16];
                tmem_ld_32x16(tS + c * 16, v);
                float ksv[16], vsv[16];
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const bool in = k0 + c * 16 + i < S;
                    const float4 t = in ? *reinterpret_cast<const float4*>(kst + c * 16 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
                    const float4 u = in ? *reinterpret_cast<const float4*>(vst + c * 16 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
                    ksv[i] = t.x; ksv[i + 1] = t.y; ksv[i + 2] = t.z; ksv[i + 3] = t.w;
                    vsv[i] = u.x; vsv[i + 1] = u.y; vsv[i + 2] = u.z; vsv[i + 3] = u.w;
                }
                tmem_ld_wait();
                uint32_t packed[4];
#pragma unroll
                for (int i4 = 0; i4 < 4; i4++) {
                    uint32_t w = 0;
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const int ii = i4 * 4 + i;
                        const float x = ((float)(int)v[ii] * qsl) * ksv[ii];
                        float pc = ex2_approx(x - mref);
                        if (diag) pc = (k0 + c * 16 + ii <= qlim) ? pc : 0.0f;
                        sum += pc;
                        uint32_t r = __float2uint_rn(pc * vsv[ii]);
                        r = r > 255u ? 255u : r;
                        w |= r << (8 * i);
                    }
                    packed[i4] = w;
                }
                const int chunk = c ^ ((row_in_tile >> 1) & 3);
                *reinterpret_cast<uint4*>(prow + chunk * 16) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
            }
            fence_proxy_async_smem();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) { mbar_arrive(bar_pfull + 8 * sb); mbar_arrive(bar_sempty + 8 * sb); }
            l = __fmaf_rn(l, alpha, sum * fj);
            m = m_new;
            // the previous tile's U.V has had this tile's softmax to finish: fold it in now
            if (j > 0 && !fold_o(j - 1)) { ok = false; break; }
            alpha_prev = alpha; f_prev = fj;
        }
        if (ok) ok = fold_o(n_kt - 1);
        if (ok && q_ok) {
            const float rl = 1.0f / l;
            const long ob = (((long)b * args.Sq + (qpos - args.q_off)) * args.HQ + hq) * 64;
#pragma unroll
            for (int i = 0; i < 64; i += 4)
                *reinterpret_cast<float4*>(args.out + ob + i) = make_float4(o[i] * rl, o[i + 1] * rl, o[i + 2] * rl, o[i + 3] * rl);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) { __nanosleep(1000); }
        if (threadIdx.x == 0 && args.error_flag) atomicOr(args.error_flag, 1);
        __syncthreads();
    }
    if (warp == 5) { tc_fence_after(); tmem_dealloc(tmem_base, ATO_TMEM_COLS); }
}

int* device_error_flag();

// fp32 front end used by the model: qkv [B*Sq][(HQ+2*HKV)*64] fp32 as the fused q/k/v projection writes it, tokens at
// positions q_off .. q_off + Sq - 1. Query heads: RoPE -> FHT-64/8 -> per-head int8, head-major [B][HQ][Sq][64] for the
// attention kernel's Q tiles. Key heads: the same arithmetic, written straight into the KV cache's pages (row = token).
// Value heads: per-head int8 quant (quant.h:527-650), token-major into a scratch that attn_v_to_pages_kernel transposes
// into the cache's V^T pages.
// Grid (head, 32 tokens, sequence): see attn_qk_prepare_kernel. Bound by memory: 32768 tokens of 32 + 2 x 8 heads 160 -> 135 us (502 MB, 77 us at the
// copy rate).
__global__ void __launch_bounds__(256) attn_qkv_prepare_f32_kernel(const float* __restrict__ qkv, const float* __restrict__ cos_t,
                                                                   const float* __restrict__ sin_t, int B, int Sq, int q_off, int HQ, int HKV,
                                                                   int8_t* __restrict__ q2, float* __restrict__ qs2,
                                                                   int8_t* __restrict__ k_pool, float* __restrict__ ks_pool,
                                                                   const int32_t* __restrict__ page_table, int max_pages,
                                                                   int8_t* __restrict__ v2, float* __restrict__ vs2) {
    pdl_sync();
    const int l8 = threadIdx.x & 7, h = blockIdx.x, b = blockIdx.z, t_mine = blockIdx.y * 32 + (threadIdx.x >> 3);
    const bool live = t_mine < Sq;
    const int t = live ? t_mine : Sq - 1;                              // the shuffles below take whole warps
    const int pos = q_off + t;
    const long bt = (long)b * Sq + t, w = bt * (HQ + 2 * HKV) + h;
    const float4* src = reinterpret_cast<const float4*>(qkv + w * 64);
    const float4 a = src[l8], c = src[8 + l8];
    const float raw[8] = {a.x, a.y, a.z, a.w, c.x, c.y, c.z, c.w};
    float x[8];
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] = raw[i];
    if (h < HQ + HKV)                                                  // value heads are quantised as they are
        head8_rotate_fht(x, reinterpret_cast<const float4*>(cos_t + (long)pos * 32)[l8], reinterpret_cast<const float4*>(sin_t + (long)pos * 32)[l8], l8);
    uint32_t lo, hi;
    const float sc = head8_quant(x, lo, hi);
    if (!live) return;
    int8_t* dst; float* sdst;
    if (h < HQ) { const long o = ((long)b * HQ + h) * Sq + t; dst = q2 + o * 64; sdst = qs2 + o; }
    else if (h < HQ + HKV) {
        const long row = (long)page_table[(long)b * max_pages + pos / 64] * HKV * 64 + (pos & 63) + (long)(h - HQ) * 64;
        dst = k_pool + row * 64; sdst = ks_pool + row;
    } else { const long o = bt * HKV + (h - HQ - HKV); dst = v2 + o * 64; sdst = vs2 + o; }
    if (l8 == 0) *sdst = sc;
    reinterpret_cast<uint32_t*>(dst)[l8] = lo;
    reinterpret_cast<uint32_t*>(dst)[8 + l8] = hi;
}

// V [B][Sq][HKV][64] (token-major scratch) -> the cache's V^T pages [page][HKV][64 dims][64 tokens] and scale pages,
// for the tokens at positions q_off .. q_off + Sq - 1 (q_off a multiple of 64: one 64-token tile = one page).
__global__ void __launch_bounds__(256) attn_v_to_pages_kernel(const int8_t* __restrict__ v, const float* __restrict__ vs, int Sq, int q_off,
                                                              int HKV, const int32_t* __restrict__ page_table, int max_pages,
                                                              int8_t* __restrict__ v_pool, float* __restrict__ vs_pool) {
    pdl_sync();
    __shared__ int8_t tile[64][64 + 4];
    const int s0 = blockIdx.x * 64, h = blockIdx.y, b = blockIdx.z;
    const long prow = ((long)page_table[(long)b * max_pages + (q_off + s0) / 64] * HKV + h) * 64;
    for (int i = threadIdx.x; i < 64 * 16; i += 256) {
        const int r = i >> 4, c4 = i & 15;   // r: token in tile, c4: group of 4 dims
        int val = 0;
        if (s0 + r < Sq) val = *reinterpret_cast<const int*>(v + (((long)b * Sq + s0 + r) * HKV + h) * 64 + c4 * 4);
        *reinterpret_cast<int*>(&tile[r][c4 * 4]) = val;
    }
    if (threadIdx.x < 64 && s0 + threadIdx.x < Sq) vs_pool[prow + threadIdx.x] = vs[((long)b * Sq + s0 + threadIdx.x) * HKV + h];
    __syncthreads();
    for (int i = threadIdx.x; i < 64 * 64; i += 256) {
        const int d = i >> 6, r = i & 63;
        if (s0 + r < Sq) v_pool[(prow + d) * 64 + r] = tile[r][d];
    }
}

static size_t align_up_(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Workspace of the stand-alone operator (contiguous head-major K, V^T).
struct PrefillWs {
    int8_t *q2, *k2, *vT, *v2;
    float *qs2, *ks2, *vsT, *vs2;
    static size_t bytes(int B, int S, int HQ, int HKV) {
        size_t n = 0;
        n += align_up_((size_t)B * HQ * S * 64, 1024);
        n += 3 * align_up_((size_t)B * HKV * S * 64, 1024);
        n += align_up_((size_t)B * HQ * S * 4, 1024);
        n += 3 * align_up_((size_t)B * HKV * S * 4, 1024);
        return n + 1024;
    }
    PrefillWs(void* ws, int B, int S, int HQ, int HKV) {
        uint8_t* w = (uint8_t*)align_up_((size_t)ws, 1024);
        q2 = (int8_t*)w; w += align_up_((size_t)B * HQ * S * 64, 1024);
        k2 = (int8_t*)w; w += align_up_((size_t)B * HKV * S * 64, 1024);
        vT = (int8_t*)w; w += align_up_((size_t)B * HKV * S * 64, 1024);
        v2 = (int8_t*)w; w += align_up_((size_t)B * HKV * S * 64, 1024);
        qs2 = (float*)w; w += align_up_((size_t)B * HQ * S * 4, 1024);
        ks2 = (float*)w; w += align_up_((size_t)B * HKV * S * 4, 1024);
        vsT = (float*)w; w += align_up_((size_t)B * HKV * S * 4, 1024);
        vs2 = (float*)w;
    }
};

// Workspace of the model path (K and V live in the KV cache): head-major Q, token-major V scratch.
struct PagedWs {
    int8_t *q2, *v2; float *qs2, *vs2;
    static size_t bytes(int B, int Sq_max, int HQ, int HKV) {
        return align_up_((size_t)B * HQ * Sq_max * 64, 1024) + align_up_((size_t)B * HKV * Sq_max * 64, 1024) +
               align_up_((size_t)B * HQ * Sq_max * 4, 1024) + align_up_((size_t)B * HKV * Sq_max * 4, 1024) + 1024;
    }
    PagedWs(void* ws, int B, int Sq_max, int HQ, int HKV) {
        uint8_t* w = (uint8_t*)align_up_((size_t)ws, 1024);
        q2 = (int8_t*)w; w += align_up_((size_t)B * HQ * Sq_max * 64, 1024);
        v2 = (int8_t*)w; w += align_up_((size_t)B * HKV * Sq_max * 64, 1024);
        qs2 = (float*)w; w += align_up_((size_t)B * HQ * Sq_max * 4, 1024);
        vs2 = (float*)w;
    }
};

// a: everything but the error flag filled in. k_rows / v_rows: rows of the [rows][64 B] (K; paged V^T) or
// [rows][v_row_bytes] (contiguous V^T) matrices the tensor maps describe.
static int mha_prefill_core(AttnArgs a, const int8_t* q2, const int8_t* kmat, uint64_t k_rows, const int8_t* vmat, uint64_t v_rows,
                            uint64_t v_row_bytes, cudaStream_t st, bool online = false) {
    CUtensorMap tq, tk, tv;
    int rc = make_tmap_2d_u8_box(&tq, q2, (uint64_t)a.B * a.HQ * a.Sq, 64, 64, 128, 64);
    if (rc != FLEXLLM_OK) return rc;
    rc = make_tmap_2d_u8_box(&tk, kmat, k_rows, 64, 64, ATT_KT, 64);
    if (rc != FLEXLLM_OK) return rc;
    rc = make_tmap_2d_u8_box(&tv, vmat, v_rows, v_row_bytes, ATT_KT, 64, 64);
    if (rc != FLEXLLM_OK) return rc;
    a.error_flag = device_error_flag();
    static std::atomic<bool> attr_set[kMaxDevices];      // the attribute belongs to (function, device)
    const int dev = current_device();
    if (dev < 0) return FLEXLLM_ECUDA;
    if (!attr_set[dev].load(std::memory_order_acquire)) {
        FLEXLLM_CHECK_CUDA(cudaFuncSetAttribute(attn_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ATT_SMEM));
        attr_set[dev].store(true, std::memory_order_release);
    }
    const int n_qt = (a.Sq + 127) / 128;
    const long grid = (long)a.B * a.HQ * n_qt;
    if (online) {
        static std::atomic<bool> attr_set_online[kMaxDevices];
        if (!attr_set_online[dev].load(std::memory_order_acquire)) {
            FLEXLLM_CHECK_CUDA(cudaFuncSetAttribute(attn_prefill_online_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ATO_SMEM));
            attr_set_online[dev].store(true, std::memory_order_release);
        }
        attn_prefill_online_kernel<<<(unsigned)grid, 192, ATO_SMEM, st>>>(tq, tk, tv, a);
        return launch_status();
    }
    const SetUpEarly early;
    launch_k(attn_prefill_kernel, dim3((unsigned)grid), dim3(192), (size_t)ATT_SMEM, st, tq, tk, tv, a);
    return launch_status();
}

size_t mha_prefill_ws_bytes(int B, int max_prefill, int max_ctx, int HQ, int HKV) {
    return PagedWs::bytes(B, max_prefill, HQ, HKV);
}

// Model path: attention of the Sq tokens at positions q_off .. q_off + Sq - 1 of every sequence, from the fp32 output of
// the fused q/k/v projection, over the paged KV cache: the new keys and values are written into the cache first (which
// is the hand-over to decode: nothing is repacked afterwards), then every query attends to cache positions 0 .. its own.
// q_off is a multiple of 128 (0 for a prompt that fits one call). max_prefill: the Sq the workspace was sized for.
int mha_prefill_paged(const float* qkv, const float* cos_t, const float* sin_t, const float* a_s, int B, int Sq, int q_off, int HQ, int HKV,
                      int max_prefill, flexllm_kv_cache* c, int layer, const int32_t* page_table, int max_pages, float* out,
                      void* workspace, cudaStream_t st) {
    if (Sq % 16 != 0 || q_off % 128 != 0 || Sq > max_prefill || c->hkv != HKV) return FLEXLLM_ENOTSUP;
    PagedWs ws(workspace, B, max_prefill, HQ, HKV);
    int8_t* k_pool = c->k + (size_t)layer * c->page_bytes; int8_t* v_pool = c->v + (size_t)layer * c->page_bytes;
    float* ks_pool = c->ks + (size_t)layer * (c->scale_bytes / 4); float* vs_pool = c->vs + (size_t)layer * (c->scale_bytes / 4);
    const SetUpEarly early;
    launch_k(attn_qkv_prepare_f32_kernel, dim3(HQ + 2 * HKV, (Sq + 31) / 32, B), dim3(256), 0, st, qkv, cos_t, sin_t, B, Sq, q_off, HQ, HKV, ws.q2, ws.qs2,
             k_pool, ks_pool, page_table, max_pages, ws.v2, ws.vs2);
    dim3 g((Sq + 63) / 64, HKV, B);
    launch_k(attn_v_to_pages_kernel, g, dim3(256), 0, st, ws.v2, ws.vs2, Sq, q_off, HKV, page_table, max_pages, v_pool, vs_pool);
    int rc = launch_status(2);
    if (rc != FLEXLLM_OK) return rc;
    AttnArgs a;
    a.B = B; a.HQ = HQ; a.HKV = HKV; a.Sq = Sq; a.q_off = q_off; a.Sk = 0;
    a.qs = ws.qs2; a.ks = ks_pool; a.vs = vs_pool; a.page_table = page_table; a.max_pages = max_pages;
    a.a_s = a_s; a.out = out; a.oacc = nullptr;
    const uint64_t rows = (uint64_t)c->n_pages * HKV * 64;
    // FLEXLLM_ATTN_ONLINE=1: the single-sweep variant (not bit-exact) in the model's prefill, for measuring what exactness costs
    static const bool online = [] { const char* e = getenv("FLEXLLM_ATTN_ONLINE"); return e && e[0] == '1'; }();
    return mha_prefill_core(a, ws.q2, k_pool, rows, v_pool, rows, 64, st, online);
}

}  // namespace flexllm

using namespace flexllm;

extern "C" size_t flexllm_mha_prefill_workspace(int B, int S, int HQ, int HKV) {
    if (B <= 0 || S <= 0 || HQ <= 0 || HKV <= 0) return 0;
    return PrefillWs::bytes(B, S, HQ, HKV);
}

static int mha_prefill_contiguous(bool online, const int8_t* q, const float* qs, const int8_t* k, const float* ks,
                                         const int8_t* v, const float* vs, const float* cos_t, const float* sin_t,
                                         const float* a_s, int B, int S, int HQ, int HKV, float* out, int32_t* oacc,
                                         void* workspace, size_t workspace_bytes, void* stream) {
    FLEXLLM_REQUIRE(B >= 0 && S > 0 && HQ > 0 && HKV > 0 && HQ % HKV == 0);
    if (B == 0) return FLEXLLM_OK;
    FLEXLLM_REQUIRE(q && qs && k && ks && v && vs && cos_t && sin_t && a_s && out && workspace);
    if (S % 16 != 0) return FLEXLLM_ENOTSUP;
    FLEXLLM_REQUIRE(workspace_bytes >= flexllm_mha_prefill_workspace(B, S, HQ, HKV));
    FLEXLLM_REQUIRE(aligned(out, 16) && (!oacc || aligned(oacc, 16)) && aligned(v, 4));
    cudaStream_t st = (cudaStream_t)stream;
    PrefillWs ws(workspace, B, S, HQ, HKV);
    auto* prepare = aligned(q, 4) && aligned(k, 4) && aligned(cos_t, 16) && aligned(sin_t, 16) ? attn_qk_prepare_kernel<true> : attn_qk_prepare_kernel<false>;
    prepare<<<dim3(HQ + 2 * HKV, (S + 31) / 32, B), 256, 0, st>>>(q, qs, k, ks, cos_t, sin_t, B, S, HQ, HKV, ws.q2, ws.qs2, ws.k2, ws.ks2, v, vs, ws.vT, ws.vsT);
    int rc = launch_status();
    if (rc != FLEXLLM_OK) return rc;
    AttnArgs a;
    a.B = B; a.HQ = HQ; a.HKV = HKV; a.Sq = S; a.q_off = 0; a.Sk = S;
    a.qs = ws.qs2; a.ks = ws.ks2; a.vs = ws.vsT; a.page_table = nullptr; a.max_pages = 0;
    a.a_s = a_s; a.out = out; a.oacc = oacc;
    return mha_prefill_core(a, ws.q2, ws.k2, (uint64_t)B * HKV * S, ws.vT, (uint64_t)B * HKV * 64, (uint64_t)S, st, online);
}

extern "C" int flexllm_mha_i8xi8_prefill(const int8_t* q, const float* qs, const int8_t* k, const float* ks,
                                         const int8_t* v, const float* vs, const float* cos_t, const float* sin_t,
                                         const float* a_s, int B, int S, int HQ, int HKV, float* out, int32_t* oacc,
                                         void* workspace, size_t workspace_bytes, void* stream) {
    return mha_prefill_contiguous(false, q, qs, k, ks, v, vs, cos_t, sin_t, a_s, B, S, HQ, HKV, out, oacc, workspace, workspace_bytes, stream);
}

extern "C" int flexllm_mha_i8xi8_prefill_online(const int8_t* q, const float* qs, const int8_t* k, const float* ks,
                                                const int8_t* v, const float* vs, const float* cos_t, const float* sin_t,
                                                int B, int S, int HQ, int HKV, float* out, void* workspace, size_t workspace_bytes,
                                                void* stream) {
    static const float unused_scale[1] = {1.0f};
    return mha_prefill_contiguous(true, q, qs, k, ks, v, vs, cos_t, sin_t, unused_scale, B, S, HQ, HKV, out, nullptr, workspace, workspace_bytes,
                                  stream);
}
