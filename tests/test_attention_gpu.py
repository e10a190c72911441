"""GPU parity of the int8 attention kernels against the CPU oracle (the prefill-attention and paged decode-attention workloads at
sizes the oracle finishes in seconds, plus edge cases)."""
import numpy as np
import pytest
import torch

import oracle
from util import assert_same, max_abs_rel, to_np

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _correctly_rounded_exp():
    """The CUDA kernels evaluate the correctly rounded expf; pin them against the oracle in the same
    mode (bit for bit). Tests that quantify the distance to the build machine's libm switch modes
    themselves."""
    with oracle.exp_mode(oracle.EXP_CORRECTLY_ROUNDED):
        yield


@pytest.fixture(scope="module")
def F():
    import flexllm_b200
    flexllm_b200.lib()
    return flexllm_b200


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def attn_inputs(B, S, HQ, HKV, seed):
    g = np.random.default_rng(seed)
    q = g.integers(-127, 128, (B, S, HQ, 64), dtype=np.int8)
    k = g.integers(-127, 128, (B, S, HKV, 64), dtype=np.int8)
    v = g.integers(-127, 128, (B, S, HKV, 64), dtype=np.int8)
    qs = g.uniform(0.005, 0.05, (B, S, HQ)).astype(np.float32)
    ks = g.uniform(0.005, 0.05, (B, S, HKV)).astype(np.float32)
    vs = g.uniform(0.005, 0.05, (B, S, HKV)).astype(np.float32)
    a_s = np.full(HQ, 0.05 / 255, np.float32)
    return q, qs, k, ks, v, vs, a_s


def check_prefill(F, B, S, HQ, HKV, seed):
    q, qs, k, ks, v, vs, a_s = attn_inputs(B, S, HQ, HKV, seed)
    cos_t, sin_t = oracle.rope_table(max(S, 16))
    out, oacc = F.MHA_i8xi8_Prefilling(dev(q), dev(qs), dev(k), dev(ks), dev(v), dev(vs), dev(cos_t), dev(sin_t),
                                       dev(a_s), want_oacc=True)
    torch.cuda.synchronize()
    ref = oracle.mha_prefill(q, qs, k, ks, v, vs, cos_t, sin_t, a_s)
    out = to_np(out); oacc = to_np(oacc)
    assert_same(oacc, ref["oacc"], "int32 P.V accumulators")
    assert_same(out, ref["out"], "fp32 output")
    # distance to the libm flavour of the oracle (a last-bit difference in exp() can move a u8 across
    # a rounding boundary): count, and require the fp32 tolerance
    with oracle.exp_mode(oracle.EXP_LIBM):
        ref_l = oracle.mha_prefill(q, qs, k, ks, v, vs, cos_t, sin_t, a_s)
    bad = np.count_nonzero(oacc != ref_l["oacc"])
    err = max_abs_rel(out, ref_l["out"])
    print(f"prefill attn B={B} S={S}: exact; vs libm expf {bad}/{oacc.size} int32 accumulators differ, max-abs-rel {err:.2e}")
    assert err < 1e-3


@pytest.mark.parametrize("B,S,HQ,HKV", [(1, 128, 4, 1), (2, 256, 8, 2), (1, 16, 4, 4), (1, 144, 4, 1), (1, 400, 8, 2)])
def test_prefill_small(F, B, S, HQ, HKV):
    check_prefill(F, B, S, HQ, HKV, 30)


def test_prefill_config3_slice(F):
    """The prefill-attention workload's shapes (S=1024, 32/8 heads) on one batch element."""
    check_prefill(F, 1, 1024, 32, 8, 31)


@pytest.mark.parametrize("what", ["peaked", "spread", "large", "saturated", "ties", "wide_scales", "tiny_scales", "zero_scales"])
def test_prefill_quantiser_ranges(F, what):
    """The probabilities' quantiser decides most values from the hardware exponential and an error bound, the rest as the reference
    does; exponentials have a short form up to 87 below the maximum. Inputs on both sides of every such line, bit for bit."""
    B, S, HQ, HKV = 1, 208, 8, 2                       # the last key tile and the last query tile are partly empty
    q, qs, k, ks, v, vs, a_s = attn_inputs(B, S, HQ, HKV, 77)
    if what == "peaked": qs *= 20                      # differences of scores up to thousands
    if what == "spread": qs *= 3                       # ... on both sides of 87 and of 104
    if what == "large": a_s[:] = 2e-6                  # U all over 0..255
    if what == "saturated": a_s[:] = 1e-8              # most of U at 255
    if what == "ties":                                 # equal scores: e = 1, P = 1/n; for n = 2^j quotients are k + 1/2 exactly
        q[:] = 0
        vs[:] = 2.0 ** g_exponents(vs.shape)
        a_s[:] = 2.0 ** -13
    if what == "wide_scales":                          # outside the bound's range: the reference's arithmetic throughout
        vs *= 2.0 ** 46
        a_s *= 2.0 ** 38
    if what == "tiny_scales":
        vs *= 2.0 ** -60
    if what == "zero_scales":
        vs[:, ::3] = 0
    cos_t, sin_t = oracle.rope_table(S)
    out, oacc = F.MHA_i8xi8_Prefilling(dev(q), dev(qs), dev(k), dev(ks), dev(v), dev(vs), dev(cos_t), dev(sin_t), dev(a_s), want_oacc=True)
    ref = oracle.mha_prefill(q, qs, k, ks, v, vs, cos_t, sin_t, a_s)
    assert_same(to_np(oacc), ref["oacc"], "int32 P.V accumulators")
    assert_same(to_np(out), ref["out"], "fp32 output")


@pytest.mark.parametrize("e", [-62, -64, -66, -70, -80])
def test_prefill_scores_below_the_normal_range(F, e):
    """Scores, or their eighths, that are subnormal or round to a zero of either sign: every exponential is 1. One visible key and many."""
    B, S, HQ, HKV = 1, 208, 8, 2
    q, qs, k, ks, v, vs, a_s = attn_inputs(B, S, HQ, HKV, 81)
    qs *= np.float32(2.0) ** e; ks *= np.float32(2.0) ** e
    cos_t, sin_t = oracle.rope_table(S)
    out, oacc = F.MHA_i8xi8_Prefilling(dev(q), dev(qs), dev(k), dev(ks), dev(v), dev(vs), dev(cos_t), dev(sin_t), dev(a_s), want_oacc=True)
    ref = oracle.mha_prefill(q, qs, k, ks, v, vs, cos_t, sin_t, a_s)
    assert_same(to_np(oacc), ref["oacc"], "int32 P.V accumulators")
    assert_same(to_np(out), ref["out"], "fp32 output")


@pytest.mark.parametrize("what", ["q", "k", "tables"])
def test_prefill_prepare_alignment(F, what):
    """Inputs whose address allows no wide loads take the other form of the preparation."""
    B, S, HQ, HKV = 1, 48, 6, 3
    q, qs, k, ks, v, vs, a_s = attn_inputs(B, S, HQ, HKV, 79)
    cos_t, sin_t = oracle.rope_table(S)

    def shifted(a):
        buf = torch.empty(a.size + 1, dtype=torch.from_numpy(a).dtype, device="cuda")
        buf[1:] = dev(a).reshape(-1)
        return buf[1:].reshape(a.shape)

    out, oacc = F.MHA_i8xi8_Prefilling(shifted(q) if what == "q" else dev(q), dev(qs), shifted(k) if what == "k" else dev(k), dev(ks), dev(v), dev(vs),
                                       shifted(cos_t) if what == "tables" else dev(cos_t), shifted(sin_t) if what == "tables" else dev(sin_t), dev(a_s),
                                       want_oacc=True)
    ref = oracle.mha_prefill(q, qs, k, ks, v, vs, cos_t, sin_t, a_s)
    assert_same(to_np(oacc), ref["oacc"], "int32 P.V accumulators")
    assert_same(to_np(out), ref["out"], "fp32 output")


def g_exponents(shape):
    return np.random.default_rng(78).integers(-9, -3, shape).astype(np.float32)


def test_prefill_rows_sum_property(F):
    """Size-independent property at the full config-3 size (B=4): with V == 1 and vs == a_s * 255
    every output equals sum_k U[q][k] * a_s and U rows sum to about 255 (P sums to 1)."""
    B, S, HQ, HKV = 4, 1024, 32, 8
    q, qs, k, ks, v, vs, a_s = attn_inputs(B, S, HQ, HKV, 32)
    v[:] = 1
    vs[:] = a_s[0] * 255
    cos_t, sin_t = oracle.rope_table(S)
    out, oacc = F.MHA_i8xi8_Prefilling(dev(q), dev(qs), dev(k), dev(ks), dev(v), dev(vs), dev(cos_t), dev(sin_t),
                                       dev(a_s), want_oacc=True)
    oacc = to_np(oacc)
    # sum_k round(255 * P_k) <= 255 + (number of keys)/2; never negative
    nkeys = np.arange(1, S + 1)[None, :, None]
    assert oacc.min() >= 0 and (oacc <= 255 + nkeys / 2).all()
    # all 64 dims of a head see the same sum
    o = oacc.reshape(B, S, HQ, 64)
    assert (o == o[..., :1]).all()
    # first token attends to itself only: U = 255 exactly
    assert (o[:, 0] == 255).all()


def _float_attention(ref, v, vs):
    """Attention of the prepared int8 Q / K (after RoPE, FHT-64 and re-quantisation) and the int8 V in float64, with no
    quantisation of P: what both kernels approximate with their 8-bit P."""
    q2, qs2, k2, ks2 = ref["q2"], ref["qs2"], ref["k2"], ref["ks2"]
    B, S, HQ, _ = q2.shape; HKV = k2.shape[2]; G = HQ // HKV
    out = np.empty((B, S, HQ * 64))
    mask = np.tril(np.ones((S, S), bool))
    for b in range(B):
        for h in range(HQ):
            kv = h // G
            x = (q2[b, :, h].astype(np.float64) @ k2[b, :, kv].astype(np.float64).T) * qs2[b, :, h, None] * ks2[b, None, :, kv] * 0.125
            x = np.where(mask, x, -np.inf)
            p = np.exp(x - x.max(axis=1, keepdims=True)); p /= p.sum(axis=1, keepdims=True)
            out[b, :, h * 64:(h + 1) * 64] = p @ (v[b, :, kv].astype(np.float64) * vs[b, :, kv, None])
    return out


@pytest.mark.parametrize("B,S,HQ,HKV", [(1, 128, 4, 1), (2, 256, 8, 2), (1, 144, 4, 1), (1, 400, 8, 2), (1, 1024, 32, 8)])
def test_prefill_online_softmax_variant_is_close(F, B, S, HQ, HKV):
    """The single-sweep online-softmax variant is NOT bit-exact (it quantises P per key tile against a dynamic scale and
    uses fast exponentials). Both it and the exact kernel approximate the unquantised-P attention with an 8-bit P; the
    variant's distance to that float64 attention must stay within 3 % of the largest output (worst element) and 0.3 %
    (mean) -- the fp32-level tolerance an 8-bit P allows -- and is printed beside the exact kernel's own distance."""
    q, qs, k, ks, v, vs, a_s = attn_inputs(B, S, HQ, HKV, 33)
    cos_t, sin_t = oracle.rope_table(max(S, 16))
    args = [dev(q), dev(qs), dev(k), dev(ks), dev(v), dev(vs), dev(cos_t), dev(sin_t)]
    exact, _ = F.MHA_i8xi8_Prefilling(*args, dev(a_s))
    online = F.MHA_i8xi8_Prefilling_online(*args)
    torch.cuda.synchronize()
    assert F.lib().flexllm_device_status() == 0
    exact = to_np(exact); online = to_np(online)
    assert np.isfinite(online).all()
    ref = _float_attention(oracle.mha_prefill(q, qs, k, ks, v, vs, cos_t, sin_t, a_s), v, vs)
    scale = np.abs(ref).max()
    d_on = np.abs(online - ref) / scale; d_ex = np.abs(exact - ref) / scale
    print(f"online softmax B={B} S={S}: distance to float64 attention, of the largest output: online max {d_on.max():.2e} mean "
          f"{d_on.mean():.2e}; exact kernel max {d_ex.max():.2e} mean {d_ex.mean():.2e}")
    assert d_on.max() < 3e-2 and d_on.mean() < 3e-3


# ------------------------------------------------------------------------------ decode (config 4)
def decode_case(F, B, ctx, HQ=32, HKV=8, seed=40, steps=1, q_gain=1.0, v_gain=1.0, a_gain=1.0, k_gain=1.0, signed_from=None):
    """signed_from n: keys before position n point against the first query head of their group, the others along it."""
    g = np.random.default_rng(seed)
    PAGE = 64
    ctx = np.asarray(ctx, np.int32)
    pages_per_seq = (ctx + steps + PAGE - 1) // PAGE + 1
    max_pages = int(pages_per_seq.max())
    n_pages = int(pages_per_seq.sum()) + 3
    perm = g.permutation(n_pages).astype(np.int32)            # seeded random page table
    page_table = np.zeros((B, max_pages), np.int32)
    o = 0
    for b in range(B):
        page_table[b, :pages_per_seq[b]] = perm[o:o + pages_per_seq[b]]; o += pages_per_seq[b]
    # cache contents for the already-present tokens (oracle layout: [n_pages][HKV][PAGE][64])
    k_pool = g.integers(-127, 128, (n_pages, HKV, PAGE, 64), dtype=np.int8)
    v_pool = g.integers(-127, 128, (n_pages, HKV, PAGE, 64), dtype=np.int8)
    ks_pool = g.uniform(0.005, 0.05, (n_pages, HKV, PAGE)).astype(np.float32)
    vs_pool = g.uniform(0.005, 0.05, (n_pages, HKV, PAGE)).astype(np.float32)
    max_ctx = int(ctx.max()) + steps
    cos_t, sin_t = oracle.rope_table(max_ctx + 1)
    a_s = np.full(HQ, 0.05 / 255 * a_gain, np.float32)
    vs_pool *= np.float32(v_gain); ks_pool *= np.float32(k_gain)
    cache = F.KVCache(1, n_pages, HKV)
    kd, ksd, vd, vsd = cache.pools(0)
    ksd.copy_(dev(ks_pool)); vsd.copy_(dev(vs_pool))
    vd.copy_(dev(np.ascontiguousarray(v_pool.transpose(0, 1, 3, 2))))
    cur = ctx.copy()
    for step in range(steps):
        q = g.integers(-127, 128, (B, HQ, 64), dtype=np.int8); k = g.integers(-127, 128, (B, HKV, 64), dtype=np.int8)
        v = g.integers(-127, 128, (B, HKV, 64), dtype=np.int8)
        qs = g.uniform(0.005, 0.05, (B, HQ)).astype(np.float32); ks = g.uniform(0.005, 0.05, (B, HKV)).astype(np.float32)
        vs = g.uniform(0.005, 0.05, (B, HKV)).astype(np.float32) * np.float32(v_gain)
        qs *= np.float32(q_gain); ks *= np.float32(k_gain)
        if signed_from is not None:
            prepared = oracle.qk_prepare(q.reshape(B, HQ, 64), qs, cur, cos_t, sin_t)[0]
            for b in range(B):
                along = np.where(prepared[b, ::HQ // HKV] < 0, -100, 100).astype(np.int8)
                for t in range(cur[b]): k_pool[page_table[b, t // PAGE], :, t % PAGE] = -along if t < signed_from else along
        if step == 0: kd.copy_(dev(k_pool))
        out, oacc = F.MHA_i8xi8_Decoding(cache, 0, dev(q), dev(qs), dev(k), dev(ks), dev(v), dev(vs), dev(cos_t), dev(sin_t),
                                         dev(a_s), dev(page_table), dev(cur), max_ctx, want_oacc=True)
        torch.cuda.synchronize()
        out_o, oacc_o = oracle.mha_decode(q, qs, k, ks, v, vs, cos_t, sin_t, a_s, k_pool, ks_pool, v_pool, vs_pool,
                                          page_table, cur)
        assert_same(to_np(oacc), oacc_o, "int32 P.V accumulators")
        assert_same(to_np(out), out_o, "fp32 output")
        cur = cur + 1
    # the appended tokens landed in the cache exactly as in the oracle
    assert_same(to_np(kd), k_pool, "K cache"); assert_same(to_np(ksd), ks_pool, "K scales")
    assert_same(to_np(vd), np.ascontiguousarray(v_pool.transpose(0, 1, 3, 2)), "V cache"); assert_same(to_np(vsd), vs_pool, "V scales")
    cache.close()


def test_decode_small(F):
    decode_case(F, 3, [0, 5, 130], steps=2)


def test_decode_page_boundaries(F):
    decode_case(F, 6, [63, 64, 65, 511, 512, 513], seed=41, steps=2)


def test_decode_config4_slice(F):
    """The decode-attention workload's shapes: contexts drawn uniformly from [512, 8192], one layer, 8 sequences."""
    g = np.random.default_rng(42)
    decode_case(F, 8, g.integers(512, 8193, 8), seed=42)


def test_decode_max_context(F):
    decode_case(F, 2, [8192, 8191], seed=43)


@pytest.mark.parametrize("what", [dict(q_gain=20.0), dict(q_gain=3.0), dict(a_gain=0.01), dict(a_gain=1e-5), dict(v_gain=2.0 ** 46, a_gain=2.0 ** 38),
                                  dict(v_gain=2.0 ** -60)], ids=["peaked", "spread", "large", "saturated", "wide_scales", "tiny_scales"])
def test_decode_quantiser_ranges(F, what):
    """Both sides of every line that the exponential and the quantiser draw (as in the prompt kernel's test), with lengths on both sides
    of a block of the ordered sums, equal lengths, and the longest sequence neither first nor last."""
    decode_case(F, 7, [62, 126, 127, 700, 62, 0, 255], seed=46, **what)


@pytest.mark.parametrize("e", [-62, -66, -70, -80])
def test_decode_scores_below_the_normal_range(F, e):
    """As in the prompt kernel's test; at 2^-80 every score is a zero, of the sign of the integer it comes from."""
    decode_case(F, 7, [62, 126, 127, 700, 62, 0, 255], seed=47, q_gain=2.0 ** e, k_gain=2.0 ** e)


def test_decode_maximum_of_either_zero(F):
    """Scores that underflow to -0 in the keys that every thread sees first and to +0 in later ones."""
    decode_case(F, 2, [300, 700], seed=48, q_gain=2.0 ** -80, k_gain=2.0 ** -80, signed_from=128)


@pytest.mark.parametrize("B,lo,hi,what", [(9, 1, 300, {}), (10, 1, 300, {}), (20, 0, 130, dict(q_gain=3.0)), (20, 60, 130, dict(a_gain=0.01)),
                                          (37, 0, 2100, {}), (38, 0, 100, {}), (38, 0, 2100, {}), (40, 126, 126, {}), (12, 1400, 1530, {}), (12, 100, 1600, dict(q_gain=20.0)),
                                          (8, 100, 5800, {}), (10, 100, 5800, {}), (10, 100, 5600, {})])
def test_decode_forms(F, B, lo, hi, what):
    """Numbers of sequences and contexts on both sides of the lines between the forms: four query heads or two to a CTA, sequences in
    their order or by length."""
    decode_case(F, B, np.append(np.random.default_rng(B).integers(lo, hi + 1, B - 1), hi), seed=50 + B, **what)


def test_kv_append_alone(F):
    """The cache managers' append on its own: the new token's K row, transposed V column and both scales land at
    position ctx[b] of the right page; everything else in the pools is untouched."""
    g = np.random.default_rng(45)
    B, HKV, PAGE = 5, 8, 64
    ctx = np.array([0, 63, 64, 200, 777], np.int32)
    pages = (ctx + 1 + PAGE - 1) // PAGE
    max_pages = int(pages.max()); n_pages = int(pages.sum()) + 2
    perm = g.permutation(n_pages).astype(np.int32)
    pt = np.zeros((B, max_pages), np.int32); o = 0
    for b in range(B):
        pt[b, :pages[b]] = perm[o:o + pages[b]]; o += pages[b]
    cache = F.KVCache(2, n_pages, HKV)
    layer = 1
    kd, ksd, vd, vsd = cache.pools(layer)
    k_pool = g.integers(-127, 128, (n_pages, HKV, PAGE, 64), dtype=np.int8); v_pool = g.integers(-127, 128, (n_pages, HKV, 64, PAGE), dtype=np.int8)
    ks_pool = g.uniform(0.005, 0.05, (n_pages, HKV, PAGE)).astype(np.float32); vs_pool = g.uniform(0.005, 0.05, (n_pages, HKV, PAGE)).astype(np.float32)
    kd.copy_(dev(k_pool)); vd.copy_(dev(v_pool)); ksd.copy_(dev(ks_pool)); vsd.copy_(dev(vs_pool))
    k = g.integers(-127, 128, (B, HKV, 64), dtype=np.int8); v = g.integers(-127, 128, (B, HKV, 64), dtype=np.int8)
    ks = g.uniform(0.005, 0.05, (B, HKV)).astype(np.float32); vs = g.uniform(0.005, 0.05, (B, HKV)).astype(np.float32)
    F.dec_KV_cache_append(cache, layer, dev(k), dev(ks), dev(v), dev(vs), dev(pt), dev(ctx), int(ctx.max()))
    torch.cuda.synchronize()
    for b in range(B):
        pg, slot = pt[b, ctx[b] // PAGE], ctx[b] % PAGE
        k_pool[pg, :, slot, :] = k[b]; v_pool[pg, :, :, slot] = v[b]; ks_pool[pg, :, slot] = ks[b]; vs_pool[pg, :, slot] = vs[b]
    assert_same(to_np(kd), k_pool, "K pool"); assert_same(to_np(vd), v_pool, "V pool")
    assert_same(to_np(ksd), ks_pool, "K scales"); assert_same(to_np(vsd), vs_pool, "V scales")
    k0 = cache.pools(0)[0]
    assert int(k0.abs().max()) == 0          # the other layer was not touched
    cache.close()


@pytest.mark.parametrize("ctx,HKV,what", [
    ([512, 0, 63, 64, 65, 127, 128, 191, 192, 256], 8, {}), ([511, 510, 100], 8, {}), ([510, 500, 100], 8, {}),     # the first length's line is 512
    ([3000, 0, 63, 64, 255, 256, 257, 3000, 1023, 1024], 2, {}), ([3000, 2999, 31], 1, dict(q_gain=20.0)),
    ([1700] + [130] * 9 + [1700] * 9 + [0], 8, {}), ([1662] + [40] * 18, 8, {}), ([1664, 1663] + [40] * 17, 8, dict(a_gain=0.01)),       # by length, with equal ones
    ([2000] + [300] * 16, 8, {}), ([2000] + [300] * 17, 8, {}),                                      # all clusters at once, and not quite
    ([10238], 8, {}), ([10239, 5], 8, {}), ([32766, 700], 1, {}), ([32767, 700], 1, {})],            # longest rows of either form
    ids=lambda v: "%d_of_%d" % (len(v), v[0]) if isinstance(v, list) else None)
def test_decode_cluster(F, ctx, HKV, what):
    """The form with a cluster of four CTAs per item: lengths around its lines, sequences of fewer pages than CTAs, page and quarter
    edges, few and many KV heads, two steps (the second reads what the first appended)."""
    decode_case(F, len(ctx), ctx, HQ=4 * HKV, HKV=HKV, seed=70 + len(ctx), steps=2 if ctx[0] < 5000 else 1, **what)


def test_decode_from_several_threads(F):
    """Calls whose shared-memory needs are far apart, from host threads on streams of their own: none takes the room of another away."""
    import threading
    lib, r = F.lib(), {}

    def work(name, max_ctx):
        g = torch.Generator(device="cuda").manual_seed(max_ctx)
        s8 = lambda *s: torch.randint(-127, 128, s, dtype=torch.int8, device="cuda", generator=g)
        u = lambda *s: torch.rand(s, device="cuda", generator=g) * 0.05
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            cache = F.KVCache(1, 2, 1)
            a = [s8(1, 4, 64), u(1, 4), s8(1, 1, 64), u(1, 1), s8(1, 1, 64), u(1, 1), u(41, 32), u(41, 32), u(4)]
            table = torch.zeros(1, max_ctx // 64 + 1, dtype=torch.int32, device="cuda")
            ctx, out = torch.tensor([40], dtype=torch.int32, device="cuda"), torch.empty(1, 256, device="cuda")
            nbytes = lib.flexllm_mha_decode_workspace(1, 4, max_ctx)
            ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
            args = [cache._h, 0, *[t.data_ptr() for t in a], table.data_ptr(), table.shape[1], ctx.data_ptr(), max_ctx, 1, 4, out.data_ptr(), None,
                    ws.data_ptr(), nbytes, stream.cuda_stream]
            call = lib.flexllm_mha_i8xi8_decode
            call(*args)
            first = out.clone()
            refused = sum(call(*args) != 0 for _ in range(20000))
            stream.synchronize()
            r[name] = refused, torch.equal(first, out)
            cache.close()

    threads = [threading.Thread(target=work, args=a) for a in (("long", 32000), ("short", 600), ("middle", 9000))]
    for t in threads: t.start()
    for t in threads: t.join()
    assert r == {k: (0, True) for k in ("long", "short", "middle")}
