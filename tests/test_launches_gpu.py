"""Which launches may start before the kernel in front has finished: read from captured graphs, whose edges say so."""
import ctypes as C
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


class EdgeData(C.Structure):
    _fields_ = [("from_port", C.c_ubyte), ("to_port", C.c_ubyte), ("type", C.c_ubyte), ("reserved", C.c_ubyte * 5)]


def edges(work):
    """(programmatic, all) edges of the graph that `work` is captured into, after one run outside of it."""
    cudart = C.CDLL("libcudart.so.12")
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        work()
        side.synchronize()
        g = torch.cuda.CUDAGraph(keep_graph=True)
        g.capture_begin()
        work()
        g.capture_end()
        n = C.c_size_t()
        graph = C.c_void_p(g.raw_cuda_graph())
        assert cudart.cudaGraphGetEdges_v2(graph, None, None, None, C.byref(n)) == 0
        a, b, d = (C.c_void_p * n.value)(), (C.c_void_p * n.value)(), (EdgeData * n.value)()
        assert cudart.cudaGraphGetEdges_v2(graph, a, b, d, C.byref(n)) == 0
        return sum(e.type == 1 for e in d), n.value


def paths(F):
    """name -> (programmatic, all) edges of the entry points that overlap launches."""
    from flexllm_b200 import synthetic
    gen = torch.Generator(device="cuda").manual_seed(1)
    s8 = lambda *n: torch.randint(-127, 128, n, dtype=torch.int8, device="cuda", generator=gen)
    u = lambda *n: torch.rand(n, device="cuda", generator=gen) * 1e-2
    x, gamma = torch.randn(4, 2048, device="cuda"), 1 + u(2048)
    lin, mlp = (s8(256, 512), u(256), s8(512, 512), u(512)), (x, gamma, s8(16384, 2048), u(16384), s8(2048, 8192), u(2048))
    att = (s8(1, 128, 4, 64), u(1, 128, 4), s8(1, 128, 1, 64), u(1, 128, 1), s8(1, 128, 1, 64), u(1, 128, 1), u(128, 32), u(128, 32), u(4))
    W = synthetic.numpy_weights(1, 256, 4, 1, 8192, 512, 140, seed=3)
    m = F.Model(1, 256, 4, 1, 8192, 512, max_batch=2, max_prefill=128, max_ctx=140)
    synthetic.load_numpy_weights(m, W)
    tok = torch.zeros(2, 128, dtype=torch.int32, device="cuda")

    def products():
        y = F.pref_Linear_Layer_i8xi8(*lin)[1]
        for _ in range(3):
            y = F.pref_Linear_Layer_i8xi8(*lin, residual=y)[1]
    r = dict(products=edges(products), attention=edges(lambda: F.MHA_i8xi8_Prefilling(*att)), mlp=edges(lambda: F.dec_MLP_block(*mlp)),
             prompt=edges(lambda: m.prefill(tok)))
    m.close()
    return r


@pytest.mark.parametrize("pdl", ["1", "0"])
def test_programmatic_launches_can_be_switched_off(pdl):
    """FLEXLLM_PDL=0 is read once in a process, so each side is one of its own."""
    code = "import sys; sys.path[:0] = [%r, %r]\nimport flexllm_b200 as F, test_launches_gpu as t\nprint(t.paths(F))" % (ROOT, os.path.join(ROOT, "tests"))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, env=dict(os.environ, FLEXLLM_PDL=pdl), cwd=ROOT, timeout=600)
    assert r.returncode == 0, r.stderr
    found = eval(r.stdout.strip().splitlines()[-1])
    assert set(found) == {"products", "attention", "mlp", "prompt"}
    for name, (programmatic, n) in found.items():
        assert n > 0 and (programmatic > 0 if pdl == "1" else programmatic == 0), (name, programmatic, n)


def chain(F, seed):
    """Inputs and the launches of a prompt's operators one after another, each on the output of the one before."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    s8 = lambda *n: torch.randint(-127, 128, n, dtype=torch.int8, device="cuda", generator=gen)
    u = lambda *n: torch.rand(n, device="cuda", generator=gen) * 1e-2
    a, w, sc = s8(256, 1024), [s8(1024, 1024) for _ in range(3)], u(1024)
    q, k, v, cos, sin, a_s = s8(2, 128, 16, 64), s8(2, 128, 4, 64), s8(2, 128, 4, 64), u(128, 32), u(128, 32), u(16)
    qs, ks, s0 = u(2, 128, 16), u(2, 128, 4), u(256)

    def work():
        y = F.pref_Linear_Layer_i8xi8(a, s0, w[0], sc)[1]
        for m in w[1:]:
            x, s = F.pref_quant_layer_fp32_qint(y)
            y = F.pref_Linear_Layer_i8xi8(x, s, m, sc, residual=y)[1]
        x, s = F.pref_quant_layer_fp32_qint(y)
        out = F.MHA_i8xi8_Prefilling(x.view(2, 128, 16, 64), qs, k, ks, v, ks, cos, sin, a_s)[0]
        return y, out, F.MHA_i8xi8_Prefilling(q, qs, k, ks, v, ks, cos, sin, a_s)[0]
    return (a, k), work


@pytest.mark.parametrize("captured", [False, True])
def test_prompt_operators_behind_another_stream(captured):
    """Inputs written late on another stream, which the first product follows through an event alone; eagerly and as a graph that is replayed
    on inputs it was not captured with."""
    import flexllm_b200 as F
    (a, k), work = chain(F, 5)
    new = [torch.randint(-127, 128, t.shape, dtype=torch.int8, device="cuda", generator=torch.Generator(device="cuda").manual_seed(i)) for i, t in enumerate((a, k))]
    old = [a.clone(), k.clone()]
    for t, n in zip((a, k), new): t.copy_(n)
    want = [t.clone() for t in work()]
    for t, n in zip((a, k), old): t.copy_(n)
    main, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()

    def forked():
        other.wait_stream(main)
        with torch.cuda.stream(other):
            torch.cuda._sleep(2_000_000)              # a millisecond: the products would be long over
            for t, n in zip((a, k), new): t.copy_(n)
        main.wait_stream(other)
        return work()
    with torch.cuda.stream(main):
        if captured:
            g = torch.cuda.CUDAGraph()
            g.capture_begin()
            got = forked()
            g.capture_end()
            for _ in range(3):
                for t, n in zip((a, k), old): t.copy_(n)
                g.replay()
        else:
            got = forked()
    torch.cuda.synchronize()
    for x, y in zip(got, want):
        assert torch.equal(x, y)
    assert F.lib().flexllm_device_status() == 0
