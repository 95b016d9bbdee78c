"""Range records around a fused attention: the queries, keys and values have them however the projections are launched."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [128, 77])
@pytest.mark.parametrize("shared_input", [True, False])
@pytest.mark.parametrize("sub_batches", [1, 2])
def test_records_of_q_k_v_are_those_of_the_unfused_graph(odla, gpu_lib, monkeypatch, S, shared_input, sub_batches):
    B, NH, D, E = 3, 2, 64, 96
    H = NH * D
    rng = np.random.default_rng(S)
    rnd = lambda a: torch.from_numpy(a.astype(np.float32)).half().float().numpy()
    ins = {n: rnd(rng.standard_normal((B, S, E))) for n in (["x"] if shared_input else ["xq", "xk", "xv"])}
    w = {n: rnd(rng.standard_normal((E, H)) / np.sqrt(E) * (i + 1)) for i, n in enumerate("qkv")}
    bias = {n: rnd(rng.standard_normal(H) + i) for i, n in enumerate("qkv")}
    tables = []
    for unfused in (False, True):
        if unfused:
            monkeypatch.setenv("ODLA_B200_NO_ATTENTION", "1")
        g = odla.Graph(gpu_lib, "ranges", fp16=True, n_gpus=1, sub_batches=sub_batches)
        args = {n: g.Reshape(g.Argument(n, (B, S, E)), (B * S, E), n + "_2d") for n in ins}
        heads = []
        for n in "qkv":
            y = g.Gemm(args["x" if shared_input else "x" + n], False, g.Constant("w" + n, w[n]), False, 1.0, 1.0, g.Constant("b" + n, bias[n]), (B * S, H), n)
            heads.append(g.Transpose(g.Reshape(y, (B, S, NH, D), n + "4"), (0, 2, 1, 3), (B, NH, S, D), n + "t"))
        q, k, v = heads
        sc = g.Mul(g.Gemm(q, False, k, True, 1.0, 0.0, None, (B, NH, S, S), "scores"), g.Constant("scale", np.array([0.125], np.float32)), "scaled")
        ctx = g.Gemm(g.Softmax(sc, -1, "probs"), False, v, False, 1.0, 0.0, None, (B, NH, S, D), "ctx")
        g.Output(g.Transpose(ctx, (0, 2, 1, 3), (B, S, NH, D), "merged"))
        g.range_profiling(True)
        g.run(ins)
        rec = {}
        for vid, ch, scale, _, mn, mx in g.quant_table():
            rec.setdefault(vid, {})[ch] = (mn, mx)
        tables.append(rec)
        assert ("softmax" in g.describe()) == unfused
        g.close()
    fused, plain = tables
    for n in "qkv":
        x = ins["x" if shared_input else "x" + n].reshape(B * S, E).astype(np.float64)
        full = (x @ w[n] + bias[n]).reshape(B * S * NH, D)
        assert set(fused[n + "t"]) == set(plain[n + "t"]) == {-D} | set(range(D))
        want = {-D: (full.min(), full.max()), **{d: (full[:, d].min(), full[:, d].max()) for d in range(D)}}
        for ch, (mn, mx) in want.items():
            np.testing.assert_allclose(fused[n + "t"][ch], (mn, mx), rtol=2.0 ** -10, atol=2.0 ** -10)   # one rounding to fp16
            np.testing.assert_allclose(plain[n + "t"][ch], (mn, mx), rtol=2.0 ** -10, atol=2.0 ** -10)


def test_launch_list_tells_launches_from_values(odla, gpu_lib):
    """The keys and values of grouped projections have entries of their own, marked as written by the launch above, and the
    profile counts no launch for them."""
    B, S, NH, D, E = 2, 32, 2, 64, 64
    rng = np.random.default_rng(0)
    g = odla.Graph(gpu_lib, "list", fp16=True, n_gpus=1)
    x = g.Argument("x", (B * S, E))
    heads = []
    for n in "qkv":
        y = g.Gemm(x, False, g.Constant("w" + n, rng.standard_normal((E, NH * D)).astype(np.float32) * 0.1), False, 1.0, 0.0, None, (B * S, NH * D), n)
        heads.append(g.Transpose(g.Reshape(y, (B, S, NH, D), n + "4"), (0, 2, 1, 3), (B, NH, S, D), n + "t"))
    sc = g.Mul(g.Gemm(heads[0], False, heads[1], True, 1.0, 0.0, None, (B, NH, S, S), "scores"), g.Constant("scale", np.array([0.125], np.float32)), "scaled")
    ctx = g.Gemm(g.Softmax(sc, -1, "probs"), False, heads[2], False, 1.0, 0.0, None, (B, NH, S, D), "ctx")
    g.Output(g.Transpose(ctx, (0, 2, 1, 3), (B, S, NH, D), "merged"))
    xin, out = rng.standard_normal((B * S, E)).astype(np.float32), np.empty((B, S, NH, D), np.float32)
    g.bind_input("x", xin.ctypes.data)
    g.bind_output("merged", out.ctypes.data)
    lines = {l.split()[1]: l for l in g.describe().splitlines() if l.startswith("  ")}
    runs = {p["name"]: p["launches"] for p in g.profile(runs=2)}
    g.close()
    for n, of_its_own in (("qt", True), ("kt", False), ("vt", False), ("merged", True)):
        assert ("(by the launch above)" in lines[n]) == (not of_its_own) and runs[n] == (2 if of_its_own else 0)
