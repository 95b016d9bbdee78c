"""The fused attention launch at sequence lengths that do not fill its 128-position blocks, behind projections (heads read
as column groups, the three projections one Gemm) and on head-split operands, against float64 numpy."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def attention(q, k, v, scale):
    s = np.einsum("bhid,bhjd->bhij", q, k) * scale
    p = np.exp(s - s.max(axis=-1, keepdims=True))
    return np.einsum("bhij,bhjd->bhid", p / p.sum(axis=-1, keepdims=True), v)


@pytest.mark.parametrize("mode", ["fp16", "bf16"])
@pytest.mark.parametrize("S", [1, 15, 16, 77, 127, 128, 129, 256, 300])
@pytest.mark.parametrize("operands", ["projections", "separate", "heads"])
def test_attention_over_any_length(odla, gpu_lib, mode, S, operands):
    B, NH, D = 3, 5, 64
    H = NH * D
    rng = np.random.default_rng(S)
    t = {"fp16": torch.float16, "bf16": torch.bfloat16}[mode]
    rnd = lambda a: torch.from_numpy(a).to(t).float().numpy()     # values the storage type holds exactly
    g = odla.Graph(gpu_lib, "att", fp16=mode == "fp16", bf16=mode == "bf16", n_gpus=1)
    ins, heads = {}, []
    if operands == "heads":
        for n in "qkv":
            ins[n] = rnd(rng.standard_normal((B, NH, S, D)).astype(np.float32))
            heads.append(g.Argument(n, (B, NH, S, D)))
        want_in = [ins[n].astype(np.float64) for n in "qkv"]
    else:
        want_in = []
        xs = {}
        for n in "qkv":
            src = "x" if operands == "projections" else "x" + n
            if src not in xs:
                ins[src] = rnd(rng.standard_normal((B * S, 96)).astype(np.float32))
                xs[src] = g.Argument(src, (B * S, 96))
            w = rnd((rng.standard_normal((96, H)) / np.sqrt(96) * (2.0 if n == "q" else 1.0)).astype(np.float32))
            b = rnd(rng.standard_normal(H).astype(np.float32) * 0.1)
            y = g.Gemm(xs[src], False, g.Constant("w" + n, w), False, 1.0, 1.0, g.Constant("b" + n, b), (B * S, H), n)
            y = g.Reshape(y, (B, S, NH, D), n + "4")
            heads.append(g.Transpose(y, (0, 2, 1, 3), (B, NH, S, D), n + "t"))
            p = rnd((ins[src].astype(np.float64) @ w + b).astype(np.float32)).astype(np.float64)
            want_in.append(p.reshape(B, S, NH, D).transpose(0, 2, 1, 3))
    q, k, v = heads
    sc = g.Mul(g.Gemm(q, False, k, True, 1.0, 0.0, None, (B, NH, S, S), "scores"), g.Constant("scale", np.array([0.125], np.float32)), "scaled")
    ctx = g.Gemm(g.Softmax(sc, -1, "probs"), False, v, False, 1.0, 0.0, None, (B, NH, S, D), "ctx")
    if operands != "heads":
        ctx = g.Transpose(ctx, (0, 2, 1, 3), (B, S, NH, D), "merged")
    g.Output(ctx)
    got = g.run(ins)["merged" if operands != "heads" else "ctx"]
    desc = g.describe(first_gpu_only=True)
    launches = g.launches()
    g.close()
    assert desc.count("attention") == 1 and "softmax" not in desc and "transpose" not in desc
    if operands == "projections":
        assert desc.count("gemm_umma") == 3 and launches <= 4          # argument and result conversions, one projection, one attention
    want = attention(*want_in, 0.125)
    want = want if operands == "heads" else want.transpose(0, 2, 1, 3)
    ulp = 2.0 ** -10 if mode == "fp16" else 2.0 ** -7
    err = np.abs(got - want)
    assert np.isfinite(got).all() and err.max() <= 6 * ulp * max(1.0, np.abs(want).max()) and err.mean() <= ulp, (err.max(), err.mean())
