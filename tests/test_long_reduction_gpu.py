"""Long reductions on the tensor cores: tiles whose reduction the CTAs of a cluster share, 192-column tiles and CTA pairs whose
second half has no rows, against float64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def run_conv(odla, lib, N, H, W, C, K, R, residual, dtype):
    rng = np.random.default_rng(N * H * W + C + K)
    pad = R // 2
    x = rng.standard_normal((N, H, W, C)).astype(np.float32)
    w = (rng.standard_normal((R, R, C, K)) / np.sqrt(R * R * C)).astype(np.float32)
    b = rng.standard_normal(K).astype(np.float32)
    r = rng.standard_normal((N, H, W, K)).astype(np.float32)
    g = odla.Graph(lib, "c", fp16=dtype == "f16", bf16=dtype == "bf16", n_gpus=1)
    io, td = (odla.FLOAT16, torch.float16) if dtype == "f16" else (odla.FLOAT32, torch.float32)
    half = torch.float16 if dtype == "f16" else torch.bfloat16
    y = g.Conv(g.Argument("x", (N, H, W, C), io), odla.CHANNELS_LAST, 1, g.Constant("w", w), odla.SIO, (1, 1), (1, 1), (pad, pad), (pad, pad), None, (N, H, W, K), "conv")
    y = g.Add(y, g.Constant("b", b.reshape(1, 1, 1, K)), "bias")
    if residual:
        y = g.Add(y, g.Argument("r", (N, H, W, K), io), "sum")
    g.Output(g.Relu(y, "y"))
    tx, tr = torch.from_numpy(x).to(half).to(td).cuda(), torch.from_numpy(r).to(half).to(td).cuda()
    o = torch.empty((N, H, W, K), dtype=td, device="cuda")
    g.bind_input("x", tx.data_ptr())
    if residual:
        g.bind_input("r", tr.data_ptr())
    g.bind_output(g.out_names[0], o.data_ptr())
    torch.cuda.synchronize()
    assert g.execute() == 0
    assert any(p["op"] == "conv_umma" for p in g.profile(runs=1))
    g.close()
    xd, wd = torch.from_numpy(x).to(half).double(), torch.from_numpy(w).to(half).double()
    ref = torch.nn.functional.conv2d(xd.permute(0, 3, 1, 2).cuda(), wd.permute(3, 2, 0, 1).cuda(), padding=pad).permute(0, 2, 3, 1).cpu().numpy() + b
    if residual:
        ref = ref + torch.from_numpy(r).to(half).double().numpy()
    return o.float().cpu().numpy(), np.maximum(ref, 0)


SIZES = [  # N, H, W, C, K, R
    (1, 7, 7, 512, 512, 3), (1, 5, 13, 256, 72, 3), (1, 1, 130, 2048, 1000, 1), (2, 7, 9, 520, 24, 3), (1, 14, 14, 1024, 256, 1), (1, 1, 1, 4096, 8, 1),   # clusters of 2 to 8
    (1, 65, 100, 768, 320, 1), (1, 64, 100, 768, 320, 1),   # 192 columns: 51 row tiles (a half-empty pair) and 50
]


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("dtype", ["f16", "bf16"])
def test_long_reductions(odla, gpu_lib, size, residual, dtype):
    got, ref = run_conv(odla, gpu_lib, *size, residual, dtype)
    # one rounding of the sum before the residual and one after it, of values below eight
    step = 2.0 ** (-10 if dtype == "f16" else -7)
    np.testing.assert_allclose(got, ref, rtol=step, atol=2 * step)


def raw_conv(odla, lib, dtype, N, H, W, C, K, R, out_kind, seed=3, **epilogue):
    """odla_b200_conv_umma over integers (int8) or values of the type; (result, the operands as float64 / int64)."""
    import ctypes
    rng = np.random.default_rng(seed)
    if dtype == "s8":
        x, w = (torch.from_numpy(rng.integers(-127, 128, s, dtype=np.int8)).cuda() for s in ((N, H, W, C), (K, R * R * C)))
    else:
        t = {"f16": torch.float16, "bf16": torch.bfloat16}[dtype]
        x, w = (torch.from_numpy(rng.standard_normal(s).astype(np.float32) * k).to(t).cuda() for s, k in (((N, H, W, C), 1.0), ((K, R * R * C), (R * R * C) ** -0.5)))
    y = torch.zeros((N, H, W, K), dtype={1: torch.float32, 2: torch.int8, 3: torch.int32}[out_kind], device="cuda")
    tensors = {n: torch.from_numpy(v).cuda() for n, v in epilogue.items() if isinstance(v, np.ndarray)}
    ptr = lambda n: tensors[n].data_ptr() if n in tensors else None
    d = odla.ConvDesc(n=N, h=H, w=W, c=C, k=K, r=R, s=R, stride_h=1, stride_w=1, pad_top=R // 2, pad_left=R // 2, p=H, q=W, dtype=["f16", "bf16", "s8"].index(dtype), out_kind=out_kind,
                      res_kind=2 if "res" in tensors else 0, act=epilogue.get("act", 0), alpha=0, res_scale=epilogue.get("res_scale", 1), out_scale=epilogue.get("out_scale", 1),
                      out_multiply=epilogue.get("out_multiply", 0))
    torch.cuda.synchronize()
    assert lib.b200_conv_umma(ctypes.byref(d), x.data_ptr(), w.data_ptr(), ptr("mul"), ptr("add"), ptr("res"), y.data_ptr(), None) == 0
    acc = torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), w.double().view(K, R, R, C).permute(0, 3, 1, 2), padding=R // 2).permute(0, 2, 3, 1)
    return y.cpu().numpy(), acc.cpu().numpy()


def test_the_switch_for_pairs_leaves_shared_reductions_on(odla, gpu_lib, monkeypatch):
    """ODLA_B200_PAIR_MIN_KB at its own default changes nothing, here for a layer whose reduction eight CTAs share."""
    size = (1, 7, 7, 512, 512, 3)
    default, _ = raw_conv(odla, gpu_lib, "f16", *size, out_kind=1)
    monkeypatch.setenv("ODLA_B200_PAIR_MIN_KB", "12")
    switched, _ = raw_conv(odla, gpu_lib, "f16", *size, out_kind=1)
    monkeypatch.setenv("ODLA_B200_NO_SPLIT", "1")
    unshared, _ = raw_conv(odla, gpu_lib, "f16", *size, out_kind=1)
    assert np.array_equal(default, switched) and not np.array_equal(default, unshared)


@pytest.mark.parametrize("chunks", ["0", "1"])
@pytest.mark.parametrize("size", [(16, 26, 26, 256, 512, 3), (1, 65, 100, 768, 320, 1), (1, 64, 128, 768, 256, 1)])
def test_epilogue_chunk_assignment_on_long_reductions(odla, gpu_lib, monkeypatch, size, chunks):
    """ODLA_B200_EPI_INTERLEAVE either way, where two boxes go round for a tile of three or four and where a tile has 192 columns."""
    monkeypatch.setenv("ODLA_B200_EPI_INTERLEAVE", chunks)
    got, ref = run_conv(odla, gpu_lib, *size, False, "f16")
    np.testing.assert_allclose(got, ref, rtol=2.0 ** -10, atol=2.0 ** -9)   # one rounding of the result, values below eight


@pytest.mark.parametrize("K", [255, 10, 64])
@pytest.mark.parametrize("residual", [False, True])
def test_shared_reductions_store_any_number_of_columns(odla, gpu_lib, K, residual):
    """Results of two-byte storage that leave as fp32: rows padded to 16 bytes inside (255 and 10 columns without a residual),
    finished value by value, or, with a residual, stored densely."""
    got, ref = run_conv(odla, gpu_lib, 1, 7, 9, 2048, K, 1, residual, "bf16")
    np.testing.assert_allclose(got, ref, rtol=2.0 ** -7, atol=2.0 ** -6)


@pytest.mark.parametrize("dtype", ["f16", "bf16", "s8"])
@pytest.mark.parametrize("K", [255, 10, 512])
def test_shared_reductions_raw_accumulators(odla, gpu_lib, dtype, K):
    """fp32 and int32 results of a reduction over 4608 products: exact integers, fp32 sums in any order."""
    got, acc = raw_conv(odla, gpu_lib, dtype, 1, 7, 7, 512, K, 3, out_kind=3 if dtype == "s8" else 1)
    if dtype == "s8":
        assert np.array_equal(got, acc.astype(np.int64))
    else:   # partial sums of up to 4608 exact products of magnitude 4608^-1/2
        np.testing.assert_allclose(got, acc, rtol=0, atol=4608 ** 0.5 * 2.0 ** -24 * 16)


@pytest.mark.parametrize("multiply", [0, 1])
@pytest.mark.parametrize("K", [512, 72, 130])
def test_shared_reductions_requantise_bit_exact(odla, gpu_lib, K, multiply):
    rng = np.random.default_rng(K)
    e = dict(mul=rng.uniform(1e-5, 1e-4, K).astype(np.float32), add=rng.standard_normal(K).astype(np.float32), res=rng.integers(-128, 128, (1, 7, 7, K), dtype=np.int8),
             act=1, res_scale=float(np.float32(0.037)), out_scale=float(np.float32(0.021)), out_multiply=multiply)
    got, acc = raw_conv(odla, gpu_lib, "s8", 1, 7, 7, 512, K, 3, out_kind=2, **e)
    v = acc.astype(np.float32) * e["mul"] + e["add"] + e["res"].astype(np.float32) * np.float32(0.037)     # numpy rounds every step to fp32, as the kernel does
    v = np.maximum(v, np.float32(0))
    scaled = v * (np.float32(1.0) / np.float32(0.021)) if multiply else v / np.float32(0.021)
    assert np.array_equal(got, np.clip(np.rint(scaled), -128, 127).astype(np.int8))


@pytest.mark.parametrize("N,transposed", [(64, False), (64, True), (96, False), (96, True)])
def test_shared_reductions_of_batched_products(odla, gpu_lib, monkeypatch, N, transposed):
    """Two run-time operands, 2 x [128, 2048] x [2048, N]: the right one read as it lies (64 columns), transposed first, or K-major."""
    B, M, K = 2, 128, 2048
    rng = np.random.default_rng(N)
    a, b = [torch.from_numpy(rng.standard_normal(s).astype(np.float32)).half() for s in ((B, M, K), (B, N, K) if transposed else (B, K, N))]
    b = (b.float() / K ** 0.5).half()
    outs = []
    for unshared in (False, True):
        if unshared:
            monkeypatch.setenv("ODLA_B200_NO_SPLIT", "1")
        g = odla.Graph(gpu_lib, "g", fp16=True, n_gpus=1)
        g.Output(g.Gemm(g.Argument("a", a.shape, odla.FLOAT16), False, g.Argument("b", b.shape, odla.FLOAT16), transposed, 1.0, 0.0, None, (B, M, N), "y"))
        outs.append(g.run({"a": a.numpy(), "b": b.numpy()})["y"])
        assert "gemm_umma" in g.describe()
        g.close()
    want = np.einsum("bmk,bnk->bmn" if transposed else "bmk,bkn->bmn", a.double().numpy(), b.double().numpy())
    for o in outs:
        np.testing.assert_allclose(o.astype(np.float64), want, rtol=2.0 ** -11, atol=4e-5)   # one rounding to fp16 of values up to five
