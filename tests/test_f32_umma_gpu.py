"""fp32 layers as three bf16 values an operand on the tensor cores (kernels_f32_umma.cu) against a float64 evaluation, and against
the CUDA-core kernels where an operand is not an ordinary number."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def conv(odla, lib, x, w, b, r=None, stride=1, pad=1, act=0.0, sub_batches=None, launch="conv_f32_umma"):
    """act: slope of a LeakyReLU (0: ReLU), None: no activation."""
    N, H, W, C = x.shape
    R, _, _, K = w.shape
    P, Q = (H + 2 * pad - R) // stride + 1, (W + 2 * pad - R) // stride + 1
    g = odla.Graph(lib, "c", n_gpus=1, sub_batches=sub_batches)
    y = g.Conv(g.Argument("x", x.shape), odla.CHANNELS_LAST, 1, g.Constant("w", w), odla.SIO, (stride, stride), (1, 1), (pad, pad), (pad, pad), None, (N, P, Q, K), "conv")
    y = g.Add(y, g.Constant("b", b.reshape(1, 1, 1, K)), "bias")
    if r is not None:
        y = g.Add(y, g.Argument("r", r.shape), "sum")
    if act is not None:
        y = g.LeakyRelu(y, act, "act") if act else g.Relu(y, "act")
    g.Output(y)
    ins = {"x": x} if r is None else {"x": x, "r": r}
    try:
        out = next(iter(g.run(ins).values()))
        assert launch in g.describe()
    finally:
        g.close()
    return out


def plain_size(x, w, pad):
    """Sums of the terms' magnitudes: what an error is to be measured against where terms cancel."""
    t = torch.nn.functional.conv2d(torch.from_numpy(np.abs(x)).double().permute(0, 3, 1, 2), torch.from_numpy(np.abs(w)).double().permute(3, 2, 0, 1), padding=pad)
    return t.permute(0, 2, 3, 1).numpy()


def float64(x, w, b, r, stride, pad, act):
    t = torch.nn.functional.conv2d(torch.from_numpy(x).double().permute(0, 3, 1, 2), torch.from_numpy(w).double().permute(3, 2, 0, 1), stride=stride, padding=pad)
    y = t.permute(0, 2, 3, 1).numpy() + b + (0 if r is None else r)
    return y if act is None else np.where(y < 0, y * np.float64(np.float32(act)), y)


# N, H, C, K, window, stride, pad: one stage and several, half stages (channels past the last 32), 64- and 128-column tiles with ragged
# rows and columns, columns that are no multiple of four, a reduction shared by a cluster, three- and four-channel images as windows
SHAPES = [(4, 56, 64, 64, 1, 1, 0), (4, 30, 96, 128, 3, 1, 1), (9, 33, 36, 72, 3, 2, 1), (3, 29, 100, 255, 1, 1, 0), (2, 14, 512, 130, 3, 1, 1), (1, 7, 2048, 512, 1, 1, 0),
          (2, 7, 512, 512, 3, 1, 1), (8, 28, 128, 512, 1, 1, 0), (2, 112, 3, 64, 7, 2, 3), (1, 200, 4, 32, 3, 1, 1), (2, 60, 68, 64, 5, 1, 2)]


@pytest.mark.parametrize("act", [0.0, 0.1, None])
@pytest.mark.parametrize("shape", SHAPES)
def test_conv_matches_float64(odla, gpu_lib, shape, act):
    N, H, C, K, R, stride, pad = shape
    P = (H + 2 * pad - R) // stride + 1
    rng = np.random.default_rng(sum(shape))
    x = rng.standard_normal((N, H, H, C)).astype(np.float32)
    w = (rng.standard_normal((R, R, C, K)) / np.sqrt(R * R * C)).astype(np.float32)
    b = rng.standard_normal(K).astype(np.float32)
    r = rng.standard_normal((N, P, P, K)).astype(np.float32) if act != 0.1 else None
    got = conv(odla, gpu_lib, x, w, b, r, stride, pad, act)
    want = float64(x, w, b, r, stride, pad, act)
    # sums of 64 products each (a few roundings of 2^-24) and the chain over them, next to the largest of the results
    n = R * R * C
    err = np.abs(got - want).max() / np.sqrt(np.mean(want ** 2))
    assert err < 4e-7 * np.sqrt(max(n / 64, 4)) + 1e-6, err


@pytest.mark.parametrize("sub_batches", [2, 3])
def test_results_do_not_depend_on_the_cut(odla, gpu_lib, sub_batches):
    rng = np.random.default_rng(1)
    x, w = rng.standard_normal((6, 14, 14, 256)).astype(np.float32), (rng.standard_normal((3, 3, 256, 200)) / 48).astype(np.float32)
    b = rng.standard_normal(200).astype(np.float32)
    assert np.array_equal(conv(odla, gpu_lib, x, w, b), conv(odla, gpu_lib, x, w, b, sub_batches=sub_batches))


@pytest.mark.parametrize("exponent", [-70, -100, 128])
@pytest.mark.parametrize("shape", [(28, 128, 512, 1), (28, 64, 260, 3)])   # tiles of 128 columns for four images and of 64 for two
def test_results_computed_again_do_not_depend_on_the_cut(odla, gpu_lib, shape, exponent):
    """Results on both sides of where they are computed again (too small for the split, sums that overflow on the way): whether a
    neighbour in the tile is on the other side makes no difference to any bit."""
    H, C, K, R = shape
    rng = np.random.default_rng(2)
    x = rng.standard_normal((4, H, H, C)).astype(np.float32) * np.float32(2.0 ** (exponent / 2))
    w = (rng.standard_normal((R, R, C, K)) / np.sqrt(R * R * C) * 2.0 ** min(exponent / 2, 19)).astype(np.float32)
    x *= np.float32(2.0 ** (exponent / 2 - 20 if exponent > 0 else 5))   # (a few of a hundred are on the other side)
    b = np.zeros(K, np.float32)
    outs = [conv(odla, gpu_lib, x, w, b, pad=R // 2, act=None, sub_batches=s) for s in (1, 2, 4)]
    with np.errstate(over="ignore"):
        size = np.abs(float64(x, w, 0, None, 1, R // 2, None))
    assert 0.01 < np.mean(size < 2.0 ** exponent) < 0.99
    for o in outs[1:]:
        assert np.array_equal(o.view(np.uint32), outs[0].view(np.uint32))


@pytest.mark.parametrize("shape", [(2, 28, 64, 128, 3), (1, 14, 256, 320, 3)])   # boxes of results; a shared reduction
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 3.4e38, 1e-30, 1e-38])
def test_values_the_split_does_not_hold(odla, gpu_lib, shape, bad, monkeypatch):
    """Infinities, NaN, the largest fp32 values and operands whose last bits no bf16 can carry: what the CUDA-core kernel gives."""
    N, H, C, K, R = shape
    rng = np.random.default_rng(5)
    x = rng.standard_normal((N, H, H, C)).astype(np.float32)
    w = (rng.standard_normal((R, R, C, K)) / np.sqrt(R * R * C)).astype(np.float32)
    b = np.zeros(K, np.float32)
    if abs(bad) < 1:
        x *= np.float32(bad)
    else:
        x[0, 3, 4, 5] = x[0, H - 1, 0, C - 1] = bad
    got = conv(odla, gpu_lib, x, w, b, act=None)
    monkeypatch.setenv("ODLA_B200_NO_F32_UMMA", "1")
    want = conv(odla, gpu_lib, x, w, b, act=None, launch="conv_simt")
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    ok = np.isfinite(want)
    # both are chains of roundings of 2^-24 (subnormal results: of 2^-149) relative to the largest terms
    assert np.abs(got[ok].astype(np.float64) - want[ok]).max() <= 2e-5 * np.abs(want[ok]).max() + 1e-43


@pytest.mark.parametrize("shape", [(2, 28, 64, 128, 3), (1, 14, 256, 320, 3)])   # boxes of results; a shared reduction
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 3.4e38, 1e-30, 1e-38, 1e-41])
def test_values_the_split_does_not_hold_next_to_their_terms(odla, gpu_lib, shape, bad, monkeypatch):
    """As above, every result next to the sum of its own terms' magnitudes."""
    N, H, C, K, R = shape
    rng = np.random.default_rng(5)
    x = rng.standard_normal((N, H, H, C)).astype(np.float32)
    w = (rng.standard_normal((R, R, C, K)) / np.sqrt(R * R * C)).astype(np.float32)
    b = np.zeros(K, np.float32)
    if abs(bad) < 1:
        x *= np.float32(bad)
    else:
        x[0, 3, 4, 5] = x[0, H - 1, 0, C - 1] = bad
    got = conv(odla, gpu_lib, x, w, b, act=None)
    monkeypatch.setenv("ODLA_B200_NO_F32_UMMA", "1")
    want = conv(odla, gpu_lib, x, w, b, act=None, launch="conv_simt")
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    ok = np.isfinite(want)
    # both are chains of roundings of 2^-24 of a result's own terms (of 2^-149 among subnormals)
    size = plain_size(np.where(np.isfinite(x), x, 0), w, 1)
    assert (np.abs(got[ok].astype(np.float64) - want[ok]) <= 2e-6 * size[ok] + 1e-43).all()


# N, H, C, K, window: boxes of results, two tiles a CTA and more, a shared reduction, columns that are no multiple of four (and shared)
@pytest.mark.parametrize("act, residual", [(None, False), (0.0, True), (0.1, True), ("gelu", False)])
@pytest.mark.parametrize("shape", [(6, 28, 64, 128, 3), (6, 56, 64, 320, 1), (6, 7, 256, 320, 3), (6, 14, 64, 255, 1), (6, 7, 512, 130, 1)])
def test_images_that_are_no_ordinary_numbers(odla, gpu_lib, monkeypatch, shape, act, residual):
    """A batch of an ordinary image, one of NaN, one of infinities, one with a single infinity and one with a single NaN, one of subnormals;
    a filter that is all zeros and one that has all but vanished.  Infinities and NaN as from the CUDA-core kernel, every other result
    next to the sum of its own terms' magnitudes."""
    N, H, C, K, R = shape
    rng = np.random.default_rng(sum(shape))
    x = rng.standard_normal((N, H, H, C)).astype(np.float32)
    w = (rng.standard_normal((R, R, C, K)) / np.sqrt(R * R * C)).astype(np.float32)
    w[..., 3] = 0
    w[..., 9] *= np.float32(1e-25)
    x[1] = np.nan
    x[2] = np.where(x[2] < 0, -np.inf, np.inf)
    x[3, 2, 3, 5] = -np.inf
    x[4, H - 1, 0, C - 1] = np.nan
    x[5] *= np.float32(1e-40)
    r = np.abs(rng.standard_normal((N, H, H, K))).astype(np.float32) if residual else None

    def layer(launch):
        if act != "gelu":
            return conv(odla, gpu_lib, x, w, np.zeros(K, np.float32), r, pad=R // 2, act=act, launch=launch)
        g = odla.Graph(gpu_lib, "c", n_gpus=1)
        y = g.Conv(g.Argument("x", x.shape), odla.CHANNELS_LAST, 1, g.Constant("w", w), odla.SIO, (1, 1), (1, 1), (R // 2, R // 2), (R // 2, R // 2), None, (N, H, H, K), "conv")
        g.Output(g.Gelu(y, False, "act"))
        try:
            out = g.run({"x": x})["act"]
            assert launch in g.describe()
        finally:
            g.close()
        return out

    got = layer("conv_f32_umma")
    monkeypatch.setenv("ODLA_B200_NO_F32_UMMA", "1")
    want = layer("conv_simt")
    for same in (np.isnan, np.isposinf, np.isneginf):
        assert np.array_equal(same(got), same(want))
    ok = np.isfinite(want)
    xf = np.where(np.isfinite(x), x, 0)
    # two fp32 chains: roundings of 2^-24 of the terms (of the residual too, of 2^-149 among subnormals), erf's 5e-7
    size = plain_size(xf, w, R // 2) + (0 if r is None else np.abs(r))
    assert (np.abs(got[ok].astype(np.float64) - want[ok]) <= 2e-6 * size[ok] + 1e-43).all()


def test_rows_computed_again_in_a_deep_product(odla, gpu_lib):
    """Several tiles a CTA over a long reduction, most rows of which are computed again while the other roles wait."""
    M, K, N = 40000, 2304, 64
    rng = np.random.default_rng(4)
    a = rng.standard_normal((M, K), dtype=np.float32)
    w = (rng.standard_normal((K, N)) / 48).astype(np.float32)
    a[:10000] *= np.float32(1e-40)
    a[10000:20000] = np.nan
    a[20000:30000, 7] = np.inf
    g = odla.Graph(gpu_lib, "g", n_gpus=1)
    g.Output(g.Gemm(g.Argument("a", a.shape), False, g.Constant("w", w), False, 1.0, 0.0, None, (M, N), "y"))
    got = g.run({"a": a})["y"]
    assert "gemm_f32_umma" in g.describe()
    g.close()
    assert np.isnan(got[10000:20000]).all()
    assert np.array_equal(got[20000:30000], np.broadcast_to(np.where(w[7] < 0, -np.inf, np.inf).astype(np.float32), (10000, N)))
    want = (torch.from_numpy(a).cuda().double() @ torch.from_numpy(w).cuda().double()).cpu().numpy()
    size = (torch.from_numpy(np.abs(a)).cuda().double() @ torch.from_numpy(np.abs(w)).cuda().double()).cpu().numpy()
    # a chain of 2304 roundings: of 2^-24 of the terms, of 2^-149 among subnormals
    for rows in (slice(0, 10000), slice(30000, M)):
        assert (np.abs(got[rows] - want[rows]) <= 1e-6 * size[rows] + K * 2.0 ** -149).all()


@pytest.mark.parametrize("gelu", [False, True])
@pytest.mark.parametrize("dims", [(6000, 256, 640), (1000, 768, 255), (130, 2048, 512), (130, 2048, 510)])   # boxes, rows, a shared reduction of either kind
def test_zeros_beside_tiny_results(odla, gpu_lib, dims, gelu):
    """One subnormal a row, so that every result is one product: where the parts' products all vanish, the product may not."""
    M, K, N = dims
    rng = np.random.default_rng(N)
    at = rng.integers(0, K, M)
    a = np.zeros((M, K), np.float32)
    a[np.arange(M), at] = rng.uniform(1, 2, M) * rng.choice([-1, 1], M) * 2.0 ** rng.integers(-136, -128, M)
    w = (rng.uniform(1, 2, (K, N)) * rng.choice([-1, 1], (K, N)) * 2.0 ** rng.integers(-20, 20, (K, N))).astype(np.float32)
    g = odla.Graph(gpu_lib, "g", n_gpus=1)
    y = g.Gemm(g.Argument("a", a.shape), False, g.Constant("w", w), False, 1.0, 0.0, None, (M, N), "y")
    g.Output(g.Gelu(y, False, "act") if gelu else y)
    got = next(iter(g.run({"a": a}).values()))
    assert "gemm_f32_umma" in g.describe()
    g.close()
    want = a[np.arange(M), at].astype(np.float64)[:, None] * w[at].astype(np.float64)
    want = np.where(gelu, 0.5, 1.0) * want
    assert (np.abs(got - want) <= 2.0 ** -24 * np.abs(want) + 2.0 ** -149).all()   # (a rounding; GELU halves them exactly, but for the last bit)


@pytest.mark.parametrize("scale, value, launch", [(2.0 ** -126, 0, "conv_simt"), (1e-40, 0, "conv_simt"), (1, 1e-36, "conv_simt"), (1, 1.5 * 2.0 ** 20, "conv_simt"),
                                                  (1, -2.0 ** 20, "conv_f32_umma"), (1, 1.2345678 * 2.0 ** -110, "conv_f32_umma"), (1, 2.0 ** -133, "conv_f32_umma"), (1, 2.0 ** -134, "conv_simt")])
def test_weights_the_split_does_not_hold(odla, gpu_lib, scale, value, launch):
    """Filters with values that are no sum of three bf16 values, or too large, stay with the CUDA-core kernel; either way the results
    are the products of the filter as given, also where large activations meet filters that are all tiny."""
    N, H, C, K, R = 2, 28, 64, 128, 3
    rng = np.random.default_rng(6)
    x = rng.standard_normal((N, H, H, C)).astype(np.float32)
    w = (rng.standard_normal((R, R, C, K)) / 24 * scale).astype(np.float32)
    if scale < 1:
        x *= np.float32(1e30)
    if value:
        w[1, 1, 7, 5] = value
    got = conv(odla, gpu_lib, x, w, np.zeros(K, np.float32), act=None, launch=launch)
    want = float64(x, w, 0, None, 1, 1, None)
    # a column against its own size (one holds the large weight); sums as in test_conv_matches_float64, on the CUDA cores a chain of all products
    err = np.abs(got - want).max(axis=(0, 1, 2)) / np.sqrt(np.mean(want ** 2, axis=(0, 1, 2)))
    assert err.max() < 4e-7 * (3 if launch == "conv_f32_umma" else 24) + 1e-6, err.max()


@pytest.mark.parametrize("dims", [(8192, 512, 640), (700, 128, 512), (130, 2048, 512), (1000, 768, 255)])   # boxes of 128 and 64 columns, a shared reduction, rows
def test_single_products(odla, gpu_lib, dims):
    """One value a row, so that every result is one product, for values whose parts are as large as they get and for subnormals."""
    M, K, N = dims
    rng = np.random.default_rng(M)
    at = rng.integers(0, K, M)
    value = (1 + rng.uniform(0, 1, M) ** 4) * rng.choice([-1, 1], M) * 2.0 ** rng.integers(-30, 30, M)
    value[7:71] *= 2.0 ** rng.integers(-136, -128, 64) / 2.0 ** np.floor(np.log2(np.abs(value[7:71])))
    a = np.zeros((M, K), np.float32)
    a[np.arange(M), at] = value
    w = ((1 + rng.uniform(0, 1, (K, N)) ** 4) * rng.choice([-1, 1], (K, N)) * 2.0 ** rng.integers(-20, 20, (K, N))).astype(np.float32)
    g = odla.Graph(gpu_lib, "g", n_gpus=1)
    g.Output(g.Gemm(g.Argument("a", a.shape), False, g.Constant("w", w), False, 1.0, 0.0, None, (M, N), "y"))
    got = g.run({"a": a})["y"]
    assert "gemm_f32_umma" in g.describe()
    g.close()
    want = a[np.arange(M), at].astype(np.float64)[:, None] * w[at].astype(np.float64)
    # in units of 2^-24 of the product: a rounding, a3 w2 of 2^-16 * 2^-8, a2 w3 of 2^-8 * 2^-17, five sums of at most 2^-7 cut off at their last bit
    assert (np.abs(got - want) <= 2.6 * 2.0 ** -24 * np.abs(want) + 2.0 ** -149).all(), (np.abs(got - want) / np.abs(want)).max() * 2.0 ** 24


@pytest.mark.parametrize("tb", [False, True])
@pytest.mark.parametrize("dims", [(2, 130, 768, 768), (1, 700, 100, 999)])   # batch, M, K, N
def test_products_match_float64(odla, gpu_lib, dims, tb):
    batch, M, K, N = dims
    rng = np.random.default_rng(M)
    lead = (batch,) if batch > 1 else ()
    a = rng.standard_normal(lead + (M, K)).astype(np.float32)
    w = (rng.standard_normal((N, K) if tb else (K, N)) / np.sqrt(K)).astype(np.float32)
    c = rng.standard_normal(N).astype(np.float32)
    g = odla.Graph(gpu_lib, "g", n_gpus=1)
    g.Output(g.Gelu(g.Gemm(g.Argument("a", a.shape), False, g.Constant("w", w), tb, 0.5, 2.0, g.Constant("c", c), lead + (M, N), "y"), False, "act"))
    got = next(iter(g.run({"a": a}).values()))
    assert "gemm_f32_umma" in g.describe()
    g.close()
    t = torch.from_numpy(0.5 * (a.astype(np.float64) @ (w.T if tb else w).astype(np.float64)) + 2.0 * c)
    want = torch.nn.functional.gelu(t).numpy()
    assert np.abs(got - want).max() / np.sqrt(np.mean(want ** 2)) < 4e-7 * np.sqrt(max(K / 64, 4)) + 1e-6


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("shape", [(8, 56, 64, 256, 1), (1, 7, 2048, 512, 1), (1, 14, 256, 320, 3), (3, 29, 100, 255, 1)])   # boxes, shared reductions, rows
def test_wait_that_runs_out(odla, gpu_lib, monkeypatch, shape, residual):
    """A stage that is never loaded: every role's bounded wait gives up after a short limit, the execute returns ODLA_TIMEOUT and the same
    layer planned without the hook is right."""
    N, H, C, K, R = shape
    rng = np.random.default_rng(3)
    x, w = rng.standard_normal((N, H, H, C)).astype(np.float32), (rng.standard_normal((R, R, C, K)) / np.sqrt(R * R * C)).astype(np.float32)
    b, r = rng.standard_normal(K).astype(np.float32), rng.standard_normal((N, H, H, K)).astype(np.float32) if residual else None
    monkeypatch.setenv("ODLA_B200_TEST_SPIN_LIMIT", "256")
    monkeypatch.setenv("ODLA_B200_TEST_SKIP_STAGE", "1")
    gpu_lib.SetLogLevel(0)
    try:
        with pytest.raises(RuntimeError, match="odla_status %d" % odla.TIMEOUT):
            conv(odla, gpu_lib, x, w, b, r, pad=R // 2)
    finally:
        gpu_lib.SetLogLevel(3)
    monkeypatch.delenv("ODLA_B200_TEST_SKIP_STAGE")
    monkeypatch.delenv("ODLA_B200_TEST_SPIN_LIMIT")
    got, want = conv(odla, gpu_lib, x, w, b, r, pad=R // 2), float64(x, w, b, r, 1, R // 2, 0.0)
    assert np.abs(got - want).max() / np.sqrt(np.mean(want ** 2)) < 4e-7 * 6 + 1e-6


def test_weights_without_memory_for_their_parts(odla, gpu_lib, monkeypatch):
    """Each allocation of a plan fails in turn (on the host, nothing touches the device): the one for the bf16 parts of the weights, half as
    much again as the weights, leaves the layer to the CUDA cores; the others are refused as before."""
    rng = np.random.default_rng(7)
    x, w = rng.standard_normal((2, 28, 28, 64)).astype(np.float32), (rng.standard_normal((3, 3, 64, 128)) / 24).astype(np.float32)
    b, launches = rng.standard_normal(128).astype(np.float32), []
    gpu_lib.SetLogLevel(0)
    try:
        for n in range(1, 9):
            monkeypatch.setenv("ODLA_B200_INJECT", "alloc@%d" % n)
            for launch in ("conv_f32_umma", "conv_simt", "refused"):
                monkeypatch.delenv("ODLA_B200_INJECT")
                conv(odla, gpu_lib, x, w, b)   # (forgets the count)
                monkeypatch.setenv("ODLA_B200_INJECT", "alloc@%d" % n)
                try:
                    got = conv(odla, gpu_lib, x, w, b, launch=launch)
                except AssertionError:
                    continue
                except RuntimeError:
                    launches.append("refused")
                    break
                launches.append(launch)
                want = float64(x, w, b, None, 1, 1, 0.0)
                assert np.abs(got - want).max() / np.sqrt(np.mean(want ** 2)) < 4e-7 * 24 + 1e-6
                break
    finally:
        gpu_lib.SetLogLevel(3)
    assert launches.count("conv_simt") == 1 and "refused" in launches and launches[-1] == "conv_f32_umma", launches


def test_refused_filters_leave_no_scratch_behind(odla, gpu_lib, monkeypatch):
    """Filters of an RGB image that stay with the CUDA cores, because the split does not hold them or because their parts find no memory: the
    plan holds no padded copy of the images (128 of 224 x 224: 420 MB)."""
    N, H, K = 128, 224, 64
    w = np.full((7, 7, 3, K), 1e-40, np.float32)

    def memory():
        g = odla.Graph(gpu_lib, "c", n_gpus=1)
        g.Output(g.Conv(g.Argument("x", (N, H, H, 3)), odla.CHANNELS_LAST, 1, g.Constant("w", w), odla.SIO, (2, 2), (1, 1), (3, 3), (3, 3), None, (N, 112, 112, K), "y"))
        before = torch.cuda.mem_get_info()[0]
        g.context()
        exe = C.c_void_p()
        done = gpu_lib.CompileComputation(g.comp, None, C.byref(exe)) == odla.SUCCESS
        taken = before - torch.cuda.mem_get_info()[0] if done and "conv_simt" in g.describe() else None
        g.close()
        return taken

    memory()   # (what the first plan of a process takes besides)
    refused = memory()
    w[:] = 1
    assert memory() is None   # on the tensor cores
    gpu_lib.SetLogLevel(0)
    failed = []
    for n in range(1, 9):
        monkeypatch.setenv("ODLA_B200_INJECT", "alloc@%d" % n)
        failed.append(memory())
        monkeypatch.delenv("ODLA_B200_INJECT")
        memory()   # (forgets the count)
    gpu_lib.SetLogLevel(3)
    failed = [taken for taken in failed if taken is not None]
    assert len(failed) == 2   # the padded images, the parts of the filter
    monkeypatch.setenv("ODLA_B200_NO_F32_UMMA", "1")
    want = memory()
    assert all(abs(taken - want) < 100e6 for taken in failed + [refused]), (failed, refused, want)
