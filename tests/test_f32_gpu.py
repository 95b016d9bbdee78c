"""The tiled fp32 kernel (kernels_f32.cu) against a float64 evaluation at the edges of its tiles, load widths and splits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def close(got, want, k):
    # a sum of k products in fp32: a few rounding steps of the result's magnitude
    err = np.abs(got.astype(np.float64) - want).max() / np.sqrt(np.mean(want ** 2))
    assert err < 4e-7 * np.sqrt(k) + 1e-6, err


# N, H, W, C, K, R, stride, pad: 3 channels and odd channels (4-byte loads), ragged pixel and channel tiles, reductions that
# leave a k-block nearly empty, few tiles over a long reduction (split over a cluster), one pixel
@pytest.mark.parametrize("shape", [(2, 17, 19, 3, 64, 7, 2, 3), (1, 9, 11, 36, 65, 3, 1, 1), (1, 7, 7, 512, 72, 3, 1, 1), (3, 13, 13, 64, 255, 1, 1, 0),
                                   (1, 8, 8, 64, 64, 1, 1, 0), (2, 8, 8, 5, 7, 2, 2, 0), (1, 1, 1, 4, 1, 1, 1, 0), (2, 28, 28, 128, 128, 3, 2, 1)])
def test_conv_f32_matches_float64(odla, gpu_lib, shape):
    N, H, W, C, K, R, stride, pad = shape
    P, Q = (H + 2 * pad - R) // stride + 1, (W + 2 * pad - R) // stride + 1
    rng = np.random.default_rng(sum(shape))
    x = rng.standard_normal((N, H, W, C)).astype(np.float32)
    w = (rng.standard_normal((R, R, C, K)) / np.sqrt(R * R * C)).astype(np.float32)
    b, r = rng.standard_normal((1, 1, 1, K)).astype(np.float32), rng.standard_normal((N, P, Q, K)).astype(np.float32)
    g = odla.Graph(gpu_lib, "c")
    xa, ra = g.Argument("x", x.shape), g.Argument("r", r.shape)
    y = g.Conv(xa, odla.CHANNELS_LAST, 1, g.Constant("w", w), odla.SIO, (stride, stride), (1, 1), (pad, pad), (pad, pad), None, (N, P, Q, K), "conv")
    g.Output(g.LeakyRelu(g.Add(g.Add(y, g.Constant("b", b), "bn"), ra, "res"), 0.1, "y"))
    got = g.run({"x": x, "r": r})["y"]
    g.close()
    t = torch.nn.functional.conv2d(torch.from_numpy(x).double().permute(0, 3, 1, 2), torch.from_numpy(w).double().permute(3, 2, 0, 1), stride=stride, padding=pad)
    want = t.permute(0, 2, 3, 1).numpy() + b + r
    close(got, np.where(want < 0, want * np.float64(np.float32(0.1)), want), R * R * C)


# batch, M, N, K, transposed A, transposed B (None: constant weights)
@pytest.mark.parametrize("dims", [(1, 64, 10, 784, 0, None), (1, 1, 1000, 2048, 0, None), (1, 65, 63, 33, 0, None), (1, 130, 70, 4, 1, None), (6, 77, 77, 64, 0, 1),
                                  (6, 77, 64, 77, 0, 0), (4, 128, 64, 128, 0, 0), (1, 3, 5, 7, 0, 0)])
def test_gemm_f32_matches_float64(odla, gpu_lib, dims):
    batch, M, N, K, ta, tb = dims
    rng = np.random.default_rng(sum(d or 0 for d in dims))
    lead = (batch,) if batch > 1 else ()
    a = rng.standard_normal(lead + ((K, M) if ta else (M, K))).astype(np.float32)
    b = rng.standard_normal(lead + ((N, K) if tb else (K, N))).astype(np.float32)
    c = rng.standard_normal(N).astype(np.float32)
    g = odla.Graph(gpu_lib, "g", n_gpus=1)
    ba = g.Constant("b", b) if tb is None else g.Argument("b", b.shape)
    aa = g.Argument("a", a.shape)
    g.Output(g.Gemm(aa, bool(ta), ba, bool(tb), 0.5, 2.0, g.Constant("c", c), lead + (M, N), "y"))
    got = g.run({"a": a, "b": b} if tb is not None else {"a": a})["y"]
    g.close()
    af, bf = a.astype(np.float64), b.astype(np.float64)
    close(got, 0.5 * ((af.swapaxes(-1, -2) if ta else af) @ (bf.swapaxes(-1, -2) if tb else bf)) + 2.0 * c, K)


def test_f32_results_do_not_depend_on_how_the_batch_is_cut(odla, gpu_lib):
    """A long convolution, a batched product and two classifiers whose shares of the reduction (and, for the last, whose
    kernel) would differ between six images and the one to five of a sub-batch: equal bits however the batch is cut."""
    B = 6
    rng = np.random.default_rng(8)
    n = lambda *s: (rng.standard_normal(s) / np.sqrt(np.prod(s[:-1]))).astype(np.float32)
    x = rng.standard_normal((B, 7, 7, 512)).astype(np.float32)
    wc, w1, w2 = n(3, 3, 512, 512), n(512, 3000), n(512, 40)
    outs = []
    for s in (1, 2, 3, 6):
        g = odla.Graph(gpu_lib, "cut", n_gpus=1, sub_batches=s)
        y = g.Conv(g.Argument("x", x.shape), odla.CHANNELS_LAST, 1, g.Constant("wc", wc), odla.SIO, (1, 1), (1, 1), (1, 1), (1, 1), None, x.shape, "conv")
        g.Output(y)
        t = g.Reshape(y, (B, 49, 512), "rows")
        g.Output(g.Gemm(t, False, t, True, 1.0, 0.0, None, (B, 49, 49), "gram"))
        v = g.Reshape(g.ReduceMean(y, (1, 2), True, (B, 1, 1, 512), "gap"), (B, 512), "flat")
        g.Output(g.Gemm(v, False, g.Constant("w1", w1), False, 1.0, 0.0, None, (B, 3000), "wide"))
        g.Output(g.Gemm(v, False, g.Constant("w2", w2), False, 1.0, 0.0, None, (B, 40), "narrow"))
        outs.append(g.run({"x": x}))
        assert g.describe().count("gpu ") == s
        g.close()
    for o in outs[1:]:
        for name in outs[0]:
            assert np.array_equal(o[name], outs[0][name]), name


@pytest.mark.parametrize("dims", [(0, 16, 8), (4, 16, 0), (0, 15, 8)])
def test_f32_product_without_results(odla, gpu_lib, dims):
    M, K, N = dims
    g = odla.Graph(gpu_lib, "none", n_gpus=1)
    g.Output(g.Gemm(g.Argument("a", (M, K)), False, g.Constant("w", np.ones((K, N), np.float32)), False, 1.0, 0.0, None, (M, N), "y"))
    assert g.run({"a": np.ones((M, K), np.float32)})["y"].shape == (M, N)
    g.close()


@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("pads", [((1, 1), (1, 1)), ((0, 0), (1, 1))])
def test_conv_f32_padding_meets_no_filter_value(odla, gpu_lib, bad, pads):
    """A filter with one infinite (or NaN) tap: pixels whose window has padding under that tap stay finite."""
    (pt, pl), (pb, pr) = pads
    H, C, K = 6, 8, 16
    P = H + pt + pb - 2
    x = np.random.default_rng(2).uniform(1, 2, (1, H, H, C)).astype(np.float32)
    w = np.full((3, 3, C, K), 0.125, np.float32)
    at = 0 if pt else 2
    w[at, at] = bad
    g = odla.Graph(gpu_lib, "c", n_gpus=1)
    g.Output(g.Conv(g.Argument("x", x.shape), odla.CHANNELS_LAST, 1, g.Constant("w", w), odla.SIO, (1, 1), (1, 1), (pt, pl), (pb, pr), None, (1, P, P, K), "y"))
    got = g.run({"x": x})["y"][0, :, :, 0]
    g.close()
    reached = np.zeros((P, P), bool)
    reached[slice(1, None) if pt else slice(None, -1), slice(1, None) if pl else slice(None, -1)] = True
    assert np.array_equal(np.isfinite(got), ~reached)
    s = np.pad(x.sum(-1)[0].astype(np.float64) * 0.125, ((pt, pb), (pl, pr)))
    want = sum(s[i:i + P, j:j + P] for i in range(3) for j in range(3))
    np.testing.assert_allclose(got[~reached], want[~reached], rtol=1e-5)


@pytest.mark.parametrize("N", [4096, 4095, 12])   # four results at a time, one at a time, a warp per 4 x 2 results
def test_f32_epilogue_rounds_every_step(odla, gpu_lib, N):
    """alpha, per-channel addend, LeakyReLU and residual on products with a single term: numpy's fp32 steps, bit for bit."""
    M, K = 8, 4
    rng = np.random.default_rng(N)
    a, w = np.zeros((M, K), np.float32), np.zeros((K, N), np.float32)
    a[:, 0], w[0] = rng.standard_normal(M), rng.standard_normal(N)
    b, r = rng.standard_normal((1, N)).astype(np.float32), rng.standard_normal((M, N)).astype(np.float32)
    alpha, slope = np.float32(0.3), np.float32(0.1)
    g = odla.Graph(gpu_lib, "r", n_gpus=1)
    aa, ra = g.Argument("a", a.shape), g.Argument("r", r.shape)
    y = g.Add(g.Gemm(aa, False, g.Constant("w", w), False, float(alpha), 0.0, None, (M, N), "gemm"), g.Constant("b", b), "bias")
    g.Output(g.Add(g.LeakyRelu(y, float(slope), "act"), ra, "y"))
    got = g.run({"a": a, "r": r})["y"]
    g.close()
    t = alpha * (a[:, :1] * w[:1]) + b
    assert np.array_equal(got, np.where(t < 0, slope * t, t) + r)


@pytest.mark.parametrize("images", [1, 4, 16])
@pytest.mark.parametrize("shape", [(9, 5, 4, 3), (9, 8, 255, 1), (14, 1, 64, 3), (20, 3, 1, 5), (28, 16, 16, 1)])   # H, C, K, window: either side of the choice
def test_short_reductions_on_whichever_kernel(odla, gpu_lib, shape, images):
    """fp32 layers at the line between the tiles and the one-thread-per-output kernel, cut in two as well."""
    H, C, K, R = shape
    rng = np.random.default_rng(H * C + K)
    x = rng.standard_normal((images, H, H, C)).astype(np.float32)
    w = (rng.standard_normal((R, R, C, K)) / np.sqrt(R * R * C)).astype(np.float32)
    outs = []
    for s in (1, 2):
        g = odla.Graph(gpu_lib, "c", n_gpus=1, sub_batches=s)
        p = R // 2
        y = g.Conv(g.Argument("x", x.shape), odla.CHANNELS_LAST, 1, g.Constant("w", w), odla.SIO, (1, 1), (1, 1), (p, p), (p, p), None, (images, H, H, K), "y")
        g.Output(y)
        rows = g.Reshape(g.ReduceMean(y, (1, 2), True, (images, 1, 1, K), "m"), (images, K), "rows")
        g.Output(g.Gemm(rows, False, g.Constant("v", w[0, 0].T.copy()), False, 1.0, 0.0, None, (images, C), "z"))
        outs.append(g.run({"x": x}))
        g.close()
    t = torch.nn.functional.conv2d(torch.from_numpy(x).double().permute(0, 3, 1, 2), torch.from_numpy(w).double().permute(3, 2, 0, 1), padding=p).permute(0, 2, 3, 1).numpy()
    close(outs[0]["y"], t, R * R * C)
    assert all(np.array_equal(outs[0][n], outs[1][n]) for n in outs[0])


@pytest.fixture
def cuda_cores(odla, monkeypatch):
    """Plans made by the test stay off the tensor cores (kernels_f32_umma.cu), which is looked up in their launches."""
    monkeypatch.setenv("ODLA_B200_NO_F32_UMMA", "1")
    launches, close = [], odla.Graph.close

    def closing(graph):
        launches.append(graph.describe())
        close(graph)

    monkeypatch.setattr(odla.Graph, "close", closing)
    yield
    assert launches and all("_simt" in text and "f32_umma" not in text for text in launches)


@pytest.mark.parametrize("shape", [(2, 17, 19, 3, 64, 7, 2, 3), (1, 9, 11, 36, 65, 3, 1, 1), (1, 7, 7, 512, 72, 3, 1, 1), (3, 13, 13, 64, 255, 1, 1, 0),
                                   (1, 8, 8, 64, 64, 1, 1, 0), (2, 28, 28, 128, 128, 3, 2, 1)])
def test_conv_f32_on_the_cuda_cores(odla, gpu_lib, cuda_cores, shape):
    test_conv_f32_matches_float64(odla, gpu_lib, shape)


@pytest.mark.parametrize("dims", [(1, 64, 10, 784, 0, None), (1, 1, 1000, 2048, 0, None), (1, 65, 63, 33, 0, None), (6, 77, 77, 64, 0, 1)])
def test_gemm_f32_on_the_cuda_cores(odla, gpu_lib, cuda_cores, dims):
    test_gemm_f32_matches_float64(odla, gpu_lib, dims)


def test_f32_results_on_the_cuda_cores_do_not_depend_on_the_cut(odla, gpu_lib, cuda_cores):
    test_f32_results_do_not_depend_on_how_the_batch_is_cut(odla, gpu_lib)
