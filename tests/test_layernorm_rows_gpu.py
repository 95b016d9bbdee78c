"""Layer normalisation of few rows (gamma and beta requested early) and of many: the same bits for the same row."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [8, 64, 128, 768, 1000, 1024])
@pytest.mark.parametrize("rows", [2369, 9475, 20001])
def test_many_rows_equal_few(odla, gpu_lib, dim, rows):
    rng = np.random.default_rng(dim + rows)
    few = rng.standard_normal((23, dim)).astype(np.float16)
    gamma, beta = rng.uniform(0.5, 1.5, dim).astype(np.float32), rng.standard_normal(dim).astype(np.float32)

    def run(x):
        g = odla.Graph(gpu_lib, "ln", fp16=True, n_gpus=1)
        g.Output(g.LayerNorm(g.Argument("x", x.shape, odla.FLOAT16), (-1,), 1e-5, g.Constant("g", gamma), g.Constant("b", beta), "ln"))
        y = g.run({"x": x})["ln"]
        g.close()
        return y

    want = run(few)
    x64 = few.astype(np.float64)
    exact = (x64 - x64.mean(1, keepdims=True)) / np.sqrt(x64.var(1, keepdims=True) + 1e-5) * gamma + beta
    np.testing.assert_allclose(want.astype(np.float64), exact, rtol=2.0 ** -10, atol=4e-3)
    got = run(few[np.arange(rows) % 23])
    np.testing.assert_array_equal(got, want[np.arange(rows) % 23])


@pytest.mark.parametrize("dim", [776, 1032, 2048])
@pytest.mark.parametrize("rows", [5, 1777, 2500])
def test_wide_rows_and_their_int8_copy(odla, gpu_lib, dim, rows):
    """Rows of 1024 values and more, for which a launch has fewer blocks and no early form, on either side of all rows under way."""
    rng = np.random.default_rng(dim)
    x = rng.standard_normal((rows, dim)).astype(np.float16)
    gamma, beta = rng.uniform(0.5, 1.5, dim).astype(np.float32), rng.standard_normal(dim).astype(np.float32)
    g = odla.Graph(gpu_lib, "ln", fp16=True, n_gpus=1)
    y = g.LayerNorm(g.Argument("x", x.shape, odla.FLOAT16), (-1,), 1e-5, g.Constant("g", gamma), g.Constant("b", beta), "ln")
    scale = np.float32(0.0625)
    g.Output(g.Quantize(y, g.Constant("s", np.array([scale])), None, 0, odla.INT8, "q"))
    g.Output(y)
    out = g.run({"x": x})
    g.close()
    x64 = x.astype(np.float64)
    exact = (x64 - x64.mean(1, keepdims=True)) / np.sqrt(x64.var(1, keepdims=True) + 1e-5) * gamma + beta
    np.testing.assert_allclose(out["ln"].astype(np.float64), exact, rtol=2.0 ** -10, atol=4e-3)
    np.testing.assert_array_equal(out["q"], np.clip(np.rint(out["ln"].astype(np.float32) / scale), -128, 127).astype(np.int8))
