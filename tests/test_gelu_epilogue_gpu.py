"""GELU in the tensor-core Gemm's two-byte epilogue: the whole range of its argument, and what is not finite."""
import numpy as np
import pytest
from scipy.special import ndtr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp16", "bf16"])
def test_gelu_epilogue_over_its_range(odla, gpu_lib, mode):
    """The addend carries the argument (the products are zero), so it reaches the function with all its fp32 bits.  Bound: the
    function's stated 5e-7 for |x| <= 12 (a few fp32 steps beyond, where the result is x or 0) and half a step of the stored type."""
    M, K, N = 300, 64, 3072
    x = np.linspace(-9, 9, N).astype(np.float32)
    x[:8] = [np.inf, -np.inf, np.nan, 0.0, 3e4, -3e4, 1e-30, -100.0]
    x[8:520] = np.random.default_rng(1).standard_normal(512)
    g = odla.Graph(gpu_lib, "m", fp16=mode == "fp16", bf16=mode == "bf16", n_gpus=1)
    y = g.Gemm(g.Argument("a", (M, K)), False, g.Constant("w", np.zeros((K, N), np.float32)), False, 1, 1, g.Constant("b", x), (M, N), "y")
    g.Output(g.Gelu(y, False, "act"))
    got = g.run({"a": np.ones((M, K), np.float32)})["act"]
    assert "gemm_umma" in g.describe()
    g.close()
    assert (got[1:].view(np.uint32) == got[0].view(np.uint32)).all()
    got = got[0].astype(np.float64)
    assert got[0] == np.inf and np.isnan(got[1]) and np.isnan(got[2]) and got[3] == 0
    x64 = x[3:].astype(np.float64)
    want = x64 * ndtr(x64)
    half = np.maximum(np.abs(want) * (2.0 ** -11 if mode == "fp16" else 2.0 ** -8), 2.0 ** -25 if mode == "fp16" else 0)
    assert (np.abs(got[3:] - want) <= 5e-7 + 1.01 * half + np.abs(x64) * 2.0 ** -23 * (np.abs(x64) > 12)).all()
