"""The two orders in which the epilogue's groups of warps fill the boxes of the staging ring."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("M,K,N", [
    (40000, 64, 256),    # a ring of two tiles' boxes
    (40000, 128, 512),   # five boxes for tiles of four: with a residual, box after box
    (40000, 192, 256),
    (12500, 256, 1024),  # a ring of exactly one tile
    (20000, 64, 128),
    (9000, 64, 64),
    (20000, 64, 384),    # tiles that lack whole boxes
    (20000, 128, 520),
    (3000, 320, 2304),
])
def test_runs_and_boxes_in_turn_agree_to_the_bit(odla, gpu_lib, monkeypatch, M, K, N, residual):
    """Only the order differs, not one operation on a value; every execute is repeated, since the orders differ in what waits for what."""
    rng = np.random.default_rng(M + N)
    a = rng.standard_normal((M, K)).astype(np.float16)
    r = rng.standard_normal((M, N)).astype(np.float16)
    w, b = (rng.standard_normal((K, N)) / np.sqrt(K)).astype(np.float32), rng.standard_normal(N).astype(np.float32)

    def run():
        g = odla.Graph(gpu_lib, "m", fp16=True, n_gpus=1)
        feeds = {"a": a}
        xr = g.Argument("r", (M, N), odla.FLOAT16) if residual else None
        y = g.Gemm(g.Argument("a", (M, K), odla.FLOAT16), False, g.Constant("w", w), False, 1, 1, g.Constant("b", b), (M, N), "y")
        if residual:
            feeds["r"] = r
            y = g.Add(y, xr, "s")
        g.Output(g.Relu(y, "act"))
        outs = [next(iter(g.run(feeds).values())).copy() for _ in range(3)]
        assert "gemm_umma    act" in g.describe() and "binary" not in g.describe()
        g.close()
        return outs

    outs = run()
    monkeypatch.setenv("ODLA_B200_EPI_INTERLEAVE", "1")
    want = run()[0]
    for got in outs:
        assert np.array_equal(got, want)
    rows = rng.integers(0, M, 50)
    t = a[rows].astype(np.float64) @ w.astype(np.float16).astype(np.float64) + b + (r[rows].astype(np.float64) if residual else 0)
    # fp32 sums of K products and one rounding to fp16 of values below 16
    assert np.abs(want[rows].astype(np.float64) - np.maximum(t, 0)).max() <= 1.01 * 2.0 ** -8
