"""The global average pool's divisions (Markstein's correction instead of a division) at their edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["f16", "f32"])
def test_global_average_pool_divides_exactly(odla, gpu_lib, kind):
    """Sums over 7 x 7 positions and their quotients as fp32 gives them one after the other: ordinary values, zeros, infinities, NaN, and
    magnitudes at which the quotient's remainder would under- or overflow."""
    dt = np.float16 if kind == "f16" else np.float32
    rng = np.random.default_rng(3)
    C = 1024
    x = rng.standard_normal((5, 7, 7, C)).astype(dt)
    x[1] = np.maximum(x[1], 0)
    x[2, :, :, :256] = 0
    x[2, 3, 3, 256], x[2, 3, 3, 257], x[2, 1, 1, 258] = np.inf, np.nan, -np.inf
    if kind == "f32":
        x[3] *= np.float32(1e-38)
        x[4] *= np.float32(3e37)
    else:
        x[3] *= np.float16(6e-8)
        x[4] *= np.float16(1e4)
    g = odla.Graph(gpu_lib, "m", fp16=kind == "f16", n_gpus=1)
    g.Output(g.ReduceMean(g.Argument("x", x.shape, odla.FLOAT16 if kind == "f16" else odla.FLOAT32), (1, 2), True, (5, 1, 1, C), "y"))
    got = next(iter(g.run({"x": x}).values()))
    g.close()
    f = x.astype(np.float32)
    with np.errstate(all="ignore"):
        u = None
        for w in range(7):
            s = f[:, 0, w].copy()
            for h in range(1, 7):
                s = s + f[:, h, w]
            m = s / np.float32(7)
            u = m if u is None else u + m
        want = (u / np.float32(7)).astype(dt)
    np.testing.assert_array_equal(got[:, 0, 0], want)
