"""Two-byte results of padded rows to dense fp32 outputs (convolutions whose channel count is no multiple of eight): every row
form of the conversion, against the same values computed with fp32 arithmetic on the rounded result."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [10, 31, 33, 100, 124, 132, 255, 257, 300])
@pytest.mark.parametrize("rows", [1, 77, 4097])
def test_padded_rows_leave_dense(odla, gpu_lib, K, rows):
    rng = np.random.default_rng(K * rows)
    x = rng.integers(-4, 5, (1, 1, rows, 16)).astype(np.float32)   # small integers: every sum is exact in fp16
    w = rng.integers(-4, 5, (1, 1, 16, K)).astype(np.float32)
    g = odla.Graph(gpu_lib, "rows", fp16=True, n_gpus=1)
    y = g.Conv(g.Argument("x", x.shape, odla.FLOAT32), odla.CHANNELS_LAST, 1, g.Constant("w", w), odla.SIO, (1, 1), (1, 1), (0, 0), (0, 0), None, (1, 1, rows, K), "y")
    g.Output(y)
    got = g.run({"x": x})["y"]
    g.close()
    np.testing.assert_array_equal(got.reshape(rows, K), torch.from_numpy(x.reshape(rows, 16)).matmul(torch.from_numpy(w.reshape(16, K))).numpy())
