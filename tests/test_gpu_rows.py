"""Row operations at the row lengths where their kernels change shape or have a remainder: argmax of rows shorter and longer
than a block's share, off the four-value loads, with equal maxima in different parts of the row."""
import numpy as np
import pytest
import torch

from oracle import ref

pytestmark = pytest.mark.gpu


def S():
    from ferrum_b200 import surface
    return surface


def dev_f32(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


@pytest.mark.parametrize("rows", [1, 5])
@pytest.mark.parametrize("n", [1, 3, 4, 31, 32, 33, 512, 1000, 4096, 4097, 16384, 32001])
def test_argmax_of_every_row_length(device, n, rows):
    s = S()
    rng = np.random.default_rng(n)
    cases = [rng.standard_normal((rows, n)).astype(np.float32), np.zeros((rows, n), np.float32), np.full((rows, n), -np.inf, np.float32)]
    for top in range(3):  # equal maxima at random places of the row, the first and the last value among them
        x = -np.abs(rng.standard_normal((rows, n))).astype(np.float32)
        for r in range(rows):
            x[r, rng.integers(0, n, 3)] = 1.0
            x[r, (0, n - 1, n // 2)[top]] = 1.0
        cases.append(x)
    for x in cases:
        out = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
        s.argmax(device, dev_f32(x), n, rows, out)
        device.synchronize()
        assert np.array_equal(out.cpu().numpy().view(np.uint32), ref.argmax_first(x))
