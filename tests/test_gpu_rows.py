"""Row operations at the row lengths where their kernels change shape or have a remainder: argmax of rows shorter and longer
than a block's share, off the four-value loads, with equal maxima in different parts of the row; normalisation and the gated unit from rows of four values to rows longer
than a block holds in registers, also in place."""
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


def rms_bound(x, w, n):
    """The sum of n squares in any order carries at most n * 2^-24 of itself, half of that reaches 1/rms; three roundings
    more make the result."""
    y = x.astype(np.float64) / np.sqrt((x.astype(np.float64) ** 2).mean(axis=1, keepdims=True) + 1e-6) * w
    return y, np.abs(y) * (n / 2 + 4) * 2.0 ** -24 + 1e-30


@pytest.mark.parametrize("rows", [1, 3, 700])
@pytest.mark.parametrize("n", [4, 128, 132, 2048, 2052, 5120, 16384, 17408])
def test_rmsnorm_of_every_row_length(device, n, rows):
    s = S()
    rng = np.random.default_rng(n + rows)
    x, r = rng.standard_normal((rows, n)).astype(np.float32), rng.standard_normal((rows, n)).astype(np.float32)
    w = (1 + 0.1 * rng.standard_normal(n)).astype(np.float32)
    dw = dev_f32(w)
    want, off = rms_bound(x, w, n)
    apart, place = torch.zeros(rows, n, device="cuda"), dev_f32(x)
    s.rmsnorm(device, dev_f32(x), dw, 1e-6, rows, apart)
    s.rmsnorm(device, place, dw, 1e-6, rows, place)
    device.synchronize()
    assert np.all(np.abs(apart.cpu().numpy() - want) <= off) and torch.equal(apart, place)
    total = x + r  # one rounding, as the kernel's
    want, off = rms_bound(total, w, n)
    h, y = torch.zeros(rows, n, device="cuda"), torch.zeros(rows, n, device="cuda")
    s.add_rmsnorm(device, dev_f32(x), dev_f32(r), dw, 1e-6, rows, h, y)
    hx, yr = dev_f32(x), dev_f32(r)  # the sum into x, the result into r
    s.add_rmsnorm(device, hx, yr, dw, 1e-6, rows, hx, yr)
    device.synchronize()
    assert np.array_equal(h.cpu().numpy(), total) and np.all(np.abs(y.cpu().numpy() - want) <= off)
    assert torch.equal(h, hx) and torch.equal(y, yr)


@pytest.mark.parametrize("n", [1, 3, 4, 777, 1024, 40002])
def test_gated_unit_of_every_length(device, n):
    s = S()
    rng = np.random.default_rng(n)
    g, u = rng.standard_normal(n).astype(np.float32) * 4, rng.standard_normal(n).astype(np.float32)
    out, place = torch.zeros(n, device="cuda"), dev_f32(g)
    s.glu(device, dev_f32(g), dev_f32(u), out)
    s.glu(device, place, dev_f32(u), place)
    device.synchronize()
    want = g.astype(np.float64) / (1 + np.exp(-g.astype(np.float64))) * u
    assert np.all(np.abs(out.cpu().numpy() - want) <= 8 * 2.0 ** -24 * np.abs(want) + 1e-30) and torch.equal(out, place)
