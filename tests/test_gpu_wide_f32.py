"""F32 projections of prompt width (bf16 tensor cores, both operands in two terms): one k-block and fewer k-blocks than
stages, row and token counts off the tiles, matrices that share a launch, and an input so wide that its split copy is
served in slices of activation rows."""
import numpy as np
import pytest
import torch

from oracle import ref

pytestmark = pytest.mark.gpu


def S():
    from ferrum_b200 import surface
    return surface


def within(got, x, dense):
    """A product misses the term lo x lo and the roundings of both lo terms, each at most 2^-18 of it; the sums over
    3 cols / 16 steps of the tensor core round by at most 2^-23 a step."""
    x, dense = x.astype(np.float64), dense.astype(np.float64)
    steps = 3 * x.shape[1] / 16
    return np.all(np.abs(got - x @ dense.T) <= (3 * 2.0 ** -18 + steps * 2.0 ** -23) * (np.abs(x) @ np.abs(dense).T))


@pytest.mark.parametrize("fmt,cols", [(ref.Q8_0, 64), (ref.Q8_0, 320), (ref.Q4_K, 256), (ref.Q5_K, 768), (ref.Q6_K, 512)])
@pytest.mark.parametrize("m", [17, 129, 384, 513])
def test_against_the_oracle(device, fmt, cols, m):
    s = S()
    shapes = (131, 260)
    packed = [ref.random_matrix(fmt, r, cols, seed=r + m) for r in shapes]
    ws = [s.Matrix.from_packed(device, r, cols, 1, fmt, p) for r, p in zip(shapes, packed)]
    x = np.random.default_rng(m).standard_normal((m, cols)).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    alone = [torch.full((m, r), float("nan"), device="cuda") for r in shapes]
    many = [torch.full((m, r), float("nan"), device="cuda") for r in shapes]
    for w, y in zip(ws, alone):
        s.project(device, w, xd, m, y)
    s.project_many(device, ws, xd, m, many)
    device.synchronize()
    for r, p, a, b in zip(shapes, packed, alone, many):
        dense = ref.dequant(fmt, p).reshape(r, cols)
        assert within(a.cpu().numpy(), x, dense)
        assert within(b.cpu().numpy(), x, dense)


def test_input_wider_than_the_scratch(device):
    s = S()
    rows, cols, m = 130, 17408, 800  # two terms of two bytes: 55.7 MB against a scratch half of 48 MiB
    packed = ref.random_matrix(ref.Q6_K, rows, cols, seed=5)
    x = np.random.default_rng(6).standard_normal((m, cols)).astype(np.float32)
    w = s.Matrix.from_packed(device, rows, cols, 1, ref.Q6_K, packed)
    y = torch.full((m, rows), float("nan"), device="cuda")
    s.project(device, w, torch.from_numpy(x).cuda(), m, y)
    device.synchronize()
    assert within(y.cpu().numpy(), x, ref.dequant(ref.Q6_K, packed).reshape(rows, cols))
