"""Projections of one to sixteen activation rows at the widths where the kernel that serves them changes: rows packed
into the columns of one MMA tile (two-plane formats up to four, four-plane IQ4 up to two) or of two (IQ4 up to four), one
tile of eight, two tiles; with row counts off the 16-row tile, one superblock and several K slices, and with the row's
norm and the gated unit folded into the activation preparation."""
import numpy as np
import pytest
import torch

from oracle import ref

pytestmark = pytest.mark.gpu

FORMATS = [ref.Q4_K, ref.Q5_K, ref.Q6_K, ref.IQ4_NL, ref.IQ4_XS]


def S():
    from ferrum_b200 import surface
    return surface


def dev_f32(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


def bound(fmt, dense, x):
    """Largest error of each output: activations rounded to 16 (IQ4: 31) bits of their superblock's maximum -- the
    integer grid's step is at most 2^-14 (2^-30) of it, half of that a value -- plus fp32 arithmetic on the products."""
    bits = 30 if fmt in (ref.IQ4_NL, ref.IQ4_XS) else 14
    top = np.abs(x).reshape(x.shape[0], -1, 256).max(axis=2)  # per row and superblock
    weight = np.abs(dense).reshape(dense.shape[0], -1, 256).sum(axis=2)
    return 0.5 * 2.0 ** -bits * (top @ weight.T) + 2e-6 * (np.abs(x) @ np.abs(dense).T)


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("rows,cols", [(37, 256), (250, 2304)])
def test_every_width_against_the_oracle(device, fmt, m, rows, cols):
    s = S()
    packed = ref.random_matrix(fmt, rows, cols, seed=rows + m)
    dense = ref.dequant(fmt, packed).reshape(rows, cols).astype(np.float64)
    x = np.random.default_rng(m).standard_normal((m, cols)).astype(np.float32)
    w = s.Matrix.from_packed(device, rows, cols, 1, fmt, packed)
    y = torch.full((m, rows), float("nan"), device="cuda")
    s.project(device, w, dev_f32(x), m, y)
    device.synchronize()
    off = np.abs(y.cpu().numpy() - x.astype(np.float64) @ dense.T)
    assert np.all(off <= bound(fmt, dense, x.astype(np.float64)))


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("m", [1, 2, 4])
def test_gated_unit_of_few_rows(device, fmt, m):
    """`dense_ffn`: the down projection's blocks compute silu(g) * u for themselves."""
    s = S()
    hidden, ffn = 512, 768
    g, u, d = (ref.random_matrix(fmt, r, c, seed=50 + i) for i, (r, c) in enumerate([(ffn, hidden), (ffn, hidden), (hidden, ffn)]))
    ws = [s.Matrix.from_packed(device, r, c, 1, fmt, p) for p, r, c in ((g, ffn, hidden), (u, ffn, hidden), (d, hidden, ffn))]
    x = (np.random.default_rng(m).standard_normal((m, hidden)) * 0.05).astype(np.float32)
    out = torch.zeros(m, hidden, device="cuda")
    s.dense_ffn(device, *ws, dev_f32(x), m, torch.zeros(3 * m * ffn, device="cuda"), out)
    device.synchronize()
    act = ref.swiglu(ref.matmul(fmt, g, ffn, hidden, x, m), ref.matmul(fmt, u, ffn, hidden, x, m))
    assert ref.rel_err(out.cpu().numpy(), ref.matmul(fmt, d, hidden, ffn, act, m)) <= 1e-3  # the op's contract


def folded(device, fmt, m, rows, cols):
    s = S()
    w = s.Matrix.from_packed(device, rows, cols, 1, fmt, ref.random_matrix(fmt, rows, cols, seed=rows + cols))
    rng = np.random.default_rng(m + cols)
    x, weight = dev_f32(rng.standard_normal((m, cols))), dev_f32(1 + 0.1 * rng.standard_normal(cols))
    normed, apart, fold = torch.zeros(m, cols, device="cuda"), torch.zeros(m, rows, device="cuda"), torch.zeros(m, rows, device="cuda")
    s.rmsnorm(device, x, weight, 1e-6, m, normed)
    s.project(device, w, normed, m, apart)
    s.rmsnorm_project_many(device, [w], x, weight, 1e-6, m, [fold], torch.zeros(m, cols, device="cuda"))
    device.synchronize()
    return fold, apart


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 16])
@pytest.mark.parametrize("rows,cols", [(37, 256), (250, 2304), (40, 17408)])
def test_norm_folded_into_the_preparation(device, fmt, m, rows, cols):
    """The same bits as the norm by itself and then the projection, whoever computes the row's sum."""
    fold, apart = folded(device, fmt, m, rows, cols)
    assert torch.equal(fold, apart) and bool(torch.isfinite(fold).all())


@pytest.mark.parametrize("fmt", [ref.Q4_K, ref.Q6_K])
@pytest.mark.parametrize("m", [2, 4])
def test_norm_of_a_slice_too_long_for_the_block_to_prepare(device, fmt, m):
    """Enough weight rows that K is not cut: twenty superblocks a row, prepared by a launch of their own."""
    fold, apart = folded(device, fmt, m, 16400, 5120)
    assert torch.equal(fold, apart) and bool(torch.isfinite(fold).all())
