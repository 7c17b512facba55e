"""The one-launch MoE block of a single token against the kernels the block is otherwise made of (`moe_ffn_ep` on a
communicator of one rank): the same bits, over shapes where its work is dealt out differently -- one and several
superblocks per row, fewer and more tiles than SMs, every format pair it serves, a gate on the shared expert, sigmoid
scores -- and what a router that yields no ranking leaves behind."""
import numpy as np
import pytest
import torch

from oracle import ref

pytestmark = pytest.mark.gpu


def S():
    from ferrum_b200 import surface
    return surface


def block(s, device, gu, dn, experts, used, hidden, ffn, shared, gate, sigmoid, seed=0):
    M = lambda fmt, rows, cols, e, i: s.Matrix.from_packed(device, rows, cols, e, fmt, ref.random_matrix(fmt, rows * e, cols, seed + i))
    w = torch.from_numpy((np.random.default_rng(seed).standard_normal(hidden) * 0.05).astype(np.float32)).cuda() if gate else None
    return s.MoeFfn(M(ref.Q8_0, experts, hidden, 1, 1), M(gu, ffn, hidden, experts, 2), M(gu, ffn, hidden, experts, 3), M(dn, hidden, ffn, experts, 4),
                    M(gu, shared, hidden, 1, 5), M(gu, shared, hidden, 1, 6), M(dn, hidden, shared, 1, 7), w, experts, used, hidden, ffn, shared,
                    sigmoid, True)


@pytest.mark.parametrize("gu,dn", [(ref.Q4_K, ref.Q6_K), (ref.Q4_K, ref.Q4_K), (ref.Q5_K, ref.Q6_K), (ref.Q5_K, ref.Q5_K), (ref.Q6_K, ref.Q6_K)])
@pytest.mark.parametrize("experts,used,hidden,ffn,shared,gate,sigmoid", [
    (16, 4, 512, 256, 256, False, False), (256, 8, 2048, 512, 512, True, False), (40, 12, 768, 768, 1024, True, True), (300, 1, 2560, 1280, 256, False, True)])
def test_same_bits_as_the_chain_of_kernels(device, gu, dn, experts, used, hidden, ffn, shared, gate, sigmoid):
    s = S()
    f = block(s, device, gu, dn, experts, used, hidden, ffn, shared, gate, sigmoid)
    n = s.moe_ffn_scratch_elems(device, f, 1)
    comm = s.Comm(device, 0, 1, 4096 + used * hidden * 4)
    for seed in range(3):
        x = torch.from_numpy((np.random.default_rng(seed).standard_normal(hidden) * 0.12).astype(np.float32)).cuda()
        one, chain = torch.zeros(hidden, device="cuda"), torch.zeros(hidden, device="cuda")
        s.moe_ffn(device, f, x, 1, torch.zeros(n, device="cuda"), one)
        s.moe_ffn_ep(device, comm, 4096, f, 0, x, 1, torch.zeros(n, device="cuda"), chain)
        device.synchronize()
        assert torch.equal(one, chain) and bool(torch.isfinite(one).all())
    comm.close()


def test_router_without_a_ranking_is_reported(device):
    s = S()
    f = block(s, device, ref.Q4_K, ref.Q6_K, 16, 4, 512, 256, 256, False, False)
    x = torch.ones(512, device="cuda")
    x[3] = float("inf")
    n = s.moe_ffn_scratch_elems(device, f, 1)
    out = torch.zeros(512, device="cuda")
    s.moe_ffn(device, f, x, 1, torch.zeros(n, device="cuda"), out)
    with pytest.raises(s.WeightError):
        device.synchronize()
    device.recover()
    x[3] = 1.0
    s.moe_ffn(device, f, x, 1, torch.zeros(n, device="cuda"), out)
    device.synchronize()
    assert bool(torch.isfinite(out).all())


@pytest.mark.parametrize("m", [1, 2, 21])
@pytest.mark.parametrize("which", ["router", "gate_exps", "up_exps", "down_exps", "shared_gate", "shared_up", "shared_down"])
def test_matrix_of_another_handle_is_refused(device, which, m):
    s = S()
    other = s.Device(0)
    f = block(s, device, ref.Q4_K, ref.Q6_K, 16, 4, 512, 256, 256, False, False)
    g = block(s, other, ref.Q4_K, ref.Q6_K, 16, 4, 512, 256, 256, False, False)
    scratch = torch.zeros(s.moe_ffn_scratch_elems(device, f, m), device="cuda")
    setattr(f, which, getattr(g, which))
    before = device.counters().dispatches
    with pytest.raises(s.DeviceMismatch):
        s.moe_ffn(device, f, torch.zeros(m * 512, device="cuda"), m, scratch, torch.zeros(m * 512, device="cuda"))
    assert device.counters().dispatches == before  # nothing was enqueued


@pytest.mark.parametrize("inside", ["x", "out", "x and out"])
def test_operands_inside_the_scratch(device, inside):
    """One token with x or the output in a part of the scratch that the block does not use at this width (the gathered
    rows, which lie before four index arrays at its end): taken, and the same bits as with buffers of their own."""
    s = S()
    experts, used, hidden = 16, 4, 512
    f = block(s, device, ref.Q4_K, ref.Q6_K, experts, used, hidden, 256, 256, True, False)
    n = s.moe_ffn_scratch_elems(device, f, 1)
    x = torch.from_numpy((np.random.default_rng(5).standard_normal(hidden) * 0.12).astype(np.float32)).cuda()
    want, out = torch.zeros(hidden, device="cuda"), torch.zeros(hidden, device="cuda")
    s.moe_ffn(device, f, x, 1, torch.zeros(n, device="cuda"), want)
    scratch = torch.zeros(n, device="cuda")
    at = n - (3 * used + (experts + 1 + 3) // 4 * 4) - used * hidden
    if "x" in inside:
        scratch[at:at + hidden] = x
        x = scratch[at:at + hidden]
    if "out" in inside:
        out = scratch[at + hidden:at + 2 * hidden]
    s.moe_ffn(device, f, x, 1, scratch, out)
    device.synchronize()
    assert torch.equal(out, want) and bool(want.abs().max() > 0)


def test_wait_for_the_other_blocks_is_bounded(device):
    """A barrier that nobody completes gives up after its time, the kernel ends and reports it, and the next block runs."""
    s = S()
    f = block(s, device, ref.Q4_K, ref.Q6_K, 16, 4, 512, 256, 256, False, False)
    x = torch.from_numpy((np.random.default_rng(2).standard_normal(512) * 0.12).astype(np.float32)).cuda()
    scratch = torch.zeros(s.moe_ffn_scratch_elems(device, f, 1), device="cuda")
    want, out = torch.zeros(512, device="cuda"), torch.zeros(512, device="cuda")
    s.moe_ffn(device, f, x, 1, scratch, want)
    device.synchronize()
    device.moe_wait_runs_out()
    s.moe_ffn(device, f, x, 1, scratch, out)
    with pytest.raises(s.TimeoutError_):
        device.synchronize()
    device.recover()
    out.zero_()
    s.moe_ffn(device, f, x, 1, scratch, out)
    device.synchronize()
    assert torch.equal(out, want)
