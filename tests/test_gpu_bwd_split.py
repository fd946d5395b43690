"""K/V tiles of the backward hop shared by several CTAs: runs that cross head boundaries or do not divide evenly, the ordered
mode (bit-reproducible with any split), and what repeats without it.  Windows: test_gpu_bwd_windows.py."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,S,Hq,Hkv,D", [(1, 640, 8, 1, 128), (1, 520, 6, 2, 64), (2, 392, 3, 1, 256), (1, 1000, 1, 1, 96)])
def test_split_tiles(B, S, Hq, Hkv, D, causal, deterministic):
    from test_gpu_kernels import run_case

    kw = dict(seed=61, deterministic=deterministic)
    first = run_case(B, S, Hq, Hkv, D, 2, causal, **kw)
    if deterministic:
        again = run_case(B, S, Hq, Hkv, D, 2, causal, **kw)
        for a, b in zip(first, again):
            assert all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,S,H,D", [(1, 2048, 4, 128), (1, 4096, 1, 64), (2, 1024, 1, 256), (1, 640, 2, 96)])
def test_mha_dk_dv_repeat_outside_the_ordered_mode(B, S, H, D, causal):
    """Without head groups only dQ is added in a varying order: dK and dV keep their bits, however small the grid is."""
    import opt_ring_flash_attn_b200 as rfa

    g = torch.Generator(device="cuda")
    g.manual_seed(S + D)
    q, k, v, dout = (torch.randn(B, S, H, D, generator=g, device="cuda").bfloat16() for _ in range(4))
    leaves = [t.requires_grad_(True) for t in (q, k, v)]

    def grads():
        return torch.autograd.grad(rfa.ring_flash_attn(*leaves, causal=causal), leaves[1:], dout)

    first = grads()
    for _ in range(8):
        assert all(torch.equal(a, b) for a, b in zip(first, grads()))


def test_mha_dk_dv_repeat_with_previous_partial_sums():
    """The same where the epilogue adds to the partial sums of the previous rank."""
    from opt_ring_flash_attn_b200 import _native as n

    B, S, H, D = 1, 1024, 1, 128
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    q, k, v, dout = (torch.randn(B, S, H, D, generator=g, device="cuda").bfloat16() for _ in range(4))
    prev = torch.randn(2, B, S, H, D, generator=g, device="cuda")
    spad, scale = n.padded_seq(S), D ** -0.5
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, lse = torch.empty_like(q), torch.empty(B, H, spad, device="cuda")
    n.fwd_hop(q, k, v, None, None, None, out, lse, scale, True, True, False, status)
    delta, lse2 = torch.empty_like(lse), torch.empty_like(lse)
    acc = torch.empty(n.dq_acc_elems(B, S, H, D), device="cuda")
    n.bwd_prepare(out, dout, lse, delta, lse2, acc, status)
    runs = [torch.empty_like(prev) for _ in range(8)]
    for r in runs:
        n.bwd_hop(q, k, v, dout, lse2, delta, acc, prev, r, scale, True, False, status)
    n.check_status(status, "bwd_hop")
    assert all(torch.equal(runs[0], r) for r in runs[1:])
