"""The backward hop's own addition of previous partial sums (``accumulate_prev``): out = prev + block, in place and into
another buffer, where the epilogue stores the sum itself (tiles of one CTA) and where several CTAs add to a copy of prev."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _hop(B, S, Hq, Hkv, D, causal, seed):
    """Inputs of a hop of a shard on itself, with the statistics of its forward."""
    from opt_ring_flash_attn_b200 import _native as n

    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    q, k, v, dout = (torch.randn(B, S, H, D, generator=g, device="cuda").bfloat16() for H in (Hq, Hkv, Hkv, Hq))
    prev = torch.randn(2, B, S, Hkv, D, generator=g, device="cuda")
    spad, scale = n.padded_seq(S), D ** -0.5
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, lse = torch.empty_like(q), torch.empty(B, Hq, spad, device="cuda")
    n.fwd_hop(q, k, v, None, None, None, out, lse, scale, True, True, causal, status)
    delta, lse2 = torch.empty_like(lse), torch.empty_like(lse)
    acc = torch.empty(n.dq_acc_elems(B, S, Hq, D), device="cuda")
    n.bwd_prepare(out, dout, lse, delta, lse2, acc, status)

    def run(prev_in, into, **kw):
        n.bwd_hop(q, k, v, dout, lse2, delta, acc, prev_in, into, scale, prev_in is not None, causal, status, **kw)
        n.check_status(status, "bwd_hop")
        return into

    return run, prev


@pytest.mark.parametrize("in_place", [True, False])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,S,Hq,Hkv,D", [
    # stored by the epilogue: fewer than four query tiles per K/V tile are never shared out, and without head groups
    # nothing is where previous sums are added
    (1, 256, 1, 1, 128), (2, 200, 2, 2, 64), (1, 384, 1, 1, 96), (1, 130, 1, 1, 256), (1, 128, 2, 1, 128), (1, 1024, 2, 2, 128),
    # added by several CTAs: 12 query tiles of a group (of 64 rows at head dim 256) on a few K/V tiles
    (1, 384, 4, 1, 128), (1, 320, 4, 2, 64), (1, 200, 6, 2, 256),
])
def test_epilogue_adds_to_the_previous_sums(B, S, Hq, Hkv, D, causal, in_place):
    run, prev = _hop(B, S, Hq, Hkv, D, causal, seed=S + D)
    block = run(None, torch.full_like(prev, float("nan")))
    given = prev.clone()
    got = run(given, given if in_place else torch.full_like(prev, float("nan")))
    if not in_place:
        assert torch.equal(given, prev)
    # sums of up to 17 fp32 terms in another order: each addition rounds by 2^-24 of a running sum of about this size
    want = prev + block
    assert ((got - want).norm() / want.norm()).item() < 2 ** -19
    assert (got - want).abs().max().item() < 2 ** -16 * want.abs().max().item()
