"""Forward hop for head dims above 128: edges of the 128-key tiles, and the state carried from one block to the next."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# P and the result are rounded to bf16 once each (2^-9 of their value): rows stay within twice that of the fp32 result in
# the 2-norm, a few rows of small norm somewhat above
ROW_REL = 2 ** -7


def _reference(q, k, v, causal):
    B, S, Hq, D = q.shape
    g = Hq // k.shape[2]
    out, lse = torch.empty(B, S, Hq, D, device=q.device), torch.empty(B, Hq, S, device=q.device)
    for b in range(B):
        for h in range(Hq):
            s = q[b, :, h].float() @ k[b, :, h // g].float().T * D ** -0.5
            if causal:
                s = s.masked_fill(torch.ones_like(s, dtype=torch.bool).triu(1), float("-inf"))
            out[b, :, h], lse[b, h] = torch.softmax(s, -1) @ v[b, :, h // g].float(), torch.logsumexp(s, -1)
    return out, lse


@pytest.mark.parametrize("B,S,Hq,Hkv,D,causal", [
    (1, 1, 1, 1, 136, True), (1, 127, 2, 1, 256, True), (2, 128, 2, 2, 160, False), (1, 129, 2, 2, 256, False),
    (1, 257, 4, 2, 256, True), (1, 385, 2, 1, 192, False), (1, 1000, 2, 2, 256, True),
    (1, 4096, 16, 16, 256, False),  # all SMs busy: the last products are still running when the softmax has finished
])
def test_tiles_and_carried_state(B, S, Hq, Hkv, D, causal):
    from opt_ring_flash_attn_b200 import _native as n

    g = torch.Generator(device="cuda")
    g.manual_seed(S + D)
    q, k, v, k2, v2 = (torch.randn(B, S, H, D, generator=g, device="cuda").bfloat16() for H in (Hq, Hkv, Hkv, Hkv, Hkv))
    spad, scale = n.padded_seq(S), D ** -0.5
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, lse = torch.empty_like(q), torch.empty(B, Hq, spad, device="cuda")

    def check(ref):
        torch.cuda.synchronize()
        n.check_status(status, "fwd_hop")
        err = (out.float() - ref[0]).norm(dim=-1) / ref[0].norm(dim=-1)
        assert err.max().item() < ROW_REL and (lse[:, :, :S] - ref[1]).abs().max().item() < 1e-3

    n.fwd_hop(q, k, v, None, None, None, out, lse, scale, True, True, causal, status)
    check(_reference(q, k, v, causal))
    if not causal:
        acc = torch.empty(n.fwd_acc_elems(B, S, Hq, D), device="cuda")
        m, l = torch.empty_like(lse), torch.empty_like(lse)
        n.fwd_hop(q, k, v, acc, m, l, out, lse, scale, True, False, False, status)
        n.fwd_hop(q, k2, v2, acc, m, l, out, lse, scale, False, True, False, status)
        check(_reference(q, torch.cat([k, k2], 1), torch.cat([v, v2], 1), False))
