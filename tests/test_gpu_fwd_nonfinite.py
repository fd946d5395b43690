"""A key with a NaN or an infinity makes every row that sees it NaN, wherever it stands in its tile (the exponentials of a
row take two routes, and only one of them passes a NaN on); rows that do not see it stay as they are."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("tile", [0, 1])  # the first tile sets the row maximum, later ones compare with it
def test_every_key_position(D, value, tile):
    from opt_ring_flash_attn_b200 import _native as n

    H, S = 128, 300
    g = torch.Generator(device="cuda")
    g.manual_seed(D)
    q, k, v = (torch.randn(1, S, H, D, generator=g, device="cuda").bfloat16() for _ in range(3))
    q = q.abs() + 0.1  # an infinite key then scores +inf
    clean, h, pos = k.clone(), torch.arange(H), tile * 128 + torch.arange(H)  # head h: key pos[h]
    k[0, pos, h] = value
    spad, scale = n.padded_seq(S), D ** -0.5
    status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def forward(keys, causal, state=None, first=True, last=True):
        out, lse = torch.zeros_like(q), torch.zeros(1, H, spad, device="cuda")
        n.fwd_hop(q, keys, v, *(state or (None, None, None)), out, lse, scale, first, last, causal, status)
        return out, lse[:, :, :S]

    out, lse = forward(k, False)
    assert out.isnan().all() and lse.isnan().all()
    out, lse = forward(k, True)
    ref, ref_lse = forward(clean, True)
    sees = torch.arange(S, device="cuda")[:, None] >= pos.cuda()[None]  # [S, H]
    assert out[0][sees].isnan().all() and lse[0].T[sees].isnan().all()
    assert torch.equal(out[0][~sees], ref[0][~sees]) and torch.equal(lse[0].T[~sees], ref_lse[0].T[~sees])
    # carried from hop to hop, in either order
    state = (torch.empty(n.fwd_acc_elems(1, S, H, D), device="cuda"), *(torch.empty(1, H, spad, device="cuda") for _ in range(2)))
    for a, b in ((k, clean), (clean, k)):
        forward(a, False, state, True, False)
        out, lse = forward(b, False, state, False, True)
        assert out.isnan().all() and lse.isnan().all()
    n.check_status(status, "fwd_hop")
