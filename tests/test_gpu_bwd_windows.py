"""Windows of the backward hop (queries from q_begin on, keys below kv_len: the zigzag layout) whose K/V tiles are shared by
several CTAs, unordered and in the ordered mode, against the fp32 restatement of the same window."""
import pytest
import torch

from oracle.ring_attn_oracle import make_inputs

pytestmark = pytest.mark.gpu

GRAD_REL_L2 = 2e-2  # the parity tests' bound: P and dS are rounded to 16 bit


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm()).item()


@pytest.mark.parametrize("ordered", [False, True])
@pytest.mark.parametrize("with_prev", [False, True])
@pytest.mark.parametrize("B,S,Hq,Hkv,D,q_begin,kv_len", [
    (1, 512, 4, 1, 128, 256, 512),  # half of the queries, all keys
    (1, 512, 4, 1, 128, 0, 256),    # all queries, half of the keys
    (2, 512, 4, 2, 128, 128, 300),  # both, the keys end inside a tile
    (1, 384, 2, 1, 256, 256, 384),
    (1, 384, 2, 1, 256, 128, 200),
    (1, 512, 6, 2, 64, 256, 130),
    (1, 512, 1, 1, 128, 384, 64),   # one query tile: not shared
])
def test_window(B, S, Hq, Hkv, D, q_begin, kv_len, with_prev, ordered):
    import fake_kernels
    from opt_ring_flash_attn_b200 import _native as n

    q, k, v, dout = make_inputs(S + kv_len, B, S, Hq, Hkv, D, dtype=torch.bfloat16)
    spad, scale = n.padded_seq(S), D ** -0.5
    # statistics and reference of the windowed problem, on the CPU
    out, lse = torch.zeros(B, S, Hq, D), torch.zeros(B, Hq, spad)
    fake_kernels.fwd_hop(q, k, v, None, None, None, out, lse, scale, True, True, False, None, q_begin=q_begin, kv_len=kv_len)
    delta, lse2 = torch.zeros(B, Hq, spad), torch.zeros(B, Hq, spad)
    fake_kernels.bwd_prepare(out, dout, lse, delta, lse2, None, None)
    dq_ref, block = torch.zeros(B * Hq * S * D), torch.zeros(2, B, S, Hkv, D)
    fake_kernels.bwd_hop(q, k, v, dout, lse2, delta, dq_ref, None, block, scale, False, False, None, q_begin=q_begin,
                         kv_len=kv_len)
    dq_ref = dq_ref.view(B, Hq, S, D).transpose(1, 2)

    q, k, v, dout, lse2, delta = (t.cuda() for t in (q, k, v, dout, lse2, delta))
    prev = torch.randn(2, B, S, Hkv, D, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def run():
        acc = torch.zeros(n.dq_acc_elems(B, S, Hq, D), device="cuda")
        dkdv = torch.full_like(prev, float("nan"))
        order = {}
        if ordered:  # scratch: cleared by the call
            order["dq_order"] = torch.full((n.dq_order_elems(B, S, Hq, D),), 7, dtype=torch.int32, device="cuda")
        n.bwd_hop(q, k, v, dout, lse2, delta, acc, prev if with_prev else None, dkdv, scale, with_prev, False, status,
                  q_begin=q_begin, kv_len=kv_len, **order)
        dq = torch.empty_like(q)
        n.dq_finalize(acc, dq)
        n.check_status(status, "bwd_hop")
        return dq, dkdv

    dq, dkdv = run()
    assert torch.equal(dq[:, :q_begin], torch.zeros_like(dq[:, :q_begin]))
    assert _rel(dq.cpu(), dq_ref) <= GRAD_REL_L2
    beyond = prev[:, :, kv_len:] if with_prev else torch.zeros_like(prev[:, :, kv_len:])
    assert torch.equal(dkdv[:, :, kv_len:], beyond)
    got = (dkdv - prev if with_prev else dkdv).cpu()
    for i in (0, 1):
        assert _rel(got[i, :, :kv_len], block[i, :, :kv_len]) <= GRAD_REL_L2
    if ordered:
        for a, b in zip((dq, dkdv), run()):
            assert torch.equal(a, b)


@pytest.mark.parametrize("W,S,Hq,Hkv,D", [(2, 512, 4, 1, 128), (3, 512, 8, 2, 64), (2, 256, 2, 1, 256)])
def test_zigzag_schedule_in_the_ordered_mode(W, S, Hq, Hkv, D):
    from inproc_ring import run_ring
    from oracle.ring_attn_oracle import zigzag_oracle, zigzag_shard

    full = [x.cuda() for x in make_inputs(81, 1, S * W, Hq, Hkv, D, dtype=torch.bfloat16)]
    shards = [zigzag_shard(x, W) for x in full]
    ref = zigzag_oracle(*full, W, head_chunk=4)

    def run():
        return run_ring(W, torch.device("cuda:0"), *shards, D ** -0.5, True, zigzag=True, deterministic=True)[2:]

    first = run()
    for r in range(W):
        for name, got in zip(("dq", "dk", "dv"), first):
            assert _rel(got[r], ref[name][r]) <= GRAD_REL_L2, f"rank {r}: {name}"
    for a, b in zip(first, run()):
        assert all(torch.equal(x, y) for x, y in zip(a, b))
