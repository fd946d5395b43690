"""The work that is timed: calls of ``ring_flash_attn`` as programs make them, over the range the operator serves.

A case is one call (forward only under ``no_grad``, or forward and backward) on one GPU.  Ring cases run one rank of
a ring: the call gets a ring handle (the duck-typed stand-in for a process group that the schedules accept) whose
transport hands over K/V blocks and partial dK/dV prepared beforehand, so the rank does exactly the hops, state
hand-overs and accumulations it does between its neighbours, without the link.
"""
from __future__ import annotations

import contextlib
import math

import torch

import opt_ring_flash_attn_b200 as rfa

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _case(name, B, S, Hq, Hkv, D, *, dtype="bf16", causal=True, backward=True, deterministic=False, world=1, rank=0,
          zigzag=False, std=1.0):
    c = dict(B=B, S=S, Hq=Hq, Hkv=Hkv, D=D, dtype=dtype, causal=causal, backward=backward, deterministic=deterministic,
             world=world, rank=rank, zigzag=zigzag, std=std)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # The smallest training call: the shard of the CPU configuration (8 heads of 64, 256 tokens per rank) in bf16.
        # Nothing but launches, gaps and host work.
        _case("train_s256_d64", 1, 256, 8, 8, 64),
        # A prompt of ragged length through a GQA layer, forward only: one wave of CTAs of unequal length.
        _case("infer_s1000_gqa", 1, 1000, 32, 8, 128, backward=False),
        # The short-shard configuration: 1024 tokens per rank, 32 heads of 128.
        _case("train_s1024_mha", 1, 1024, 32, 32, 128),
        # Dense (not causal) training of a batch with a ragged length and a head dim that needs padding, fp16.
        _case("train_dense_s1500_d96", 2, 1500, 16, 4, 96, dtype="fp16", causal=False),
        # Bit-reproducible gradients (debugging, regression runs) at the reference grid's GQA shape.
        _case("train_det_s2048_gqa", 1, 2048, 16, 2, 128, deterministic=True),
        # Head dim 64 at the reference grid's 4096 tokens.
        _case("train_s4096_d64", 1, 4096, 16, 16, 64),
        # The large-head-dim configuration.
        _case("train_s4096_d256", 2, 4096, 16, 16, 256),
        # The Llama-3-8B-shaped configuration, the one bench.py times.
        _case("train_s8192_gqa", 1, 8192, 32, 8, 128),
        # Prefill of a long prompt through the same layer, fp16, forward only.
        _case("infer_s16384_gqa", 1, 16384, 32, 8, 128, dtype="fp16", backward=False),
        # The last rank of a ring of four over contiguous shards: one diagonal and three full blocks, running state
        # carried between hops, partial dK/dV folded in.
        _case("ring4_s2048_gqa", 1, 2048, 32, 8, 128, world=4, rank=3),
        # One rank of a ring of four over zigzag shards: every hop is a window of half the queries or half the keys.
        _case("zigzag4_s4096_gqa", 1, 4096, 32, 8, 128, world=4, rank=1, zigzag=True),
        # The long-context shard length with one GQA group of its 64/8 heads.
        _case("train_s131072_gqa", 1, 131072, 8, 1, 128, std=0.5),
    ]


_MAX_FLOPS = 3.5 * 2 * 8 * 131072 * 131072 * 128  # of the largest listed case


def draw(rng):
    while True:
        S = int(round(math.exp(rng.uniform(math.log(128), math.log(131072)))))
        if rng.random() < 0.6:  # lengths are multiples of something in most programs, ragged in many
            S = max(128, S // 128 * 128)
        D = rng.choice([64, 64, 128, 128, 128, 128, 256, 32, 96, 160])
        Hkv = rng.choice([1, 2, 4, 8, 16, 32])
        Hq = Hkv * rng.choice([1, 1, 2, 4, 8])
        B = rng.choice([1, 1, 1, 2, 3, 4])
        kind = rng.random()
        kw = dict(dtype=rng.choice(["bf16", "bf16", "fp16"]), causal=rng.random() < 0.75,
                  backward=rng.random() < 0.7, std=rng.choice([1.0, 1.0, 0.5]))
        if kind < 0.12:
            kw.update(deterministic=True, backward=True)
        elif kind < 0.3:
            world = rng.choice([2, 3, 4, 8])
            kw.update(world=world, causal=True)
            if rng.random() < 0.5:
                S = max(256, S // 256 * 256)
                kw.update(zigzag=True, rank=rng.randrange(world))
            else:
                kw.update(rank=world - 1)
        c = _case(None, B, S, Hq, Hkv, D, **kw)
        # as much work as the largest listed case at most, and no more data than fits comfortably
        if Hq <= 64 and work(c)["flops"] <= _MAX_FLOPS and work(c)["bytes"] <= 4e9:
            return c


class _Neighbours:
    """The two neighbours of a rank on one of its rings, as a transport: ``wait`` delivers the next prepared message,
    ``post`` takes the outgoing one (kept where it is a result: the partial dK/dV that travel on)."""

    def __init__(self, world, inbox, outbox):
        self.world_size = world
        self.inbox, self.outbox = inbox, outbox
        self._recv, self._sent, self._taken = [], 0, 0

    def post(self, send, recv):
        if self.outbox:
            self.outbox[self._sent % len(self.outbox)].copy_(send)
        self._sent += 1
        self._recv.append(recv)

    def wait(self):
        self._recv.pop(0).copy_(self.inbox[self._taken % len(self.inbox)])
        self._taken += 1


class _Rank:
    def __init__(self, world, rank, transports):
        self.world_size, self.ring_rank = world, rank
        self.workspace_key = ("perf", world, rank)
        self._transports = transports

    def transport(self, name):
        return self._transports[name]


def prepare(case, seed):
    B, S, Hq, Hkv, D, W = case["B"], case["S"], case["Hq"], case["Hkv"], case["D"], case["world"]
    dev, dt = torch.device("cuda"), _DTYPES[case["dtype"]]
    g = torch.Generator(device=dev)
    g.manual_seed(seed)

    def normal(*shape, std=1.0, dtype=dt):
        return (torch.randn(*shape, generator=g, device=dev, dtype=torch.float32) * std).to(dtype)

    st = {"case": case}
    for name, H in (("q", Hq), ("k", Hkv), ("v", Hkv)):
        st[name] = normal(B, S, H, D, std=case["std"]).requires_grad_(case["backward"])
    if case["backward"]:
        st["dout"] = normal(B, S, Hq, D)
    if W > 1:
        kv = [normal(2, B, S, Hkv, D, std=case["std"]) for _ in range(W - 1)]
        tr = {"fwd_kv": _Neighbours(W, kv, []), "bwd_kv": _Neighbours(W, kv, [])}
        if case["backward"]:
            part = [normal(2, B, S, Hkv, D, dtype=torch.float32) for _ in range(W - 1)]
            sent = [torch.empty_like(part[0]) for _ in range(W)]
            # the last message is this rank's own block coming home, as it was first sent
            tr["bwd_dkdv"] = _Neighbours(W, part + [sent[0]], sent)
            st["sent"] = sent
        st["group"] = _Rank(W, case["rank"], tr)
    return st


def run(state):
    c = state["case"]
    q, k, v = state["q"], state["k"], state["v"]
    kw = dict(causal=c["causal"], zigzag=c["zigzag"], group=state.get("group"))
    if not c["backward"]:
        with torch.no_grad():
            return rfa.ring_flash_attn(q, k, v, **kw)
    with rfa.deterministic() if c["deterministic"] else contextlib.nullcontext():
        out = rfa.ring_flash_attn(q, k, v, **kw)
    grads = torch.autograd.grad(out, (q, k, v), state["dout"])
    # what travels on to the next rank is a result too (the first message comes back as dk, dv)
    return (out.detach(), *grads, *state["sent"][1:]) if "sent" in state else (out.detach(), *grads)


def work(case):
    B, S, Hq, Hkv, D, W = case["B"], case["S"], case["Hq"], case["Hkv"], case["D"], case["world"]
    if W == 1:
        blocks = 0.5 if case["causal"] else 1.0
    elif case["zigzag"]:
        blocks = W / 2
    else:
        blocks = W - 0.5
    flops = (3.5 if case["backward"] else 1.0) * blocks * 4 * B * Hq * S * S * D
    qb, kvb = 2 * B * S * Hq * D, 2 * 2 * B * S * Hkv * D
    nbytes = 2 * qb + W * kvb  # q, K/V blocks in; out
    if case["backward"]:
        nbytes += 2 * qb + kvb  # dout in; dq, dk, dv out
        if W > 1:
            nbytes += (2 * (W - 1) + 2) * 2 * kvb  # fp32 partial dK/dV in and out, own block out and home
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # The same attention in fp64 on these shapes: out 2.1e-3, dq and dk 3.0e-3, dv 2.3e-3 in bf16; 2.9e-4, 3.6e-4 and
    # 3.0e-4 in fp16 (rounding of P, dS and the results).  Four times the largest.
    return {"rel": 1.2e-2 if case["dtype"] == "bf16" else 1.5e-3}
