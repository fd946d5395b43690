"""K/V tiles of the backward hop shared by several CTAs: runs that cross head boundaries, do not divide evenly, or start
inside a window, and the ordered mode (bit-reproducible with any split)."""
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
