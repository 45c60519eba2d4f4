"""Expert pools on host memory: what a layer keeps of them lives as long as the pools do."""
import pytest
import torch

from moonep_b200.parallel.symm import SymmetricHeap
from moonep_b200.pools import ExpertPools, pool_layout

SHAPES = (64, 32), (64, 32), (32, 64)


def make_pools(with_grads=True, dtype=torch.bfloat16):
    _, _, nbytes = pool_layout(2, dict(zip(("gate", "up", "down"), SHAPES)), dtype, with_grads)
    return ExpertPools(2, *SHAPES, dtype=dtype, with_grads=with_grads, world=1, rank=0, heap=SymmetricHeap.local(1, nbytes, "cpu"))


def test_addresses_are_those_of_the_compute_views():
    p = make_pools()
    for _ in range(2):
        assert p.addresses(2, 64, 32) == tuple(p.compute_weight(n).data_ptr() for n in ("gate", "up", "down"))
        assert p.addresses(2, 64, 32, grads=True) == tuple(p.compute_grad(n).data_ptr() for n in ("gate", "up", "down"))
    for size in ((4, 64, 32), (2, 32, 64)):
        with pytest.raises(AssertionError, match="the layer needs"):
            p.addresses(*size)
    with pytest.raises(AssertionError, match="bf16"):
        make_pools(dtype=torch.float16).addresses(2, 64, 32)


def test_no_addresses_without_memory():
    p = make_pools(with_grads=False)
    p.addresses(2, 64, 32)
    with pytest.raises(KeyError):
        p.addresses(2, 64, 32, grads=True)
    p.kept("anything", lambda: p.local_weight("up"))
    p.destroy()
    for ask in (lambda: p.addresses(2, 64, 32), lambda: p.local_weight("up"), lambda: p.kept("anything", lambda: p.local_weight("up"))):
        with pytest.raises(AttributeError):
            ask()


@pytest.mark.parametrize("view", ["local_weight", "compute_weight", "local_grad", "compute_grad"])
def test_views_share_memory_and_nothing_else(view):
    p = make_pools()
    a = getattr(p, view)("gate")
    shape = a.shape
    a.requires_grad_(True)
    (a * 2).sum().backward()
    b = getattr(p, view)("gate")
    assert b is not a and not b.requires_grad and b.grad is None and b.shape == shape
    b[1].fill_(3)
    c = getattr(p, view)("gate")
    c.unsqueeze_(0)
    d = getattr(p, view)("gate")
    assert d.shape == shape and bool((d[1] == 3).all()) and bool((d[0] == 0).all())
