"""cp_polymul where both forward transforms share a launch, against the transforms and the product as
separate calls: every kind of CUDA-core plan, operands in either order in memory, c aliasing them."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nphi,k,npolys", [(4, 1, 1), (64, 3, 2), (2048, 2, 5), (4096, 2, 1), (4096, 3, 16), (4096, 7, 7),
                                           (8192, 5, 1), (16384, 8, 1), (16384, 3, 3), (32768, 16, 1), (65536, 2, 1)])
@pytest.mark.parametrize("cluster", [False, True])
def test_polymul_equals_its_parts(gpu, nphi, k, npolys, cluster):
    import torch

    from cupoly_b200.engine import FORWARD, INVERSE, UNIFORM, Engine, QBase
    e = Engine(k, 0, nphi, 256)
    if cluster:
        if nphi < 16384:
            pytest.skip("no cluster form")
        e.set_split_mode(1)
    mem = e.empty(QBase, 2 * npolys)
    e.sample(mem, QBase, UNIFORM, 5, 0, 2 * npolys, to_dgt=False)
    ws = e.polymul_workspace(QBase, npolys)
    want = e.empty(QBase, npolys)
    fa, fb = mem[:npolys].clone(), mem[npolys:].clone()
    e.dgt(fa, QBase, FORWARD, npolys)
    e.dgt(fb, QBase, FORWARD, npolys)
    e.mul_batch(want, fa, fb, QBase, npolys)
    e.dgt(want, QBase, INVERSE, npolys)
    c = e.empty(QBase, npolys)
    e.polymul(c, mem[:npolys], mem[npolys:], QBase, ws, npolys)
    assert torch.equal(c, want)
    e.polymul(c, mem[npolys:], mem[:npolys], QBase, ws, npolys)  # the second operand below the first
    assert torch.equal(c, want)
    a = mem[:npolys].clone()
    e.polymul(a, a, mem[npolys:], QBase, ws, npolys)
    assert torch.equal(a, want)
