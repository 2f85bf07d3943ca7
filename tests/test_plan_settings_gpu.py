"""Which transforms run where: the plan settings made after an engine's creation take effect in its
launches although the engine has tensor-core transforms, and cp_engine_set_tensor takes them
back; what the tensor cores cannot do is refused.  Results are equal on every route."""
import pytest

pytestmark = pytest.mark.gpu


def _transformed(e, x, units):
    from cupoly_b200.engine import FORWARD, INVERSE, QBase
    y = x.clone()
    e.dgt(y, QBase, FORWARD, units)
    z = y.clone()
    e.dgt(z, QBase, INVERSE, units)
    return y, z


@pytest.mark.parametrize("nphi", (32768, 65536))
def test_cluster_form_goes_before_the_tensor_cores(gpu, nphi):
    import torch
    from cupoly_b200.engine import Engine
    e = Engine(1, 0, nphi, 256)
    x = torch.randint(0, 1 << 62, (3, 1, nphi // 2, 2), device="cuda", dtype=torch.int64)
    assert e.dgt_launches(3) == (2, True)  # split stage, tensor-core blocks
    want = _transformed(e, x, 3)
    for setting, arg, route in (("set_split_mode", 1, (1, False)), ("set_tensor", 1, (2, True)),
                                ("set_split_mode", 1, (1, False)), ("set_split_mode", 0, (2, True)),
                                ("set_split_mode", 1, (1, False)), ("set_tensor", 2, (2, True)),
                                ("set_tensor", 0, (1, False))):
        getattr(e, setting)(arg)
        assert e.dgt_launches(3) == route, (setting, arg)
        assert all(torch.equal(a, b) for a, b in zip(_transformed(e, x, 3), want)), (setting, arg)
    e.check()


def test_small_launch_plan_goes_before_the_tensor_cores(gpu):
    import torch
    from cupoly_b200.engine import Engine
    e = Engine(1, 0, 8192, 256)
    x = torch.randint(0, 1 << 62, (97, 1, 4096, 2), device="cuda", dtype=torch.int64)
    assert e.dgt_launches(64)[1] is False and e.dgt_launches(65) == (1, True)
    want = {n: _transformed(e, x[:n], n) for n in (96, 97)}
    e.set_narrow_plan(2, 10, 96)
    for tensor in (False, True):
        if tensor:
            e.set_tensor(1)
        assert e.dgt_launches(96) == ((1, True) if tensor else (2, False)) and e.dgt_launches(97) == (1, True)
        for n in (96, 97):
            assert all(torch.equal(a, b) for a, b in zip(_transformed(e, x[:n], n), want[n])), (tensor, n)
    e.set_narrow_plan(2, 10, 96)
    e.set_narrow_plan(0, 0, 0)
    assert e.dgt_launches(96) == (1, True)
    e.check()


def test_tensor_transforms_that_cannot_be_had_are_refused(gpu):
    from cupoly_b200 import _lib
    from cupoly_b200.engine import Engine
    e = Engine(1, 0, 32768, 256)
    e.set_plan(3, 13)  # one split bit
    for eng in (e, Engine.ckks(2, 0, 4096, 55), Engine(1, 0, 1024, 256)):
        with pytest.raises(_lib.CupolyError) as ei:
            eng.set_tensor(2)
        assert ei.value.code == 3
        eng.set_tensor(1)  # in the launches that gain from them: none
        assert not eng.get_tensor() and not eng.dgt_launches(1000)[1]
    e.set_plan(3, 12)
    e.set_tensor(2)
    assert e.get_tensor() and e.dgt_launches(1) == (2, True)


@pytest.mark.parametrize("nphi,k,npolys", [(16384, 8, 1), (16384, 3, 3), (32768, 4, 2), (65536, 2, 1)])
def test_polymul_pair_in_the_cluster_form(gpu, nphi, k, npolys):
    """Both forward transforms of cp_polymul in one cluster launch with two sources."""
    import torch
    from cupoly_b200.engine import Engine, QBase
    e, o = Engine(k, 0, nphi, 256), Engine(k, 0, nphi, 256)
    e.set_narrow_plan(0, 0, 0)
    e.set_split_mode(1)
    o.set_tensor(2)
    assert e.dgt_launches(2 * npolys * k) == (1, False) and o.dgt_launches(npolys * k)[1]
    mem = torch.randint(0, 1 << 62, (2 * npolys, k, nphi // 2, 2), device="cuda", dtype=torch.int64)
    ws = e.polymul_workspace(QBase, npolys)
    want, c = o.empty(QBase, npolys), e.empty(QBase, npolys)
    o.polymul(want, mem[:npolys], mem[npolys:], QBase, ws, npolys)
    for a, b in ((mem[:npolys], mem[npolys:]), (mem[npolys:], mem[:npolys])):
        c.fill_(-1)
        e.polymul(c, a, b, QBase, ws, npolys)
        assert torch.equal(c, want)
    a = mem[:npolys].clone()
    e.polymul(a, a, mem[npolys:], QBase, ws, npolys)
    assert torch.equal(a, want)
    e.check()


@pytest.mark.parametrize("nphi,k", [(16384, 3), (32768, 2)])
def test_single_multiplication_in_the_cluster_form(gpu, nphi, k):
    """The last transform of cp_bfv_mul writes three separate results from its clusters."""
    import torch
    from cupoly_b200.engine import Engine, QBase
    e, o = Engine(k, 0, nphi, 256), Engine(k, 0, nphi, 256)
    e.set_narrow_plan(0, 0, 0)
    e.set_split_mode(1)
    assert e.dgt_launches(3 * k) == (1, False)
    ins = [torch.randint(0, 1 << 62, (1, k, nphi // 2, 2), device="cuda", dtype=torch.int64) for _ in range(4)]
    outs = [[eng.empty(QBase) for _ in range(3)] for eng in (e, o)]
    e.bfv_mul(*outs[0], *ins)
    o.bfv_mul(*outs[1], *ins)
    assert all(torch.equal(a, b) for a, b in zip(*outs))
    e.check()
