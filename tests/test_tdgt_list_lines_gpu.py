"""Work lists on both sides of their lines between CUDA and tensor cores, where the two directions of nphi 2048
have lines of their own: cp_polymul_list and cp_dgt_list against the same rows on the CUDA cores."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nphi,n", [(2048, 320), (2048, 1150), (2048, 1151), (2048, 2600), (2048, 2601), (4096, 148),
                                    (4096, 149), (8192, 74), (8192, 75), (16384, 74), (16384, 75)])
def test_lists_around_their_lines(gpu, nphi, n):
    import torch
    from cupoly_b200 import _lib
    from cupoly_b200.engine import Engine, _ptr, _stream
    e, o = Engine(3, 0, nphi, 256), Engine(3, 0, nphi, 256)
    o.set_tensor(0)
    forward, products = {2048: (2600, 1150), 4096: (148, 148), 8192: (74, 74), 16384: (74, 74)}[nphi]
    assert e.dgt_launches(n, True)[1] == (n > forward)
    assert e.products_apart(n, True) == (n > products)
    g = torch.Generator(device="cuda").manual_seed(n)
    rid = torch.randint(0, 3, (n,), generator=g, device="cuda", dtype=torch.int32)
    a, b = (torch.randint(0, 1 << 62, (n, nphi // 2, 2), generator=g, device="cuda", dtype=torch.int64) for _ in "ab")
    res = []
    for eng in (e, o):
        wa, wb, c, x = (torch.empty_like(a) for _ in range(4))
        _lib.call("cp_polymul_list", eng.handle, _ptr(c), _ptr(a), _ptr(b), _ptr(wa), _ptr(wb), _ptr(rid), n, _stream())
        x.copy_(a)
        _lib.call("cp_dgt_list", eng.handle, _ptr(x), _ptr(rid), n, 0, _stream())
        y = x.clone()
        _lib.call("cp_dgt_list", eng.handle, _ptr(y), _ptr(rid), n, 1, _stream())
        res.append((c, x, y))
    for p, q in zip(*res):
        assert torch.equal(p, q)
    assert torch.equal(res[0][2], a)
    e.check()
