"""Work lists of more rows than one tensor-core launch takes (4096): the later launches' offsets into the
rows, the operands and the primes.  The rows after 4096 have primes that the first ones have not."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nphi,n", [(2048, 4097), (2048, 8193), (4096, 4099), (8192, 4100), (16384, 4097)])
def test_lists_of_several_launches(gpu, nphi, n):
    import torch
    from cupoly_b200 import _lib
    from cupoly_b200.engine import Engine, _ptr, _stream
    e, o = Engine(8, 0, nphi, 256), Engine(8, 0, nphi, 256)
    e.set_tensor(2)
    o.set_tensor(0)
    assert n > 4096 and e.dgt_launches(n, True) == ((n + 4095) // 4096, True)
    g = torch.Generator(device="cuda").manual_seed(n)
    rid = torch.randint(0, 5, (n,), generator=g, device="cuda", dtype=torch.int32)
    rid[4096:] = torch.randint(5, 8, (n - 4096,), generator=g, device="cuda", dtype=torch.int32)
    a, b = (torch.randint(0, 1 << 62, (n, nphi // 2, 2), generator=g, device="cuda", dtype=torch.int64) for _ in "ab")
    res = []
    for eng in (e, o):
        wa, wb, c = (torch.empty_like(a) for _ in range(3))
        _lib.call("cp_polymul_list", eng.handle, _ptr(c), _ptr(a), _ptr(b), _ptr(wa), _ptr(wb), _ptr(rid), n, _stream())
        wa.copy_(a)
        _lib.call("cp_dgt_list", eng.handle, _ptr(wa), _ptr(rid), n, 0, _stream())
        wb.copy_(wa)
        _lib.call("cp_dgt_list", eng.handle, _ptr(wb), _ptr(rid), n, 1, _stream())
        res.append((c, wa, wb))
    for p, q in zip(*res):
        assert torch.equal(p, q)
    assert torch.equal(res[0][2], a)  # values below every prime come back
    e.check()
