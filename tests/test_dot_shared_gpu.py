"""cp_dot_batch with shared keys (runs of polynomials per thread, the keys held in registers) against
the call with a copy of the keys per polynomial, which sums one element per thread."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nphi,k,n,npolys", [(8, 1, 1, 1), (64, 3, 2, 5), (512, 2, 3, 701), (256, 4, 4, 2),
                                             (2048, 5, 5, 37), (1024, 6, 6, 3), (128, 7, 7, 300), (4096, 2, 8, 9),
                                             (256, 9, 9, 4)])
def test_dot_shared_equals_per_polynomial_keys(gpu, nphi, k, n, npolys):
    import torch

    from cupoly_b200.engine import UNIFORM, Engine, QBase
    e = Engine(k, 0, nphi, 256)
    a, b = e.empty(QBase, npolys * n), e.empty(QBase, n)
    e.sample(a, QBase, UNIFORM, 11, 0, npolys * n, to_dgt=False)
    e.sample(b, QBase, UNIFORM, 12, 0, n, to_dgt=False)
    top = torch.tensor([p - 1 for p in e.Q], dtype=torch.int64, device="cuda").view(k, 1, 1)
    a.view(npolys * n, k, nphi // 2, 2)[:, :, :2] = top     # the largest sums
    b.view(n, k, nphi // 2, 2)[:, :, :2] = top
    got, want = e.empty(QBase, npolys), e.empty(QBase, npolys)
    e.dot_batch(got, a, b, n, npolys, QBase, b_shared=True)
    each = b.reshape(1, -1).expand(npolys, -1).contiguous()
    e.dot_batch(want, a, each, n, npolys, QBase)
    assert torch.equal(got, want)
