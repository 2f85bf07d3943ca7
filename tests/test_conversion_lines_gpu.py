"""The batched chain on both sides of the lines between its conversions on CUDA and tensor cores, against the
same pairs one at a time: 4 residues to 3 or 4 from 2^17 elements on, 3 residues from 2^18."""
import pytest

pytestmark = pytest.mark.gpu


# 3 P x 4096 elements pass 2^17 at P 11, 4 P x 4096 at P 8; 2^18 at P 22 and 16
@pytest.mark.parametrize("k,kl", [(3, 4), (4, 4), (4, 3), (4, 5)])
@pytest.mark.parametrize("P", (7, 8, 10, 11, 16, 22))
def test_batches_equal_single_pairs(gpu, k, kl, P):
    import torch
    from cupoly_b200.engine import Engine, QBase
    e = Engine(k, kl, 8192, 256)
    ins = [torch.randint(0, 1 << 62, (P, k, 4096, 2), device="cuda", dtype=torch.int64) for _ in range(4)]
    c, one = e.empty(QBase, 3 * P), e.empty(QBase, 3)
    e.bfv_mul_batch(c, *ins, P, e.bfv_mul_batch_workspace(P))
    ws = e.bfv_mul_batch_workspace(1)
    for q in range(P):
        e.bfv_mul_batch(one, *(x[q:q + 1] for x in ins), 1, ws)
        for v in range(3):
            assert torch.equal(c[v * P + q], one[v]), (q, v)
    e.check()
