"""cp_bfv_mul runs the batched chain's launches on separate operands and results: equal to
cp_bfv_mul_batch at sizes on each transform path, for bases smaller and larger than Q, with
results apart from each other or in the operands' own buffers."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nphi, k, kl, t", [(64, 1, 2, 256), (2048, 2, 1, 256), (4096, 2, 3, 65537), (8192, 5, 6, 256),
                                            (8192, 24, 24, 256), (16384, 3, 7, 256), (16384, 24, 24, 256),
                                            (32768, 2, 3, 65537), (65536, 1, 2, 256)])
def test_single_multiplication_equals_the_batched_one(gpu, nphi, k, kl, t):
    import torch
    from cupoly_b200.engine import Engine, QBase
    e = Engine(k, kl, nphi, t)
    N = nphi // 2
    ins = [torch.randint(0, 1 << 62, (1, k, N, 2), device="cuda", dtype=torch.int64) for _ in range(4)]
    want = e.empty(QBase, 3)
    e.bfv_mul_batch(want, *ins, 1, e.bfv_mul_batch_workspace(1))
    # three results at uneven distances in one buffer
    room = torch.full((3 * k * N + 37, 2), -1, device="cuda", dtype=torch.int64)
    at = [(0, 3), (k * N + 3, 30), (2 * k * N + 33, 4)]
    outs = [room[o:o + k * N].view(1, k, N, 2) for o, _ in at]
    keep = [x.clone() for x in ins]
    e.bfv_mul(*outs, *ins)
    for v in range(3):
        assert torch.equal(outs[v][0], want[v])
        assert (room[at[v][0] + k * N:at[v][0] + k * N + at[v][1]] == -1).all()  # nothing written beyond
    assert all(torch.equal(a, b) for a, b in zip(keep, ins))
    e.bfv_mul(ins[1], ins[0], ins[3], *ins)  # results in the operands' buffers
    for v, x in enumerate((ins[1], ins[0], ins[3])):
        assert torch.equal(x[0], want[v])
    e.check()
