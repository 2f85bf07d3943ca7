"""The base conversions on the tensor cores, through the multiplication chain: against the
oracle at base sizes around the groups of 8 targets, the K steps of 4 residues and the registers
of the early loads, on the fast path and with every coefficient sent to the exact path."""
import numpy as np
import pytest

from tests.common import fold, random_poly_residues, unfold

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nphi, k, kl, P", [(256, 4, 5, 1), (256, 7, 8, 3), (256, 8, 9, 2), (512, 11, 12, 1),
                                            (256, 12, 17, 2), (256, 16, 17, 1), (256, 23, 24, 1), (256, 4, 16, 1),
                                            (16384, 3, 4, 11)])
def test_chain_conversions_match_the_oracle(gpu, nphi, k, kl, P):
    from cupoly_b200.engine import FORWARD, INVERSE, Engine, QBase, from_u64, to_u64
    from oracle import coracle
    e = Engine(k, kl, nphi, 256)
    rows = [np.stack([random_poly_residues(100 * v + q, e.Q, nphi) for q in range(P)]) for v in range(4)]
    rows[0][0][:, :2] = 0
    for r, p in enumerate(e.Q):
        rows[1][0][r, :5] = p - 1
    ins = []
    for a in rows:
        x = from_u64(np.stack([fold(q) for q in a]))
        e.dgt(x, QBase, FORWARD)
        ins.append(x)
    want = coracle.bfv_mul(*rows, e.Q, e.B, 256)
    ws = e.bfv_mul_batch_workspace(P)
    for exact in (False, True):
        e.set_hps_force_exact(exact)
        c = e.empty(QBase, 3 * P)
        e.bfv_mul_batch(c, *ins, P, ws)
        e.dgt(c, QBase, INVERSE)
        got = unfold(to_u64(c)).reshape(3, P, k, nphi)
        for v in range(3):
            assert np.array_equal(got[v], want[v]), (exact, v)
    e.check()
