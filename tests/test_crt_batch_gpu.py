"""cp_crt / cp_icrt over batches, bit-exact against Python big integers: enough blocks that each takes
every residue of its elements, bases that are no multiple of the four residues taken at a time, ring
degrees below one block's elements, limb counts at the changes of the block size (23, 47), and the
byte matrix products with their largest limb counts and bases (32, 16) and one more."""
import numpy as np
import pytest

from oracle import pyoracle as O
from tests.common import splitmix64, unfold

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,nphi,npolys,nlimbs", [(5, 8, 640, 5), (4, 64, 600, 23), (3, 1024, 300, 24), (9, 16, 601, 47),
                                                  (2, 256, 600, 48), (1, 512, 600, 1), (6, 2048, 2, 7),
                                                  (1, 32768, 300, 1), (2, 16384, 150, 2), (3, 4096, 256, 3),
                                                  (5, 8192, 48, 33), (7, 1024, 200, 7), (8, 256, 1, 8),
                                                  (16, 1024, 40, 32), (17, 512, 30, 32)])
def test_crt_icrt_batches(gpu, k, nphi, npolys, nlimbs):
    import torch

    from cupoly_b200.engine import Engine, from_u64, limbs_to_ints, to_u64
    e = Engine(k, 0, nphi, 256)
    w = splitmix64(k * 131 + nlimbs, 3, npolys * nphi * nlimbs).reshape(npolys, nphi, nlimbs)
    Q = O.prod(e.Q)
    w[0, 0] = np.uint64(0xFFFFFFFFFFFFFFFF)
    for at, v in ((1, 0), (2, 1), (3, Q - 1), (4, Q), (5, Q // 2)):    # and around multiples of Q
        if at < nphi and v < 1 << (64 * nlimbs):
            w[0, at] = [(v >> (64 * i)) & 0xFFFFFFFFFFFFFFFF for i in range(nlimbs)]
    x = e.empty(0, npolys)
    e.crt(x, from_u64(w), 0)
    got = to_u64(x).reshape(npolys, k, nphi // 2, 2)
    polys = sorted({0, npolys // 4, npolys // 2, npolys - 1})
    ints = {q: limbs_to_ints(w[q]) for q in polys}
    for q in polys:
        res = unfold(got[q:q + 1])[0]
        for r, p in enumerate(e.Q):
            assert np.array_equal(res[r], np.array([v % p for v in ints[q]], dtype=np.uint64)), (q, r)
    nl = max(nlimbs, k)
    back = torch.full((npolys, nphi, nl), -1, dtype=torch.int64, device="cuda")
    e.icrt(back, x, 0)
    host = to_u64(back)
    for q in polys:
        assert limbs_to_ints(host[q]) == [v % Q for v in ints[q]], q
