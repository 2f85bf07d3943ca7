"""CKKS modulus raising and reduction at the ends of the compiled base sizes (1 and 24 source residues),
against the same big-integer restatement as the other sizes."""
import pytest

from tests import test_ckks_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,kl,nphi,prec,level", [(24, 24, 64, 55, 23), (13, 9, 512, 45, 6), (2, 1, 16, 48, 0),
                                                  (17, 12, 256, 52, 16)])
def test_ckks_base_sizes(gpu, k, kl, nphi, prec, level):
    test_ckks_gpu.test_ckks_modulus_raising_and_reduction(gpu, k, kl, nphi, prec, level)
