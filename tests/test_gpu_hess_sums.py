"""What the Hessian's sums over millions of quartets leave of translational invariance: every quartet's block
is invariant to its own rounding, so the row sums over the atoms show the rounding of the accumulation.

Bound: an entry is the sum of partial sums, each rounded to half an eps of its size at each of its additions
with random signs; 64 eps of the largest entry covers the 26 blocks of a row.  One sum over all quartets
exceeds it about four times.
"""
import numpy as np
import pytest

from hfscf_b200 import basis as B
from hfscf_b200 import engine as E
from hfscf_b200 import molecules as M

pytestmark = pytest.mark.gpu


def test_translational_residual_of_a_large_hessian():
    Z, x = M.n_alkane(8)
    bs = B.build_basis("6-31g**", Z, np.asarray(x) * B.ANGSTROM_TO_BOHR)
    A = np.random.default_rng(3).normal(size=(bs.nbf, bs.nbf))
    with E.Engine(bs) as eng:
        H = eng.hess2e((A + A.T) / bs.nbf)
    residual = np.max(np.abs(H.reshape(len(H), -1, 3).sum(axis=1)))
    assert residual < 64 * np.finfo(float).eps * np.max(np.abs(H))
