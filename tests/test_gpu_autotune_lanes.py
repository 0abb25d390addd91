"""The schedule that hfgpu_autotune keeps and returns names the lanes of every class: a class that the tuner
did not time, or a starting schedule that it kept, leaves no -1 (the rule by size), and builds agree with
the default's (1e-11, as in test_gpu_schedule).
"""
import numpy as np
import pytest

from hfscf_b200 import basis as B
from hfscf_b200 import engine as E
from hfscf_b200 import molecules as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [E.FP64, E.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("name", ["sto-3g", "6-31g*"])  # without and with d shells
def test_autotuned_schedule_names_its_lanes(name, precision):
    Z, x = M.water(np.random.default_rng(1))
    bs = B.build_basis(name, Z, np.asarray(x) * B.ANGSTROM_TO_BOHR, pure=False)
    A = np.random.default_rng(2).normal(size=(bs.nbf, bs.nbf))
    D = (A + A.T) / bs.nbf
    with E.Engine(bs) as eng:
        J0, K0 = eng.jk(D, [D])
        sched = eng.autotune(D, precision, repeats=1)
        assert np.isin(sched[:, 1], (0, 1, 4, 8, 16, 32)).all(), sched[:, 1]
        assert (eng.get_schedule() == sched).all()
        J, K = eng.jk(D, [D])
    assert np.max(np.abs(J - J0)) < 1e-11
    assert np.max(np.abs(K[0] - K0[0])) < 1e-11
