"""The FP64 Boys function (hfgpu_boys): its accuracy over the table, and beyond it.

Over [0, 70], against the series in 80-bit arithmetic.  The interpolation error of F_M is at most
(1/64)^6 / (6! 2^5) F_{M+6} = 6e-16 F_M, the 32-bit coefficients cost 1e-16 and the dropped e^-T 1e-16; Horner's
rule, the downward recursion and the reciprocal powers add a few roundings per order.  1e-14 of every
value bounds their sum, and 4e-16 their mean: the errors fill their bounds on average to a tenth (below
the 1.1e-15 of a Taylor row at M = 10).

Beyond the table every finite T >= 0 is accepted, and for large T the value is the complete integral
F_n(T) = (2n-1)!! / 2^(n+1) sqrt(pi) T^-(n+1/2) (the rest, below e^-T, is far below the last digit).
Tolerance: the evaluation takes two or three rounded operations per order, below 1e-14 relative in all, and
1e-307 absolute where F_n is subnormal (above T = 1e307, where 1/T is, every F_n but F_0 is zero).
"""
import numpy as np
import pytest

from hfscf_b200 import basis as B
from hfscf_b200 import engine as E
from hfscf_b200 import molecules as M

pytestmark = pytest.mark.gpu


def _engine():
    Z, x = M.water(np.random.default_rng(1))
    return E.Engine(B.build_basis("sto-3g", Z, np.asarray(x) * B.ANGSTROM_TO_BOHR))


@pytest.mark.parametrize("m", range(11))
def test_boys_accuracy_over_the_table(m):
    T = np.random.default_rng(5).uniform(0.0, 70.0, 20000)
    with _engine() as eng:
        F = eng.boys(m, T)
    t = T.astype(np.longdouble)
    errors = []
    for n in range(m + 1):
        term = np.full_like(t, 1 / np.longdouble(2 * n + 1))
        ref = term.copy()
        for i in range(500):
            term = term * 2 * t / (2 * n + 2 * i + 3)
            ref += term
        ref *= np.exp(-t)
        errors.append(np.abs(F[:, n] - ref) / ref)
    assert np.max(errors) < 1e-14
    assert np.mean(errors) < 4e-16


@pytest.mark.parametrize("m", range(11))
def test_boys_of_large_arguments(m):
    T = np.concatenate([10.0 ** np.arange(2, 308, 7), [3e28, 2e29, 3e35, 1e200, 1.7e308]])
    with _engine() as eng:
        F = eng.boys(m, T)
    t = T.astype(np.longdouble)
    ref = np.sqrt(np.longdouble("3.14159265358979323846264338327950288") / t) / 2
    for n in range(m + 1):
        assert np.all(np.abs(F[:, n] - ref) <= 1e-14 * ref + np.longdouble(1e-307)), n
        ref = ref * (n + np.longdouble(0.5)) / t


@pytest.mark.parametrize("carbons,name", [(4, "6-31g**"), (3, "cc-pvdz")])
def test_staged_rows_match_the_global_ones(carbons, name):
    """J/K in the staged form (its own grid, eight coefficients) against one thread per quartet on the global
    rows: both Boys functions are within 1e-14 of the exact value and 4e-16 on average, and an entry sums
    thousands of integrals up to a few times its size: 5e-14 of the largest entry."""
    Z, x = M.n_alkane(carbons)
    bs = B.build_basis(name, Z, np.asarray(x) * B.ANGSTROM_TO_BOHR, pure=name == "cc-pvdz")
    A = np.random.default_rng(11).normal(size=(bs.nbf, bs.nbf))
    D = (A + A.T) / bs.nbf
    with E.Engine(bs) as eng:
        eng.set_schedule(np.tile(np.array((64, 0, 0, 0), dtype=np.int32), (E.NUM_CLASSES, 1)))
        J0, K0 = eng.jk(D, [D])
        eng.set_schedule(np.tile(np.array((64, 0, 0, 2), dtype=np.int32), (E.NUM_CLASSES, 1)))
        J, K = eng.jk(D, [D])
    assert np.max(np.abs(J - J0)) < 5e-14 * np.max(np.abs(J0))
    assert np.max(np.abs(K[0] - K0[0])) < 5e-14 * np.max(np.abs(K0[0]))
