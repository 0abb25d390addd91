"""The forms that a launch takes by its size, against the general ones: J/K (primitive-split lanes and Rys
quadrature in small builds) against one thread per quartet, derivatives (thread triples, Rys groups)
against the thread forms, and the Boys rows at the edges of their intervals.

Tolerances.  J/K: the forms' integrals differ by at most the Boys rows' 6e-14 (relative) and rounding, the
matrices hold sums of them up to a few tens: 1e-11 of the largest entry.  Mixed builds: 1e-6, gradients
1e-10 and Hessians 1e-9 as in test_gpu_parity and test_gpu_hessian.  Boys: the polynomials' 6e-14 at most,
2e-14 for the asymptotic side, and rounding: 1e-13.
"""
import numpy as np
import pytest

from hfscf_b200 import basis as B
from hfscf_b200 import engine as E
from hfscf_b200 import molecules as M

pytestmark = pytest.mark.gpu


def _basis(kind, n, name):
    rng = np.random.default_rng(41)
    if kind == "water":
        Z, x = M.water_cluster(n, 2.9, rng, 0.1)
    elif kind == "alkane":
        Z, x = M.n_alkane(n) if n > 1 else M.methane()
    else:
        Z, x = [1, 1], [[0.0, 0.0, 0.0], [0.0, 0.1, 0.74]]
    x = np.asarray(x) * B.ANGSTROM_TO_BOHR
    return B.build_basis(name, Z, x, pure=name == "cc-pvdz")


def _density(rng, n):
    A = rng.normal(size=(n, n))
    return (A + A.T) / n


# one class only; one long primitive loop; both sides of the small builds' line, on both kinds of shells
CASES = [("h2", 2, "sto-3g"), ("water", 1, "cc-pvdz"), ("alkane", 1, "6-31g**"), ("alkane", 3, "6-31g**"),
         ("water", 5, "cc-pvdz"), ("water", 6, "cc-pvdz")]


@pytest.mark.parametrize("precision", [E.FP64, E.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("case", CASES, ids=["-".join(map(str, c)) for c in CASES])
def test_jk_forms_by_size_match_one_thread_per_quartet(case, precision):
    bs = _basis(*case)
    rng = np.random.default_rng(43)
    D, Db = _density(rng, bs.nbf), _density(rng, bs.nbf)
    for density_tol in (0.0, 1e-9):
        with E.Engine(bs, density_tol=density_tol) as eng:
            got = [eng.jk(D, [D, Db], precision), eng.jk(1e-4 * D, [1e-4 * D], precision)]
            eng.set_schedule(np.tile(np.array((64, 0, 0, 0), dtype=np.int32), (E.NUM_CLASSES, 1)))
            want = [eng.jk(D, [D, Db], precision), eng.jk(1e-4 * D, [1e-4 * D], precision)]
        for (J, K), (J0, K0) in zip(got, want):
            for a, b in [(J, J0), *zip(K, K0)]:
                tol = 1e-11 * np.max(np.abs(b)) if precision == E.FP64 else 1e-6
                assert np.max(np.abs(a - b)) < tol


@pytest.mark.parametrize("case", CASES[:4], ids=["-".join(map(str, c)) for c in CASES[:4]])
def test_derivative_forms_by_size_match_thread_forms(case):
    bs = _basis(*case)
    D = _density(np.random.default_rng(47), bs.nbf)
    with E.Engine(bs) as eng:
        g, H = eng.grad2e(D), eng.hess2e(D)
        eng.set_hess_form(0)
        H0 = eng.hess2e(D)
    with E.Engine(bs, grad_warp_max_waves=0) as eng:
        g0 = eng.grad2e(D)
    assert np.max(np.abs(g - g0)) < 1e-10
    assert np.max(np.abs(H - H0)) < 1e-9


TMAX = [36, 38, 40, 45, 45, 50, 50, 53, 53, 56, 56]   # end of the polynomials by order


@pytest.mark.parametrize("m", range(11))
def test_boys_rows_at_interval_edges(m):
    k = np.arange(0, TMAX[m] * 16, 7)
    h = 1 / 32
    T = np.concatenate([k / 16, k / 16 + h, np.nextafter(k / 16 + h, 0), np.nextafter(k / 16 + h, 99), [0.0, 5e-324, 1e-9],
                        np.nextafter(TMAX[m], [0, 99]), [TMAX[m], TMAX[m] + h, 80.0]])
    with E.Engine(_basis(*CASES[0])) as eng:
        F = eng.boys(m, T)
    t = T.astype(np.longdouble)
    for n in range(m + 1):
        term = np.full_like(t, 1 / np.longdouble(2 * n + 1))
        ref = term.copy()
        for i in range(400):
            term = term * 2 * t / (2 * n + 2 * i + 3)
            ref += term
        ref *= np.exp(-t)
        assert np.max(np.abs(F[:, n] - ref) / ref) < 1e-13
