"""The thread-triple forms of the derivative kernels (ten triples per quartet where quartets are few, one where
they are many) against values that do not run them: gradients against the CPU oracle, Hessians against the
op tables, each with one and two exchange densities and without a Coulomb density, whole and in parts
(whose shorter lists change a class from one triple per quartet to ten).

1e-10 and 1e-9 as in test_gpu_parity and test_gpu_hessian.
"""
import numpy as np
import pytest

import oracle
from hfscf_b200 import basis as B
from hfscf_b200 import engine as E
from hfscf_b200 import molecules as M

pytestmark = pytest.mark.gpu


def _basis(kind, n, name):
    if kind == "water":
        Z, x = M.water_cluster(n, 2.9, np.random.default_rng(41), 0.1)
    elif kind == "alkane":
        Z, x = M.n_alkane(n) if n > 1 else M.methane()
    else:
        Z, x = [1, 1], [[0.0, 0.0, 0.0], [0.0, 0.1, 0.74]]
    return B.build_basis(name, Z, np.asarray(x) * B.ANGSTROM_TO_BOHR, pure=name == "cc-pvdz")


def _densities(n, seed):
    rng = np.random.default_rng(seed)
    A, C = rng.normal(size=(2, n, n))
    return (A + A.T) / n, (C + C.T) / n


def _derivative(eng, order, DJ, DKs):
    """Order 1: gradient, 2: Hessian, with cJ = 2 and cK = 1, on device matrices."""
    import torch
    dj = torch.from_numpy(DJ).cuda() if DJ is not None else None
    dk = torch.from_numpy(np.stack(DKs)).cuda()
    n = eng.basis.natoms
    out = torch.zeros((n, 3) if order == 1 else (3 * n, 3 * n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    call = eng.grad2e_device if order == 1 else eng.hess2e_device
    stream = torch.cuda.Stream()
    eng.set_stream(stream.cuda_stream)
    call(dj.data_ptr() if dj is not None else 0, 2.0, len(DKs), dk.data_ptr(), 1.0, out.data_ptr())
    torch.cuda.synchronize()
    eng.set_stream(None)
    return out.cpu().numpy()


def _weights(kind, n):
    D, Db = _densities(n, 47)
    return {"rhf": (D, [D]), "uhf": (D + Db, [D, Db]), "exchange": (None, [D])}[kind]


@pytest.mark.parametrize("weights", ["rhf", "uhf", "exchange"])
@pytest.mark.parametrize("case", [("h2", 2, "sto-3g"), ("water", 1, "cc-pvdz"), ("water", 1, "6-31g**"),
                                  ("alkane", 1, "6-31g**")], ids=lambda c: "-".join(map(str, c)))
def test_gradients_of_small_molecules_match_the_oracle(case, weights):
    bs = _basis(*case)
    DJ, DKs = _weights(weights, bs.nbf)
    want = oracle.grad2e(bs, np.zeros((bs.nbf, bs.nbf)) if DJ is None else DJ, 0.0 if DJ is None else 2.0, DKs, 1.0)
    with E.Engine(bs) as eng:
        got = _derivative(eng, 1, DJ, DKs)
    assert np.max(np.abs(got - want)) < 1e-10


@pytest.mark.parametrize("weights", ["rhf", "uhf", "exchange"])
@pytest.mark.parametrize("case", [("water", 2, "6-31g**"), ("alkane", 3, "6-31g**"), ("alkane", 3, "cc-pvdz")],
                         ids=lambda c: "-".join(map(str, c)))
@pytest.mark.parametrize("order", [1, 2], ids=["gradient", "hessian"])
def test_whole_lists_match_the_sum_of_their_parts(case, weights, order):
    bs = _basis(*case)
    DJ, DKs = _weights(weights, bs.nbf)
    parts = 48
    with E.Engine(bs) as eng:
        whole = _derivative(eng, order, DJ, DKs)
        total = np.zeros_like(whole)
        for p in range(parts):
            eng.set_partition(p, parts)
            total += _derivative(eng, order, DJ, DKs)
        eng.set_partition(0, 1)
        if order == 2:
            eng.set_hess_form(0)
            assert np.max(np.abs(whole - _derivative(eng, 2, DJ, DKs))) < 1e-9
    assert np.max(np.abs(whole - total)) < (1e-10 if order == 1 else 1e-9)
