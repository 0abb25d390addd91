"""What hfgpu_autotune_hess keeps is not slower than the defaults it started from: they are among the forms
that it times.  Device time of whole Hessians (median of seven); classes that were timed alone share
the GPU here, so a quarter more is allowed.  Without the three-thread form of the defaults to choose, tuning
made these Hessians take 1.4 and 1.5 times as long.
"""
import numpy as np
import pytest

from hfscf_b200 import basis as B
from hfscf_b200 import engine as E
from hfscf_b200 import molecules as M

pytestmark = pytest.mark.gpu


def _ms(eng, D):
    import torch
    n3 = 3 * eng.basis.natoms
    H = torch.zeros(n3, n3, dtype=torch.float64, device="cuda")
    stream = torch.cuda.Stream()
    eng.set_stream(stream.cuda_stream)
    times = []
    for _ in range(8):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        e0.record(stream)
        eng.hess2e_device(D.data_ptr(), 2.0, 1, D.data_ptr(), 1.0, H.data_ptr())
        e1.record(stream)
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1))
    eng.set_stream(None)
    return float(np.median(times[1:]))


@pytest.mark.parametrize("name,carbons", [("6-31g**", 6), ("cc-pvdz", 4)])
def test_tuned_hessian_is_not_slower_than_the_default(name, carbons):
    import torch
    Z, x = M.n_alkane(carbons)
    bs = B.build_basis(name, Z, np.asarray(x) * B.ANGSTROM_TO_BOHR, pure=name == "cc-pvdz")
    A = np.random.default_rng(3).normal(size=(bs.nbf, bs.nbf))
    D = torch.from_numpy((A + A.T) / bs.nbf).cuda()
    with E.Engine(bs) as eng:
        default = _ms(eng, D)
        forms = eng.autotune_hess(D, repeats=3)
        tuned = _ms(eng, D)
        eng.set_hess_forms(forms)
        again = _ms(eng, D)
    print(forms, default, tuned, again)
    assert tuned < 1.25 * default
    assert again < 1.25 * default
