"""Two handles on two host threads: a kernel's attributes belong to the kernel, so what one handle's launch
sets must suit the other's.  Gradients of molecules of different size run in loops at the same time; every
call succeeds and agrees with the same call alone (1e-10, the summation order of the atomic adds).
"""
import threading

import numpy as np
import pytest

from hfscf_b200 import basis as B
from hfscf_b200 import engine as E
from hfscf_b200 import molecules as M

pytestmark = pytest.mark.gpu


def _case(carbons):
    Z, x = M.n_alkane(carbons) if carbons > 1 else M.methane()
    bs = B.build_basis("6-31g**", Z, np.asarray(x) * B.ANGSTROM_TO_BOHR)
    A = np.random.default_rng(carbons).normal(size=(bs.nbf, bs.nbf))
    return bs, (A + A.T) / bs.nbf


def test_gradients_of_two_handles_on_two_threads():
    cases = [_case(1), _case(2), _case(4)]
    engines = [E.Engine(bs) for bs, _ in cases]
    try:
        alone = [eng.grad2e(D) for eng, (_, D) in zip(engines, cases)]
        failures = []
        start = threading.Barrier(len(cases))

        def loop(k):
            start.wait()
            for _ in range(400):
                try:
                    g = engines[k].grad2e(cases[k][1])
                except E.HfgpuError as e:
                    failures.append((k, str(e)))
                    return
                if np.max(np.abs(g - alone[k])) > 1e-10:
                    failures.append((k, "value"))
                    return

        threads = [threading.Thread(target=loop, args=(k,)) for k in range(len(cases))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not failures, failures
    finally:
        for eng in engines:
            eng.close()
