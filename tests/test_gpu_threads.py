"""Two handles on two host threads: a kernel's attributes belong to the kernel, so what one handle's launch
sets must suit the other's.  Gradients of molecules of different size, or the batched eigensolver and
purification, run in loops at the same time; every call succeeds, and gradients agree with the same call
alone (1e-10, the summation order of the atomic adds).
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


def test_batched_linear_algebra_of_two_handles_on_two_threads():
    import torch

    from hfscf_b200 import batch
    cases = []
    for carbons in (2, 3):  # 60 and 85 functions: both kernels above 48 KB of shared memory, in different size
        bs = _case(carbons)[0]
        n = bs.nbf
        A = np.random.default_rng(carbons).normal(size=(n, n))
        cases.append((batch.BatchEngine([bs]), torch.from_numpy((A + A.T) / 2).cuda().reshape(1, n, n).contiguous(),
                      torch.empty((1, n), dtype=torch.float64, device="cuda"),
                      torch.empty((1, n, n), dtype=torch.float64, device="cuda"),
                      torch.tensor([n // 3], dtype=torch.int32, device="cuda"),
                      torch.empty(1, dtype=torch.float64, device="cuda")))
    torch.cuda.synchronize()
    failures = []
    start = threading.Barrier(len(cases))

    def loop(be, A, W, V, nocc, err):
        start.wait()
        try:
            for _ in range(400):
                be.eigh(A, W, V)
                be.purify(A, nocc, V, err)
        except E.HfgpuError as e:
            failures.append(str(e))

    threads = [threading.Thread(target=loop, args=c) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for c in cases:
        c[0].close()
    assert not failures, failures
