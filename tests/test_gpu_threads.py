"""Several host threads, each with a context of its own, in the same kernels at
different sizes (GPU)."""
import threading

import numpy as np
import pytest

from mbx_b200 import capi, system as msys, workloads
from mbx_b200.specs import SPECS

pytestmark = pytest.mark.gpu


def together(*bodies):
    """Runs the bodies on threads of their own; raises what any of them raised."""
    errors, start = [], threading.Barrier(len(bodies))

    def guarded(body):
        try:
            start.wait()
            body()
        except Exception as e:   # reported by the test's thread
            errors.append(e)

    threads = [threading.Thread(target=guarded, args=(b,)) for b in bodies]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def nmers(name, n):
    rng = np.random.default_rng(n)
    parts = []
    for k, m in enumerate(SPECS[name].monomers):
        v = rng.normal(size=(n, 3))
        r = rng.uniform(3.0, 5.0, size=n) * (k > 0)
        parts.append(workloads.place(rng, workloads.BODIES[m](), v / np.linalg.norm(v, axis=1, keepdims=True) * r[:, None]))
    return np.ascontiguousarray(np.concatenate(parts, 1).reshape(n, -1))


def test_fits_of_two_evaluators():
    """The coefficient adjoint's shared memory: 50 KB (MB-pol 3b) and 101 KB
    (CH4-CH4) a block."""
    import torch
    calls = 4000

    def fit(name):
        c = capi.Context(0)
        x = torch.tensor(nmers(name, 8), device="cuda")
        first = torch.tensor(c.evaluate_dcoef(name, x.cpu().numpy()), device="cuda")
        out = torch.zeros_like(first)

        def body():
            for _ in range(calls):
                c.evaluate_dcoef(name, x, None, out)
            torch.cuda.synchronize()
            # a sum of equal values, rounded at every addition
            assert torch.all(torch.abs(out - calls * first) <= calls ** 2 * 2.0 ** -53 * torch.abs(first))
        return body

    together(*[fit(name) for name in ("mbpol3b", "ch4ch42b", "mbpol3b", "ch4ch42b")])


def test_searches_of_two_sizes():
    """The match staging of the neighbour search: 72 and 130 KB a block."""
    def search(n):
        side = int(np.ceil((1.3 * n) ** (1 / 3)))
        ids, xyz, _ = workloads.water_box(side, n, 39.44 * (n / 2048) ** (1 / 3), seed=n)
        s = msys.from_arrays(ids, xyz, None, 400.0, 4.0)
        first = s.TwoBodyEnergy(False)

        def body():
            for _ in range(150):
                e = s.TwoBodyEnergy(False)
                assert abs(e - first) <= 1e-10 * abs(first)
                assert s.NmerCounts(2)[0] == n * (n - 1) // 2
        return body

    together(search(1100), search(2000))
