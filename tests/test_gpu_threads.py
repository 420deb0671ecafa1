"""Several host threads read arrays and states of one handle at once: each gets what it gets alone
(ocfd_get_array and ocfd_get_state pass through one staging area of the handle)."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
def test_reads_from_several_threads(gpu, prec):
    from ocfd_b200 import cases
    p, case = cases.config2_small(precision=prec)
    s = gpu.Solver(p, case)
    s.advance(2)
    s.synchronize()
    jobs = [(b, name) for b in range(s.nblk) for name in ("U", "Res", "DU", "mu", "vol", "ni1", "state")]

    def read(job):
        b, name = job
        return s.get_state(b) if name == "state" else s.get_array(b, name)[0]

    alone = [read(j) for j in jobs]
    with ThreadPoolExecutor(8) as pool:
        for got in (list(pool.map(read, jobs)) for _ in range(20)):
            for x, y, j in zip(got, alone, jobs):
                assert np.array_equal(x, y), j
    s.close()


def test_reads_beside_the_first_step(gpu):
    """The first step is captured into a graph; an array that does not change, read by another thread all
    the while, is right and leaves the step as it is."""
    from ocfd_b200 import cases
    p, case = cases.config2_small()
    ref = gpu.Solver(p, case)
    ref.advance(3)
    for _ in range(5):
        s = gpu.Solver(p, case)
        vol = s.get_array(0, "vol")[0]
        with ThreadPoolExecutor(2) as pool:
            reads = [pool.submit(lambda: s.get_array(0, "vol")[0]) for _ in range(40)]
            s.advance(3)
            assert all(np.array_equal(r.result(), vol) for r in reads)
        assert s.launches_per_step() == ref.launches_per_step()
        for b in range(s.nblk):
            assert np.array_equal(s.get_state(b), ref.get_state(b))
        s.close()
    ref.close()
