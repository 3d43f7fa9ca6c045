"""The FP64 integrator's two kernels (one electron per lane; eight lanes per electron)
against the oracle, bit for bit, around the number of electrons where a job moves from
one to the other, for state sizes 4 to 7."""
import numpy as np
import pytest

import _oracle as O
import etraj_gb300 as et
from etraj_gb300 import abi
from test_gpu_parity import job_of

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = et.Engine(device=0)
    yield e
    e.close()


@pytest.mark.parametrize("dim,phase,target", [(2, "CTMC", "H"), (2, "SCTS", "Ar"), (3, "CTMC", "Ar"), (3, "QTMC", "H")])
def test_electron_counts_around_the_hand_over(eng, dim, phase, target):
    job = job_of(method="SPANE", dim=dim, phase=phase, target=target, nt=60, nkd=21, nkz=5, laser="cos2",
                 ellip=1.0 if dim == 2 else 0.5)
    init = O.sample_all(job)
    assert len(init) > 200
    ref, rs, rn = O.integrate(job, init)
    # the second kernel alone, then the first with a hand-over of all but a few, of half, and
    # of a small part of the electrons (7,296 is the bound on 152 SMs)
    for n in (1, 7, 9, len(init), 7296, 7297, 12000, 40000):
        k = np.arange(n) % len(init)
        fin, st, steps = eng.integrate(job, init[k])
        assert np.array_equal(fin, ref[k]) and np.array_equal(st, rs[k]) and np.array_equal(steps, rn[k]), n


@pytest.mark.parametrize("dim,phase", [(2, "SCTS"), (3, "QTMC")])
def test_whole_jobs_use_the_same_values(eng, dim, phase):
    """A run (no final-state buffer: the states go through the sample arrays) against the
    same electrons through integrate, few and many."""
    for nt in (40, 1200):
        job = job_of(method="SPANE", dim=dim, phase=phase, target="H", nt=nt, nkd=21, nkz=3, laser="cos2",
                     ellip=1.0 if dim == 2 else 0.5)
        eng.keep_final_states(True)
        res, _, _ = eng.run(job)
        n = res.num_effective_traj
        steps = eng.dump_step_counts(n)
        _, _, st = eng.dump_final_states(n)
        rmin = eng.dump_min_radius(n)
        eng.keep_final_states(False)
        init = eng.sample_all(job)
        assert len(init) == n
        fin, status, counts = eng.integrate(job, init)
        assert np.array_equal(counts, steps) and np.array_equal(status, st & 0xff)
        assert np.all(rmin <= np.sqrt((init[:, :dim] ** 2).sum(axis=1)) * (1 + 1e-15)) and np.all(rmin > 0)


@pytest.mark.parametrize("dim,phase,target", [(2, "SCTS", "Ar"), (3, "QTMC", "H")])
def test_electron_counts_around_blocks_in_step(eng, dim, phase, target):
    """Up to two warps per sub-partition (38,912 electrons on 152 SMs) the first kernel's warps
    run freely, above that a block's go in step; 97,281 are one more than all its lanes."""
    job = job_of(method="SPANE", dim=dim, phase=phase, target=target, nt=60, nkd=21, nkz=5, laser="cos2",
                 ellip=1.0 if dim == 2 else 0.5)
    init = O.sample_all(job)
    ref, rs, rn = O.integrate(job, init)
    for n in (38912, 38913, 97281):
        k = np.arange(n) % len(init)
        fin, st, steps = eng.integrate(job, init[k])
        assert np.array_equal(fin, ref[k]) and np.array_equal(st, rs[k]) and np.array_equal(steps, rn[k]), n
