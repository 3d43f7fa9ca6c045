"""A whole FP64 run's values, electron by electron, against the oracle's solve of the same
initial conditions: a run keeps no final-state buffer, so the states pass through the sample
arrays and a 3D z through the contributions, and the larger job's last electrons change
kernels on the way.  Tolerance: none, every bit."""
import numpy as np
import pytest
import torch

import _oracle as O
import etraj_gb300 as et
from test_gpu_parity import job_of, same_bits

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = et.Engine(device=0)
    yield e
    e.close()


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("nt", [40, 1200])
@pytest.mark.parametrize("dim,phase,target", [(2, "CTMC", "H"), (2, "SCTS", "Ar"), (3, "QTMC", "H"), (3, "SCTS", "Ar")])
def test_run_against_the_oracle(eng, dim, phase, target, nt):
    job = job_of(method="SPANE", dim=dim, phase=phase, target=target, nt=nt, nkd=21, nkz=3, laser="cos2",
                 ellip=1.0 if dim == 2 else 0.5)
    eng.keep_final_states(True)
    try:
        res, spec, amp = eng.run(job, want_amplitude=phase != "CTMC")
        n = res.num_effective_traj
        p_inf, ph, st = eng.dump_final_states(n)
        steps, rmin = eng.dump_step_counts(n), eng.dump_min_radius(n)
    finally:
        eng.keep_final_states(False)
    # 48 electrons per SM: below, the second kernel alone; above, both
    assert (n > 48 * sms()) == (nt == 1200)
    init = O.sample_all(job)
    assert len(init) == n
    fin, status, counts, least = O.integrate_rmin(job, init)
    rspec, ramp, _, rp, _ = O.collect(job, init, fin, status, counts)
    assert np.array_equal(st & 0xff, status) and np.array_equal(steps, counts)
    assert same_bits(rmin, least) and same_bits(p_inf, rp) and same_bits(spec, rspec)
    if phase == "CTMC":
        return
    assert same_bits(amp, ramp)
    if phase == "QTMC":  # (SCTS adds the post-pulse term, seen through the contributions)
        ok = status == 0
        assert same_bits(ph[ok], fin[ok, -1])
    key, cre, cim = O.contributions(job, init, fin, status)
    hit = key < job.grid_size
    assert hit.sum() > n // 2
    w = np.sqrt(init[hit, 2 * dim + 1])
    assert same_bits(w * O.detmath("cos", ph[hit]), cre[hit]) and same_bits(w * O.detmath("sin", ph[hit]), cim[hit])


def edges():
    """Around each bound of the FP64 launches: 48 electrons per SM, two warps per sub-partition
    (8 warps of 32 per SM), and all lanes (five blocks of 128 per SM, or four)."""
    m = sms() if torch.cuda.is_available() else 1
    return [48 * m - 1, 48 * m, 48 * m + 1, 256 * m, 256 * m + 1, 512 * m, 512 * m + 1, 640 * m, 640 * m + 1]


@pytest.mark.parametrize("dim,phase,target", [(2, "SCTS", "Ar"), (3, "QTMC", "H")])
def test_electron_counts_around_every_bound(eng, dim, phase, target):
    job = job_of(method="SPANE", dim=dim, phase=phase, target=target, nt=60, nkd=21, nkz=5, laser="cos2",
                 ellip=1.0 if dim == 2 else 0.5)
    init = O.sample_all(job)
    ref, rs, rn = O.integrate(job, init)
    for n in edges():
        k = np.arange(n) % len(init)
        fin, st, steps = eng.integrate(job, init[k])
        assert same_bits(fin, ref[k]) and np.array_equal(st, rs[k]) and np.array_equal(steps, rn[k]), n
