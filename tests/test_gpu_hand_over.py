"""The last electrons of an FP64 or a double-float job leave the kernel with one electron per
lane whatever warp they are in.  It takes two to three times as long per attempt as the kernel
they go to, so a warp that kept its slow electrons would show in the time of the call."""
import time

import numpy as np
import pytest
import torch

import etraj_gb300 as et

pytestmark = pytest.mark.gpu


def timed(eng, job, init):
    """(least time of three calls, the result of one before them)"""
    out, took = eng.integrate(job, init), []
    for _ in range(3):
        t = time.perf_counter()
        eng.integrate(job, init)
        took.append(time.perf_counter() - t)
    return min(took), out


@pytest.mark.parametrize("precision,slower", [("fp64", 1.8), ("fp32_df", 1.4)])
@pytest.mark.parametrize("slow", [28, 30, 31, 32])
def test_slow_electrons_of_one_warp(slow, precision, slower):
    """`slow` electrons that circle the core among one warp's 32, in a job whose others are far
    from it; against the same 32 alone, all in the second kernel."""
    L = et.Cos4Laser(peak_int=1e10, wave_len=800.0, cyc_num=2, ellip=1.0)
    T = L.Period()
    job = et.make_job(init_cond_method="ADK", laser=L, target=et.get_atom("H"), dimension=2, sample_t_intv=(-T, T),
                      sample_t_num=10, traj_t_final=3 * T, final_p_max=(1.5, 1.5), final_p_num=(32, 32), ss_kd_max=1.0,
                      ss_kd_num=9, traj_phase_method="CTMC", seed=1, precision=precision)
    n = 256 * torch.cuda.get_device_properties(0).multi_processor_count  # every warp's first electrons are all there are
    init = np.zeros((n, job.rows))
    init[:, 0] = 1e4 + np.arange(n)
    init[:, 4] = -T
    init[:, 5] = 1e-3
    r = 0.5 + 0.001 * np.arange(slow)
    init[:slow, 0] = r
    init[:slow, 3] = 1.0 / np.sqrt(r)
    eng = et.Engine(device=0)
    few, (f0, s0, n0) = timed(eng, job, init[:32])
    rest, _ = timed(eng, job, init[32:])
    many, (f1, s1, n1) = timed(eng, job, init)
    eng.close()
    assert np.array_equal(f1[:32], f0) and np.array_equal(n1[:32], n0) and np.array_equal(s1[:32], s0)
    assert n0[:slow].min() > 2000 and n1[slow:].max() < 200
    # the others take a few attempts, so the slow ones leave almost at once; kept to their end by
    # the first kernel they would take about three times `few` (FP64), or twice (double-float);
    # `slower` is half-way on a logarithmic scale
    assert many < slower * few + rest
