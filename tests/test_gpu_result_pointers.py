"""Result pointers of the C entry points that the Python layer does not combine: a CTMC job
with an amplitude array gets its real sums in the real halves (they are as many doubles as
bins, half of what a coherent job's amplitude takes)."""
import ctypes as C

import numpy as np
import pytest

import etraj_gb300 as et
from etraj_gb300 import abi
from test_gpu_parity import job_of, same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_FP32_DF, abi.PRECISION_FP32_BULK])
@pytest.mark.parametrize("empty", [False, True])
def test_amplitude_pointer_of_a_ctmc_job(precision, empty):
    job = job_of(phase="CTMC", ellip=1.0, pnum=(33, 31), cutoff=1e3 if empty else 1e-16)
    job.precision = precision
    eng = et.Engine(device=0)
    spec, amp = np.full(job.grid_size, 7.0), np.full(2 * job.grid_size, 7.0)
    res = abi.Result()
    res.momentum_spec, res.amplitude = abi.dptr(spec), abi.dptr(amp)
    assert eng.lib.etraj_run(eng.ctx, C.byref(job), C.byref(res)) == abi.OK
    r, s, _ = eng.run(job)
    assert (r.num_effective_traj == 0) == empty and (s.sum() == 0.0) == empty
    assert same_bits(spec, s) and same_bits(amp[0::2].copy(), s) and not amp[1::2].any()
    eng.close()
