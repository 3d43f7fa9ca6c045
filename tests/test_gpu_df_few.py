"""The double-float integrator's main pass and its eight-lanes-per-electron kernel give an
electron the same bits: jobs of one electron to more than the hand-over bound (7,296 on 152
SMs) against the host build, for every state size and both target kinds."""
import numpy as np
import pytest

import etraj_gb300 as et
from etraj_gb300 import abi
from test_df_host import dfhost, host_integrate  # noqa: F401  (dfhost: fixture)
from test_gpu_parity import job_of

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = et.Engine(device=0)
    yield e
    e.close()


@pytest.mark.parametrize("dim,phase,target", [(2, "CTMC", "H"), (2, "SCTS", "Ar"), (2, "QTMC", "H"), (3, "CTMC", "Ar"),
                                              (3, "QTMC", "H"), (3, "SCTS", "Ar")])
def test_electron_counts_around_the_hand_over(eng, dfhost, dim, phase, target):  # noqa: F811
    job = job_of(method="SPANE", dim=dim, phase=phase, target=target, nt=40, nkd=15, nkz=5, laser="cos2",
                 ellip=1.0 if dim == 2 else 0.5)
    job.precision = abi.PRECISION_FP32_DF
    init = eng.sample_all(job)
    assert len(init) > 100
    # integrate places the field table at the earliest electron given, the first of every subset here
    ref, rs, rn = host_integrate(dfhost, job, init, tmin=float(init[:, 2 * dim].min()))
    for n in (1, 5, len(init), 7296, 7297, 30000):
        k = np.arange(n) % len(init)
        fin, st, steps = eng.integrate(job, init[k])
        assert np.array_equal(fin, ref[k]) and np.array_equal(st, rs[k]) and np.array_equal(steps, rn[k]), n
