"""Time samples outside a cos^n pulse, where the field is exactly zero: an exponential
rate of zero is kept when the cut-off is zero, and its rows carry the direction of a zero
field (atan2 of signed zeros), which the device takes from the same signs as the oracle."""
import numpy as np
import pytest

import _oracle as O
import etraj_gb300 as et

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = et.Engine(device=0)
    yield e
    e.close()


@pytest.mark.parametrize("laser", [et.Cos4Laser, et.Cos2Laser])
@pytest.mark.parametrize("ellip,azi", [(0.0, 0.0), (1.0, 0.0), (0.6, 0.7)])
@pytest.mark.parametrize("dim", [2, 3])
def test_samples_outside_the_pulse(eng, laser, ellip, azi, dim):
    L = laser(peak_int=1e14, wave_len=800.0, cyc_num=2, ellip=ellip, azi=azi)
    T = L.Period()
    job = et.make_job(init_cond_method="ADK", laser=L, target=et.get_atom("H"), dimension=dim,
                      sample_t_intv=(-1.9 * T, 1.9 * T), sample_t_num=41, traj_t_final=2.5 * T,
                      final_p_max=(1.5,) * dim, final_p_num=(32,) * dim, ss_kd_max=1.0, ss_kd_num=9,
                      ss_kz_max=1.0, ss_kz_num=3 if dim == 3 else 0, rate_prefix="Exp", sample_cutoff_limit=0.0,
                      traj_phase_method="SCTS", seed=1)
    ref = O.sample_all(job)
    assert (np.abs(ref[:, 2 * dim]) > 1.3 * T).sum() > 20  # rows of a zero field are there
    got = eng.sample_all(job)
    assert got.shape == ref.shape
    # every bit, but for the payloads of NaN
    assert np.all((got.view(np.uint64) == ref.view(np.uint64)) | (np.isnan(got) & np.isnan(ref)))
