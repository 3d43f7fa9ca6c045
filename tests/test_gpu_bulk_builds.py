"""The bulk integrator's builds -- a single job's first round and its later ones, a batch's, and
the two register budgets of each -- give an electron the same bits, for every dimension,
phase and kind of target: where an electron runs is a matter of scheduling alone."""
import numpy as np
import pytest

import etraj_gb300 as et
from etraj_gb300 import abi

pytestmark = pytest.mark.gpu
PHASES = {"CTMC": abi.PHASE_CTMC, "QTMC": abi.PHASE_QTMC, "SCTS": abi.PHASE_SCTS}


def job_for(dim, phase, target, seed):
    # 9.2 cycles of field table (512 pieces each): more than shared memory holds, so that the
    # later rounds use the build that reads the table ahead
    L = et.Cos2Laser(peak_int=1.5e14, wave_len=800.0, cyc_num=8, ellip=0.3)
    T = L.Period()
    return et.make_job(init_cond_method="ADK", laser=L, target=et.get_atom(target), dimension=dim,
                       sample_t_intv=(-4 * T, 2 * T), sample_t_num=60, traj_t_final=5.2 * T,
                       final_p_max=(2.0,) * dim, final_p_num=(60,) * 2 + (8,) * (dim - 2), sample_monte_carlo=True,
                       mc_kt_num=200, mc_kd_max=1.0, mc_kz_max=1.0 if dim == 3 else 0.0, traj_phase_method=phase,
                       seed=seed, precision="fp32_bulk")


@pytest.mark.parametrize("target", ["H", "Ar"])
@pytest.mark.parametrize("phase", sorted(PHASES))
@pytest.mark.parametrize("dim", [2, 3])
def test_every_build_gives_the_same_bits(dim, phase, target):
    jobs = [job_for(dim, phase, target, s) for s in (1, 2)]
    kind = abi.TARGET_HYDROGEN_LIKE if target == "H" else abi.TARGET_SAE
    amp = phase != "CTMC"
    ref = None
    for blocks in (2, 3):  # 256-thread blocks per SM: 128 and 85 registers a thread
        for chunk in (0, 16):  # one round, or rounds that electrons leave after 16, 256, 4096 steps
            e = et.Engine(device=0)
            e.set_straggler_repack(chunk > 0)
            for multi in (False, True):
                e.set_bulk_tile(dim, PHASES[phase], kind, 256, blocks, 4, multi=multi)
                if chunk:
                    e.set_bulk_step_chunk(dim, PHASES[phase], kind, chunk, multi=multi)
            e.keep_final_states(True)
            got = []
            for j in jobs:
                r, s, a = e.run(j, want_amplitude=amp)
                n = r.num_effective_traj
                p, f, st = e.dump_final_states(n)
                steps = e.dump_step_counts(n)
                assert n > 1000 and (steps > 256).sum() > 0
                got.append((r.num_steps, r.ion_prob, s, a, p, f, st, steps))
            e.keep_final_states(False)
            outs, _ = e.run_batch(jobs, want_spectrum=True, want_amplitude=amp)
            e.close()
            if ref is None:
                ref = got
            for g, q in zip(got, ref):
                for x, y in zip(g, q):
                    assert np.array_equal(x, y), (blocks, chunk)
            for (r, s, a), q in zip(outs, ref):
                assert r.num_steps == q[0] and r.ion_prob == q[1], (blocks, chunk)
                assert np.array_equal(s, q[2]) and (not amp or np.array_equal(a, q[3])), (blocks, chunk)
