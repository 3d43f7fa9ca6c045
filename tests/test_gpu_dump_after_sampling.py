"""The final states a context keeps of its last job stay as they are while initial conditions
are sampled on the same context."""
import numpy as np
import pytest

import etraj_gb300 as et
from test_gpu_parity import job_of, same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["ADK", "SPANE", "SPA"])
def test_sampling_leaves_kept_states(method):
    job = job_of(method="SPANE", laser="cos2", ellip=1.0, phase="SCTS", nt=24)
    other = job_of(method=method, nt=6, nkd=5)  # fewer electrons, so that a dump by its count is short
    eng = et.Engine(device=0)
    eng.keep_final_states(True)
    r, _, _ = eng.run(job)
    n = r.num_effective_traj
    before = eng.dump_final_states(n) + (eng.dump_step_counts(n), eng.dump_min_radius(n))
    assert n > 50 and before[3].min() > 0
    assert len(eng.sample_all(other)) < n
    eng.sample_batch(other, 3)
    after = eng.dump_final_states(n) + (eng.dump_step_counts(n), eng.dump_min_radius(n))
    for a, b in zip(before, after):
        assert same_bits(a, b)
    eng.close()
