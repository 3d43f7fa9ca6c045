"""The double-float roofline record of bench.py: issue and busy fractions of the FMA pipe under
names of their own, and a rate that counts the operations of all it names."""
import importlib.util
import os

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_module", os.path.join(ROOT, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_two_quantities_two_names(bench):
    r = bench.df_roofline(1.6e8, 62.0, 4.0e6, 152, 2070.0, True)
    issue, busy = r["fma_pipe_issue_frac_ncu"], r["fma_pipe_busy_frac_ncu"]
    assert set(issue) == set(busy) == {"start_up", "main", "few"}
    for k in issue:  # a pair's instruction keeps the pipe for two cycles
        assert 0 < issue[k] < busy[k] < 2 * issue[k]


def test_rate_counts_operations(bench):
    r = bench.df_roofline(1.6e8, 62.0, 4.0e6, 152, 2070.0, True)
    assert "operations" in r["unit"] and "instructions" not in r["unit"] and "k_integrate_df_few" in r["kernel"]
    assert r["achieved"] == pytest.approx(1.6e8 * r["fp32_ops_per_step_attempt"] / 62.0e-3 / 1e12)
    assert r["peak"] == pytest.approx(152 * 128 * 2070e6 / 1e12)
    assert bench.df_roofline(1.6e8, 62.0, 4.0e6, 152, 2070.0, False)["achieved"] is None


def test_fp64_time_is_of_a_warm_run(bench):
    """The first FP64 run loads its kernels; the speed the others are compared with does not
    count that."""
    class Job:
        dimension, final_p_num, traj_rtol, precision = 1, [100], 1e-6, "fp64"

        def copy(self):
            return Job()

    class Result:
        num_effective_traj, ion_prob = 1000, 0.5

    class Engine:
        runs = 0

        def run(self, job, want_spectrum=True):
            Engine.runs += 1
            r = Result()
            r.elapsed_ms = 20.0 if Engine.runs == 1 else 5.0
            return r, np.ones(100) if want_spectrum else None, None

    out = bench.accuracy_report(Engine(), Job(), Job())
    assert out["fp64_plain"]["ms_per_step"] == 5.0 and out["fp64_plain"]["value"] == 1000 / 5.0e-3
