"""The double-float roofline record of bench.py: issue and busy fractions of the FMA pipe under
names of their own, and a rate that counts the operations of all it names."""
import importlib.util
import os

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
