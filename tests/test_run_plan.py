"""The rules by which a run's kernels wait for their peers, on the host: none
beside a lane's run, each form where its CTAs are resident together, and the runs
of several contexts together only where all of them fit."""
import pytest

from test_split_launch import run_host_test


@pytest.mark.parametrize("name", ["test_run_plan", "test_gate"])
def test_rules(tmp_path, name):
    run_host_test(tmp_path, name)
