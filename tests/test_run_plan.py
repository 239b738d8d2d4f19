"""The rules by which a run's kernels wait for their peers, on the host: none
beside a lane's run, each form where its CTAs are resident together."""
from test_split_launch import run_host_test


def test_run_plan(tmp_path):
    run_host_test(tmp_path, "test_run_plan")
