"""The FEM assembly takes the faster of its two forms, on the host."""
from test_split_launch import run_host_test


def test_rule_takes_the_faster_form(tmp_path):
    run_host_test(tmp_path, "test_fem_rule")
