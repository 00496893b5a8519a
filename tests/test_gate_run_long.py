"""Grouping a plan's gates takes time in proportion to their number
(tests/cpp/gate_run_long_check.cpp)."""
from test_host_logic import _link_against_library, gxx  # noqa: F401


def test_long_plans_are_grouped_in_linear_time(gxx, tmp_path):  # noqa: F811
    import subprocess
    r = subprocess.run([_link_against_library(gxx, tmp_path, "gate_run_long_check")], capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0 and r.stdout.splitlines()[-1] == "bad 0", r.stdout
