"""The tile-pass model counts the SMs of its device (tests/cpp/gate_run_sms_check.cpp)."""
from test_host_logic import _link_against_library, _run, gxx  # noqa: F401


def test_tile_passes_are_chosen_for_the_devices_sms(gxx, tmp_path):  # noqa: F811
    out = _run(_link_against_library(gxx, tmp_path, "gate_run_sms_check"))
    assert out.startswith("bad 0"), out
