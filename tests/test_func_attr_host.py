"""Kernel settings that apply to one device at a time
(curfp_b200/csrc/func_attr.h): every device gets them on its first use, and a
failure is not remembered.  No GPU needed: the setter is a stand-in."""
import ctypes
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "curfp_b200" / "csrc"
OK, RAN = 1, 2


def calls(hs, devices, fail_at=-1):
    out = (ctypes.c_int * len(devices))()
    assert hs.hs_once_per_device(len(devices), (ctypes.c_int * len(devices))(*devices), fail_at,
                                 out) == 0
    return list(out)


def test_every_device_is_set_once(hostsim):
    assert calls(hostsim, [0, 0, 3, 0, 63, 3]) == [OK + RAN, OK, OK + RAN, OK, OK + RAN, OK]
    assert calls(hostsim, [64, 64]) == [OK + RAN, OK + RAN]


def test_failure_is_tried_again(hostsim):
    assert calls(hostsim, [0, 0, 0], fail_at=0) == [RAN, OK + RAN, OK]
    assert calls(hostsim, [0, 1, 1, 0], fail_at=1) == [OK + RAN, RAN, OK + RAN, OK]


def test_no_launch_remembers_the_setting_for_the_process():
    for src in CSRC.glob("*.cu"):
        assert "cudaFuncSetAttribute" not in src.read_text(), src.name
