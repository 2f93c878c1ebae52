"""A wait that ran out inside an int8 product is the status of the call it ran out in (tests/cpp/check_wait_status.cpp), and
stages with the int8 products off agree with them on."""
import subprocess

import pytest

from test_cpp_api import build

pytestmark = pytest.mark.gpu


def test_wait_status_is_reported_by_its_call(tmp_path):
    exe = build(str(tmp_path), "check_wait_status")
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip().endswith("OK")


def test_int8_products_off_agree(tmp_path):
    """What a stage does when an int8 workspace does not fit (tests/cpp/check_int8_off.cpp)."""
    exe = build(str(tmp_path), "check_int8_off")
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip().endswith("OK")
