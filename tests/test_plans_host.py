"""Context buffers, graph keys and launch plans without a GPU (csrc/plan_tests.cpp)."""
import subprocess

from conftest import PKG_DIR


def test_plan_tests_binary(cmc):
    subprocess.run(["make", "-C", str(PKG_DIR), "-j4"], check=True, stdout=subprocess.DEVNULL)
    r = subprocess.run([str(PKG_DIR / "plan_tests")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr + r.stdout
    assert "ALL PLAN TESTS PASSED" in r.stdout
