"""Native test of the noise kernel's launch plan (no GPU)."""
from test_native_host import test_native as _run


def test_noise_plan(tmp_path):
    _run("noise_plan_test", tmp_path)
