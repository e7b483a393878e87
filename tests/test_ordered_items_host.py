"""Native test of the work items that the device orders (no GPU)."""
from test_native_host import test_native as _run


def test_work_items_for_the_device_to_order(tmp_path):
    _run("work_items_ordered_test", tmp_path)
