"""Native test of the work items of small steps (no GPU)."""
from test_native_host import test_native as _run


def test_work_items_of_few_views(tmp_path):
    _run("work_items_few_test", tmp_path)
