"""Native tests of the renderer's host runtime on a fake CUDA runtime (no GPU)."""
import pytest
from test_native_host import test_native as _run


@pytest.mark.parametrize("name", ["draw_stream_test", "step_graphs_test", "plain_items_test", "tuning_test", "queue_fill_test", "work_items_plan_test", "two_streams_test"])
def test_renderer_runtime(name, tmp_path):
    _run(name, tmp_path)
