"""The benchmark's printed line: every key of the metric, short enough to survive
in the last few thousand characters of a log, whatever the whole result holds;
that goes to a file."""
import json

import bench


def full_result():
    trials = [dict(threads=512, region_width=128, region_height=64, raster_ms=1.2345678901234567)] * 60
    e2e = dict(value=385432.123456789, unit="frames/s", h2d_bytes_per_step=98304, d2h_bytes_per_step=201326592,
               ms_per_step=2.65, call_ms=[0.123] * 100, timing="host clock " * 30)
    roof = dict(bound="hbm", achieved=150.0, peak=6782.8, unit="GB/s", frac=0.022, issue_active_frac=0.65,
                avg_launch_ms=1.5, issue_note="note " * 30, bytes_breakdown=dict(a=1, b=2))
    parity = dict(envs_checked=64, pixels=1 << 20, mismatched_pixels=0, max_linear_depth_err_m=0.0,
                  depth_tolerance_m=1e-4)
    block = dict(value=123456.7890123, e2e=e2e, plain=dict(value=1.0, ms_per_step=2.0, form="form " * 20), roofline=roof,
                 parity=parity, autotune=dict(trials=trials))
    return dict(metric=bench.METRIC, value=650000.123, unit="frames/s", n_gpus=1, steps=20, warmup=5, ms_per_step=1.57,
                p50_ms=1.57, p99_ms=1.6, higher_is_better=True, scaling="weak", vs_baseline=None, dtype="f32",
                data="synthetic",
                config=dict(workload=bench.WORKLOADS["config1"], envs=1024, resolution=[128], planes=bench.PLANES),
                details=dict(form="batched: prepare + persistent raster per step, CUDA graph", l2="flushed " * 8,
                             autotune=dict(trials=trials)),
                plain=block["plain"], batched_over_plain=1.2, e2e=e2e, roofline=roof, gpu_launches=60,
                clocks=dict(sm_mhz=2070.0, sm_max_mhz=2070.0, reasons=[], samples=99), parity=parity,
                cpu_baseline=dict(value=1252.0, unit="frames/s", cores=16, cpu_model="model " * 10),
                configs=dict(config0=block, config2=block, config3=block),
                serving=dict(saturation=dict(requests_per_s=250000.0, steps=1), sweep=[dict(trials[0])] * 10),
                replay=dict(value=200000.0, timing="t " * 50), postprocess=dict(hbao=block))


def test_printed_line_is_short_and_complete(tmp_path):
    full = full_result()
    path = tmp_path / "d.json"
    stored = bench.write_details(full, str(path))
    line = bench.headline(full, stored)
    text = json.dumps(line)
    assert len(text) < 2600 and "\n" not in text
    assert json.loads(path.read_text()) == json.loads(json.dumps(full)) and line["details"] == "d.json"
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "clocks", "gpu_launches"):
        assert line[k] == full[k], k
    assert line["l2"] == full["details"]["l2"]
    assert line["e2e"] == {k: full["e2e"][k] for k in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step",
                                                       "ms_per_step")}
    assert set(line["configs"]) == {"config0", "config2", "config3"}


def test_legs_that_were_left_out(tmp_path):
    full = full_result()
    full.update(plain=None, e2e=None, parity=None, cpu_baseline=None, configs={}, serving=None, replay=None,
                postprocess=None)
    line = bench.headline(full, bench.write_details(full, "none"))
    assert line["value"] == full["value"] and line["e2e"] is None and line["serving"] is None
    assert bench.write_details(full, str(tmp_path / "missing" / "d.json")) is None
