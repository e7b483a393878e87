"""The autotuner's choice of the per-scene region, on a renderer that only keeps
its tuning (no GPU): the library's own region is among the candidates, so that
tuning never makes the per-scene form slower than leaving it alone."""
import pytest

import __graft_entry__ as graft


class Renderer:
    def __init__(self, own):
        self.set = {}
        self.own = own

    def tuning(self):
        return dict(threads=512, region_width=128, region_height=64, small_area=4, ctas_per_sm=2,
                    plain_region_width=self.own[0], plain_region_height=self.own[1], occlusion_culling=1,
                    queue_fill_percent=75) | self.set

    def setTuning(self, **kw):
        self.set.update(kw)

    def setKernelTiming(self, on):
        pass

    def sceneCount(self):
        return 1

    def sceneViewport(self, s):
        return (0, 0, 128, 128)


@pytest.mark.parametrize("own,best", [((64, 128), (64, 128)), ((64, 128), (16, 64)), ((16, 32), (16, 32))])
def test_plain_region(monkeypatch, tmp_path, own, best):
    graft.load_package()
    from habitat_sim_gb300 import autotune
    monkeypatch.setattr(autotune, "_time_batched", lambda r, poses, draws: float(r.tuning()["threads"] != 512))
    tried = []

    def plain(r, poses, draws):
        t = r.tuning()
        tried.append((t["plain_region_width"], t["plain_region_height"]))
        return 1.0 if tried[-1] == best else 2.0
    monkeypatch.setattr(autotune, "_time_plain", plain)
    r = Renderer(own)
    tuning, report = autotune.tune(r, [], 1000, cache=str(tmp_path / "cache.json"))
    assert own in tried and len(set(tried)) == len(tried)
    assert (tuning["plain_region_width"], tuning["plain_region_height"]) == best
    # A second renderer takes the stored choice as it is.
    again, report = autotune.tune(Renderer((32, 32)), [], 1000, cache=str(tmp_path / "cache.json"))
    assert report["cached"] and again == tuning
