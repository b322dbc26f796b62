"""Simulators take the fastest measured tile: every class of the committed
timings names the tile of its smallest time, and so does a new measurement."""

import json

import numpy as np

from finitevolumegpu_b200 import Autotuner as module
from finitevolumegpu_b200.Autotuner import DEFAULT_CACHE, Autotuner


def test_cached_tile_is_the_fastest_measured_one():
    for device, schemes in json.load(open(DEFAULT_CACHE)).items():
        for key, entry in schemes.items():
            for cls, best in [("", entry)] if key.startswith("batch:") else entry.items():
                fastest = min(best["all"].values())
                assert best["all"][str(best["tile"])] == fastest == best["ms_per_step"], (device, key, cls)


def test_benchmark_records_the_fastest_and_peak_reports_the_widest_known(tmp_path, monkeypatch):
    """A stand-in simulator whose 12 x 12 tile is the fastest at 256 x 256."""
    import finitevolumegpu_b200 as fv

    class Sim(object):
        def __init__(self, context, *args):
            self.tile = context.autotuner.get_tile("KP07_dimsplit", 256, 256)

        def advance(self, n):
            pass

        def last_advance_ms(self):
            return {11: 0.5, 12: 0.75}.get(self.tile, 1.0 + self.tile)

        def tile_info(self):
            return {"tile_w": 12 if self.tile == 11 else 28, "tile_h": 28}

    class Context(object):
        device_name, autotuner = "Dev", None

    monkeypatch.setitem(fv.SCHEMES, "KP07_dimsplit", Sim)
    Sim.__name__ = "KP07_dimsplit"
    tuner = Autotuner(nx=256, ny=256, cache_file=str(tmp_path / "cache.json"))
    tuner._context = Context()
    peak = tuner.get_peak_performance(Sim)
    assert Autotuner(cache_file=str(tmp_path / "cache.json")).get_tile("KP07_dimsplit", 256, 256, "Dev") == 11
    assert peak["block_width"] == 28 and np.isclose(peak["megacells"], 256 * 256 / 0.75e-3 / 1e6)
    assert set(module.SMALL_TILES) <= set(module.TILE_CONFIGS)


def test_no_batched_kernel_is_listed_twice():
    """The tuner times every row of the batched kernels' table."""
    import os
    import re

    from conftest import ROOT

    src = open(os.path.join(ROOT, "finitevolumegpu_b200", "csrc", "fv_api.cu")).read()
    rows = re.findall(r"batch_fn<([^>]*)>\(\)", re.search(r"BEntry kBatchTable\[\] = \{(.*?)\n\};", src, re.S).group(1))
    rows = [tuple((r.replace(" ", "").split(",") + ["0", "1"])[:6]) for r in rows]
    assert len(rows) > 20 and len(set(rows)) == len(rows)
