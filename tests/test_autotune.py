"""The autotuner's choices, with a fake library and fake plans (no GPU): segment
and tier split come from the lone call that users make, the bucket split from
plans, and the shipped table lies within the candidates."""
import json
import re
import time
import types

import pytest

from conftest import ROOT, build_library


@pytest.fixture(scope="module")
def at():
    build_library()
    from voss_gb300 import autotune
    return autotune


def test_what_is_timed(at, monkeypatch):
    import torch
    import voss_gb300.plan
    now = {}

    class Lib:
        @staticmethod
        def voss_primes_range_stats(a, b, out):
            # the lone call is fastest with segments of 98304 and a split of 1024
            slow = (now["seg"] != 98304) + (now["split"] != 1024)
            end = time.perf_counter() + 2e-4 * (1 + 2 * slow)
            while time.perf_counter() < end:
                pass
            return 0

    def set_tuning(n, entries):
        now.update(seg=entries[0].seg_bytes, split=entries[0].tier_split, bucket=entries[0].bucket_split)
        return 0

    class Plan:
        def __init__(self, ranges): pass
        def launch(self, stream=0): pass
        def results(self, stream=0): pass
        def close(self): pass
        def kernel_ms(self):
            # plans are fastest with other segments, and with lists from 1327104 on
            return (1.0 + (now["seg"] != 65536) + (now["split"] != 512) - 0.5 * (now["bucket"] == 1327104), 0.0)

    Lib.voss_gb300_set_tuning = staticmethod(set_tuning)
    monkeypatch.setattr(torch.cuda, "Stream", lambda: types.SimpleNamespace(cuda_stream=0))
    monkeypatch.setattr(voss_gb300.plan, "SievePlan", Plan)
    monkeypatch.setattr("voss_gb300._capi._lib", Lib)
    monkeypatch.setattr(at, "REGIMES", [(10**14, 10**9, [(0, 10)])])
    assert at.run() == [(10**14, 10**9, 98304, 1024, 1327104)]


def test_shipped_table_lies_within_the_candidates(at):
    table = json.loads((ROOT / "voss_gb300" / "tune_table.json").read_text())
    assert [(e["b_max"], e["width_max"]) for e in table] == [r[:2] for r in at.REGIMES]
    for e in table:
        assert e["seg_bytes"] in at.SEGS and e["tier_split"] in at.SPLITS and e["bucket_split"] in at.BUCKETS, e
    rows = re.findall(r"^\{(\d+)ull, (\d+)ull, (\d+), (\d+), (\d+), 0\},$",
                      (ROOT / "voss_gb300" / "csrc" / "tune_table.inc").read_text(), re.M)
    assert [tuple(map(int, r)) for r in rows] == [tuple(e.values()) for e in table]
