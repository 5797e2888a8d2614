"""The autotuner's tensor-core tile times are the GEMM kernel's alone: between the
events around it, all operands packed before, and nothing estimated and taken off."""
import pytest

pytestmark = pytest.mark.gpu

import batchgemm_gb300 as bg  # noqa: E402
from batchgemm_gb300 import autotune  # noqa: E402
from batchgemm_gb300.batch import DeviceBatch  # noqa: E402

PACKING_BEFORE = 1


@pytest.mark.parametrize("mode,cfg", [("tf32", 8), ("tf32x3", 1), ("tf32x3", 10), ("bf16x3", 13)])
@pytest.mark.parametrize("K", [32, 2048])
def test_tile_time_is_the_kernels(cuda, monkeypatch, mode, cfg, K):
    seen = []
    packing, events = bg.lib().bgemm_debug_plan_packing, bg.Plan.set_kernel_events
    execute = DeviceBatch.execute

    def on_packing(h, who):
        seen.append(("packing", who))
        return packing(h, who)

    def on_events(self, start=None, stop=None):
        seen.append(("events", start, stop))
        return events(self, start, stop)

    def on_execute(self, p, *args, **kw):
        seen.append(("execute", p.info()["grid"], p.info()["num_tiles"]))
        return execute(self, p, *args, **kw)

    monkeypatch.setattr(bg.lib(), "bgemm_debug_plan_packing", on_packing)
    monkeypatch.setattr(bg.Plan, "set_kernel_events", on_events)
    monkeypatch.setattr(DeviceBatch, "execute", on_execute)
    t, ms = autotune.measure(mode, cfg, K, bg.device_info()["num_sms"] // (2 if cfg >= 8 else 1))
    assert seen[0] == ("packing", PACKING_BEFORE)
    assert [s[1] for s in seen if s[0] == "packing"] == [PACKING_BEFORE]
    timed = [s[1:] for s in seen if s[0] == "events" and s[1] is not None]
    assert timed and ms == min(a.elapsed_time(b) for a, b in timed)
    grid, tiles = seen[1][1:]
    lanes = grid // 2 if cfg >= 8 else grid
    assert t == pytest.approx(ms * 1e6 * lanes / tiles, rel=1e-12)
