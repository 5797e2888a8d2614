"""Queues of about as many tiles as CTAs: how they spread over the chip, as a
ratio of times within one run.  512 tiles of 32 x 32 have two warps per CTA, on
four different quarters of each SM, and take about as long as 256 (1.05 times
measured; 1.6 with the two on one quarter of the SM, 2.8 when the warps of the
first CTAs take all that is left of the queue).  One matrix of 1024 x 1024 x
1024 takes less than a quarter of the time of one of 2048 (0.16; 0.26)."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from batchgemm_gb300.batch import DeviceBatch  # noqa: E402


def ms(n, mn, k, cfg=-1):
    db = DeviceBatch([mn] * n, [mn] * n, [k] * n).fill_fast()
    with db.plan("simt", force_tile_config=cfg) as p:
        for _ in range(3):
            db.execute(p)
        t = []
        for _ in range(9):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            for _ in range(4):
                db.execute(p)
            e1.record()
            e1.synchronize()
            t.append(e0.elapsed_time(e1) / 4)
    return sorted(t)[4]


def test_second_tile_per_cta_runs_beside_the_first(cuda):
    few, many = ms(4, 256, 4096, cfg=1), ms(8, 256, 4096, cfg=1)
    assert many < 1.35 * few, (few, many)


def test_one_matrix_uses_the_whole_chip(cuda):
    small, large = ms(1, 1024, 1024), ms(1, 2048, 2048)
    assert small < 0.21 * large, (small, large)
