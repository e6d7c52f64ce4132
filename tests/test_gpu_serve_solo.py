"""Served sphere jobs on both sides of the edge above which they step by themselves: the results of the job run alone."""
import pytest

pytestmark = pytest.mark.gpu

wb = pytest.importorskip("wake_b200")
from test_gpu_serve import _assert_same  # noqa: E402
from wake_b200 import serve as S  # noqa: E402


def test_solo_and_batched_jobs_together():
    jobs = S.mixed_jobs(8, 400.0, d3q19_frac=1.0, n_range=(S.SOLO_MIN_EDGE - 8, S.SOLO_MIN_EDGE + 8), median_steps=40.0,
                        p5_steps=20.0, steps_range=(10, 80))
    keys = [S._class_key(j)[0] for j in jobs]
    assert "solo" in keys and 19 in keys
    rep = S.Server(sum(S.job_bytes(j, "f32") for j in jobs), max_tick_steps=16).run(jobs, realtime=False)
    assert len(rep.results) == len(jobs)
    for r in rep.results:
        _assert_same(r, S.run_alone(next(j for j in jobs if j.id == r.id)))
