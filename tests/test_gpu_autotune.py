"""The batch autotuner where the jobs run in one kernel: its pool, refill and
shading coordinates do nothing there, so it must leave them at their defaults
whatever its trials measure."""
import pytest

from tinypt_b200 import scenes

pytestmark = pytest.mark.gpu


def _tune(work):
    import torch

    from tinypt_b200.render import BatchScenes

    films = [(torch.empty(3 * c.film_pixels, dtype=torch.float64, device="cuda"),
              torch.empty(c.film_pixels, dtype=torch.float64, device="cuda")) for _, c in work]
    jobs = [(k, c, a.data_ptr(), w.data_ptr()) for k, ((_, c), (a, w)) in enumerate(zip(work, films))]
    with BatchScenes([s for s, _ in work]) as bs:
        best, trials = bs.autotune(jobs)
        st = bs.render(jobs, tuning=best)
    return best, trials, st


@pytest.mark.parametrize("seed", [1, 2, 3, 4])
def test_loop_settings_stay_where_no_loop_runs(gpu, monkeypatch, seed):
    for k in ("TPT_POOL", "TPT_TASK_SPP", "TPT_TRACE_CHUNK", "TPT_SHADE_CTAS", "TPT_TAIL_SLOTS"):
        monkeypatch.delenv(k, raising=False)
    work = scenes.batch_workload(4, seed=seed, tri_range=(200, 2000), res_range=(24, 48), spp_range=(4, 16), max_depth=8)
    (pool, _, chunk, ctas), trials, st = _tune(work)
    assert st.iterations == 0 and (pool, chunk, ctas) == (64 << 20, 16, 8) and len(trials) >= 9
