"""Workers that a launch of the persistent engine holds at once.

The reference's compute threads run side by side (dsgl.hpp:783-826, one slice each) under one
learning-rate schedule, so a launch shape must hold all the workers of a call: a worker that
starts when another has ended trains its whole slice at the low end of the schedule.  An SM
holds at most three teams (128 registers x 160 threads each) and eight one-warp workers (up
to 255 registers a thread), in whole CTAs."""
import re

import numpy as np
import pytest

import sgns

pytestmark = pytest.mark.gpu


def small_corpus(V, n_walks, seed):
    rng = np.random.default_rng(seed)
    walks = np.hstack([rng.integers(0, V, (n_walks, 30)), -np.ones((n_walks, 1), np.int64)]).ravel().astype(np.int32)
    return walks, np.maximum(np.bincount(walks[walks >= 0], minlength=V), 1).astype(np.int32)


def held(team, per_cta):
    import torch

    return (3 if team else 8) // per_cta * per_cta * torch.cuda.get_device_properties(0).multi_processor_count


def train(V, walks, counts, **options):
    opt = sgns.default_options(iter=1, engine="persistent", table_size=1000000, sample=0.0, **options)
    with sgns.Trainer(opt) as t:
        t.set_vocab(counts)
        return t.train_corpus(walks)


@pytest.mark.parametrize("V,d,window,negative,storage,workers", [
    (400_000, 200, 7, 3, "bf16", 0), (1_100_000, 128, 10, 5, "bf16", 0), (190_000, 256, 10, 10, "fp32", 0),
    (20_000, 128, 10, 5, "fp32", 700), (20_000, 64, 5, 5, "bf16", 5000)])
def test_tried_shapes_hold_every_worker(V, d, window, negative, storage, workers, sgns_lib, capfd):
    """The autotuner tries shapes that hold all the workers of the call; when none does, it tries
    the one-warp shapes."""
    walks, counts = small_corpus(V, 6000, seed=V)
    st = train(V, walks, counts, size=d, window=window, negative=negative, storage=storage, workers=workers, debug=3)
    trials = re.findall(r"trial team (\d), (\d) per CTA.*?: (\d+) workers", capfd.readouterr().err)
    assert trials and st.workers == (workers or int(trials[0][2]))
    for team, per_cta, n in trials:
        assert int(n) == st.workers
        assert int(n) <= held(int(team), int(per_cta)) or (not int(team) and workers == 5000), (team, per_cta, n)


@pytest.mark.parametrize("per_cta,per_sm,more,warps", [(1, 1, 0, 5), (1, 3, 0, 5), (1, 3, 1, 1), (2, 2, 0, 5), (2, 2, 1, 1),
                                                       (3, 3, 0, 5), (3, 3, 1, 1), (4, 1, 0, 1)])
def test_given_cta_shape_takes_teams_where_all_run_at_once(per_cta, per_sm, more, warps, sgns_lib):
    walks, counts = small_corpus(20_000, 6000, seed=5)
    workers = held(0, 1) // 8 * per_sm + more
    st = train(20_000, walks, counts, size=64, window=5, negative=5, storage="bf16", workers=workers,
               warps_per_cta=per_cta, debug=0)
    assert (st.workers, st.warps_per_cta, st.warps_per_worker) == (workers, per_cta, warps)


def test_given_cta_shape_at_the_default_count(sgns_lib):
    """400,000 vertices, CTAs of two: a count of its own rule, above the teams that run at once."""
    walks, counts = small_corpus(400_000, 6000, seed=6)
    st = train(400_000, walks, counts, size=128, window=10, negative=5, storage="bf16", warps_per_cta=2, debug=0)
    assert held(1, 1) < st.workers <= held(0, 2) and st.warps_per_worker == 1


def test_untimed_shape_is_the_faster_engine(sgns_lib):
    """No room for the autotuner's copies of the tables: teams where the GPU holds all of them
    (here 450 workers), which the timings prefer at every count of theirs."""
    import torch

    from test_gpu_parity import _hold_all_but

    V = 180_000
    walks, counts = small_corpus(V, 6000, seed=7)
    opt = sgns.default_options(size=256, window=5, negative=5, iter=1, debug=0, table_size=1000000, sample=0.0)
    with sgns.Trainer(opt) as t:
        t.set_vocab(counts)  # two tables of 184 MB
        t.upload(walks)
        hold = _hold_all_but(276 << 20)
        try:
            st = t.train()
        finally:
            del hold
            torch.cuda.empty_cache()
    assert st.workers == V // 400 and st.warps_per_worker == 5
