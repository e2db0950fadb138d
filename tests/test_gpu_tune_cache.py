"""What the autotuner records: a choice holds for the runs that may choose from the same
shapes, and for the kernels it was timed with."""
import numpy as np
import pytest

import sgns
from test_gpu_residency import small_corpus, train

pytestmark = pytest.mark.gpu
V = 20_000


@pytest.fixture
def run(tmp_path, monkeypatch, sgns_lib):
    cache = tmp_path / "tune.txt"
    monkeypatch.setenv("SGNS_TUNE_CACHE", str(cache))
    walks, counts = small_corpus(V, 6000, seed=8)

    def go(**options):
        return train(V, walks, counts, size=128, window=5, negative=5, storage="bf16", debug=0, **options)

    go.lines = lambda: cache.read_text().splitlines()
    go.plant = lambda line: cache.write_text(line + "\n")
    return go


@pytest.mark.parametrize("other", [dict(compute_loss=1), dict(forward_tile=1), dict(windows_per_step=1)])
def test_other_runs_leave_the_recorded_shape(run, other):
    first = run()
    assert first.warps_per_worker == 5 and len(run.lines()) == 1
    st = run(**other)
    assert st.warps_per_worker == 1 and len(run.lines()) == 2
    again = run()
    assert (again.warps_per_worker, again.warps_per_cta) == (5, first.warps_per_cta)
    assert run(**other).warps_per_cta == st.warps_per_cta and len(run.lines()) == 2


def test_recorded_team_shape_is_taken(run):
    run()
    run.plant(run.lines()[0].split("\t")[0] + "\tteam\t3\t1")
    st = run()
    assert (st.warps_per_worker, st.warps_per_cta) == (5, 3) and len(run.lines()) == 1


def test_lines_of_earlier_kernels_are_not_taken(run):
    """Their key ends with the vertex count, and their shape was timed before teams were."""
    run()
    run.plant(run.lines()[0].split("|V=")[0] + "|V=%d\t4\t1" % V)
    assert run().warps_per_worker == 5 and len(run.lines()) == 2
