"""The persistent engine's two kernels -- a team of warps per worker (1 to 3 workers per CTA)
and one warp per worker (a forward tile given) -- at the edges of their row splits: hidden
sizes of one chunk, of an odd number of chunks, with and without quarters (d % 16), the
widest; windows of 1 and 15; 0, 5 and 10 negatives; corpora whose walks revisit vertices and
meet in the same vertices.  One worker, bit for bit the oracle's window policy; several
workers on disjoint components, row for row."""
import numpy as np
import pytest

from test_gpu_hogwild import component_corpus
from test_gpu_parity import gpu_train, oracle_train

pytestmark = pytest.mark.gpu


def small_walks(V, hot, n_walks, seed):
    """Short walks over few hot vertices: repeats within a window, shared rows between walks."""
    rng = np.random.default_rng(seed)
    toks = []
    for _ in range(n_walks):
        n = int(rng.integers(2, 48))
        toks += np.where(rng.random(n) < 0.5, rng.integers(0, hot, n), rng.integers(0, V, n)).tolist() + [-1]
    return np.array(toks, np.int32)


SHAPES = [(4, 1, 0), (8, 2, 5), (16, 15, 10), (36, 5, 5), (48, 3, 10), (64, 10, 5), (100, 15, 5), (112, 7, 10),
          (128, 15, 10), (132, 4, 5), (200, 6, 10), (240, 10, 5), (252, 5, 10), (256, 10, 5)]


@pytest.mark.parametrize("kernel", ["team1", "team3", "warp"])
@pytest.mark.parametrize("storage", ["fp32", "bf16"])
@pytest.mark.parametrize("d,window,negative", SHAPES)
def test_kernels_match_the_oracle(d, window, negative, storage, kernel, sgns_lib, oracle_mod):
    corpus = small_walks(300, 12, 90, seed=d + window)
    cfg = dict(V=300, d=d, window=window, negative=negative, iter=2, sample=0.0 if d % 8 else 1e-2, alpha=0.05)
    tile = 1 if kernel == "warp" else 0
    wih, woh, st, _ = gpu_train(cfg, corpus, "persistent", storage, wpc=3 if kernel == "team3" else 1, tile=tile)
    owih, owoh, ost = oracle_train(oracle_mod, cfg, corpus, oracle_mod.POLICY_WINDOW, storage)
    assert st.warps_per_worker == (1 if kernel == "warp" else 5)
    assert (st.steps, st.pairs, st.word_count_actual) == (ost["steps"], ost["pairs"], ost["word_count_actual"])
    assert np.array_equal(wih.view(np.uint32), owih.view(np.uint32)), np.abs(wih - owih).max()
    assert np.array_equal(woh.view(np.uint32), owoh.view(np.uint32)), np.abs(woh - owoh).max()


@pytest.mark.parametrize("storage,wpc", [("fp32", 2), ("bf16", 3)])
def test_disjoint_teams_match_the_oracle(storage, wpc, sgns_lib, oracle_mod):
    """Seven workers over CTAs of two and three (the last CTA partly empty), no shared row."""
    W, n = 7, 60
    corpus = component_corpus(W, n, 1500, seed=23)
    cfg = dict(V=W * n, d=128, window=10, negative=0, iter=1, sample=0.0, alpha=0.05)
    wih, woh, st, _ = gpu_train(cfg, corpus, "persistent", storage, workers=W, wpc=wpc)
    owih, owoh, ost = oracle_train(oracle_mod, cfg, corpus, oracle_mod.POLICY_WINDOW, storage, workers=W)
    assert st.workers == W and st.warps_per_worker == 5
    assert (st.steps, st.pairs) == (ost["steps"], ost["pairs"])
    assert np.array_equal(wih.view(np.uint32), owih.view(np.uint32))
    assert np.array_equal(woh.view(np.uint32), owoh.view(np.uint32))
