"""Explicit minibatch steps where the block's work split can go wrong, bit for bit the oracle:
1 to 64 inputs, 2 to 12 outputs, one column chunk to 64, calls on both sides of the size at
which the row offsets come from a prefix kernel."""
import numpy as np
import pytest

from test_gpu_minibatch import run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d", [(1, 4), (65, 252), (1024, 8), (1025, 12), (2600, 36)])
def test_minibatch_edges_bit_exact(n, d, sgns_lib, oracle_mod):
    rng = np.random.default_rng(n)
    batches = []
    for b in range(n):
        I, O = (1, 2) if b % 7 == 0 else (64, 12) if b % 7 == 1 else (int(rng.integers(1, 65)), int(rng.integers(2, 13)))
        batches.append(((rng.standard_normal((I, d)) * 3 / np.sqrt(d)).astype(np.float32),
                        rng.standard_normal((O, d)).astype(np.float32), rng.integers(1, 4, O).astype(np.int32),
                        int(rng.integers(0, I + 1)), np.float32(0.03)))
    gi, go = run_gpu(batches, d)
    oi = oo = 0
    for xin, xout, meta, first, alpha in batches:
        want_in, want_out = oracle_mod.minibatch(xin, xout, meta, first, float(alpha), acc64=False)
        I, O = xin.shape[0], xout.shape[0]
        assert np.array_equal(gi[oi:oi + I], want_in.astype(np.float32))
        assert np.array_equal(go[oo:oo + O], want_out.astype(np.float32))
        oi += I
        oo += O
