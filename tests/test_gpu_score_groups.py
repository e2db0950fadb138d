"""Link scores at the edges of the kernel's groups of pairs: counts around a group, ids outside the
table anywhere in a group, pair arrays that start between 8-byte boundaries.  Every score has the
oracle's bits; a pair that names a row outside the table scores 0 and is refused."""
import numpy as np
import pytest

import sgns


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("d", [4, 124, 128, 132, 256])
def test_scores_in_groups(d, dtype, sgns_lib, oracle_mod):
    import torch

    rng = np.random.default_rng(7 * d + dtype)
    V = 61
    t = rng.standard_normal((V, d)).astype(np.float32)
    table = (t.view(np.uint32) >> 16).astype(np.uint16) if dtype else t
    dev = torch.from_numpy(table.view(np.int16) if dtype else table).cuda()
    for n in (1, 2, 3, 4, 5, 7, 8, 9, 31, 32, 33, 70001):
        pr = rng.integers(0, V, size=(n, 2)).astype(np.int32)
        ref, _ = oracle_mod.link_scores(table, pr)
        flat = torch.empty(2 * n + 1, dtype=torch.int32, device="cuda")
        for off in (0, 1):
            pairs = flat[off:off + 2 * n].view(n, 2)
            pairs.copy_(torch.from_numpy(pr))
            sc = torch.full((n + 3,), 5.0, device="cuda")
            sgns.link_scores(dtype, d, dev, V, pairs, sc[:n])
            got = sc.cpu().numpy()
            assert np.array_equal(got[:n].view(np.uint32), ref.view(np.uint32)) and (got[n:] == 5.0).all(), (n, off)
    for n, at, side, row in [(1, 0, 1, V), (6, 3, 0, -1), (6, 5, 1, V), (9, 8, 0, 2 ** 31 - 1)]:
        pr = rng.integers(0, V, size=(n, 2)).astype(np.int32)
        ref, _ = oracle_mod.link_scores(table, pr)
        pr[at, side] = row
        sc = torch.full((n,), 5.0, device="cuda")
        with pytest.raises(sgns.SgnsError) as e:
            sgns.link_scores(dtype, d, dev, V, torch.from_numpy(pr).cuda(), sc)
        assert e.value.status == sgns.EINVAL
        ref[at] = 0.0
        assert np.array_equal(sc.cpu().numpy(), ref)
