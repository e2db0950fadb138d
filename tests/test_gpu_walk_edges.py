"""The walker's shortcuts and the common-neighbour kernel's splits at their edges, bit for bit
the oracle: caps at multiples of the history's groups of four and up to the limit, stop
thresholds where the cheap test cannot decide (0, 1, negative) and where it does, hubs whose
lists the whole warp searches, edge counts around the tile."""
import numpy as np
import pytest

import sgns

pytestmark = pytest.mark.gpu


def clique_and_tail(n, tail):
    """A clique of n vertices, a path of `tail` more behind it, an isolated vertex at the end."""
    V = n + tail + 1
    adj = [set() for _ in range(V)]
    for i in range(n):
        adj[i] |= set(range(n)) - {i}
    for i in range(n - 1, n + tail - 1):
        adj[i].add(i + 1)
        adj[i + 1].add(i)
    ip = np.zeros(V + 1, np.int64)
    ip[1:] = np.cumsum([len(a) for a in adj])
    return ip, np.array([v for a in adj for v in sorted(a)], np.int32)


def on_gpu(ip, ix):
    import torch

    return torch.from_numpy(ip).cuda(), torch.from_numpy(ix).cuda()


@pytest.mark.parametrize("n,tail", [(2, 0), (16, 14), (17, 0), (24, 3), (26, 1), (60, 5)])
def test_common_neighbors_of_cliques(n, tail, sgns_lib, oracle_mod):
    import torch

    ip, ix = clique_and_tail(n, tail)
    dip, dix = on_gpu(ip, ix)
    cn = torch.empty(len(ix), dtype=torch.int32, device="cuda")
    sgns.edge_common_neighbors(dip, dix, cn)
    assert np.array_equal(cn.cpu().numpy(), oracle_mod.edge_common_neighbors(ip, ix))


@pytest.mark.parametrize("trace", [0, 1])
@pytest.mark.parametrize("min_length,max_length,r_th", [
    (0, 1, 0.9), (0, 2, 0.9), (1, 4, 0.5), (2, 5, 1.0), (3, 8, 0.0), (5, 81, -1.0), (0, 60, 2.0), (20, 80, 0.84),
    (4, 63, 1e-9), (10, 250, 0.97), (30, 1000, 0.7)])
def test_walks_at_the_edges(min_length, max_length, r_th, trace, sgns_lib, oracle_mod):
    ip, ix = clique_and_tail(9, 40)
    cn = oracle_mod.edge_common_neighbors(ip, ix)
    dip, dix = on_gpu(ip, ix)
    import torch

    got, n = sgns.info_walks(dip, dix, torch.from_numpy(cn).cuda(), 777, min_length, max_length, r_th, 11, trace=trace)
    want, _ = oracle_mod.info_walks(ip, ix, cn, 777, min_length, max_length, r_th, 11, trace=trace)
    assert n == len(want) and np.array_equal(got.cpu().numpy(), want)
