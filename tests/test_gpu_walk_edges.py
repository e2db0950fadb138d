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


def test_walks_without_a_corpus_take_its_room_only(sgns_lib):
    """A new corpus costs its own bytes and the walks' offsets, not those of the longest walks
    (here 800 MB for about 20): what torch keeps, the library cannot allocate."""
    import torch

    V, n_walks = 4000, 200_000
    ip = torch.arange(0, 2 * V + 1, 2, dtype=torch.int64, device="cuda")
    i = torch.arange(V, dtype=torch.int32, device="cuda")
    ix = torch.stack([(i + V - 1) % V, (i + 1) % V], 1).sort(1).values.reshape(-1).contiguous()
    cn = torch.zeros(2 * V, dtype=torch.int32, device="cuda")
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()

    def asked():  # bytes asked for, without the allocator's rounding
        return torch.cuda.memory_stats()["requested_bytes.all.peak"]

    before, reserved = asked(), torch.cuda.memory_reserved()
    out, n = sgns.info_walks(ip, ix, cn, n_walks, 20, 1000, 0.999, 3, trace=0)
    peak, kept = asked() - before, torch.cuda.max_memory_reserved() - reserved
    room = 4 * n + 8 * (n_walks + 1) + (1 << 16)
    assert n == out.numel() and 8 * room < 4 * 1001 * n_walks
    assert peak <= room and kept <= 2 * room + (64 << 20)
    assert int((out == -1).sum()) == n_walks


def test_walk_tokens_refuse_a_small_corpus(sgns_lib, oracle_mod):
    """The two calls by themselves: offsets as the corpus's walks, a corpus one entry short
    refused and left as it was."""
    import ctypes

    import torch

    ip, ix = clique_and_tail(9, 40)
    cn = oracle_mod.edge_common_neighbors(ip, ix)
    want, _ = oracle_mod.info_walks(ip, ix, cn, 500, 5, 40, 0.9, 11, trace=1)
    dip, dix, dcn = *on_gpu(ip, ix), torch.from_numpy(cn).cuda()
    o = sgns.WalkOptions(walker_num=500, min_length=5, max_length=40, r_threshold=0.9, seed=11, trace_steps=1)
    graph = (ctypes.byref(o), dip.data_ptr(), dix.data_ptr(), dcn.data_ptr(), len(ip) - 1, len(ix))
    offsets, n = torch.empty(501, dtype=torch.int64, device="cuda"), ctypes.c_int64()
    assert sgns_lib.sgns_info_walk_offsets(*graph, offsets.data_ptr(), ctypes.byref(n), None) == sgns.OK
    ends = np.flatnonzero(want == -1) + 1
    assert n.value == len(want) and np.array_equal(offsets.cpu().numpy(), np.append(0, ends))
    corpus = torch.full((len(want),), -9, dtype=torch.int32, device="cuda")
    tokens = lambda cap: sgns_lib.sgns_info_walk_tokens(*graph, offsets.data_ptr(), corpus.data_ptr(), cap, None)
    assert tokens(len(want) - 1) == sgns.EINVAL and bool((corpus == -9).all())
    assert tokens(len(want)) == sgns.OK and np.array_equal(corpus.cpu().numpy(), want)
    assert sgns_lib.sgns_info_walk_offsets(*graph, None, ctypes.byref(n), None) == sgns.EINVAL


@pytest.mark.parametrize("at,value", [(0, 3), (0, -1), (1, -4), (1, 0), (250, 1 << 40), (250, -(1 << 62)), (499, 1),
                                      (500, 7), (500, -1)])
def test_walk_tokens_refuse_offsets_that_are_not_walks(at, value, sgns_lib, oracle_mod):
    """The walks are written where the offsets say: any that would lead outside the corpus is
    refused before the first token."""
    import ctypes

    import torch

    ip, ix = clique_and_tail(9, 40)
    dip, dix, dcn = *on_gpu(ip, ix), torch.from_numpy(oracle_mod.edge_common_neighbors(ip, ix)).cuda()
    o = sgns.WalkOptions(walker_num=500, min_length=5, max_length=40, r_threshold=0.9, seed=11, trace_steps=1)
    graph = (ctypes.byref(o), dip.data_ptr(), dix.data_ptr(), dcn.data_ptr(), len(ip) - 1, len(ix))
    offsets, n = torch.empty(501, dtype=torch.int64, device="cuda"), ctypes.c_int64()
    assert sgns_lib.sgns_info_walk_offsets(*graph, offsets.data_ptr(), ctypes.byref(n), None) == sgns.OK
    offsets[at] = value
    corpus = torch.full((n.value,), -9, dtype=torch.int32, device="cuda")
    assert sgns_lib.sgns_info_walk_tokens(*graph, offsets.data_ptr(), corpus.data_ptr(), n.value, None) == sgns.EINVAL
    assert bool((corpus == -9).all())


def test_walks_from_another_stream_wait_for_their_corpus(sgns_lib):
    """Torch's current stream still writes the memory that the new corpus gets: the walks, on the
    default stream, come after that."""
    import torch

    ip, ix = on_gpu(*clique_and_tail(40, 0))
    cn = torch.empty(ix.numel(), dtype=torch.int32, device="cuda")
    sgns.edge_common_neighbors(ip, ix, cn)
    walks = lambda: sgns.info_walks(ip, ix, cn, 100_000, 20, 60, 0.9, 5)
    want, n = walks()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        held = torch.empty(n, dtype=torch.int32, device="cuda")
        side.synchronize()
        place = held.data_ptr()
        torch.cuda._sleep(400_000_000)  # 0.2 s
        held.fill_(-7)
        del held
        got, _ = walks()
    torch.cuda.synchronize()
    assert got.data_ptr() == place and torch.equal(got, want)


@pytest.mark.parametrize("past", [0, 1])
def test_common_neighbors_around_the_small_graphs(past, sgns_lib, oracle_mod):
    """Up to 4 x 64 edges per SM lists of three entries go to a warp, above those of 25."""
    import torch

    edges = 256 * torch.cuda.get_device_properties(0).multi_processor_count + 2 * past
    ip, ix = clique_and_tail(30, (edges - 30 * 29) // 2)
    assert len(ix) == edges
    cn = torch.empty(edges, dtype=torch.int32, device="cuda")
    sgns.edge_common_neighbors(*on_gpu(ip, ix), cn)
    assert np.array_equal(cn.cpu().numpy(), oracle_mod.edge_common_neighbors(ip, ix))


def test_common_neighbors_take_as_long_in_any_order_of_the_vertices(sgns_lib, oracle_mod):
    """The same power-law graph with its ids by degree and shuffled: the same searches, so about
    the same time, though by degree the hubs' edges follow one another (1.5 is far above the
    scatter of a median; hubs' edges on a few SMs take several times as long)."""
    import torch

    import synth

    V = 20_000
    ip, ix = synth.chung_lu(V, 54_600, 2.1, seed=3, device="cuda")
    src = torch.repeat_interleave(torch.arange(V, device="cuda"), ip.diff())
    new = torch.randperm(V, generator=torch.Generator().manual_seed(1)).cuda()
    key, order = torch.sort(new[src] * V + new[ix.long()])
    sip = torch.searchsorted(torch.div(key, V, rounding_mode="floor"), torch.arange(V + 1, device="cuda"))
    six = (key % V).to(torch.int32)
    counts, medians = [], []
    for p, x in ((ip, ix), (sip, six)):
        cn = torch.empty_like(x)
        times = []
        for _ in range(15):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            sgns.edge_common_neighbors(p, x, cn)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        counts.append(cn)
        medians.append(sorted(times)[len(times) // 2])
    assert np.array_equal(counts[0].cpu().numpy(), oracle_mod.edge_common_neighbors(ip.cpu().numpy(), ix.cpu().numpy()))
    assert torch.equal(counts[0][order], counts[1])
    assert medians[0] < 1.5 * medians[1], medians


def test_walks_over_a_bad_graph_make_nothing(sgns_lib):
    """A neighbour outside the graph, and an indptr that leads past the edges: each of the walk
    calls refuses it and leaves the corpus as it was."""
    import ctypes

    import torch

    good = clique_and_tail(9, 40)
    cn = torch.zeros(len(good[1]), dtype=torch.int32, device="cuda")
    o = sgns.WalkOptions(walker_num=500, min_length=5, max_length=40, r_threshold=0.9, seed=11, trace_steps=0)
    offsets, n = torch.empty(501, dtype=torch.int64, device="cuda"), ctypes.c_int64()
    corpus = torch.full((500 * 41,), -9, dtype=torch.int32, device="cuda")
    graph = lambda ip, ix: (ctypes.byref(o), ip.data_ptr(), ix.data_ptr(), cn.data_ptr(), ip.numel() - 1, ix.numel())
    whole = on_gpu(*good)
    assert sgns_lib.sgns_info_walk_offsets(*graph(*whole), offsets.data_ptr(), ctypes.byref(n), None) == sgns.OK
    far, past = on_gpu(*good), on_gpu(*good)
    far[1][7] = len(good[0]) - 1
    past[0][20] = len(good[1]) + 1
    for g in (far, past):
        calls = ((sgns_lib.sgns_info_walk_tokens, offsets.data_ptr(), corpus.data_ptr(), corpus.numel(), None),
                 (sgns_lib.sgns_info_walks, corpus.data_ptr(), corpus.numel(), ctypes.byref(n), None),
                 (sgns_lib.sgns_info_walk_offsets, torch.empty_like(offsets).data_ptr(), ctypes.byref(n), None))
        for call, *args in calls:
            n.value = 5
            assert call(*graph(*g), *args) == sgns.EINVAL and (n.value == 0 or call == calls[0][0])
        assert bool((corpus == -9).all())
    assert sgns_lib.sgns_info_walk_tokens(*graph(*whole), offsets.data_ptr(), corpus.data_ptr(), corpus.numel(), None) == sgns.OK
