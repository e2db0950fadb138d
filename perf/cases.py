"""The work a user of this library has it do, as measurable cases.

Each case goes through the public Python binding (gdistger-re_gb300/sgns.py): training a
corpus to embeddings, replaying one worker exactly, stepping explicit minibatches, the loss
and its adjoint, scoring held-out pairs, parsing walk text, and producing a corpus of
information-oriented walks.  Sizes are the benchmark's and the tests' (the LiveJournal-sized
Chung-Lu graph, the labelled SBM, the shape sweep, the 4M-vertex adjoint), the smallest
ones those of a first try or a check.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gdistger-re_gb300"))

import sgns  # noqa: E402
import synth  # noqa: E402

BF16, FP32, FP64 = "bf16", "fp32", "fp64"
DTYPE_CODE = {FP32: 0, BF16: 1, FP64: 2}
TORCH_TYPE = {FP32: torch.float32, BF16: torch.bfloat16, FP64: torch.float64}


def listed():
    return [
        # a check against the reference: one worker replayed exactly, the default options
        # (d = 100, window 5, 5 negatives, fp32) on a small walk corpus
        dict(name="replay_d100_fp32", kind="train", graph="cl", V=1500, E=8000, walkers=1500, cap=40, d=100, w=5, K=5,
             storage=FP32, workers=1, exact_mode=True, table=1_000_000),
        # the link-prediction corpus: labelled SBM, information-oriented walks, bf16 tables,
        # the library's own worker count and launch shape
        dict(name="train_sbm100k_d128_bf16", kind="train", graph="sbm", V=100_000, E=273_000, walkers=200_000, cap=80,
             d=128, w=10, K=5, storage=BF16, workers=0, exact_mode=False, table=10_000_000),
        # its largest size with every resident worker: tokens from pinned host memory in,
        # embeddings into pinned host memory out
        dict(name="train_sbm1m_d128_bf16", kind="train", graph="sbm", V=1_100_000, E=3_000_000, walkers=1_100_000,
             cap=80, d=128, w=10, K=5, storage=BF16, workers=1064, exact_mode=False, table=100_000_000),
        # the wide end of the shape sweep: d = 256, 10 negatives, fp32 tables
        dict(name="train_sbm120k_d256_k10_fp32", kind="train", graph="sbm", V=120_000, E=327_000, walkers=30_000,
             cap=200, d=256, w=10, K=10, storage=FP32, workers=0, exact_mode=False, table=10_000_000),
        # a handful of explicit reference steps: a caller stepping its own minibatches
        dict(name="minibatch_64_d100", kind="minibatch", n=64, d=100, w=5, K=5, rounded=False),
        # the bf16 write-back of many steps (the per-minibatch error statement's call)
        dict(name="minibatch_20k_d128_bf16", kind="minibatch", n=20_000, d=128, w=10, K=5, rounded=True),
        # loss and gradient of a small batch over fp32 tables
        dict(name="adjoint_1k_d100_fp32", kind="adjoint", n=1_000, V=20_000, d=100, w=5, K=5, dtype=FP32),
        # loss and gradient of 200k minibatches over 4M-vertex bf16 tables
        dict(name="adjoint_200k_d128_bf16", kind="adjoint", n=200_000, V=4_000_000, d=128, w=10, K=5, dtype=BF16),
        # scoring the held-out pairs of the headline graph
        dict(name="scores_20m_d128_bf16", kind="scores", n=20_000_000, V=2_238_731, d=128, dtype=BF16),
        # one small walk file, and a gigabyte of walk text
        dict(name="parse_9k_tokens", kind="parse", tokens=9_000, V=5_000, mean=40, cap=80),
        dict(name="parse_160m_tokens", kind="parse", tokens=160_000_000, V=2_238_731, mean=40, cap=80),
        # the corpus producer: common-neighbour counts, then 10 walks per vertex
        dict(name="walks_sbm200k", kind="walks", graph="sbm", V=200_000, E=546_000, walks=10, min_length=20,
             max_length=80, r=0.84, trace=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "minibatch", "adjoint", "adjoint", "scores", "parse", "walks"])
    if kind == "train":
        # racing updates of hub rows differ from run to run, so power-law graphs are for the
        # replayed runs; the others train a part of their walks over an SBM, at a low rate
        exact = rng.random() < 0.2
        V = _log(rng, 1_000, 2_500) if exact else _log(rng, 15_000, 400_000)
        return dict(kind=kind, graph="cl" if exact else "sbm", V=V, E=int(V * rng.uniform(2.5, 8)),
                    walkers=V if exact else -(-V // rng.choice([3, 4, 6])), cap=40 if exact else rng.choice([60, 80, 200]),
                    d=rng.choice([64, 100, 128, 128, 128, 200, 256]), w=rng.choice([5, 7, 10]),
                    K=rng.choice([5, 5, 5, 3, 10]), storage=rng.choice([BF16, FP32]), workers=1 if exact else 0,
                    exact_mode=exact, table=1_000_000 if exact else 10_000_000)
    if kind == "minibatch":
        return dict(kind=kind, n=_log(rng, 10, 20_000), d=rng.choice([64, 100, 128, 200, 256]),
                    w=rng.choice([5, 7, 10]), K=rng.choice([3, 5, 5, 10]), rounded=rng.random() < 0.5)
    if kind == "adjoint":
        dtype = rng.choice([BF16, BF16, FP32, FP32, FP64])
        n = _log(rng, 100, 10_000 if dtype == FP64 else 200_000)
        return dict(kind=kind, n=n, V=_log(rng, 5_000, 4_000_000), d=rng.choice([36, 64, 100, 128, 128]),
                    w=rng.choice([5, 7, 10]), K=rng.choice([3, 5, 5, 10]), dtype=dtype)
    if kind == "scores":
        return dict(kind=kind, n=_log(rng, 1_000, 20_000_000), V=_log(rng, 5_000, 2_238_731),
                    d=rng.choice([64, 100, 128, 128, 256]) if rng.random() < 0.7 else 4 * rng.randint(1, 32),
                    dtype=rng.choice([BF16, FP32]))
    if kind == "parse":
        return dict(kind=kind, tokens=_log(rng, 1_000, 160_000_000), V=_log(rng, 1_000, 2_238_731),
                    mean=rng.choice([10, 40, 60]), cap=rng.choice([80, 200]))
    V = _log(rng, 2_000, 200_000)
    return dict(kind=kind, graph=rng.choice(["sbm", "cl"]), V=V, E=int(V * rng.uniform(2.5, 8)),
                walks=rng.choice([1, 5, 10]), min_length=20, max_length=rng.choice([60, 80, 100]),
                r=rng.choice([0.78, 0.84, 0.999]), trace=rng.choice([0, 1]))


# ---- inputs ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _graph(case, seed):
    if case["graph"] == "sbm":
        ip, ix, _ = synth.sbm(case["V"], case["E"], 4, 20.0, seed=seed, device="cuda")
        return ip, ix
    return synth.chung_lu(case["V"], case["E"], 2.1, seed=seed, device="cuda")


def _lengths(n, mean, cap, g):
    """Walk lengths: geometric with the given mean, capped."""
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64).clamp_min(1e-300)
    return (torch.floor(torch.log(u) / math.log(1.0 - 1.0 / mean)).long() + 1).clamp(1, cap)


def _popular(V, n, g):
    """n row ids with a power law's popularity (rows sorted by frequency)."""
    w = (torch.arange(V, dtype=torch.float64, device="cuda") + max(1.0, V ** 0.25)) ** (-1.0 / 1.1)
    cdf = torch.cumsum(w / w.sum(), 0)
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    for i in range(0, n, 1 << 25):
        m = min(n - i, 1 << 25)
        out[i:i + m] = torch.searchsorted(cdf, torch.rand(m, generator=g, device="cuda", dtype=torch.float64)).clamp_max(V - 1).to(torch.int32)
    return out


def _corpus(case, seed):
    """Walks over the case's graph: tokens on the GPU, -1 after each walk."""
    ip, ix = _graph(case, seed)
    V, n = case["V"], case["walkers"]
    if case["graph"] == "sbm" and n >= V:  # the labelled corpus: information-oriented walks
        cn = torch.empty(ix.numel(), dtype=torch.int32, device="cuda")
        sgns.edge_common_neighbors(ip, ix, cn)
        return sgns.info_walks(ip, ix, cn, n, 20, case["cap"], 0.84, seed, trace=0)[0]
    # uniform walks of geometric length from the first n vertices of a shuffled order
    L = _lengths(V, 12 if case["graph"] == "cl" else 40, case["cap"], _gen(seed + 1))
    c = synth.random_walks(ip, ix, 1, L, seed=seed + 2)
    return c[:int(torch.nonzero(c == -1)[n - 1]) + 1]


def _shared_draws(n, K, V, t1, g):
    """K shared negatives per minibatch, equal draws merged, draws of target 1 dropped:
    (ids [n, K], multiplicities [n, K], kept [n, K])."""
    if K == 0:
        z = torch.zeros((n, 0), dtype=torch.int32, device="cuda")
        return z, z, z.bool()
    s = torch.sort(_popular(V, n * K, g).view(n, K), 1).values
    same = s.unsqueeze(2) == s.unsqueeze(1)
    earlier = torch.tril(torch.ones((K, K), dtype=torch.bool, device="cuda"), -1)
    first = ~(same & earlier).any(2)
    return s, same.sum(2).to(torch.int32), first & (s != t1.unsqueeze(1))


def _minibatches(n, w, K, V, g):
    """n reference-shaped steps: the windows of two walks around their targets (the shrink
    drawn once per step), target 1, the shared negatives, target 2."""
    b = torch.randint(0, w, (n,), generator=g, device="cuda")
    sides = []
    for _ in range(2):
        L = _lengths(n, 40, 80, g).clamp_min(2)
        pos = (torch.rand(n, generator=g, device="cuda") * L).long().clamp_max(L - 1)
        sides.append(torch.minimum(pos, w - b) + torch.minimum(L - 1 - pos, w - b))
    first, count = sides[0].to(torch.int32), (sides[0] + sides[1]).to(torch.int32)
    t = _popular(V, 2 * n, g).view(n, 2)
    s, m, kept = _shared_draws(n, K, V, t[:, 0], g)
    one = torch.ones((n, 1), dtype=torch.int32, device="cuda")
    keep = torch.cat([one.bool(), kept, one.bool()], 1)
    out_ids = torch.cat([t[:, :1], s, t[:, 1:]], 1)[keep]
    meta = torch.cat([one, m, one], 1)[keep]
    in_ids = _popular(V, int(count.sum()), g)
    ptr = lambda c: torch.cat([torch.zeros(1, dtype=torch.int32, device="cuda"), torch.cumsum(c, 0).to(torch.int32)])
    return in_ids, ptr(count), first, out_ids, ptr(keep.sum(1)), meta


def _walk_text(case, g):
    """Walk text (" %u" per vertex, newline per walk) of about case["tokens"] tokens."""
    n = case["tokens"]
    L = _lengths(max(2, n // 8), case["mean"], case["cap"], g)
    ends = torch.cumsum(L + 1, 0)
    tok = _popular(case["V"], n, g)
    tok[ends[ends <= n - 2] - 1] = -1
    tok[n - 1] = -1
    is_id = tok >= 0
    digits = torch.ones(n, dtype=torch.int64, device="cuda")
    for k in range(1, 8):
        digits += tok >= 10 ** k
    end = torch.cumsum(torch.where(is_id, digits + 1, 1), 0)
    text = torch.full((int(end[-1]),), ord(" "), dtype=torch.uint8, device="cuda")
    text[(end - 1)[~is_id]] = ord("\n")
    rest = tok.clamp_min(0)
    for k in range(8):
        m = is_id & (digits > k)
        text[(end - 1 - k)[m]] = (48 + rest % 10)[m].to(torch.uint8)
        rest = rest // 10
    return text


def prepare(case, seed):
    kind = case["kind"]
    g = _gen(seed)
    s = dict(case=case)
    if kind == "train":
        corpus = _corpus(case, seed)
        counts = torch.bincount(corpus[corpus >= 0].long(), minlength=case["V"]).to(torch.int32).cpu().numpy()
        s["tokens"] = torch.empty(corpus.numel(), dtype=torch.int32, pin_memory=True)
        s["tokens"].copy_(corpus)
        opt = sgns.default_options(size=case["d"], window=case["w"], negative=case["K"], iter=1, sample=1e-3,
                                   alpha=0.01 if case["exact_mode"] else 0.0025, threads=12, table_size=case["table"], storage=case["storage"],
                                   engine="persistent", workers=case["workers"], debug=0, device=0,
                                   mode="exact" if case["exact_mode"] else "hogwild")
        s["trainer"] = sgns.Trainer(opt)
        s["trainer"].set_vocab(counts)
        s["wih"] = torch.empty((case["V"], case["d"]), dtype=torch.float32, pin_memory=True)
        s["woh"] = torch.empty((case["V"], case["d"]), dtype=torch.float32, pin_memory=True) if case["exact_mode"] else None
    elif kind == "minibatch":
        n, d = case["n"], case["d"]
        ii, ip, first, oi, op, meta = _minibatches(n, case["w"], case["K"], 100_000, g)
        s.update(in_count=ip.diff(), first=first, out_count=op.diff(), meta=meta,
                 alpha=torch.full((n,), 0.025, device="cuda"))
        # rows of a table that has been trained for a while
        s["x"] = torch.randn((ii.numel(), d), generator=g, device="cuda") * (1.5 / math.sqrt(d))
        s["o"] = torch.randn((oi.numel(), d), generator=g, device="cuda") * (1.5 / math.sqrt(d))
        kind_of = torch.int16 if case["rounded"] else torch.float32
        # buffers for the largest steps of this shape, kept by the caller from call to call
        s["dx"] = torch.zeros((4 * case["w"] * n, d), dtype=kind_of, device="cuda")
        s["do"] = torch.zeros(((case["K"] + 2) * n, d), dtype=kind_of, device="cuda")
    elif kind == "adjoint":
        V, d, ty = case["V"], case["d"], TORCH_TYPE[case["dtype"]]
        s["batch"] = _minibatches(case["n"], case["w"], case["K"], V, g)
        rows = lambda: ((torch.rand((V, d), generator=g, device="cuda") - 0.5) * (4.0 / math.sqrt(d))).to(ty)
        s["wih"], s["woh"] = rows(), rows()
        acc = torch.float64 if case["dtype"] == FP64 else torch.float32
        # buffers for the largest steps of this shape, kept by the caller from call to call
        n_in, n_out = 4 * case["w"] * case["n"], (case["K"] + 2) * case["n"]
        s["loss"] = torch.zeros(1, dtype=torch.float64, device="cuda")
        s["in_ids"] = torch.zeros(n_in, dtype=torch.int32, device="cuda")
        s["out_ids"] = torch.zeros(n_out, dtype=torch.int32, device="cuda")
        s["g_in"] = torch.zeros((n_in, d), dtype=acc, device="cuda")
        s["g_out"] = torch.zeros((n_out, d), dtype=acc, device="cuda")
    elif kind == "scores":
        V, d = case["V"], case["d"]
        s["table"] = (torch.randn((V, d), generator=g, device="cuda") / math.sqrt(d)).to(TORCH_TYPE[case["dtype"]])
        s["pairs"] = torch.randint(0, V, (case["n"], 2), generator=g, device="cuda", dtype=torch.int32)
        s["scores"] = torch.empty(case["n"], dtype=torch.float32, device="cuda")
    elif kind == "parse":
        s["text"] = _walk_text(case, g)
    else:
        s["graph"] = _graph(case, seed)
        s["seed"] = seed
        # the program's own buffers: a count per directed edge, a corpus of the longest walks
        s["cn"] = torch.zeros(2 * int(1.08 * case["E"]) + 32, dtype=torch.int32, device="cuda")
        s["corpus"] = torch.zeros(case["walks"] * case["V"] * (case["max_length"] + 1), dtype=torch.int32, device="cuda")
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "train":
        t = s["trainer"]
        t.reset_model()
        st = t.train_corpus_ptr(s["tokens"].data_ptr(), s["tokens"].numel())
        t.embeddings_to(0, s["wih"].data_ptr())
        out = {"wih": s["wih"], "steps": int(st.steps), "pairs": int(st.pairs), "words": int(st.word_count_actual)}
        if case["exact_mode"]:  # (racing workers leave an output table of their own every time)
            t.embeddings_to(1, s["woh"].data_ptr())
            out["woh"] = s["woh"]
        return out
    if kind == "minibatch":
        if case["rounded"]:
            sgns.minibatch_update_bf16(case["d"], s["in_count"], s["first"], s["out_count"], s["meta"], s["alpha"],
                                       s["x"], s["o"], s["dx"], s["do"], 0x5EED)
            return {"in": s["dx"].view(torch.bfloat16), "out": s["do"].view(torch.bfloat16)}
        sgns.minibatch_update(case["d"], s["in_count"], s["first"], s["out_count"], s["meta"], s["alpha"], s["x"],
                              s["o"], s["dx"], s["do"])
        return {"in": s["dx"], "out": s["do"]}
    if kind == "adjoint":
        ii, ip, first, oi, op, meta = s["batch"]
        n_in, n_out = sgns.loss_adjoint(DTYPE_CODE[case["dtype"]], case["d"], case["V"], ip, ii, first, op, oi, meta,
                                        s["wih"].data_ptr(), s["woh"].data_ptr(), s["loss"], s["in_ids"], s["g_in"],
                                        s["out_ids"], s["g_out"])
        # the loss in the precision of the arithmetic that made it
        return {"loss": s["loss"].to(s["g_in"].dtype), "n_in": n_in, "in_ids": s["in_ids"], "g_in": s["g_in"],
                "n_out": n_out, "out_ids": s["out_ids"], "g_out": s["g_out"]}
    if kind == "scores":
        sgns.link_scores(DTYPE_CODE[case["dtype"]], case["d"], s["table"], case["V"], s["pairs"], s["scores"])
        return s["scores"]
    if kind == "parse":
        n = sgns.parse_walks_count(s["text"])
        tokens = torch.empty(n, dtype=torch.int32, device="cuda")
        _, max_id = sgns.parse_walks(s["text"], tokens)
        return {"tokens": tokens, "max_id": max_id}
    ip, ix = s["graph"]
    sgns.edge_common_neighbors(ip, ix, s["cn"])
    corpus, n = sgns.info_walks(ip, ix, s["cn"], case["walks"] * case["V"], case["min_length"], case["max_length"],
                                case["r"], s["seed"], trace=case["trace"])
    s["corpus"][:n].copy_(corpus)
    return {"cn": s["cn"], "corpus": s["corpus"], "n": n}


def _pairs_per_step(w):
    """Input rows of a two-walk step: the mean window after the shrink, less the walk ends."""
    return 2 * 0.87 * (w + 1)


def work(case):
    kind = case["kind"]
    if kind == "train":
        tokens = case["walkers"] * (12 if case["graph"] == "cl" else 40)
        el = 2 if case["storage"] == BF16 else 4
        flops = tokens / 2 * _pairs_per_step(case["w"]) * (case["K"] + 2) * case["d"] * 6.0
        return dict(bytes=4.0 * tokens + case["V"] * case["d"] * (4.0 * el + 4.0), flops=flops)
    if kind == "minibatch":
        i, o = case["n"] * _pairs_per_step(case["w"]), case["n"] * (case["K"] + 2)
        return dict(bytes=(i + o) * case["d"] * (4.0 + (2.0 if case["rounded"] else 4.0)) + 4.0 * o + 16.0 * case["n"],
                    flops=i * (case["K"] + 2) * case["d"] * 6.0)
    if kind == "adjoint":
        i, o = case["n"] * _pairs_per_step(case["w"]), case["n"] * (case["K"] + 2)
        rows = sum(case["V"] * 0.5 * (1.0 - math.exp(-2.0 * r / case["V"])) for r in (i, o))  # distinct rows, about
        el, ga = {BF16: (2, 4), FP32: (4, 4), FP64: (8, 8)}[case["dtype"]]
        return dict(bytes=rows * (case["d"] * float(el + ga) + 4.0) + 4.0 * (i + 2 * o) + 12.0 * case["n"],
                    flops=i * (case["K"] + 2) * case["d"] * 6.0)
    if kind == "scores":
        el = 2 if case["dtype"] == BF16 else 4
        rows = min(2.0 * case["n"], float(case["V"])) if case["V"] * case["d"] * el < 100e6 else 2.0 * case["n"]
        return dict(bytes=rows * case["d"] * el + 12.0 * case["n"], flops=2.0 * case["n"] * case["d"])
    if kind == "parse":
        text = case["tokens"] * (1.0 + 0.85 * math.log10(case["V"]))
        return dict(bytes=text + 4.0 * case["tokens"], flops=0.0)
    tokens = case["walks"] * case["V"] * (case["min_length"] + case["max_length"]) * 0.42
    return dict(bytes=4.0 * tokens + 8.0 * case["V"] + 4.0 * 4 * case["E"], flops=30.0 * tokens)


# ---- the same results in 64 bits, by plain torch -----------------------------------------
def _segments(ptr):
    c = ptr.diff().long()
    return torch.repeat_interleave(torch.arange(c.numel(), device=ptr.device), c)


def _dense_steps(ii, ip, first, oi, op, meta, x, o):
    """Per minibatch b: inputs X [n, I, d], outputs O [n, O, d] (zero padded), multiplicities,
    and labels [n, O, I]; with the places of the real rows."""
    n, ib, ob = first.numel(), _segments(ip), _segments(op)
    ic, oc = ip.diff().long(), op.diff().long()
    ij = torch.arange(ib.numel(), device="cuda") - ip.long()[ib]
    oj = torch.arange(ob.numel(), device="cuda") - op.long()[ob]
    I, O = int(ic.max()), int(oc.max())
    X = torch.zeros((n, I, x.shape[1]), dtype=torch.float64, device="cuda")
    Y = torch.zeros((n, O, o.shape[1]), dtype=torch.float64, device="cuda")
    M = torch.zeros((n, O), dtype=torch.float64, device="cuda")
    X[ib, ij], Y[ob, oj], M[ob, oj] = x.double(), o.double(), meta.double()
    i, j = torch.arange(O, device="cuda").view(1, O, 1), torch.arange(I, device="cuda").view(1, 1, I)
    f = first.long().view(n, 1, 1)
    label = (((i == 0) & (j < f)) | ((i == oc.view(n, 1, 1) - 1) & (j >= f))).double()
    real = (j < ic.view(n, 1, 1)).double()
    return X, Y, M, label, real, (ib, ij), (ob, oj)


def exact(case, seed):
    kind = case["kind"]
    if kind == "scores":
        s = prepare(case, seed)
        out = torch.empty(case["n"], dtype=torch.float64, device="cuda")
        for i in range(0, case["n"], 1 << 20):
            p = s["pairs"][i:i + (1 << 20)].long()
            out[i:i + (1 << 20)] = (s["table"][p[:, 0]].double() * s["table"][p[:, 1]].double()).sum(1)
        return out
    if kind == "minibatch":
        s = prepare(case, seed)
        step = torch.arange(1001, dtype=torch.float32)
        e = torch.exp(((step / 1000.0 * 2 - 1) * 6.0).double())
        table = (e / (e + 1)).cuda()  # the sigmoid table of the step, 1001 entries on [-6, 6]
        ptr = lambda c: torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), torch.cumsum(c, 0)])
        dx, do = (torch.zeros(s[k].shape, dtype=torch.float64, device="cuda") for k in ("dx", "do"))
        ip, op = ptr(s["in_count"]), ptr(s["out_count"])
        for b0 in range(0, case["n"], 4096):
            b1 = min(case["n"], b0 + 4096)
            i0, i1, o0, o1 = int(ip[b0]), int(ip[b1]), int(op[b0]), int(op[b1])
            X, Y, M, label, real, at_i, at_o = _dense_steps(None, ip[b0:b1 + 1] - i0, s["first"][b0:b1], None,
                                                            op[b0:b1 + 1] - o0, s["meta"][o0:o1], s["x"][i0:i1], s["o"][o0:o1])
            f = Y @ X.transpose(1, 2)
            sig = table[((f + 6.0) * 83.0).long().clamp(0, 1000)]
            sig = torch.where(f > 6.0, 1.0, torch.where(f < -6.0, 0.0, sig))
            c = (label - sig) * s["alpha"][b0:b1].double().view(-1, 1, 1) * M.unsqueeze(2) * real
            dx[i0:i1], do[o0:o1] = (c.transpose(1, 2) @ Y)[at_i], (c @ X)[at_o]
        if case["rounded"]:  # the rows themselves
            dx[:s["x"].shape[0]] += s["x"]
            do[:s["o"].shape[0]] += s["o"]
        return {"in": dx, "out": do}
    if kind == "adjoint":
        s = prepare(case, seed)
        ii, ip, first, oi, op, meta = s["batch"]
        ids_in, slot_in = torch.unique(ii, return_inverse=True)
        ids_out, slot_out = torch.unique(oi, return_inverse=True)
        g_in, g_out = (torch.zeros(s[k].shape, dtype=torch.float64, device="cuda") for k in ("g_in", "g_out"))
        loss = torch.zeros(1, dtype=torch.float64, device="cuda")
        for b0 in range(0, case["n"], 8192):
            b1 = min(case["n"], b0 + 8192)
            i0, i1, o0, o1 = int(ip[b0]), int(ip[b1]), int(op[b0]), int(op[b1])
            X, Y, M, label, real, at_i, at_o = _dense_steps(None, ip[b0:b1 + 1] - i0, first[b0:b1], None,
                                                            op[b0:b1 + 1] - o0, meta[o0:o1], s["wih"][ii[i0:i1].long()],
                                                            s["woh"][oi[o0:o1].long()])
            f = Y @ X.transpose(1, 2)
            w = M.unsqueeze(2) * real
            loss += (w * torch.nn.functional.softplus(-(2 * label - 1) * f, threshold=700.0)).sum()
            c = w * (torch.sigmoid(f) - label)
            g_in.index_add_(0, slot_in[i0:i1], (c.transpose(1, 2) @ Y)[at_i])
            g_out.index_add_(0, slot_out[o0:o1], (c @ X)[at_o])
        pad = lambda v, n: torch.nn.functional.pad(v, (0, n - v.numel()))
        return {"loss": loss, "n_in": ids_in.numel(), "in_ids": pad(ids_in, g_in.shape[0]), "g_in": g_in,
                "n_out": ids_out.numel(), "out_ids": pad(ids_out, g_out.shape[0]), "g_out": g_out}
    return None  # training orders its own rounding; the other outputs are whole numbers
