"""The adjoint's sparse rows: vocabularies at the edges of the mark words (32 rows) and tiles
(32,768 rows), rows referenced once, twice in one minibatch, and by every minibatch; row ids,
loss and gradients against numpy in 64 bits."""
import numpy as np
import pytest

import sgns

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# fp32 sums of at most a few hundred terms of size <= 1: error below 300 * 2^-24 of the largest
TOL = {0: 2e-5, 1: 2e-5, 2: 1e-12}


def batch(V, n, seed):
    rng = np.random.default_rng(seed)
    ins, outs, first, ip, op, meta = [], [], [], [0], [0], []
    for b in range(n):
        I, O = int(rng.integers(1, 41)), int(rng.integers(2, 13 if b % 2 else 8))
        i = rng.integers(0, V, I)
        i[0] = V - 1 if b % 3 == 0 else 0          # the last row, the first row
        if I > 3:
            i[2] = i[1]                            # the same row twice
        o = rng.integers(0, V, O)
        o[0] = min(V - 1, 32 * (V // 64))          # one row of every minibatch
        ins += i.tolist()
        outs += o.tolist()
        first.append(int(rng.integers(0, I + 1)))
        ip.append(len(ins))
        op.append(len(outs))
        meta += rng.integers(1, 4, O).tolist()
    return ins, ip, first, outs, op, meta


@pytest.mark.parametrize("dtype", [0, 1, 2])
@pytest.mark.parametrize("V,d,n", [(2, 8, 3), (31, 12, 9), (32, 16, 20), (33, 128, 40), (32767, 36, 60), (32768, 64, 60),
                                   (32769, 100, 300), (100_003, 5, 50), (131_072, 256, 30)])
def test_sparse_rows(V, d, n, dtype, sgns_lib):
    ins, ip, first, outs, op, meta = batch(V, n, seed=V + d)
    rng = np.random.default_rng(d)
    scale = 1.0 / np.sqrt(d)
    wih, woh = (torch.tensor(rng.standard_normal((V, d)) * scale) for _ in range(2))
    ty = {0: torch.float32, 1: torch.bfloat16, 2: torch.float64}[dtype]
    wih, woh = wih.to(ty), woh.to(ty)
    x, o = wih.double().numpy(), woh.double().numpy()
    g_in, g_out, loss = np.zeros((V, d)), np.zeros((V, d)), 0.0
    for b in range(n):
        i, j, m = np.array(ins[ip[b]:ip[b + 1]]), np.array(outs[op[b]:op[b + 1]]), np.array(meta[op[b]:op[b + 1]])
        label = np.zeros((len(j), len(i)))
        label[0, :first[b]] = 1
        label[-1, first[b]:] = 1
        f = o[j] @ x[i].T
        loss += (m[:, None] * np.logaddexp(0.0, -(2 * label - 1) * f)).sum()
        c = m[:, None] * (1 / (1 + np.exp(-f)) - label)
        np.add.at(g_in, i, c.T @ o[j])
        np.add.at(g_out, j, c @ x[i])
    dev = lambda a: torch.tensor(np.asarray(a, np.int32), device="cuda")
    acc = torch.float64 if dtype == 2 else torch.float32
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    ids = [torch.full((len(a),), -1, dtype=torch.int32, device="cuda") for a in (ins, outs)]
    grads = [torch.full((len(a), d), float("nan"), dtype=acc, device="cuda") for a in (ins, outs)]
    wih, woh = wih.cuda(), woh.cuda()
    for _ in range(2):  # the second call finds the first one's scratch and results
        n_in, n_out = sgns.loss_adjoint(dtype, d, V, dev(ip), dev(ins), dev(first), dev(op), dev(outs), dev(meta),
                                        wih.data_ptr(), woh.data_ptr(), out, ids[0], grads[0], ids[1], grads[1])
    assert abs(float(out) - loss) <= TOL[dtype] * abs(loss)
    for got_n, got_ids, got, want, refs in ((n_in, ids[0], grads[0], g_in, ins), (n_out, ids[1], grads[1], g_out, outs)):
        rows = np.unique(refs)
        assert got_n == len(rows) and np.array_equal(got_ids[:got_n].cpu().numpy(), rows)
        err = np.abs(got[:got_n].double().cpu().numpy() - want[rows])
        assert err.max() <= TOL[dtype] * max(1.0, np.abs(want[rows]).max())
