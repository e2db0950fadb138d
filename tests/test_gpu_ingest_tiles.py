"""Walk-text parsing where its two paths through a tile (8192 bytes, 32 to a thread) meet: ids
of every length, dense tiles, newlines off the short path, every alignment of the text's start.
Tokens are whole numbers: they equal the oracle's."""
import numpy as np
import pytest

import sgns


def _ids(rng, length, count):
    lo = 10 ** (length - 1) if length > 1 else 0
    return rng.integers(lo, min(10 ** length, 2 ** 31), count)


def _text(kind, rng):
    if kind.startswith("digits"):  # " %u" per id, a newline directly behind every seventh
        ids = _ids(rng, int(kind[6:]), 6000)
        return b"".join(b" %d" % v + (b"\n" if k % 7 == 6 else b"") for k, v in enumerate(ids))
    if kind == "dense_ids":  # 4096 outputs to a tile
        return b"1 " * 9000
    if kind == "dense_walks":  # 8192 outputs to a tile
        return b"7\n" * 9000
    if kind == "zeros":  # leading zeros up to ten digits
        return b"".join(b" %0*d" % (int(rng.integers(1, 11)), int(rng.integers(0, 10))) for _ in range(5000)) + b"\n"
    if kind == "late_newlines":  # one newline behind a blank in each of several tiles, at its edges too
        t = bytearray(b" 12345\n" * 9000)
        for at in (8191, 8192, 3 * 8192 - 1, 3 * 8192, 4 * 8192 + 4000):
            t[at:at + 1] = b" \n"[at % 2:at % 2 + 1]
            t[at - 1:at] = b" "
        return bytes(t)
    if kind == "tabs":  # a tab or a CR in some tiles only
        t = bytearray(b" 123 45\n" * 7000)
        for at in (100 * 8, 8192, 5 * 8192 + 24):
            t[at] = 9 if at % 3 else 13
        return bytes(t)
    if kind == "blank_tile_end":  # a tile whose last 40 bytes are blank, the newline in the next
        return (b" 42" * 2730)[:8152] + b" " * 40 + b"\n" + b" 5 6\n" * 2000
    raise AssertionError(kind)


KINDS = ["digits%d" % k for k in range(1, 11)] + ["dense_ids", "dense_walks", "zeros", "late_newlines", "tabs",
                                                 "blank_tile_end"]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_parse_matches_oracle(kind, sgns_lib, oracle_mod):
    import torch

    rng = np.random.default_rng(sum(kind.encode()))
    text = _text(kind, rng)
    # the whole text, ends just before, at and behind a thread's and a tile's last byte
    for n, off in [(len(text), 0), (len(text), 5), (31, 0), (32, 0), (33, 1), (8191, 0), (8192, 0), (8193, 0),
                   (8200, 16), (16384, 7)]:
        part = text[:n]
        code, want, mx, _ = oracle_mod.parse_walks(part)
        assert code == 0
        buf = torch.tensor(np.frombuffer(b"9" * off + part, np.uint8).copy(), device="cuda")[off:]
        assert sgns.parse_walks_count(buf) == len(want)
        tok = torch.full((len(want) + 8,), -7, dtype=torch.int32, device="cuda")
        assert sgns.parse_walks(buf, tok) == (len(want), mx)
        got = tok.cpu().numpy()
        assert np.array_equal(got[:len(want)], want) and (got[len(want):] == -7).all(), (kind, n, off)
