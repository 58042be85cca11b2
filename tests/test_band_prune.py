"""The band rules of the alignment kernels (band_advance, tile.cuh), restated
step by step, against the oracle's whole-band scores: a pair whose score
reaches the cutoff gets exactly that score over the rows the rules keep, a
pair that does not is rejected, and no window is wider than window_need says.
Lengths around multiples of 32, skipped characters (net < raw), either record
the longer one, similarities from 0.1 to 1."""
from __future__ import annotations

import math

import numpy as np
import pytest

import ngia
from oracle import oracle
from tests.helpers import seqs_to_db

M32 = 0xFFFFFFFF


def _codes(rec, db_type):
    hw, P = (6, 2) if db_type == 0 else (30, 5)
    net = int(rec[1])
    out = []
    for k in range(net):
        w = hw + (k >> 5) * P
        out.append(sum(((int(rec[w + p]) >> (k & 31)) & 1) << p for p in range(P)))
    return out


def _pruned(r, q, L1, L2, s, B, cut):
    """(passes, score, widest window) by the kernels' rules."""
    net1, net2 = len(r), len(q)
    nb1, nq = (net1 + 31) // 32, (net2 + 31) // 32
    if B < 0 or nb1 == 0 or nq == 0:
        return 0 >= cut, 0, 0
    eq = {}
    for j, c in enumerate(r):
        eq.setdefault(c, [0] * nb1)[j >> 5] |= 1 << (j & 31)
    vlast = (1 << (net1 & 31)) - 1 if net1 & 31 else M32
    row = [M32] * nb1
    js, je = 0, min(B, nb1 - 1, max(0, (32 + net1 - cut) >> 5))
    frozen, i, widest = 0, 0, 0

    def zeros(j, mask=True):
        z = ~row[j] & M32
        return bin(z & vlast if mask and j == nb1 - 1 else z).count("1")

    while True:
        widest = max(widest, je - js + 1)
        for c in q[32 * i:32 * i + 32]:
            carry, e = 0, eq.get(c)
            for j in range(js, je + 1):
                x = row[j] & (e[j] if e else 0)
                t = row[j] + x + carry
                carry, row[j] = t >> 32, (t & M32) | (row[j] ^ x)
        i += 1
        if i >= nq:
            break
        left = net2 - 32 * i
        zw = sum(zeros(j, False) for j in range(js, je + 1))
        while js <= je and not (js >= i - B and frozen + zeros(js) + left >= cut):
            frozen += zeros(js)
            zw -= zeros(js, False)
            js += 1
        if frozen + zw + left < cut or frozen + max(net1 - 32 * js, 0) < cut:
            return False, None, widest
        while je > js and frozen + zw - zeros(je, False) + 32 + net1 - 32 * je < cut:
            zw -= zeros(je, False)
            je -= 1
        if je < min(i + B, nb1 - 1) and frozen + zw + net1 - 32 * je >= cut:
            je += 1
            row[je] = M32
        if js > je:
            break
    score = frozen + sum(zeros(j) for j in range(js, je + 1))
    return score >= cut, score, widest


def _mutate(rng, seq, rate, alpha):
    out = bytearray()
    for b in seq:
        u = rng.random()
        if u < rate / 4:
            continue
        if u < rate / 2:
            out.append(alpha[int(rng.integers(0, len(alpha)))])
        out.append(alpha[int(rng.integers(0, len(alpha)))] if rng.random() < rate else b)
    return bytes(out)


@pytest.mark.parametrize("db_type", [0, 1])
@pytest.mark.parametrize("s", [0.1, 0.5, 0.7, 0.85, 0.95, 1.0])
def test_pruned_band_gives_the_oracles_accepted_scores(db_type, s):
    alpha = b"ACGT" if db_type == 0 else b"ACDEFGHIKLMNPQRSTVWY"
    rng = np.random.default_rng(1000 * db_type + int(100 * s))
    seqs = []
    for L in (1, 15, 31, 32, 33, 64, 95, 160, 257, 300, 410):
        base = bytes(alpha[int(k)] for k in rng.integers(0, len(alpha), L))
        seqs.append(base)
        for rate in (0.02, 0.1, 0.3):
            m = _mutate(rng, base, rate, alpha)
            a = int(rng.integers(0, max(1, len(m) // 5)))
            m = m[a:]  # a window of the sequence
            if len(m) > 3 and rng.random() < 0.4:  # skipped characters
                k = int(rng.integers(0, len(m)))
                m = m[:k] + b"#" * int(rng.integers(1, 9)) + m[k:]
            seqs.append(m or b"A")
    db = seqs_to_db(db_type, seqs)
    w = 5 if db_type == 0 else 3
    sf = np.float32(s)
    codes = [_codes(db.record(i), db_type) for i in range(db.n)]
    accepted = 0
    for a in range(db.n):
        for b in range(db.n):
            if rng.random() < 0.6:
                continue
            L1, L2 = int(db.read_len[a]), int(db.read_len[b])
            _, _, score, B = (int(v) for v in oracle.pair(db.words, db.rec_off, db_type, s, w, a, b)[:4])
            cut = math.ceil(float(np.float32(L2) * sf))
            ok, got, widest = _pruned(codes[a], codes[b], L1, L2, s, B, cut)
            assert ok == (score >= cut), (a, b, score, cut, got)
            if ok:
                accepted += 1
                assert got == score, (a, b, score, got)
            nb1 = (len(codes[a]) + 31) // 32
            need = min(min(2 * B + 1, nb1) if B >= 0 else 0, max(0, L2 - cut) // 32 + max(0, L1 - cut) // 32 + 3)
            assert widest <= need, (a, b, widest, need)
    assert accepted > 20


@pytest.mark.parametrize("cap,widest", [(64, 48), (128, 112)])
def test_row_indices_stay_inside_the_shared_rows(cap, widest):
    """SmemRing::fit (tile.cuh) restated: every row a tile touches, and the row
    of the block that enters next, lie within the CAP rows of a lane."""
    rng = np.random.default_rng(cap)
    for _ in range(300):
        off, js, je = 0, 0, int(rng.integers(0, widest))
        for _ in range(150):
            slots = int(rng.integers(je - js + 1, widest + 1))  # the warp's widest window
            if not js - off + slots < cap:
                assert je - off < cap
                off = js
            assert js >= off and js + slots - 1 - off < cap
            js = min(js + int(rng.integers(0, 4)), je)
            je -= int(rng.integers(0, je - js + 1)) if rng.random() < 0.2 else 0
            if rng.random() < 0.8 and je - js + 1 < widest:
                je += 1
                assert je - off < cap
