"""The short-word filter (tables of 1, 2 or 4 words per lookup, counting that
stops once the answer is settled, a thread or a warp per candidate) against the
oracle's tests of every pair of the first iteration: lengths around blocks,
around the four and two blocks of a step, and around the length from which a
warp takes a candidate; candidates from unrelated to nearly equal, so that
counts lie on both sides of the least that passes."""
from __future__ import annotations

import numpy as np
import pytest

import ngia
from oracle import oracle
from tests.helpers import seqs_to_db

pytestmark = pytest.mark.gpu

LENGTHS = (16, 17, 31, 32, 33, 63, 64, 65, 95, 97, 127, 128, 129, 160, 161, 255, 257, 1023, 1025, 2047, 2048, 2049,
           2081, 3071, 3073, 4095)


@pytest.mark.parametrize("db_type,w,s", [(0, 4, 0.9), (0, 5, 0.9), (0, 5, 0.97), (0, 6, 0.9), (0, 7, 0.93),
                                         (0, 8, 0.95), (1, 2, 0.7), (1, 3, 0.8), (1, 3, 0.9)])
def test_word_passes_of_one_iteration(cuda_device, db_type, w, s):
    rng = np.random.default_rng(100 * w + db_type)
    alpha = np.frombuffer(b"ACGT" if db_type == 0 else b"ACDEFGHIKLMNPQRSTVWY", np.uint8)
    unit = min(4100, 2 * len(alpha) ** w // 5)  # the representative holds at most 2 of 5 words
    base = np.resize(alpha[rng.integers(0, len(alpha), unit)], 4100)
    seqs = [base.tobytes()]
    for L in LENGTHS:
        for frac in (0.0, 0.02, 0.05, 0.1, 0.2, 0.4, 1.0):  # share of residues replaced
            o = int(rng.integers(0, len(base) - L + 1))
            x = base[o:o + L].copy()
            hit = rng.random(L) < frac
            x[hit] = alpha[rng.integers(0, len(alpha), int(hit.sum()))]
            seqs.append(x.tobytes())
    db = seqs_to_db(db_type, seqs)
    p = ngia.params_clamp(db_type, s, w, 0)
    assert p.word_length == w
    exp = np.stack([oracle.pair(db.words, db.rec_off, db_type, p.similarity, w, 0, i) for i in range(1, db.n)])
    base_ok = exp[:, 4] != 0
    word_ok = base_ok & (exp[:, 5] != 0)
    assert 0 < word_ok.sum() < base_ok.sum()
    with ngia.Context(db) as ctx:
        for mode in (ngia.MODE_PLAIN, ngia.MODE_GRAPH):
            ctx.set_tuning(1, 32, -1)
            ctx.begin(p, mode)
            ctx.step(1)
            st = ctx.stats()
            cl, ident = ctx.end()[:2]
            # the representative itself is a candidate of its own iteration
            assert st["base_pass"] - 1 == base_ok.sum()
            assert sum(st["class_pairs"]) - 1 == word_ok.sum()
            member = word_ok & (exp[:, 6] != 0)
            assert ((cl[1:] == 0) == member).all()


@pytest.mark.parametrize("db_type,w,s", [(0, 5, 0.97), (1, 3, 0.9)])
def test_word_passes_of_records_in_any_order(cuda_device, db_type, w, s):
    """Long records behind short ones (the filter gives a warp each to those in
    front): candidates of one representative, the rest in random order."""
    rng = np.random.default_rng(7 + db_type)
    alpha = np.frombuffer(b"ACGT" if db_type == 0 else b"ACDEFGHIKLMNPQRSTVWY", np.uint8)
    base = np.resize(alpha[rng.integers(0, len(alpha), 400 if db_type == 0 else 3200)], 4100)
    seqs = [base.tobytes()]
    for L in (40, 300, 2040, 2049, 2600, 4000) * 20:
        x = base[:L].copy()
        hit = rng.random(L) < rng.choice([0.0, 0.02, 0.1, 1.0])
        x[hit] = alpha[rng.integers(0, len(alpha), int(hit.sum()))]
        seqs.append(x.tobytes())
    db = seqs_to_db(db_type, seqs)
    order = np.concatenate([[0], 1 + rng.permutation(db.n - 1)])
    recs = ngia.Records(db_type, np.ascontiguousarray(db.words), np.ascontiguousarray(db.rec_off[order]))
    p = ngia.params_clamp(db_type, s, w, 0)
    exp = np.stack([oracle.pair(db.words, db.rec_off, db_type, p.similarity, w, 0, i) for i in order])
    ok = (exp[:, 4] != 0) & (exp[:, 5] != 0)
    ok[0] = True
    with ngia.Context(recs) as ctx:
        ctx.set_tuning(1, 32, -1)
        ctx.begin(p, ngia.MODE_GRAPH)
        ctx.step(1)
        st = ctx.stats()
        cl = ctx.end()[0]
    assert sum(st["class_pairs"]) == ok.sum()
    assert ((cl == 0) == (ok & ((exp[:, 6] != 0) | (np.arange(len(ok)) == 0)))).all()
