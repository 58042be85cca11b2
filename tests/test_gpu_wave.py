"""The group-per-pair kernels (a warp, a CTA or 16 threads per pair) at the
edges of their forms: band widths around each row-word count, queries of 16
and 17 blocks, last blocks of 1, 16, 17 and 32 columns, against the oracle's
scores; and whole clusterings of widely spread lengths, every class forced to
either kernel."""
from __future__ import annotations

import numpy as np
import pytest

import ngia
from oracle import oracle
from tests.helpers import seqs_to_db

pytestmark = pytest.mark.gpu


def _seq(rng, alpha, L, base=None):
    out = np.frombuffer(alpha, np.uint8)[rng.integers(0, len(alpha), L)]
    if base is not None:  # a copy with one residue in six replaced
        b = np.frombuffer(base, np.uint8)
        keep = rng.random(min(L, len(b))) < 5 / 6
        out[:len(keep)][keep] = b[:len(keep)][keep]
    return out.tobytes()


# (rep length, similarity, query lengths): the bands cover one row word per
# thread of a warp (up to 47 blocks), two (64), one of a CTA (128), and 2, 4,
# 8 and 16 of a CTA; short queries take the 16-thread form.
@pytest.mark.parametrize("db_type,rep,s,queries", [
    (0, 1505, 0.99, (1505, 1500, 1489, 1473, 1472, 1441, 800)),
    (0, 2040, 0.6, (2040, 2033, 1700, 1025, 513, 512, 497, 33, 1)),
    (0, 4097, 0.5, (4096, 4081, 2100, 530, 512, 480, 16)),
    (0, 10001, 0.6, (9999, 6000, 1010, 512, 511, 65)),
    (0, 60003, 0.5, (50000, 20000, 500, 31)),
    (0, 20000, 0.97, (19990, 19500)),  # long pairs: every form's code ring wraps many times
    (0, 16000, 0.95, (15990, 15600)),
    (0, 30000, 0.93, (29990, 28500)),
    (1, 33000, 0.9, (32990, 31000)),
    (1, 40000, 0.8, (39000,)),
    (1, 1520, 0.9, (1520, 1400, 1040, 512, 500)),
    (1, 4100, 0.6, (4100, 2049, 544, 512, 496, 17)),
    (1, 9000, 0.5, (8990, 3000, 513, 512, 90)),
])
def test_scores_at_the_edges_of_the_forms(cuda_device, db_type, rep, s, queries):
    alpha = b"ACGT" if db_type == 0 else b"ACDEFGHIKLMNPQRSTVWY"
    rng = np.random.default_rng(rep)
    base = _seq(rng, alpha, rep)
    db = seqs_to_db(db_type, [base] + [_seq(rng, alpha, L, base if k % 2 else None) for k, L in enumerate(queries)])
    w = 5 if db_type == 0 else 3
    p = ngia.params_clamp(db_type, s, w, 0)
    with ngia.Context(db) as ctx:
        got = ctx.pair_scores(p, 0, np.arange(db.n))
    for i in range(db.n):
        exp = oracle.pair(db.words, db.rec_off, db_type, p.similarity, p.word_length, 0, i)
        assert got[i, 2] == exp[2] and got[i, 3] == exp[3], (i, int(db.read_len[i]), got[i].tolist(), exp.tolist())


@pytest.mark.parametrize("warp_pairs", ["0", "100000000"])
@pytest.mark.parametrize("db_type,s,w,precise", [(0, 0.8, 5, 0), (0, 0.9, 6, 1), (1, 0.5, 2, 0), (1, 0.8, 2, 1)])
def test_spread_lengths_cluster_as_the_oracle(cuda_device, monkeypatch, db_type, s, w, precise, warp_pairs):
    monkeypatch.setenv("NGIA_WARP_PAIRS", warp_pairs)
    kw = dict(type=0, len_dist=2, len_a=30.0, len_b=7000.0, len_min=30, len_max=7000) if db_type == 0 else \
        dict(type=1, len_dist=1, len_a=400.0, len_b=1.2, len_min=20, len_max=7000)
    seqs = ngia.synth(n_seqs=160, n_ancestors=9, subst_max=0.3, seed=7 + db_type, **kw)
    db = ngia.DB.pack(db_type, seqs, seqs.off)
    p = ngia.params_clamp(db_type, s, w, precise)
    ocl, oid, ost = oracle.cluster(db.words, db.rec_off, db_type, p.similarity, p.word_length, p.precise)
    with ngia.Context(db) as ctx:
        for mode in (ngia.MODE_PLAIN, ngia.MODE_GRAPH, ngia.MODE_SPEC):
            cl, ident, st = ctx.cluster(p, mode)
            assert np.array_equal(cl, ocl) and np.array_equal(ident, oid), mode
            assert st["iterations"] == ost["iterations"]
