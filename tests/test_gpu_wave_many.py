"""Wide pairs by a warp each (more queued than a CTA each is for): bands on both
sides of what 4, 8 and 16 row words per thread hold and beyond all of them (a
CTA takes those), in clustering iterations and in speculative rounds, against
the oracle's clusters and scores."""
from __future__ import annotations

import numpy as np
import pytest

import ngia
from oracle import oracle
from tests.helpers import seqs_to_db

pytestmark = pytest.mark.gpu


def _copies(rng, alpha, base, n, frac, shorter):
    """n copies with a share of residues replaced, and up to `shorter` dropped at one place."""
    out = []
    for _ in range(n):
        x = base.copy()
        hit = rng.random(len(x)) < frac * rng.random()
        x[hit] = alpha[rng.integers(0, len(alpha), int(hit.sum()))]
        cut = int(rng.integers(0, shorter + 1))
        o = int(rng.integers(0, len(x) - cut + 1))
        out.append(np.delete(x, slice(o, o + cut)).tobytes())
    return out


# (type, similarity, length): blocks a query block's band covers
@pytest.mark.parametrize("db_type,s,L", [
    (0, 0.5, 4000),    # 127: 4 words, the class of windows up to 112 and the next
    (0, 0.5, 4200),    # 133
    (0, 0.6, 10000),   # 253: 8 words
    (0, 0.6, 10400),   # 263: 16 words
    (0, 0.5, 15500),   # 487
    (0, 0.5, 16300),   # 511, a representative of 510 blocks
    (0, 0.5, 20000),   # 629: too wide for a warp
    (1, 0.5, 4600),
    (1, 0.5, 17000),   # 535
])
def test_many_wide_pairs(cuda_device, db_type, s, L):
    rng = np.random.default_rng(L)
    alpha = np.frombuffer(b"ACGT" if db_type == 0 else b"ACDEFGHIKLMNPQRSTVWY", np.uint8)
    base = alpha[rng.integers(0, len(alpha), L)]
    seqs = [base.tobytes()] + _copies(rng, alpha, base, 7, 1.0, 40) + _copies(rng, alpha, base, 6, 1.0, int(L * (1 - s)))
    db = seqs_to_db(db_type, seqs)
    p = ngia.params_clamp(db_type, s, 5 if db_type == 0 else 2, 1)
    exp = np.stack([oracle.pair(db.words, db.rec_off, db_type, p.similarity, p.word_length, 0, i) for i in range(db.n)])
    member = (exp[:, 4] != 0) & (exp[:, 6] != 0)
    member[0] = True
    with ngia.Context(db) as ctx:
        for warp_pairs in (56, 10 ** 6):  # a warp per pair from two pairs on; a CTA per pair
            ctx.set_tuning(2, 32, warp_pairs)
            ctx.begin(p, ngia.MODE_PLAIN)
            ctx.step(1)
            cl, ident = ctx.end()[:2]
            assert ((cl == 0) == member).all()
            assert (ident[1:][member[1:]] == exp[1:, 2][member[1:]]).all()


@pytest.mark.parametrize("L", [5500, 9000])  # windows up to 112 blocks, and wider
def test_many_wide_pairs_in_rounds(cuda_device, L):
    rng = np.random.default_rng(L)
    alpha = np.frombuffer(b"ACGT", np.uint8)
    seqs = []
    for _ in range(3):
        base = alpha[rng.integers(0, 4, L)]
        seqs += _copies(rng, alpha, base, 90, 0.4, 60)
    db = seqs_to_db(0, seqs)
    p = ngia.params_clamp(0, 0.7, 5, 1)
    ocl, oid, _ = oracle.cluster(db.words, db.rec_off, 0, p.similarity, p.word_length, p.precise)
    with ngia.Context(db) as ctx:
        cl, ident = ctx.cluster(p, ngia.MODE_SPEC)[:2]
    assert (cl == ocl).all() and (ident == oid).all()


# (type, similarity, length, dropped): blocks a query block's band covers
@pytest.mark.parametrize("db_type,s,L,drop", [
    (0, 0.9, 300, 20),     # one chunk row per thread and fewer
    (0, 0.7, 1000, 200),   # 21, 32 blocks: 4 words
    (0, 0.8, 2200, 300),   # 29
    (0, 0.75, 2100, 300),  # 35: 8 words
    (0, 0.6, 2047, 300),   # 53, 64 blocks
    (0, 0.6, 2200, 60),    # 57: 16 words, the class of windows up to 112 and the narrower
    (0, 0.6, 3900, 100),   # 99
    (0, 0.7, 4090, 100),   # 79, 128 blocks
    (0, 0.7, 5400, 100),   # 103: too wide for 8 threads
    (0, 0.9, 12000, 100),  # 77, long records
    (1, 0.5, 380, 100),
    (1, 0.7, 900, 200),
    (1, 0.7, 5400, 60),
])
def test_many_pairs_of_common_width(cuda_device, db_type, s, L, drop):
    rng = np.random.default_rng(L + db_type)
    alpha = np.frombuffer(b"ACGT" if db_type == 0 else b"ACDEFGHIKLMNPQRSTVWY", np.uint8)
    base = alpha[rng.integers(0, len(alpha), L)]
    seqs = [base.tobytes()] + _copies(rng, alpha, base, 30, 3 * (1 - s), 3) + _copies(rng, alpha, base, 17, 1 - s, drop)
    db = seqs_to_db(db_type, seqs)
    w = 5 if db_type == 0 else 2
    for precise in (1, 0):  # 0: the short-word test follows the alignment
        p = ngia.params_clamp(db_type, s, w, precise)
        exp = np.stack([oracle.pair(db.words, db.rec_off, db_type, p.similarity, p.word_length, 0, i)
                        for i in range(db.n)])
        member = (exp[:, 4] != 0) & (exp[:, 6] != 0) & ((exp[:, 5] != 0) | (precise == 1))
        member[0] = True
        with ngia.Context(db) as ctx:
            ctx.set_tuning(2, 32, 56)
            for mode in (ngia.MODE_PLAIN, ngia.MODE_GRAPH):
                ctx.begin(p, mode)
                ctx.step(1)
                cl, ident = ctx.end()[:2]
                assert ((cl == 0) == member).all()
                assert (ident[1:][member[1:]] == exp[1:, 2][member[1:]]).all()


@pytest.mark.parametrize("db_type,s,L", [(0, 0.85, 700), (0, 0.8, 2400), (0, 0.7, 5200), (1, 0.6, 500)])
def test_rounds_and_scores_of_common_width(cuda_device, db_type, s, L):
    rng = np.random.default_rng(L)
    alpha = np.frombuffer(b"ACGT" if db_type == 0 else b"ACDEFGHIKLMNPQRSTVWY", np.uint8)
    seqs = []
    for _ in range(8):
        base = alpha[rng.integers(0, len(alpha), L)]
        seqs += _copies(rng, alpha, base, 70, 1.5 * (1 - s), 40)
    db = seqs_to_db(db_type, seqs)
    p = ngia.params_clamp(db_type, s, 5 if db_type == 0 else 2, 0)
    ocl, oid, _ = oracle.cluster(db.words, db.rec_off, db_type, p.similarity, p.word_length, p.precise)
    with ngia.Context(db) as ctx:
        cl, ident = ctx.cluster(p, ngia.MODE_SPEC)[:2]
        got = ctx.pair_scores(p, 0, np.arange(db.n))
    assert (cl == ocl).all() and (ident == oid).all()
    exp = np.stack([oracle.pair(db.words, db.rec_off, db_type, p.similarity, p.word_length, 0, i)
                    for i in range(db.n)])
    assert (got[:, 2] == exp[:, 2]).all()
