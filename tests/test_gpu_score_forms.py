"""Every form of the score calls against the oracle's scores, the numbers of
pairs following the rules that choose between the forms (pairs per SM):
ngia_rep_scores_noalloc with a warp or a CTA, 8 threads and one thread per
pair, and with its fixed rows (several queries per thread); ngia_pair_scores
with four pairs per warp and with a thread per pair."""
from __future__ import annotations

import numpy as np
import pytest

import ngia
from oracle import oracle
from tests.helpers import seqs_to_db

pytestmark = pytest.mark.gpu

ALPHA = {0: np.frombuffer(b"ACGT", np.uint8), 1: np.frombuffer(b"ACDEFGHIKLMNPQRSTVWY", np.uint8)}


def _mutants(rng, db_type, base, lengths):
    """Windows of the given lengths of a sequence (longer ones go on at random), a share of residues replaced."""
    alpha, out = ALPHA[db_type], []
    for L in lengths:
        o = int(rng.integers(0, max(0, len(base) - L) + 1))
        b = np.concatenate([base[o:o + L], alpha[rng.integers(0, len(alpha), max(0, L - len(base)))]])
        hit = rng.random(L) < 0.4 * rng.random()
        b[hit] = alpha[rng.integers(0, len(alpha), int(hit.sum()))]
        out.append(b.tobytes())
    return out


def _noalloc(torch, db, rep, s, pick):
    words = torch.from_numpy(np.ascontiguousarray(db.words).view(np.int32)).cuda()
    off = torch.from_numpy(db.rec_off[pick].astype(np.int64)).cuda()
    out = torch.full((len(pick),), -7, dtype=torch.int32, device="cuda")
    ngia.rep_scores_noalloc(words.data_ptr(), int(db.rec_off[rep]), off.data_ptr(), len(pick), db.type, s,
                            out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _oracle(db, s, rep, w):
    return np.array([oracle.pair(db.words, db.rec_off, db.type, s, w, rep, i)[2] for i in range(db.n)], dtype=np.int32)


# per SM: 1 and 10 are groups of 32 or 128 threads (of 8 for 10 and more than
# 64 blocks), 30 and 60 of 8 or a thread by the length, 130 a thread for up to
# 112 blocks
@pytest.mark.parametrize("per", [1, 10, 30, 60, 130])
@pytest.mark.parametrize("blocks", [4, 16, 17, 33, 48, 49, 65, 97, 112, 113, 128, 129])
@pytest.mark.parametrize("db_type", [0, 1])
def test_noalloc_forms_by_pairs_per_sm(cuda_device, db_type, blocks, per):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(1000 * blocks + per)
    net = 32 * blocks - int(rng.integers(0, 32))  # last blocks of any width
    alpha = ALPHA[db_type]
    base = alpha[rng.integers(0, len(alpha), net)]
    lengths = [net, net - 1, net + 33, 1, 15, 32, 33] + [int(x) for x in rng.integers(max(1, net // 2), net + 1, 9)]
    db = seqs_to_db(db_type, [base.tobytes()] + _mutants(rng, db_type, base, lengths))
    rep = next(i for i in range(db.n) if db.read_len[i] == net)
    s = 0.7
    exp = _oracle(db, s, rep, 5 if db_type == 0 else 3)
    pick = rng.integers(0, db.n, per * sms + int(rng.integers(1, 32)))
    got = _noalloc(torch, db, rep, s, pick)
    wrong = np.flatnonzero(got != exp[pick])
    assert wrong.size == 0, (int(db.read_len[pick[wrong[0]]]), int(got[wrong[0]]), int(exp[pick[wrong[0]]]), wrong.size)


@pytest.mark.parametrize("rep_len", [56000, 65536])  # 599 and 512 rows of the fixed array: 512 threads
def test_noalloc_fixed_rows_take_several_queries_per_thread(cuda_device, rep_len):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(rep_len)
    base = ALPHA[1][rng.integers(0, 20, rep_len)]
    db = seqs_to_db(1, [base.tobytes()] + _mutants(rng, 1, base, [1, 31, 32, 33, 64, 65, 90, 120]))
    exp = _oracle(db, 0.5, 0, 3)
    pick = 1 + rng.integers(0, db.n - 1, 1300)
    got = _noalloc(torch, db, 0, 0.5, pick)
    assert np.array_equal(got, exp[pick])


# (type, length, similarity): windows of few, up to 48, up to 112 and of 103
# blocks (which 8 threads cannot hold), and wider
@pytest.mark.parametrize("db_type,L,s", [(0, 300, 0.9), (0, 1450, 0.85), (0, 2040, 0.7), (0, 3500, 0.6), (0, 5400, 0.7),
                                         (0, 4200, 0.5), (1, 380, 0.7), (1, 1500, 0.6), (1, 3500, 0.6), (1, 5400, 0.7)])
@pytest.mark.parametrize("warp_pairs", ["1120", "0"])  # four pairs per warp from 180 or 400 pairs on; a thread each
def test_pair_scores_of_many_pairs(cuda_device, monkeypatch, db_type, L, s, warp_pairs):
    monkeypatch.setenv("NGIA_WARP_PAIRS", warp_pairs)
    rng = np.random.default_rng(L)
    alpha = ALPHA[db_type]
    base = alpha[rng.integers(0, len(alpha), L)]
    kinds = _mutants(rng, db_type, base, [L - int(x) for x in rng.integers(0, min(L // 8, 70), 24)])
    db = seqs_to_db(db_type, [base.tobytes()] + [kinds[k % len(kinds)] for k in range(700)])
    w = 5 if db_type == 0 else 3
    p = ngia.params_clamp(db_type, s, w, 0)
    known = {}
    exp = np.empty((db.n, 2), dtype=np.int64)
    for i in range(db.n):
        key = db.record(i).tobytes()
        if key not in known:
            o = oracle.pair(db.words, db.rec_off, db_type, p.similarity, p.word_length, 0, i)
            known[key] = (int(o[2]), int(o[3]))
        exp[i] = known[key]
    with ngia.Context(db) as ctx:
        got = ctx.pair_scores(p, 0, np.arange(db.n))
    assert np.array_equal(got[:, 2], exp[:, 0]) and np.array_equal(got[:, 3], exp[:, 1])
