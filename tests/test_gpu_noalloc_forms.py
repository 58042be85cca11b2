"""The three kernels behind ngia_rep_scores_noalloc (a group per pair, a
thread per pair with a row ring, a protein too long for the shared-memory
match table) against the oracle's scores: representatives of up to 64, 128
and more blocks, few and many queries (offsets repeat, so that many queries
need few records), queries longer than the representative, damaged records."""
from __future__ import annotations

import numpy as np
import pytest

import ngia
from oracle import oracle
from tests.helpers import seqs_to_db

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("db_type,longest,rep_len,n", [
    (0, 2300, 1450, 1), (0, 2300, 1450, 700), (0, 2300, 1450, 9001), (0, 2300, 33, 9001), (0, 4100, 3000, 9001),
    (0, 9000, 9000, 40), (1, 900, 380, 500), (1, 900, 380, 9001), (1, 4000, 3500, 9001), (1, 56000, 56000, 150), (1, 62000, 62000, 150),
])
def test_scores_of_every_form(cuda_device, db_type, longest, rep_len, n):
    torch = pytest.importorskip("torch")
    alpha = b"ACGT" if db_type == 0 else b"ACDEFGHIKLMNPQRSTVWY"
    rng = np.random.default_rng(longest + n)
    rep = np.frombuffer(alpha, np.uint8)[rng.integers(0, len(alpha), longest)].tobytes()
    seqs = [rep, rep[:rep_len] + b"#"]
    for L in (1, 31, 32, 33, 160, 481, 512, 513, rep_len - 1, min(longest, rep_len + 40)):
        b = np.frombuffer(rep, np.uint8)[:max(L, 1)].copy()
        hit = rng.random(len(b)) < 0.15
        b[hit] = np.frombuffer(alpha, np.uint8)[rng.integers(0, len(alpha), int(hit.sum()))]
        seqs.append(b.tobytes())
    db = seqs_to_db(db_type, seqs)
    r = int(np.flatnonzero(db.read_len == rep_len + 1)[0])
    s = 0.85
    exp = np.array([oracle.pair(db.words, db.rec_off, db_type, s, 5 if db_type == 0 else 3, r, i)[2]
                    for i in range(db.n)], dtype=np.int32)
    words = np.ascontiguousarray(db.words).copy()
    bad = len(words)
    words = np.concatenate([words, np.array([5, 9], np.uint32), np.zeros(64, np.uint32)])  # net > raw: not a record
    pick = rng.integers(0, db.n + 1, n)
    off = np.where(pick < db.n, db.rec_off[np.minimum(pick, db.n - 1)], bad).astype(np.int64)
    expect = np.where(pick < db.n, exp[np.minimum(pick, db.n - 1)], -1)
    d_words = torch.from_numpy(words.view(np.int32)).cuda()
    d_off = torch.from_numpy(off).cuda()
    out = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    ngia.rep_scores_noalloc(d_words.data_ptr(), int(db.rec_off[r]), d_off.data_ptr(), n, db_type, s, out.data_ptr(),
                            torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    wrong = np.flatnonzero(got != expect)
    assert wrong.size == 0, (int(wrong[0]), int(got[wrong[0]]), int(expect[wrong[0]]), wrong.size)
