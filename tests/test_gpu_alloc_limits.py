"""Sizes that no allocation can hold are refused as such, and leave nothing
behind: the next database opens and clusters."""
from __future__ import annotations

import numpy as np
import pytest

import ngia
from oracle import oracle
from tests.helpers import family_db

pytestmark = pytest.mark.gpu

NGIA_E_NOMEM = -4


@pytest.mark.parametrize("db_type,n_words", [(1, 2 ** 61), (0, 2 ** 61), (1, 2 ** 62), (0, 2 ** 62), (0, 2 ** 63 - 1)])
def test_more_words_than_any_device_holds(cuda_device, db_type, n_words):
    db = family_db(db_type, n=40, anc=3, seed=5)
    huge = ngia.Records.subset(db, np.arange(db.n))
    huge.view.n_words = n_words  # refused before anything is copied
    with pytest.raises(ngia.NgiaError) as e:
        ngia.Context(huge)
    assert e.value.code == NGIA_E_NOMEM
    p = ngia.params_clamp(db_type, 0.8, 5 if db_type == 0 else 2, 0)
    ocl, oid, _ = oracle.cluster(db.words, db.rec_off, db_type, p.similarity, p.word_length, p.precise)
    with ngia.Context(db) as ctx:
        cl, ident, _ = ctx.cluster(p, ngia.MODE_SPEC)
    assert np.array_equal(cl, ocl) and np.array_equal(ident, oid)
