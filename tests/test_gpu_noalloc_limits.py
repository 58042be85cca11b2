"""ngia_rep_scores_noalloc at the largest number of queries it accepts: the
thread-per-pair kernel and the one of four pairs per warp stride over them past
the end of the 32-bit range."""
from __future__ import annotations

import numpy as np
import pytest

import ngia
from oracle import oracle
from tests.helpers import seqs_to_db

pytestmark = pytest.mark.gpu

MOST = 2 ** 31 - 1


@pytest.mark.parametrize("rep_len", [9, 3600])  # a thread per pair; 113 blocks: four pairs per warp
def test_most_queries(cuda_device, rep_len):
    torch = pytest.importorskip("torch")
    if torch.cuda.mem_get_info()[0] < 40 * 2 ** 30:
        pytest.skip("26 GB of offsets and scores")
    rng = np.random.default_rng(rep_len)
    rep = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, rep_len)].tobytes()
    db = seqs_to_db(0, [rep, rep[:2], rep[:1]])
    exp = [oracle.pair(db.words, db.rec_off, 0, 0.5, 5, 0, i)[2] for i in range(3)]
    assert exp[1] != exp[2]
    words = torch.from_numpy(np.ascontiguousarray(db.words).view(np.int32)).cuda()
    off = torch.full((MOST,), int(db.rec_off[1]), dtype=torch.int64, device="cuda")
    others = torch.tensor([0, 1, MOST // 2, MOST - 40000, MOST - 2, MOST - 1], device="cuda")
    off[others] = int(db.rec_off[2])
    out = torch.full((MOST,), -7, dtype=torch.int32, device="cuda")
    ngia.rep_scores_noalloc(words.data_ptr(), int(db.rec_off[0]), off.data_ptr(), MOST, 0, 0.5, out.data_ptr(),
                            torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert (out[others] == exp[2]).all()
    out[others] = exp[1]
    wrong = 0
    for k in range(0, MOST, 1 << 28):
        wrong += int((out[k:k + (1 << 28)] != exp[1]).sum())
    assert wrong == 0
