"""GPU: the serving path (ngia_serve_*) — batches assigned to a resident
representative set, leftovers clustered among themselves — against the
oracle's replay of the same batches (ora_assign), and every batch's result
identical alone and in a mix of batches running side by side."""
from __future__ import annotations

import numpy as np
import pytest

import ngia
from oracle import oracle
from tests.helpers import seqs_to_db, split

pytestmark = pytest.mark.gpu

GEN = {
    0: dict(type=0, len_a=600.0, len_b=80.0, len_min=300, len_max=900, subst_max=0.2, indel_max=3),
    1: dict(type=1, len_dist=1, len_a=200.0, len_b=0.5, len_min=20, len_max=1500, subst_max=0.5, indel_max=5),
}


def _workload(db_type: int, s: float, w: int, n_res: int, anc: int, sizes: list[int], seed: int):
    """Resident representatives (the clustering of n_res sequences, in
    creation order) and query batches drawn from the same ancestors beyond
    them, 10% of them from novel ancestors."""
    p = ngia.params_clamp(db_type, s, w, 0)
    total = n_res + sum(sizes)
    seq, off = ngia.synth(**GEN[db_type], n_seqs=total, n_ancestors=anc, novel_frac=0.1, seed=seed)
    seqs = split(seq, off)
    res_seq, res_off = ngia.synth(**GEN[db_type], n_seqs=n_res, n_ancestors=anc, seed=seed)
    res_db = ngia.DB.pack(db_type, res_seq, res_off)
    cl, _, _ = oracle.cluster(res_db.words, res_db.rec_off, db_type, p.similarity, p.word_length, p.precise)
    reps = ngia.Records.subset(res_db, np.flatnonzero(cl == np.arange(res_db.n)))
    batches, k = [], n_res
    for m in sizes:
        batches.append(seqs_to_db(db_type, seqs[k:k + m]))
        k += m
    return p, reps, batches


def _expected(p, reps, b):
    return oracle.assign(reps.words, reps.rec_off, b.words, b.rec_off, b.type, p.similarity, p.word_length,
                         p.precise)


@pytest.mark.parametrize("db_type,s,w", [(0, 0.9, 5), (0, 0.95, 5), (1, 0.9, 3)])
def test_serve_matches_oracle_alone_and_mixed(cuda_device, db_type, s, w):
    sizes = [1, 7, 64, 250, 33, 400, 2, 120, 17, 90]
    p, reps, batches = _workload(db_type, s, w, 500 if db_type == 0 else 400, 10, sizes, seed=81 + db_type)
    exp = [_expected(p, reps, b) for b in batches]
    assert sum(int((e[0] >= 0).sum()) for e in exp) > 50  # queries do join resident representatives
    with ngia.Server(reps, p, slots=4, max_batch=512) as srv:
        assert srv.slots == 4
        # the mix: everything submitted at once, batches run side by side
        tickets = [srv.submit(b) for b in batches]
        mixed = [srv.wait(t) for t in tickets]
        # alone: one batch at a time
        alone = [srv.wait(srv.submit(b)) for b in batches]
    for b, e, m, a in zip(batches, exp, mixed, alone):
        assert np.array_equal(m[0], e[0]) and np.array_equal(m[1], e[1]), f"batch of {b.n}: mixed != oracle"
        assert np.array_equal(a[0], m[0]) and np.array_equal(a[1], m[1]), f"batch of {b.n}: alone != mixed"
        info = m[2]
        assert info["done"] == 1 and info["resident"] == int((e[0] >= 0).sum()) and info["new_reps"] == e[2]
    assert len({m[2]["slot"] for m in mixed}) > 1  # the mix did use several slots


def test_serve_poll_and_errors(cuda_device):
    p, reps, batches = _workload(0, 0.9, 5, 300, 6, [40, 5], seed=91)
    with ngia.Server(reps, p, slots=2, max_batch=64) as srv:
        t = srv.submit(batches[0])
        got = None
        for _ in range(10000):
            got = srv.poll(t, wait_ms=5)
            if got is not None:
                break
        assert got is not None
        e = _expected(p, reps, batches[0])
        assert np.array_equal(got[0], e[0]) and np.array_equal(got[1], e[1])
        with pytest.raises(ngia.NgiaError) as ex:  # a released ticket
            srv.poll(t)
        assert ex.value.code == -1
        big = _workload(0, 0.9, 5, 10, 6, [80], seed=92)[2][0]
        with pytest.raises(ngia.NgiaError) as ex:  # more records than a slot holds
            srv.submit(big)
        assert ex.value.code == -8
        prot = _workload(1, 0.9, 3, 10, 3, [5], seed=93)[2][0]
        with pytest.raises(ngia.NgiaError) as ex:  # another sequence type
            srv.submit(prot)
        assert ex.value.code == -1
        assert srv.wait(srv.submit(batches[1]))[2]["done"] == 1


def test_large_batches_of_services_side_by_side(cuda_device):
    """A service for batches that take several tiles of the filter, and one of
    other limits opened after it: full batches, whole tiles and one query more."""
    rng = np.random.default_rng(96)
    alpha = np.frombuffer(b"ACGT", np.uint8)
    base = alpha[rng.integers(0, 4, (7, 64))]  # four representatives, three novel families
    p = ngia.params_clamp(0, 0.8, 4, 0)
    reps = seqs_to_db(0, [b.tobytes() for b in base[:4]])

    def batch(n):
        x = base[np.where(rng.random(n) < 0.002, rng.integers(4, 7, n), rng.integers(0, 4, n))]
        hit = rng.random(x.shape) < 0.12 * rng.random((n, 1))
        x[hit] = alpha[rng.integers(0, 4, int(hit.sum()))]
        length = rng.integers(52, 65, n)
        return seqs_to_db(0, [r[:k].tobytes() for r, k in zip(x, length)])

    with ngia.Server(reps, p, slots=1, max_batch=240_000, max_record_blocks=4) as large, \
            ngia.Server(reps, p, slots=1, max_batch=60_000, max_record_blocks=4) as small:
        for srv, n in ((large, 240_000), (small, 60_000), (large, 65_536), (large, 65_537), (large, 3)):
            b = batch(n)
            got = srv.wait(srv.submit(b))
            exp = _expected(p, reps, b)
            assert np.array_equal(got[0], exp[0]) and np.array_equal(got[1], exp[1]), n


@pytest.mark.parametrize("max_batch,blocks", [(512, 128), (64, 1024), (4096, 96), (4096, 256)])
def test_slots_stay_within_the_memory_budget(cuda_device, max_batch, blocks):
    torch = pytest.importorskip("torch")
    p, reps, batches = _workload(0, 0.9, 5, 300, 6, [40], seed=91)
    with ngia.Server(reps, p, slots=1, max_batch=64, max_record_blocks=blocks) as srv:  # what loads once
        srv.wait(srv.submit(batches[0]))
    free = torch.cuda.mem_get_info()[0]
    budget = 1 << 30
    with ngia.Server(reps, p, slots=64, max_batch=max_batch, max_record_blocks=blocks, memory_budget=budget) as srv:
        used = free - torch.cuda.mem_get_info()[0]
        assert srv.slots >= 1
        assert used <= budget + (64 << 20)  # the representatives are not counted
        e = _expected(p, reps, batches[0])
        got = srv.wait(srv.submit(batches[0]))
        assert np.array_equal(got[0], e[0]) and np.array_equal(got[1], e[1])
