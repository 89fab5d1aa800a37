"""A device wait that ran out is reported by every call that hands out the result.
No wait runs out here: "fail_mma_after" sets the status word behind one launch, as
its kernel does when a wait runs out, and the last test writes it directly."""
import numpy as np
import pytest

from conftest import memcpy_h2d, rand_u64, to_dev

pytestmark = pytest.mark.gpu

LOGN, COLS = 16, 16  # tensor-core passes K1, K2, K3, row hash, and five tree levels
MMA_LAUNCHES = 9


@pytest.fixture(autouse=True)
def no_injection_left(tv):
    yield
    left = tv.get_tuning("fail_mma_after")
    tv.set_tuning("fail_mma_after", 0)
    assert left == 0, "the launch meant to fail was never made"
    assert tv.get_tuning("mma_timeouts") == 0


def readers(c):
    r = [c.root, c.sync, lambda: c.auth_paths([3]), lambda: c.auth_structure([3]), c.leaves, c.nodes, c.root]
    if c.device_lde():
        r += [lambda: c.read_rows([1]), lambda: c.read_columns(0, 1), c.lde, lambda: c.lde(row_major=True)]
    return r


def assert_refused(tv, c):
    for read in readers(c):
        with pytest.raises(tv.Timeout):
            read()


@pytest.mark.parametrize("k", range(1, MMA_LAUNCHES + 1))
def test_every_launch_of_a_commit(tv, k):
    t = rand_u64(1, (COLS, 1 << LOGN))
    d = to_dev(t)
    tv.set_tuning("fail_mma_after", k)
    with tv.Commitment(d.data_ptr(), width=COLS, trace_len=1 << LOGN, device_ptr=True) as c:
        assert_refused(tv, c)
    with tv.Commitment(t) as good:
        for read in readers(good):
            read()


def _kinds(tv):
    t = rand_u64(2, (COLS, 1 << LOGN))
    d = to_dev(t)
    n = dict(width=COLS, trace_len=1 << LOGN, device_ptr=True)
    return {
        "host trace": lambda: tv.Commitment(t),
        "row major": lambda: tv.Commitment(np.ascontiguousarray(t.T), row_major=True),
        "randomized": lambda: tv.Commitment(t, randomizers=rand_u64(3, (COLS, 9)), trace_offset=3),
        "discard": lambda: tv.Commitment(d.data_ptr(), discard_lde=True, **n),
        "frugal": lambda: tv.Commitment(d.data_ptr(), frugal=True, **n),
        "rows": lambda: tv.Commitment.from_rows(t),
        "digests": lambda: tv.Commitment.from_digests(rand_u64(4, (1 << 15, 5))),
        "multi": lambda: tv.commit_multi([t])[0],
    }


@pytest.mark.parametrize("kind", ["host trace", "row major", "randomized", "discard", "frugal", "rows", "digests",
                                  "multi"])
def test_kinds_of_commitment(tv, kind):
    make = _kinds(tv)[kind]
    tv.set_tuning("fail_mma_after", 1)
    c = make()
    assert_refused(tv, c)
    c.free()
    c = make()
    c.root()
    c.free()


def test_synchronous_commits_fail_themselves(tv):
    t, lv = rand_u64(2, (COLS, 1 << LOGN)), rand_u64(4, (1 << 15, 5))
    for call in (lambda: tv.Commitment(t, sync=True), lambda: tv.commit_multi([t], sync=True),
                 lambda: tv.Commitment.from_digests(lv, sync=True)):
        tv.set_tuning("fail_mma_after", 1)
        with pytest.raises(tv.Timeout):
            call()


def test_batch(tv):
    shapes = [(1 << LOGN, COLS), (64, 3)]
    tv.set_tuning("fail_mma_after", 4)  # the row hash of both tables; captured, so every run of this batch
    with tv.Batch(shapes) as b:
        for (n, w), i in zip(shapes, range(2)):
            memcpy_h2d(b.input_ptr(i), rand_u64(5 + i, (w, n)))
        for _ in range(2):
            b.run()
            with pytest.raises(tv.Timeout):
                b.tables[0].root()


def test_batch_before_its_first_run_has_not_failed(tv):
    """Whatever the tables' memory held before."""
    with tv.Batch([(64, 3)] * 8) as a:
        for t in a.tables:
            memcpy_h2d(t.device_tree(), np.ones(1, dtype=np.uint64))
    with tv.Batch([(64, 3)] * 8) as b:
        for t in b.tables:
            t.sync()


def test_server(tv):
    t = rand_u64(2, (COLS, 1 << LOGN))
    with tv.Server() as s:
        tv.set_tuning("fail_mma_after", 1)
        rid = s.submit(t)
        with pytest.raises(tv.TvmcError) as e:
            s.wait(rid)
        assert not isinstance(e.value, tv.Timeout)  # waiting again would not help
        with pytest.raises(tv.TvmcError):
            s.open(rid, [0])
        s.release(rid)


def test_host_calls(tv):
    rows = rand_u64(6, (1 << 14, 11))
    pairs = rand_u64(7, (1 << 13, 5))
    t = rand_u64(8, (COLS, 1 << LOGN))
    calls = [lambda: tv.ntt(rand_u64(9, (48, 1 << 16))), lambda: tv.ntt(rand_u64(9, (48, 1 << 16)), inverse=True),
             lambda: tv.lde(t), lambda: tv.lde_randomized(t, rand_u64(3, (COLS, 9)), 4, 7, 3),
             lambda: tv.evaluate_on_coset(t, 1 << 18, 7), lambda: tv.hash_varlen_rows(rows),
             lambda: tv.hash_pairs(pairs, pairs), lambda: tv.tip5_permutations(rand_u64(10, (1 << 13, 16))),
             lambda: tv.merkle_heap(rand_u64(11, (1 << 15, 5)))]
    for call in calls:
        want = call()
        tv.set_tuning("fail_mma_after", 1)
        with pytest.raises(tv.Timeout):
            call()
        assert (call() == want).all()


def test_status_word_is_looked_at_by_every_reader(tv):
    """The marker as a kernel leaves it, before anything was read from the commitment."""
    import torch
    with tv.Commitment(rand_u64(12, (3, 64))) as c:
        torch.cuda.synchronize()
        memcpy_h2d(c.device_tree(), np.ones(1, dtype=np.uint64))
        assert_refused(tv, c)
