"""The two forms of the Tip5 kernels -- tensor-core (128 states per tile) and
sixteen lanes per state -- at the edges of their tiles and of the rule between
them, and the tensor-core LDE passes, bit for bit against the oracle."""
import numpy as np
import pytest

from conftest import EDGE_VALUES, P, dev_empty, from_dev, rand_u64, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 7, 8, 9, 127, 128, 129, 12287, 12289, 20001])
@pytest.mark.parametrize("width", [0, 1, 9, 10, 23])
def test_hash_rows_at_tile_edges(tv, oracle, rows, width):
    t = rand_u64(rows * 31 + width, (max(width, 1), rows), hi=2**64 - 1)
    t.ravel()[: EDGE_VALUES.size] = EDGE_VALUES[: t.size]
    d, out = to_dev(t), dev_empty(rows, 5)
    tv.hash_rows_gpu(d.data_ptr(), rows, width, out.data_ptr())
    assert (from_dev(out) == oracle.hash_rows_cm(t[:width] % P if width else np.zeros((0, rows), np.uint64))).all()


@pytest.mark.parametrize("n", [2, 4, 128, 256, 1 << 14, 1 << 15, 1 << 17])
def test_merkle_levels_of_both_forms(tv, oracle, n):
    lv = rand_u64(n, (n, 5))
    assert (tv.merkle_heap(lv)[1:] == oracle.merkle(lv)[1:]).all()


@pytest.mark.parametrize("count", [1, 8, 9, 8191, 8192, 20000])
def test_pairs_and_permutations_of_both_forms(tv, oracle, count):
    a, b = rand_u64(count, (count, 5)), rand_u64(count + 1, (count, 5))
    got = tv.hash_pairs(a, b)
    s = rand_u64(count + 2, (count, 16), hi=2**64 - 1)
    perm = tv.tip5_permutations(s)
    pick = sorted({0, 1 % count, count // 2, count - 1})
    for i in pick:
        assert (got[i] == oracle.hash_pair(a[i], b[i])).all()
        assert (perm[i] == oracle.permutation(s[i] % P)).all()


@pytest.mark.parametrize("count", [8192, 8193])
@pytest.mark.parametrize("shift", [0, 1])
def test_permutations_at_any_word_of_an_array(tv, oracle, count, shift):
    """The tensor-core form moves pairs of words where the array's alignment allows it."""
    s = rand_u64(count + shift, (count, 16), hi=2**64 - 1)
    d = dev_empty(16 * count + 2)
    d[shift: shift + 16 * count] = to_dev(s).reshape(-1)
    d[shift + 16 * count:] = 5
    tv.tip5_permutations_gpu(d.data_ptr() + 8 * shift, count)
    got = from_dev(d)
    for i in (0, 1, 127, 128, count - 1):
        assert (got[shift + 16 * i: shift + 16 * i + 16] == oracle.permutation(s[i] % P)).all()
    assert (got[shift + 16 * count:] == 5).all()


@pytest.mark.parametrize("logn", [16, 17, 18, 19, 20, 21])
@pytest.mark.parametrize("cols,exp,offset", [(1, 4, 7), (3, 2, 3), (2, 1, 7), (1, 8, 11)])
def test_lde_with_tensor_core_passes(tv, oracle, logn, cols, exp, offset):
    t = rand_u64(logn * 7 + cols, (cols, 1 << logn))
    t.ravel()[: EDGE_VALUES.size] = EDGE_VALUES % P
    assert (tv.lde(t, exp, offset) == oracle.lde(t, exp, offset)).all()


@pytest.mark.parametrize("logn,cols,exp", [(12, 256, 4), (13, 128, 2), (14, 64, 4), (15, 32, 8), (16, 16, 1), (16, 37, 16),
                                           (17, 1, 16), (18, 2, 2), (20, 1, 4), (22, 1, 4)])
def test_lde_of_any_representatives_where_the_tensor_cores_pay(tv, oracle, logn, cols, exp):
    """The shortest columns and fewest of them that take these passes, the 10 + 12 split
    of 2^22 and K2 with sixteen cosets; inputs that are not canonical."""
    t = rand_u64(logn * 9 + cols, (cols, 1 << logn), hi=2**64 - 1)
    t[0, : EDGE_VALUES.size] = EDGE_VALUES
    t[-1, -3:] = [2**64 - 1, P, P + 1]
    got = tv.lde(t, exp, 7)
    for c in sorted({0, cols // 2, cols - 1}):
        assert (got[c] == oracle.lde(t[c: c + 1] % P, exp, 7)[0]).all()


def test_lde_column_count_beyond_one_unit(tv, oracle):
    """More columns than one unit of the tensor-core passes holds, and an odd count."""
    t = rand_u64(99, (37, 1 << 20))
    d, out = to_dev(t), dev_empty(37, 1 << 21)
    tv.lde_gpu(d.data_ptr(), 37, 1 << 20, out.data_ptr(), 1 << 21)
    for c in (0, 15, 16, 31, 36):
        assert (from_dev(out[c]) == oracle.lde(t[c: c + 1], 2, 7)[0]).all()


@pytest.mark.parametrize("logn,cols,R,exp", [(12, 256, 98, 4), (16, 16, 5, 2), (17, 2, 300, 4), (20, 1, 98, 4), (18, 2, 1, 8)])
def test_randomized_lde_with_tensor_core_passes(tv, oracle, logn, cols, R, exp):
    t, r = rand_u64(logn + cols, (cols, 1 << logn)), rand_u64(logn + R, (cols, R))
    got = tv.lde_randomized(t, r, exp, 7, 3)
    for c in sorted({0, cols // 2, cols - 1}):
        assert (got[c] == oracle.lde_randomized(t[c: c + 1], r[c: c + 1], exp, 7, 3)[0]).all()


@pytest.mark.parametrize("logn,cols", [(1, 300), (5, 33), (6, 5), (8, 379), (9, 3), (11, 2)])
@pytest.mark.parametrize("exp", [1, 2, 8, 16])
def test_short_columns_with_any_number_of_cosets(tv, oracle, logn, cols, exp):
    t = rand_u64(logn * cols + exp, (cols, 1 << logn))
    assert (tv.lde(t, exp, 7) == oracle.lde(t, exp, 7)).all()


@pytest.mark.parametrize("logn,cols", [(12, 800), (13, 400), (16, 48), (18, 13), (20, 3), (21, 2), (22, 1)])
@pytest.mark.parametrize("inverse", [False, True])
def test_ntt_with_tensor_core_passes(tv, oracle, logn, cols, inverse):
    a = rand_u64(logn + cols, (cols, 1 << logn), hi=2**64 - 1)
    got = tv.ntt(a, inverse=inverse)
    for c in sorted({0, cols // 2, cols - 1}):
        assert (got[c] == oracle.ntt(a[c] % P, inverse=inverse)).all()


def test_no_wait_ran_out(tv):
    assert tv.get_tuning("mma_timeouts") == 0
