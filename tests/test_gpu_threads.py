"""Host threads calling the library at the same time, each on its own stream."""
import threading

import pytest

from conftest import dev_empty, from_dev, rand_u64, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logn,cols,rounds", [(11, 1, 4000), (17, 2, 1500)])
def test_ldes_of_different_expansions_from_two_threads(tv, oracle, logn, cols, rounds):
    """The dynamic shared memory of these kernels depends on the expansion, and
    the limit it is checked against belongs to the function: no call may lower
    it under another thread's launch."""
    import torch
    t = rand_u64(logn, (cols, 1 << logn))
    d = to_dev(t)
    out = {e: dev_empty(cols, e << logn) for e in (1, 4)}
    torch.cuda.synchronize()
    errors = []

    def work(e):
        s = torch.cuda.Stream()
        try:
            for _ in range(rounds):
                tv.lde_gpu(d.data_ptr(), cols, 1 << logn, out[e].data_ptr(), e << logn, stream=s)
            s.synchronize()
        except Exception as x:  # noqa: BLE001 - reported in the main thread
            errors.append(x)
        finally:
            tv.forget_stream(s)

    threads = [threading.Thread(target=work, args=(e,)) for e in out]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors[0]
    for e, o in out.items():
        assert (from_dev(o) == oracle.lde(t, e, 7)).all()
