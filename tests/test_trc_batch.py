"""The tracers that one batch of the horizontal advection takes: up to four, but
its work fields (one set a tracer) leave most of the free device memory alone."""
import pytest


@pytest.mark.parametrize("nq", [1, 2, 3, 4, 17, 32])
def test_batch_size_follows_the_memory_that_is_left(pkg, nq):
    batch = pkg.runtime.load_library().nc_trc_batch
    one = 3 * 10 ** 9
    assert batch(180 * 10 ** 9, one, nq) == min(nq, 4)
    assert batch(0, one, nq) == batch(one, one, nq) == batch(16 * one - 16, one, nq) == 1
    last = 1
    for free in range(0, 40 * one, one // 4):
        n = batch(free, one, nq)
        assert last <= n <= min(nq, 4)
        assert (n - 1) * one * 6 <= free + 6 * 3      # at most a sixth of what is left
        last = n
    assert last == min(nq, 4)
    assert batch(-1, one, nq) < 0 and batch(one, 0, nq) < 0 and batch(one, one, 0) < 0
