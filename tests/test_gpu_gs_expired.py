"""A block Gauss-Seidel sweep whose wait runs out ends with an error status:
all lanes of a warp take the same verdict, so that none stays behind in a
warp-wide synchronisation.  The wait is made to run out by a barrier that
expects one item more than its level has."""
import time

import pytest

import xamg


@pytest.mark.gpu
@pytest.mark.parametrize("blocks", [2, 64])
def test_expired_block_sweep_reports_code_3(gpu, blocks):
    L = xamg.lib()
    t0 = time.perf_counter()
    rc = L.XAMG_b200_wait_selftest(2, blocks, 0.2)
    dt = time.perf_counter() - t0
    assert rc == 3, L.XAMG_b200_last_error()
    assert b"block sweep" in L.XAMG_b200_last_error()
    assert 0.15 <= dt < 10.0
    assert L.XAMG_b200_synchronize() == 0
