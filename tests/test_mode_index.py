"""The row of a mode in the update kernel (k_rk_update): j = floor((q + 1/2) * (1 / NKK)) in 32-bit
floating point, for every mode q of the largest plane that a z length can meet."""
import numpy as np
import pytest

LENGTHS = sorted(2 ** a * f for a in range(3, 11) for f in (1, 3, 5, 7) if 16 <= 2 ** a * f <= 1024)


@pytest.mark.parametrize("nz", LENGTHS)
def test_row_of_a_mode(nz):
    nkk, nkj = 2 * (nz // 3) + 1, 2 * (1024 // 3) + 1
    q = np.arange(nkj * nkk, dtype=np.int64)
    assert q.size < 1 << 19
    inv = np.float32(1.0) / np.float32(nkk)
    j = ((q.astype(np.float32) + np.float32(0.5)) * inv).astype(np.int64)
    assert np.array_equal(j, q // nkk)
