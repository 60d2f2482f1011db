"""The division of the row quantisers (three multiply-adds with the rounded reciprocal, row_quant.cuh) against IEEE
division, in numpy.  Values are fp16 and the divisor is a row maximum (fp16) over 448 or 127 in fp32.  Scaling x or
the maximum by a power of two scales the quotient and every intermediate by it (fp16 over its whole range keeps
them in fp32's normal range), so the 1024 significands of each stand for all values; subnormal ones are among them."""
import numpy as np
import pytest

F32, F64 = np.float32, np.float64


def _round_sum(a, b):
    """a + b rounded once to fp32, for doubles: the error of the double sum decides where it is halfway."""
    s = a + b
    t = s - a
    err = (a - (s - t)) + (b - t)
    near = s.astype(F32)
    up = np.where(near.astype(F64) > s, near, np.nextafter(near, F32(np.inf), dtype=F32))
    down = np.where(near.astype(F64) > s, np.nextafter(near, F32(-np.inf), dtype=F32), near)
    halfway = (s - down.astype(F64)) == (up.astype(F64) - s)
    return np.where(halfway & (err > 0), up, np.where(halfway & (err < 0), down, near))


@pytest.mark.parametrize("top", [448, 127])
def test_row_division_is_ieee_division(top):
    significands = (1 + np.arange(1024, dtype=F32) / 1024)
    s = (significands / F32(top))[:, None]
    y = F32(1) / s
    x = significands[None, :]
    q = x * y
    # (the 48-bit product and the difference are exact in a double; the fused multiply-add rounds the difference once)
    r = (x.astype(F64) - q.astype(F64) * s.astype(F64)).astype(F32)
    got = _round_sum(q.astype(F64), r.astype(F64) * y.astype(F64))
    want = x / s
    assert not np.array_equal(q, want)                             # (the product alone is not enough)
    assert np.array_equal(got, want)
