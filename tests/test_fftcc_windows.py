"""Tensor-core FFT-CC over every window size, with batches that the POIs do not
fill (the operand rows past them are never written): integer displacements
equal the oracle's, ZNCC within the FP32 oracle's own rounding (3e-5)."""
import numpy as np
import pytest

from oracle import oracle as O
from tw_gb300 import PATH_FAST, cuFFTCC2D, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", range(4, 32))
def test_every_window_size_partial_batches(r):
    w, h, grid = 150, 141, 9
    pair, _ = synth.small_case(h=h, w=w, r=max(r, 8), grid=grid, seed=r, u0=0.6 if r < 8 else 1.6,
                               v0=-0.4 if r < 8 else -2.4)
    for margin in ((w - 2 - 2 * r) // 2, 6):  # one or a few POIs, then several batches and a rest
        f = cuFFTCC2D(w, h, w - 2, h - 2, 1, 1, r, r, grid, grid, margin, 6, path=PATH_FAST)
        u, v, z = f.InitializeFFTCC(pair.ref)
        status = np.zeros(f.GetNumPOIs(), np.uint8)
        f.ComputeFFTCC(u, v, z, pair.tar, status)
        uo, vo, zo, so = O.fftcc(pair.ref, pair.tar, f.POIPositions(), r)
        np.testing.assert_array_equal(status, so)
        # (a mismatch would have to be an exact tie of the integer correlation)
        for i in np.flatnonzero((u.ravel() != uo) | (v.ravel() != vo)):
            py, px = f.POIPositions()[i]
            c = O.exact_surface(pair.ref, pair.tar, py, px, r)
            assert c[int(v.ravel()[i]) % (2 * r), int(u.ravel()[i]) % (2 * r)] == c[int(vo[i]) % (2 * r), int(uo[i]) % (2 * r)]
        np.testing.assert_allclose(z.ravel(), zo, atol=3e-5, rtol=0)
