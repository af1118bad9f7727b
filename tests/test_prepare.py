"""The neighbourhood table at the edges of the ROI and of the image (its column
pieces of eight rows, whole and in part; the bicubic table's zero last row and
column; the B-spline table's zero bytes outside the image): IC-GN from the table
agrees with IC-GN from the float coefficient LUT, flags exactly, displacements
within the parity bar of 1e-3 px.  Guesses push the subsets of margin-0 POIs onto
the ROI's last rows and columns."""
import numpy as np
import pytest

from tw_gb300 import INTERP_BICUBIC, INTERP_BSPLINE, PATH_FAST, SAMPLER_LUT, SAMPLER_NBHD, dic, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("interp", [INTERP_BICUBIC, INTERP_BSPLINE])
@pytest.mark.parametrize("w,h", [(101, 74), (102, 75), (103, 76), (104, 77), (97, 78), (98, 79), (99, 80), (100, 81)])
def test_table_edges_match_lut(w, h, interp):
    r, grid = 6, 5
    pair, _ = synth.small_case(h=h, w=w, r=r, grid=grid, seed=w)
    p = dic.make_params(w, h, 1, 1, w - 2, h - 2, r, r, grid, grid, 0, 0, 20, 0.001, PATH_FAST)
    outs = []
    for sampler in (SAMPLER_NBHD, SAMPLER_LUT):
        f = dic.DICFrame(p)
        f.set_interpolation(interp)
        f.set_guess_mode(1)
        f.set_reference(pair.ref)
        b = dic.DICBatch()
        b.set_tuning(1024, 0, sampler, icgn_chunk=32)
        o = f.alloc_outputs()
        pos = f.poi_positions()
        # towards the nearer edge of the ROI by up to the last row or column
        o["u"][:] = np.clip(w - 2 - r - pos[:, 1], -1, 2)
        o["v"][:] = np.clip(h - 2 - r - pos[:, 0], -1, 2)
        b.process([f], [pair.tar], [o])
        outs.append(o)
    a, l = outs
    np.testing.assert_array_equal(a["flags"], l["flags"])
    ok = (a["flags"] == 0) & (a["iters"] == l["iters"])
    assert ok.sum() > 50 and (a["iters"] != l["iters"]).sum() <= max(2, a["iters"].size // 50)
    np.testing.assert_allclose(a["u"][ok], l["u"][ok], atol=1e-3, rtol=0)
    np.testing.assert_allclose(a["v"][ok], l["v"][ok], atol=1e-3, rtol=0)
