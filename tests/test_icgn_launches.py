"""The IC-GN launch shapes chosen by the number of POIs (a CTA of eight warps
per POI, CTAs of four one-POI warps, one CTA of 32 per SM) give bit for bit the
outputs of the one-warp-per-CTA kernel, whose agreement with the oracle other
tests hold: the smallest to the largest subsets, POIs that leave the ROI, whole
and fractional guesses, both interpolants."""
import numpy as np
import pytest

from tw_gb300 import INTERP_BICUBIC, INTERP_BSPLINE, PATH_FAST, SAMPLER_NBHD, dic, synth

pytestmark = pytest.mark.gpu

# image, subset radius, POI step, margin: 180, 221 and 576 POIs (a CTA per POI up
# to 608 on 152 SMs), 676 and 2,378 (four-warp CTAs up to 2,432), 2,790 and
# 6,084.  A margin of 0 gives POIs whose subsets leave the ROI under the warp.
SHAPES = [(192, 160, 4, 13, 0), (192, 160, 31, 8, 0), (256, 256, 5, 10, 4), (256, 256, 10, 9, 2),
          (400, 300, 8, 6, 20), (400, 300, 16, 6, 0), (512, 512, 4, 6, 20)]


def _run(ref, tar, params, interp, one_warp, guess):
    f = dic.DICFrame(params)
    f.set_interpolation(interp)
    f.set_reference(ref)
    b = dic.DICBatch()
    o = f.alloc_outputs()
    if guess is not None:
        f.set_guess_mode(1)
        o["u"][:], o["v"][:] = guess
    if one_warp:
        f.set_tuning(32, 0, SAMPLER_NBHD, 1, icgn_chunk=0)
        b.set_tuning(32, 0, SAMPLER_NBHD, icgn_chunk=0)
    if guess is None:
        f.process(tar, **o)
    else:
        b.process([f], [tar], [o])
    return o


@pytest.mark.parametrize("interp", [INTERP_BICUBIC, INTERP_BSPLINE])
@pytest.mark.parametrize("guessed", [False, True])
@pytest.mark.parametrize("w,h,r,grid,margin", SHAPES)
def test_launch_shapes_bit_identical(w, h, r, grid, margin, guessed, interp):
    pair, _ = synth.small_case(h=h, w=w, r=r, grid=grid)
    ref = pair.ref.copy()
    ref[:3 * h // 10, :3 * w // 10] = 20  # dark subsets: a flat corner of the reference
    p = dic.make_params(w, h, 1, 1, w - 2, h - 2, r, r, grid, grid, margin, margin, 20, 0.001, PATH_FAST)
    guess = None
    if guessed:
        n = int(np.prod(dic.num_pois(p)))
        rng = np.random.default_rng(r)
        guess = (np.float32(1.6) + rng.uniform(-0.7, 0.7, n).astype(np.float32),
                 np.float32(-2.4) + rng.uniform(-0.7, 0.7, n).astype(np.float32))
        guess[0][::5] = 2.0  # whole-pixel guesses among them
        guess[1][::5] = -2.0
    a = _run(ref, pair.tar, p, interp, False, guess)
    b = _run(ref, pair.tar, p, interp, True, guess)
    for k in a:
        if guessed and k == "zncc":
            continue  # not an output of a guessed frame
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    assert (a["flags"] == 0).any()
