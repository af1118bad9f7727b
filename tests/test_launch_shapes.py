"""A launch shape that the caller sets is the one that runs; the shapes chosen
by the number of POIs are those of handles that set none."""
import numpy as np
import pytest

from launches import launches
from tw_gb300 import INTERP_BSPLINE, SAMPLER_LUT, SAMPLER_NBHD, dic, synth

pytestmark = pytest.mark.gpu


def _frame(w, h, r, grid, margin=10):
    pair, _ = synth.small_case(h=h, w=w, r=r, grid=grid)
    f = dic.DICFrame(dic.make_params(w, h, 1, 1, w - 2, h - 2, r, r, grid, grid, margin, margin, 20, 0.001))
    f.set_reference(pair.ref)
    return f, pair.tar


def _icgn(f, tar, batch=None):
    o = f.alloc_outputs()
    if batch is None:
        call = lambda: f.process(tar, **o)  # noqa: E731
    else:
        call = lambda: batch.process([f], [tar], [o])  # noqa: E731
    call()
    found = [x for x in launches(call) if x.name.startswith("k_icgn")]
    assert len(found) == 1, found
    return found[0]


# 320 POIs (at most four per SM of 152) and 2,300 (at most 16)
FEW, SOME = (192, 160, 10, 8, 6), (440, 410, 12, 8, 10)


@pytest.mark.parametrize("geometry", [FEW, SOME])
@pytest.mark.parametrize("threads,chunk,unroll", [(1024, 32, 8), (1024, 32, 4), (1024, 32, 2), (1024, 7, 8),
                                                  (512, 32, 8), (256, 32, 8), (128, 32, 8)])
def test_the_shape_asked_for_runs(geometry, threads, chunk, unroll):
    f, tar = _frame(*geometry)
    for sampler, name in ((SAMPLER_NBHD, "2"), (SAMPLER_LUT, "1")):
        f.set_tuning(threads, 0, sampler, 1, icgn_chunk=chunk)
        f.set_icgn_unroll(unroll)
        k = _icgn(f, tar)
        assert k.name == "k_icgn_warp" and k.threads == threads, k
        assert k.args[:2] == [str(threads // 32), name], k
        assert k.args[3] == str(unroll if threads == 1024 else 4), k


def test_the_shape_asked_of_a_batch_runs():
    f, tar = _frame(*FEW)
    b = dic.DICBatch()
    assert _icgn(f, tar, b).name == "k_icgn_team"  # none asked for: by the number of POIs
    for setter in (lambda: b.set_tuning(1024, 0, SAMPLER_NBHD, icgn_chunk=None), lambda: b.set_icgn_layout(32),
                   lambda: b.set_icgn_unroll(2)):
        b = dic.DICBatch()
        setter()
        k = _icgn(f, tar, b)
        assert k.name == "k_icgn_warp" and k.threads == 1024, k


@pytest.mark.parametrize("interp", [None, INTERP_BSPLINE])
def test_shapes_by_the_number_of_pois(interp):
    for geometry, name in ((FEW, "k_icgn_team"), (SOME, "k_icgn_warp")):
        f, tar = _frame(*geometry)
        if interp is not None:
            f.set_interpolation(interp)
        k = _icgn(f, tar)
        assert k.name == name and k.threads == (256 if name == "k_icgn_team" else 128), k


def test_autotuned_shape_by_the_number_of_pois(tmp_path):
    """The rule is one of the autotuner's shapes: a cached choice of it, and a
    line of ten values, apply it; a choice of a shape applies that shape."""
    f, tar = _frame(*FEW)
    cache = tmp_path / "tuning.txt"
    f.autotune(tar, cache_path=cache)
    key, vals = cache.read_text().strip().split(" ", 1)
    v = vals.split()
    assert len(v) == 11 and v[10] in ("0", "1")
    v[:5] = "1024 0 2 32 2".split()
    for values, name in ((v[:10] + ["1"], "k_icgn_team"), (v[:10], "k_icgn_team"), (v[:10] + ["0"], "k_icgn_warp")):
        cache.write_text(key + " " + " ".join(values) + "\n")
        g, _ = _frame(*FEW)
        assert g.autotune(tar, cache_path=cache)["from_cache"] == 1
        k = _icgn(g, tar)
        assert k.name == name, (values, k)
        if name == "k_icgn_warp":
            assert k.args[0] == "32" and k.args[3] == "2", k


@pytest.mark.parametrize("r,step,twiddles", [(13, 25, 0), (13, 26, 0), (12, 29, 1), (15, 22, 1), (12, 3, 0)])
def test_fftcc_groups_of_small_windows(r, step, twiddles):
    """Five groups per CTA where five fit with eight POIs per batch, whatever
    the POI step (a batch of more never costs a group)."""
    nx = 64
    side = 2 + 2 * r + 16 + step * (nx - 1)
    f = dic.DICFrame(dic.make_params(side, side, 1, 1, side - 2, side - 2, r, r, step, step, 8, 8, 20, 0.001))
    f.set_fftcc_twiddles(twiddles)
    img = np.random.default_rng(r).integers(0, 255, (side, side), np.uint8)
    f.set_reference(img)
    o = f.alloc_outputs()
    f.process(img, **o)
    found = [x for x in launches(lambda: f.process(img, **o)) if x.name == "k_fftcc_tc"]
    assert len(found) == 1 and found[0].threads == 640, found
