"""A per-reference FFT-CC pass that gave up on a bounded wait leaves incomplete
spectra: the call that returns host results reports it, and the spectra are
computed again by the next call, whatever its kind.  The failure is made on the
host (twdic_frame_fail_reference_pass)."""
import numpy as np
import pytest

from launches import launches
from tw_gb300 import dic, synth
from tw_gb300._lib import TWDICError, check

pytestmark = pytest.mark.gpu


@pytest.fixture
def frame():
    pair, g = synth.small_case()
    f = dic.DICFrame(dic.make_params(g.img_w, g.img_h, g.start_x, g.start_y, g.roi_w, g.roi_h, g.subset_r, g.subset_r,
                                     g.grid, g.grid, g.margin, g.margin, g.max_iter, g.delta_p))
    f.set_reference(pair.ref)
    want = f.alloc_outputs()
    f.process(pair.tar, **want)
    return f, pair.tar, want


def _fail(f):
    check(f._lib.twdic_frame_fail_reference_pass(f._h))


def _passes(call):
    """Per-reference passes among the call's FFT-CC launches."""
    return sum(x.args[4] in ("true", "1") for x in launches(call) if x.name == "k_fftcc_tc")


def _equal(o, want):
    for k in want:
        a = o[k] if isinstance(o[k], np.ndarray) else o[k].cpu().numpy()
        np.testing.assert_array_equal(a, want[k], err_msg=k)


def test_needs_a_pass():
    pair, g = synth.small_case()
    f = dic.DICFrame(dic.make_params(g.img_w, g.img_h, g.start_x, g.start_y, g.roi_w, g.roi_h, g.subset_r, g.subset_r,
                                     g.grid, g.grid, g.margin, g.margin, g.max_iter, g.delta_p))
    with pytest.raises(TWDICError):
        _fail(f)


def test_host_results_report_it_once(frame):
    f, tar, want = frame
    o = f.alloc_outputs()

    def reported():
        with pytest.raises(TWDICError, match="TIMEOUT"):
            f.process(tar, **o)

    _fail(f)
    assert _passes(reported) == 1
    _equal(o, want)
    assert _passes(lambda: f.process(tar, **o)) == 0
    _equal(o, want)


def test_device_results_compute_the_spectra_again(frame):
    import torch
    f, tar, want = frame
    t, o = torch.from_numpy(tar).cuda(), f.alloc_outputs("cuda")
    _fail(f)
    assert _passes(lambda: f.process(t, **o)) == 1
    _equal(o, want)
    assert _passes(lambda: f.process(t, **o)) == 0
    # the next call with host results reports it, its own results are good
    h = f.alloc_outputs()
    with pytest.raises(TWDICError, match="TIMEOUT"):
        f.process(tar, **h)
    _equal(h, want)
    f.process(tar, **h)


def test_batches(frame):
    import torch
    f, tar, want = frame
    b = dic.DICBatch()
    h = f.alloc_outputs()
    _fail(f)
    with pytest.raises(TWDICError, match="TIMEOUT"):
        b.process([f], [tar], [h])
    _equal(h, want)
    b.process([f], [tar], [h])
    # a captured graph reads the spectra: it is not replayed over incomplete ones
    t, o = torch.from_numpy(tar).cuda(), f.alloc_outputs("cuda")
    g = dic.DICBatch(graph=True)
    for replayed in (False, True):
        g.process([f], [t], [o])
        assert g.replayed == replayed
    _fail(f)
    assert _passes(lambda: g.process([f], [t], [o])) == 1
    assert not g.replayed
    g.process([f], [t], [o])
    torch.cuda.synchronize()
    assert g.replayed
    _equal(o, want)
