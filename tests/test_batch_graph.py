"""A batch's captured graph holds frame state in its launches' parameters (the
per-frame table's address, the box widths of the tensor maps).  A call of a
frame alone that moves it makes the next batch call run and be captured anew."""
import numpy as np
import pytest

from tw_gb300 import SAMPLER_LUT, SAMPLER_NBHD, dic, synth

pytestmark = pytest.mark.gpu


def _table_moved(f):
    # the float LUT takes four times the neighbourhood table's bytes
    f.set_tuning(1024, 0, SAMPLER_LUT, 1, icgn_chunk=32)


def _maps_encoded_anew(f):
    # another batch size: boxes of another width
    f.set_tuning(1024, 0, SAMPLER_NBHD, 1, icgn_chunk=32)
    f.set_fftcc_tuning(1, 0, 2)


@pytest.mark.parametrize("change", [_table_moved, _maps_encoded_anew])
def test_graph_recaptured_after_a_frame_call_moved_its_state(change):
    import torch
    frames, tars, want = [], [], []
    for k, (h, w, r, grid) in enumerate([(160, 192, 10, 7), (200, 150, 16, 9)]):
        pair, g = synth.small_case(h=h, w=w, r=r, grid=grid, seed=21 + k)
        f = dic.DICFrame(dic.make_params(g.img_w, g.img_h, g.start_x, g.start_y, g.roi_w, g.roi_h, r, r, grid, grid,
                                         g.margin, g.margin, g.max_iter, g.delta_p))
        f.set_reference(pair.ref)
        frames.append(f)
        tars.append(torch.from_numpy(pair.tar).cuda())
        want.append(f.alloc_outputs())
        f.process(pair.tar, **want[-1])
    outs = [f.alloc_outputs(device="cuda") for f in frames]
    b = dic.DICBatch(graph=True)

    def check(replayed):
        for o in outs:
            for a in o.values():
                a.zero_()
        torch.cuda.synchronize()
        b.process(frames, tars, outs)
        torch.cuda.synchronize()
        assert b.replayed == replayed
        for o, w in zip(outs, want):
            for k in w:
                np.testing.assert_array_equal(o[k].cpu().numpy(), w[k], err_msg=k)

    check(False)
    check(True)
    change(frames[0])
    o = frames[0].alloc_outputs()
    frames[0].process(tars[0].cpu().numpy(), **o)
    check(False)
    check(True)
