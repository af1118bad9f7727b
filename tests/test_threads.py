"""Handles of different threads at the same time, with launches of one kernel
that take different amounts of shared memory: none refuses the other's."""
import threading

import numpy as np
import pytest

from tw_gb300 import PATH_PLAIN, SAMPLER_WINDOW, dic, synth

pytestmark = pytest.mark.gpu


def _frame(w, h, r, grid, margin=8, path=None):
    pair, _ = synth.small_case(h=h, w=w, r=r, grid=grid)
    f = dic.DICFrame(dic.make_params(w, h, 1, 1, w - 2, h - 2, r, r, grid, grid, margin, margin, 20, 0.001,
                                     *([] if path is None else [path])))
    f.set_reference(pair.ref)
    return f, pair.tar


def _fftcc(big):
    f, tar = _frame(512, 512, 20, 5) if big else _frame(128, 128, 20, 12)
    if not big:
        f.set_fftcc_tuning(1, 1, 1)
    return lambda o: f.process(tar, **o), [f]


def _icgn(big):
    f, tar = _frame(192, 160, 31 if big else 8, 9)
    f.set_tuning(128, 0, SAMPLER_WINDOW, 1, icgn_chunk=0)
    return lambda o: f.process(tar, **o), [f]


def _plain(big):
    f, tar = _frame(160, 160, 31 if big else 8, 9, path=PATH_PLAIN)
    return lambda o: f.process(tar, **o), [f]


def _segments(big):
    pairs = [_frame(160, 160, r, 9) for r in ((20, 30) if big else (5, 6))]
    b = dic.DICBatch()
    frames = [f for f, _ in pairs]
    return lambda o: b.process(frames, [t for _, t in pairs], o), frames


@pytest.mark.parametrize("kind", [_fftcc, _icgn, _plain, _segments])
def test_threads_with_different_shared_memory(kind):
    errors, results = [], {}
    start, done = threading.Barrier(2), threading.Event()

    def work(big):
        try:
            call, frames = kind(big)
            outs = [f.alloc_outputs() for f in frames]
            arg = outs if kind is _segments else outs[0]
            call(arg)
            results[big] = [{k: a.copy() for k, a in o.items()} for o in outs]
            start.wait()
            if big:
                for _ in range(400):
                    call(arg)
            else:
                while not done.is_set():
                    call(arg)
            for o, w in zip(outs, results[big]):
                for k in o:
                    np.testing.assert_array_equal(o[k], w[k], err_msg=k)
        except BaseException as e:  # noqa: BLE001
            errors.append(e)
            start.abort()
        finally:
            done.set()

    threads = [threading.Thread(target=work, args=(big,)) for big in (True, False)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
