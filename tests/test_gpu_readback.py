"""State read-back (fesomc_gpu_sync_to_host) through the staging slots: the
same values as the snapshot path (its own copies and buffers) below and above
the size from which worker threads take part, in both precision forms and
storage orders, and with two threads reading at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(cfg, fp32, sfc):
    from fesomc import cases, model
    g = model.GpuModel(cases.estuary(cfg, fp32_form=fp32, sfc_order=sfc))
    g.step(2)
    return g


@pytest.mark.parametrize("cfg,fp32,sfc", [("small", 0, 0), ("small", 1, 1), ("medium", 0, 1), ("medium", 1, 0)])
def test_readback_equals_snapshot(built, cfg, fp32, sfc):
    g = _model(cfg, fp32, sfc)
    try:
        got = g.state()
        g.snapshot_begin()
        snap = g.snapshot_end()
        assert set(got) == set(snap)
        for k, v in snap.items():
            assert np.array_equal(got[k], v), k
    finally:
        g.close()


def test_two_threads_read_at_once(built):
    models = [_model("medium", 0, 0), _model("medium", 1, 1)]
    try:
        want = [g.state() for g in models]
        got = [[], []]

        def read(i):
            for _ in range(4):
                got[i].append(models[i].state())

        ts = [threading.Thread(target=read, args=(i,)) for i in range(2)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        for i in range(2):
            assert len(got[i]) == 4
            for s in got[i]:
                for k, v in want[i].items():
                    assert np.array_equal(s[k], v), k
    finally:
        for g in models:
            g.close()
