"""The library's host side without a GPU: its own objects linked with a
stand-in for the CUDA runtime (fake_cuda), which logs launches and copies and
holds copies to the host back until something waits for them."""
import ctypes as C

import numpy as np
import pytest


@pytest.fixture(scope="module")
def fake_lib(built):
    import fake_cuda
    from fesomc import abi, build
    lib = abi.load(fake_cuda.build(build))
    assert not lib.missing_symbols
    return lib


@pytest.fixture
def fake(fake_lib, monkeypatch):
    """The stand-in's log; models made meanwhile run on it."""
    import fake_cuda
    from fesomc import abi
    monkeypatch.setattr(abi, "_lib", fake_lib)
    return fake_cuda.Log(fake_lib)


def _model(**kw):
    from fesomc import cases, model
    return model.GpuModel(cases.estuary("small", **kw))


@pytest.mark.parametrize("fp32,sfc", [(0, 0), (1, 1)])
def test_failed_readback_leaves_no_copy_pending(fake, fp32, sfc):
    """A read-back that fails after some of its fields were enqueued waits
    for their copies before it returns: the staging memory they go to is the
    whole process's, and the next read-back, of another model and stream,
    uses it at once."""
    a, b = _model(fp32_form=fp32, sfc_order=sfc), _model()
    try:
        want = b.state()
        for after in (1, 7):
            fake.lib.fake_fail_copy(after)
            with pytest.raises(RuntimeError):
                a.state()
            assert fake.lib.fake_pending() == 0
            got = b.state()
            assert all(np.array_equal(got[k], v) for k, v in want.items())
        if not sfc:   # (the reordering is a kernel)
            assert np.array_equal(a.state()["TF"].astype(np.float32), b.state()["TF"].astype(np.float32))
    finally:
        fake.lib.fake_fail_copy(-1)
        a.close()
        b.close()
