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


def _check_starts(fake):
    """Every kernel started early directly follows a kernel on its stream (or
    opens a captured step, which as a graph waits for all before it)."""
    before, early = {}, 0
    for o in fake.ops():
        if o.early:
            early += 1
            prev = before.get((o.stream, o.captured), "k" if o.captured else "")
            assert prev == "k", (o.name, prev)
        before[(o.stream, o.captured)] = o.kind
    return early


@pytest.mark.parametrize("kw", [{}, {"fp32_form": 1, "sfc_order": 1}, {"T_potential": 1}, {"atm": {"qns": -50.0}},
                                {"bih_3D": 1, "bih_2D": 1, "Abh0": 1e4}])
@pytest.mark.parametrize("device_forcing", [False, True])
def test_early_starts_follow_kernels(fake, kw, device_forcing):
    """What makes an early start safe is the kernel before it; behind a copy
    or a fill (the forcing's upload, a snapshot, a halo, the status) a kernel
    is launched plainly: in first, captured, replayed and harvesting steps."""
    from fesomc import abi, cases, closure
    fake.clear()
    g = _model(**kw)
    c = closure.Closure(g.case.mesh.NS, capacity=4096)
    try:
        if "atm" in kw and not device_forcing:
            g.set_atm_fields(*cases.atm_coefficients(g.case.mesh, g.case.params.time_jd0))
        if device_forcing:
            f = g.case.forcing_fn(1, g.case.params.time_jd0 + 20.0)
            g.set_forcing(f)
            base = np.ascontiguousarray(f["runoff_rivers"])
            abi.check(g.lib.fesomc_gpu_set_device_forcing(g.h, abi.dptr(base), 1))
        g.snapshot_begin()            # its copies on the step's stream are not waited for
        g.step(1)
        g.snapshot_end()
        g.step(2)
        g.snapshot_begin()
        c.harvest(g, 2)
        g.snapshot_end()
        g.energy()
        n = np.arange(1, 40, dtype=np.int32)
        h, m = C.c_void_p(), C.c_int64()
        abi.check(g.lib.fesomc_gpu_halo_plan(g.h, len(n), abi.iptr(n), len(n), abi.iptr(n), C.byref(h)))
        abi.check(g.lib.fesomc_gpu_halo_size(h, C.byref(m)))
        buf = np.zeros(m.value)
        abi.check(g.lib.fesomc_gpu_halo_pack(g.h, h, buf.ctypes.data))
        abi.check(g.lib.fesomc_gpu_halo_unpack(g.h, h, buf.ctypes.data))
        g.lib.fesomc_gpu_halo_free(h)
        assert _check_starts(fake) > 50
    finally:
        c.close()
        g.close()


def _kernels(fake):
    return sum(o.kind == "k" for o in fake.ops())


@pytest.mark.parametrize("kw", [{}, {"fp32_form": 1}, {"tracer_adv": 1}, {"tracer_adv": 4}, {"T_potential": 1},
                                {"atm": {"qns": -50.0}}, {"bih_3D": 1, "Abh0": 1e4}, {"bih_2D": 1, "Abh0": 1e4},
                                {"bih_2D": 1, "mom_adv_2D": 0, "Abh0": 1e4}, {"mom_adv_3D": 0},
                                {"filt_bi_3D": 1, "filt_bi_2D": 1}, {"im_vert_visc": 1, "im_vert_visc_fic": 0},
                                {"im_vert_visc": 1, "im_vert_visc_fic": 1}, {"im_vert_visc_fic": 0}])
def test_counted_launches_are_the_launches(fake, kw):
    """fesomc_gpu_kernel_launches against the launches made: the first step
    and the captured one."""
    from fesomc import cases
    g = _model(**kw)
    try:
        if "atm" in kw:
            g.set_atm_fields(*cases.atm_coefficients(g.case.mesh, g.case.params.time_jd0))
        for _ in range(2):
            f = g.case.forcing_fn(1, g.time_jd)
            g.set_forcing(f)
            fake.clear()
            n0 = g.kernel_launches()
            assert g.lib.fesomc_gpu_step(g.h, 1) == 0
            assert g.kernel_launches() - n0 == _kernels(fake)
    finally:
        g.close()


@pytest.mark.parametrize("fp32", [0, 1])
def test_page_locked_arrays_receive_the_copy_directly(fake, fp32):
    """A read-back into page-locked arrays (here the ones a snapshot locked)
    copies its FP64 fields straight into them; the FP32 fields, which are
    widened on the host, and pageable arrays go through the staging slots."""
    from fesomc import abi
    g = _model(fp32_form=fp32)
    try:
        want = g.state()
        g.snapshot_begin()
        g.snapshot_end()
        arrays, st = g._snap
        fp64 = {"eta_n", "eta_n_1", "eta_n_2", "etaAB", "ssh_gp"} if fp32 else set(arrays)
        for pageable in (False, True):
            if pageable:
                arrays = {k: np.empty_like(v) for k, v in arrays.items()}
                st = g.case.state_struct(arrays, 0.0)
            for v in arrays.values():
                v[...] = -1.0
            fake.clear()
            abi.check(g.lib.fesomc_gpu_sync_to_host(g.h, abi.F_ALL, C.byref(st)))
            assert fake.lib.fake_pending() == 0
            to = {o.dst for o in fake.ops() if o.kind == "h"}
            for k, v in arrays.items():
                assert np.array_equal(v, want[k]), k
                assert (v.ctypes.data in to) == (k in fp64 and not pageable), k
    finally:
        g.close()


@pytest.mark.parametrize("fp32", [0, 1])
def test_staging_memory_grows_with_use_and_is_given_back(fake, fp32):
    """The page-locked slots are made as read-backs justify them (1.5 MB for
    small ones, more with the volume of larger ones, 16 MB at most), shared by
    the process's models and freed with the last of them; the values are the
    same at every stage."""
    from fesomc import cases, model
    MB = 1 << 20
    base = fake.lib.fake_pinned_bytes()
    events = fake.lib.fake_live_events()
    a = _model()
    held = fake.lib.fake_pinned_bytes()          # a model's own small buffers
    try:
        want = a.state()
        assert fake.lib.fake_pinned_bytes() - held == 3 * MB // 2
        case = cases.estuary_case("e", 200, 100, 300.0, 21, 2.0, 25.0, fp32_form=fp32)
        b = model.GpuModel(case)
        held = fake.lib.fake_pinned_bytes() - 3 * MB // 2
        sizes = []
        first = b.state()
        assert 64 * MB < sum(v.nbytes for k, v in first.items() if k != "_time_jd") < 128 * MB
        for _ in range(4):
            sizes.append((fake.lib.fake_pinned_bytes() - held) / MB)
            got = b.state()
            for k, v in got.items():
                assert np.array_equal(v, first[k]), k
        assert sizes == [4.5, 16.5, 16.5, 16.5]
        got = a.state()
        assert all(np.array_equal(got[k], v) for k, v in want.items())
        b.close()
        assert fake.lib.fake_pinned_bytes() - base >= 16 * MB
    finally:
        a.close()
    assert fake.lib.fake_pinned_bytes() == base and fake.lib.fake_live_events() == events


@pytest.mark.parametrize("fp32,nsigma,early", [(1, 40, True), (1, 41, False), (1, 127, False), (0, 63, False), (0, 127, False)])
def test_column_kernel_with_large_local_arrays_is_not_started_early(fake, fp32, nsigma, early):
    """d3_end with one thread per column and local arrays for more than 40
    levels: started early its few blocks crowd the first SMs that have room,
    and their arrays leave the cache."""
    from fesomc import cases, model
    g = model.GpuModel(cases.estuary_case("e", 20, 10, 300.0, nsigma, 2.0, 25.0, fp32_form=fp32))
    try:
        fake.clear()
        g.step(2)
        got = {o.early for o in fake.ops() if "k_d3endILi" in o.name}
        assert got == {early}
    finally:
        g.close()


def _launched(fake, nx, ny, nsigma, fp32, **kw):
    """Names of the kernels of a step."""
    from fesomc import cases, model
    g = model.GpuModel(cases.estuary_case("e", nx, ny, 300.0, nsigma, 2.0, 25.0, fp32_form=fp32, **kw))
    try:
        fake.clear()
        g.step(1)
        return " ".join(o.name for o in fake.ops() if o.kind == "k")
    finally:
        g.close()


# 160x100: 16,261 nodes; 280x150: 42,431; 310x160: 50,071
@pytest.mark.parametrize("nx,ny,nsigma,fp32,reg", [(160, 100, 11, 0, False), (280, 150, 11, 0, True), (280, 150, 11, 1, False),
                                                   (310, 160, 11, 1, True), (310, 160, 5, 1, True), (280, 150, 9, 0, True),
                                                   (310, 160, 12, 0, False), (280, 150, 21, 1, True), (160, 100, 21, 0, False)])
def test_vertical_diffusion_form(fake, nx, ny, nsigma, fp32, reg):
    """Register tiles for few layers (and 20) on grids that fill the device."""
    names = _launched(fake, nx, ny, nsigma, fp32)
    assert ("k_vdiff_regILi%dE" % (nsigma - 1) in names) == reg and ("k_vdiff_tile" in names) != reg


# 160x100: about 21 k elements; 200x120: 31 k; 280x150: 55 k
@pytest.mark.parametrize("nx,ny,nsigma,fp32,reg", [(160, 100, 11, 0, False), (160, 100, 7, 1, False), (200, 120, 7, 1, True),
                                                   (200, 120, 7, 0, False), (280, 150, 11, 0, True), (280, 150, 11, 1, True),
                                                   (280, 150, 5, 1, True), (280, 150, 12, 0, False), (280, 150, 21, 1, False)])
def test_implicit_viscosity_form(fake, nx, ny, nsigma, fp32, reg):
    """Register tiles for few layers on grids that fill the device."""
    names = _launched(fake, nx, ny, nsigma, fp32)
    assert ("k_implvisc_fic_regILi%dE" % (nsigma - 1) in names) == reg and ("k_implvisc_fic_tile" in names) != reg


@pytest.mark.parametrize("nx,ny,nsigma,fp32,tiles", [(160, 100, 11, 0, True), (280, 150, 11, 0, False), (280, 150, 5, 0, False),
                                                     (280, 150, 12, 0, True), (280, 150, 11, 1, False), (160, 100, 21, 1, False)])
def test_d3end_form(fake, nx, ny, nsigma, fp32, tiles):
    """Tiles of columns, or one thread per column: FP32, and few levels on
    grids that fill the device; the knob reports the form."""
    from fesomc import autotune, cases, model
    case = cases.estuary_case("e", nx, ny, 300.0, nsigma, 2.0, 25.0, fp32_form=fp32)
    g = model.GpuModel(case)
    try:
        for form in (None, 1) if fp32 else (None, 1, 2):
            if form:
                autotune.apply(g, {"d3end_arrays": form})
            else:
                assert autotune.get(g)[0]["d3end_arrays"] == (2 if tiles else 1)
            fake.clear()
            g.step(1)
            names = " ".join(o.name for o in fake.ops() if o.kind == "k")
            want = tiles if form is None else form == 2
            assert ("k_d3end_tileILi" in names) == want and ("k_d3endILi" in names) != want
    finally:
        g.close()


@pytest.mark.parametrize("nsigma,fp32,cols", [(55, 0, 32), (56, 0, 16), (106, 0, 16), (107, 0, 8), (127, 0, 8), (127, 1, 32)])
def test_implicit_viscosity_tile(fake, nsigma, fp32, cols):
    """FP64 tiles of 16 and 8 columns where 32 and 16 leave an SM fewer than
    four."""
    assert "k_implvisc_fic_tileILi%dE" % cols in _launched(fake, 20, 10, nsigma, fp32)


@pytest.mark.parametrize("nsigma,columns,pressure,p1", [(11, 16, 16, 16), (21, 8, 8, 8), (25, 6, 8, 8), (45, 3, 5, 5),
                                                        (54, 3, 3, 3), (55, 2, 4, 4), (81, 2, 4, 2), (84, 3, 4, 3), (97, 1, 4, 2),
                                                        (106, 3, 4, 3), (108, 1, 4, 2), (120, 1, 4, 2), (121, 1, 4, 1),
                                                        (127, 1, 4, 1)])
def test_columns_per_block(fake, nsigma, columns, pressure, p1):
    """Entities per block of the column kernels, by the level count."""
    from fesomc import cases, model
    g = model.GpuModel(cases.estuary_case("e", 20, 10, 300.0, nsigma, 2.0, 25.0))
    try:
        fake.clear()
        g.step(1)
        block = {o.name: o.block for o in fake.ops() if o.kind == "k"}
        for k, b in (("k_pressure_col", pressure), ("k_bpg_elem", columns), ("k_update3d", columns), ("k_wvel", columns),
                     ("k_p1_elem", p1)):
            assert {v for n, v in block.items() if k in n} == {b * (nsigma - 1)}, k
    finally:
        g.close()


@pytest.mark.parametrize("nsigma", [11, 21, 40, 41])
@pytest.mark.parametrize("form", [2, 3, 4, 5, 6])
def test_d3end_forms_of_fp32(fake, nsigma, form):
    """The knob's forms of FP32: arrays in shared memory, a set-up and a sweep
    kernel up to 40 levels (in registers for 21), all counted; the arrays
    between the two kernels are made when a form asks for them, and a refusal
    changes nothing."""
    from fesomc import autotune, cases, model
    g = model.GpuModel(cases.estuary_case("e", 20, 10, 300.0, nsigma, 2.0, 25.0, fp32_form=1))
    try:
        split = form >= 3 and nsigma <= 40
        fake.lib.fake_fail_malloc(2)
        if split:
            with pytest.raises(RuntimeError):
                autotune.apply(g, {"d3end_arrays": form})
            assert autotune.get(g)[0]["d3end_arrays"] == 1
        fake.lib.fake_fail_malloc(-1)
        autotune.apply(g, {"d3end_arrays": form})
        fake.clear()
        n0 = g.kernel_launches()
        g.step(1)
        assert g.kernel_launches() - n0 == _kernels(fake)
        names = " ".join(o.name for o in fake.ops() if o.kind == "k")
        assert ("k_d3end_setup" in names) == split
        assert ("k_d3end_sweep_regILi21ELi%dE" % (8 if form == 6 else 6) in names) == (form >= 5 and nsigma == 21)
        assert ("k_d3end_sweep_sm" in names) == (split and not (form >= 5 and nsigma == 21))
        assert ("k_d3end_sm" in names) == (form == 2)
        assert ("k_d3endILi" in names) == (form >= 3 and not split)
    finally:
        fake.lib.fake_fail_malloc(-1)
        g.close()


def test_search_leaves_out_what_nothing_reads(fake, monkeypatch):
    """The autotuner's search tries no knob that no launch reads, or whose
    kernels the case does not run; the shapes name every knob all the same."""
    from fesomc import autotune, cases
    tried = set()
    apply = autotune.apply
    monkeypatch.setattr(autotune, "apply", lambda g, shapes: (tried.update(shapes), apply(g, shapes)))
    shapes, report = autotune.search(cases.estuary("small"), steps=1, warmup=1)
    assert set(shapes) == {n for n, _ in autotune.knobs(fake.lib)} and all(v > 0 for v in shapes.values())
    assert not tried & {"zero_filt", "vdiff_form", "implvisc_form", "upwind_h", "velgrad2d"}
    assert {"velrhs", "columns", "d3end_arrays", "muscl_h"} <= tried and report["trials"] > 0


def test_readback_with_another_device_current(fake):
    """A model is read back on its own device's events whatever device is
    current in the calling thread, which stays current."""
    from fesomc import cases, model
    rt = fake.lib
    g = model.GpuModel(cases.estuary_case("e", 200, 100, 300.0, 21, 2.0, 25.0))
    try:
        assert rt.fesomc_gpu_set_device(1) == 0
        events = rt.fake_live_events()
        got = g.state()
        assert rt.fake_live_events() > events          # the slots' own
        now = C.c_int(-1)
        rt.cudaGetDevice(C.byref(now))
        assert now.value == 1
        assert all(np.array_equal(got[k], v) for k, v in g.case.state0.items())
    finally:
        rt.fesomc_gpu_set_device(0)
        g.close()


@pytest.mark.parametrize("batch,rows", [(1, 64), (4608, 64), (4609, 128), (8192, 128)])
def test_network_tile(fake, batch, rows):
    """The FP32 network's products (256 hidden units): tiles of 128 rows where
    they give every SM a block, else of 64; the weight gradients, split over
    the batch, of 128."""
    from fesomc import closure
    c = closure.Closure(21)
    try:
        fake.clear()
        c.grad(np.zeros((batch, c.n_in), dtype=np.float32), np.zeros((batch, c.n_out), dtype=np.float32))
        hidden = [o for o in fake.ops() if "k_sgemmILb0ELb1ELi2E" in o.name]
        parts = [o for o in fake.ops() if "k_sgemmILb1ELb0ELi0E" in o.name]
        assert len(hidden) == 3 and {("ELi%dE" % rows) in o.name[-60:] for o in hidden} == {True}
        assert len(parts) == 4 and all("Li0ELi128E" in o.name for o in parts)
        assert all((o.grid >= 148) == (rows == 128) or rows == 64 for o in hidden)
    finally:
        c.close()
