"""Host arrays as callers may hold them, against ordinary ones bit for bit: off the 8-byte boundaries of their
doubles (a field inside a packed record), which only the copy engines can move; with pages missing, or page-locked."""
import numpy as np
import pytest

from simplebubblyflowsolver_gb300 import SYNC_ALL, SYNC_NONE, SYNC_STATE, ic

from ._helpers import clone, new_state, set_env

pytestmark = pytest.mark.gpu

FIELDS = ("ux", "uy", "p", "psi0", "psi1", "vof")


@pytest.fixture(scope="module")
def libs():
    import oracle
    from simplebubblyflowsolver_gb300 import load_library
    return load_library(), oracle.Oracle()


def _start(libs, nx, ny):
    gpu, orc = libs
    wl = ic.single_bubble(nx, ny)
    set_env(wl)
    for lib in libs:
        lib.set_dt_coefs(wl.coef_dt_adv, wl.coef_dt_dif, wl.coef_dt_int)
    gpu.set_autotune(False)
    gpu.set_sync_mode(SYNC_STATE)
    return new_state(wl, orc)


def _move(st, slots, offset):
    """the arrays of `slots` in buffers of their own, `offset` bytes past an 8-byte boundary"""
    for s in slots:
        old = st.field(s)
        raw = np.zeros(old.nbytes + 16, dtype=np.uint8)
        at = -raw.ctypes.data % 8 + offset
        new = raw[at:at + old.nbytes].view(np.float64).reshape(old.shape)
        new[...] = old
        st._buffers[new.ctypes.data] = new
        st._array_t(s).data = new.ctypes.data


def _same(a, b, slots):
    for s in slots:
        assert np.array_equal(a.field(s), b.field(s), equal_nan=True), s


CALLS = {
    "decide_dt": lambda g, s, dt: g.decide_dt(s),
    "density": lambda g, s, dt: g.compute_density(s, 0),
    "curvature": lambda g, s, dt: g.compute_curvature_tensor(s),
    "force": lambda g, s, dt: g.compute_force(s),
    "vof": lambda g, s, dt: g.update_vof(s, 0, dt),
    "predict": lambda g, s, dt: g.predict_field(s, 0, dt),
    "potential": lambda g, s, dt: g.compute_potential(s, 0.2 * dt, 0.5 * dt),
    "correct": lambda g, s, dt: g.correct_velocity(s, 0.2 * dt, 0.5 * dt),
    "pressure": lambda g, s, dt: g.update_pressure(s),
}


@pytest.mark.parametrize("offset", [1, 4])
def test_off_boundary_single_calls(libs, offset):
    gpu = libs[0]
    a = _start(libs, 37, 16)
    dt = gpu.integrate(a)
    b = clone(a)
    _move(b, b.slots(), offset)
    for call in CALLS.values():
        call(gpu, a, dt)
        call(gpu, b, dt)
        _same(a, b, a.slots())


@pytest.mark.parametrize("mode", [SYNC_STATE, SYNC_ALL])
def test_off_boundary_steps(libs, mode):
    gpu = libs[0]
    a = _start(libs, 37, 16)
    b = clone(a)
    _move(b, b.slots(), 4)
    gpu.set_sync_mode(mode)
    try:
        da = [gpu.integrate(a) for _ in range(3)]
        assert gpu.host_link_used() == (mode == SYNC_STATE)
        db = [gpu.integrate(b) for _ in range(3)]
        assert not gpu.host_link_used()
    finally:
        gpu.set_sync_mode(SYNC_STATE)
    assert da == db
    _same(a, b, a.slots())


def test_off_boundary_downloads(libs):
    """one array of the six is enough; of a batch's cases, one"""
    gpu = libs[0]
    st = _start(libs, 37, 16)
    out = [clone(st) for _ in range(2)]
    _move(out[1], ["psi1"], 4)
    batch = [[clone(st) for _ in range(3)] for _ in range(2)]
    _move(batch[1][2], ["vof"], 4)
    gpu.set_sync_mode(SYNC_NONE)
    try:
        gpu.invalidate_device()
        gpu.run_steps_timed(st, 2)
        for o in out:
            gpu.sync_to_host(o)
        for b in batch:
            gpu.batch_release()
            gpu.integrate_batch(b)
            gpu.batch_sync_to_host(b)
    finally:
        gpu.set_sync_mode(SYNC_STATE)
        gpu.batch_release()
    _same(out[0], out[1], FIELDS)
    for x, y in zip(*batch):
        _same(x, y, FIELDS)


# 640 x 1024: 5.3 MB an array, so pages are looked at
@pytest.mark.parametrize("pages", ["untouched", "some", "locked"])
def test_large_arrays_with_missing_pages(libs, pages):
    """downloads and steps into arrays that have no pages, some, or page-locked ones, as into ordinary ones"""
    gpu = libs[0]
    st = _start(libs, 640, 1024)
    ordinary, other = clone(st), clone(st)
    for s in FIELDS:
        ordinary.field(s)[...] = 1.0  # every page written
    if pages != "locked":
        for s in FIELDS:
            shape = other.field(s).shape
            new = np.zeros(shape)  # fresh mapping, no page of it touched
            if pages == "some":
                new[:shape[0] // 3] = 1.0
            other._buffers[new.ctypes.data] = new
            other._array_t(s).data = new.ctypes.data
    else:
        gpu.pin_host_state(other)
    gpu.set_sync_mode(SYNC_NONE)
    try:
        gpu.invalidate_device()
        gpu.run_steps_timed(st, 1)
        for o in (ordinary, other):
            gpu.sync_to_host(o)
        _same(ordinary, other, FIELDS)
        for mode in (SYNC_ALL, SYNC_STATE):
            gpu.set_sync_mode(mode)
            assert gpu.integrate(ordinary) == gpu.integrate(other)
            _same(ordinary, other, FIELDS)
    finally:
        gpu.set_sync_mode(SYNC_STATE)
        if pages == "locked":
            gpu.unpin_host_state(other)
        gpu.release()
