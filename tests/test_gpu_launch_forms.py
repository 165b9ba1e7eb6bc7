"""Forms a launch takes by its size or its arrays, against each other bit for bit: a case alone (one part of a cell a
thread, transforms over lanes, FP64 alone) and in batches whose cells pass each line (shared with the integer pipes,
in halves and whole; transforms and tridiagonal solves shared); the fine-grained calls' and downloads' copies in one
launch and one by one."""
import numpy as np
import pytest

from simplebubblyflowsolver_gb300 import RK_GAMMA, SYNC_NONE, SYNC_STATE, ic

from ._helpers import clone, new_state, set_env

pytestmark = pytest.mark.gpu

STATE = ("ux", "uy", "p", "psi0", "psi1", "vof")


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


# cells of the batch: 49k to 98k, 98k to 262k, above; nx leaves ragged blocks, 64 rows take the radix-8 stage, 128 not
@pytest.mark.parametrize("nx,ny,cases", [(125, 64, 7), (125, 64, 13), (125, 64, 33), (61, 128, 7), (61, 128, 35)])
def test_batched_case_steps_as_alone(libs, nx, ny, cases):
    gpu = libs[0]
    st = _start(libs, nx, ny)
    alone = clone(st)
    batch = [clone(st) for _ in range(cases)]
    for _ in range(3):
        dt = gpu.integrate(alone)
        dts = gpu.integrate_batch(batch)
        assert (np.asarray(dts) == dt).all()
    gpu.batch_release()
    for b in (batch[0], batch[-1]):
        for s in STATE:
            assert np.array_equal(b.field(s), alone.field(s)), s


CALLS = {
    "density": lambda g, s, dt: g.compute_density(s, 0),
    "viscosity": lambda g, s, dt: g.compute_viscosity(s),
    "curvature": lambda g, s, dt: g.compute_curvature_tensor(s),
    "force": lambda g, s, dt: g.compute_force(s),
    "vof": lambda g, s, dt: g.update_vof(s, 1, dt),
    "mass_flux": lambda g, s, dt: g.compute_mass_flux(s),
    "predict": lambda g, s, dt: g.predict_field(s, 1, dt),
    "potential": lambda g, s, dt: g.compute_potential(s, RK_GAMMA[0] * dt, RK_GAMMA[1] * dt),
    "correct": lambda g, s, dt: g.correct_velocity(s, RK_GAMMA[0] * dt, RK_GAMMA[1] * dt),
    "pressure": lambda g, s, dt: g.update_pressure(s),
}
SLOTS = STATE + ("den0", "den1", "visux", "visuy", "dvof", "normal", "curv", "ifrcx", "ifrcy", "fluxx", "fluxy")


@pytest.mark.parametrize("nx,ny", [(37, 16), (130, 64)])
def test_calls_copy_in_one_launch_as_one_by_one(libs, nx, ny):
    gpu = libs[0]
    st = _start(libs, nx, ny)
    dt = gpu.integrate(st)
    a, b = clone(st), clone(st)
    for name, call in CALLS.items():
        for state, link in ((a, True), (b, False)):
            gpu.set_host_link(link)
            try:
                call(gpu, state, dt)
            finally:
                gpu.set_host_link(True)
        for s in SLOTS:
            assert np.array_equal(a.field(s), b.field(s), equal_nan=True), (name, s)


@pytest.mark.parametrize("nx,ny", [(37, 16), (130, 64)])
def test_download_in_one_launch_as_one_by_one(libs, nx, ny):
    gpu = libs[0]
    st = _start(libs, nx, ny)
    gpu.set_sync_mode(SYNC_NONE)
    try:
        gpu.invalidate_device()
        gpu.run_steps_timed(st, 3)
        out = []
        for link in (True, False):
            gpu.set_host_link(link)
            o = clone(st)
            for s in STATE:
                o.field(s)[...] = np.nan
            gpu.sync_to_host(o)
            out.append(o)
    finally:
        gpu.set_host_link(True)
        gpu.set_sync_mode(SYNC_STATE)
    for s in STATE:
        a, b = out[0].field(s), out[1].field(s)
        assert np.isfinite(a[2:-2]).all() and np.array_equal(a, b, equal_nan=True), s
