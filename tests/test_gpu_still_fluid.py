"""Fluid at rest, or moving along y only: ux is zero everywhere, and the momentum kernels leave the integer forms at
the start of the step.  Cases of a batch that shares its arithmetic with the integer pipes, each against itself alone
(FP64 alone), beside cases in motion; then the first forms of the same kernels by a grid's own size."""
import numpy as np
import pytest

from simplebubblyflowsolver_gb300 import SYNC_NONE, SYNC_STATE, ic

from ._helpers import clone, compare_state, new_state, set_env

pytestmark = pytest.mark.gpu

STATE = ("ux", "uy", "p", "psi0", "psi1", "vof")


@pytest.fixture(scope="module")
def libs():
    import oracle
    from simplebubblyflowsolver_gb300 import load_library
    return load_library(), oracle.Oracle()


def _states(libs, nx, ny):
    """at rest without and with a bubble, moving along y as one and sheared, in motion"""
    gpu, orc = libs
    wl = ic.single_bubble(nx, ny)
    wl.Fr = np.inf
    set_env(wl)
    for lib in libs:
        lib.set_dt_coefs(wl.coef_dt_adv, wl.coef_dt_dif, wl.coef_dt_int)
    gpu.set_autotune(False)
    gpu.set_sync_mode(SYNC_STATE)
    x = np.linspace(0.0, 1.0, nx)
    out = {}
    for name in ("rest", "bubble", "uniform", "shear", "moving"):
        f = wl.fields()
        if name in ("rest", "uniform", "shear"):
            f["vof"][...] = 0.0
        f["uy"][:, 1:-1] = {"uniform": 0.1 + 0 * x, "shear": 0.1 * x * (1 - x)}.get(name, 0 * x)
        if name == "moving":
            y = 2 * np.pi * np.arange(ny) / ny
            f["ux"][:, 1:-1] = 0.05 * np.outer(np.cos(y), np.sin(np.pi * np.arange(1, nx) / nx) ** 2)
        out[name] = new_state(wl, orc, f)
    return out


@pytest.mark.parametrize("nx,ny,cases", [(125, 64, 7), (125, 64, 33)])
def test_cases_in_a_batch_as_alone(libs, nx, ny, cases):
    gpu = libs[0]
    start = _states(libs, nx, ny)
    names = [list(start)[i % len(start)] for i in range(cases)]
    batch = [clone(start[n]) for n in names]
    want = {}
    for n, st in start.items():
        alone = clone(st)
        want[n] = ([gpu.integrate(alone) for _ in range(3)], alone)
    dts = [gpu.integrate_batch(batch) for _ in range(3)]
    gpu.batch_release()
    for i, (n, b) in enumerate(zip(names, batch)):
        assert [d[i] for d in dts] == want[n][0], (i, n)
        for s in STATE:
            assert np.array_equal(b.field(s), want[n][1].field(s)), (i, n, s)
    # what rests stays at rest; the bubble at rest starts to move along x as well
    assert not want["rest"][1].field("ux").any() and not want["rest"][1].field("uy").any()
    assert not want["shear"][1].field("ux").any() and want["bubble"][1].field("ux").any()


# one block of the finishing kernel, and several
@pytest.mark.parametrize("nx", [256, 600])
def test_flow_in_one_column(libs, nx):
    """a single cell's ux says that there is flow: resident steps as the oracle's"""
    gpu, orc = libs
    st = _states(libs, nx, 512)["uniform"]
    st.interior_rows("ux")[3, nx // 2] = 1e-3
    orc.apply_initial_boundaries(st)
    a, b = clone(st), clone(st)
    gpu.set_sync_mode(SYNC_NONE)
    try:
        gpu.invalidate_device()
        gpu.run_steps_timed(a, 2)
        gpu.sync_to_host(a)
    finally:
        gpu.set_sync_mode(SYNC_STATE)
    for _ in range(2):
        orc.integrate(b)
    err = compare_state(a, b, ("ux", "uy", "vof"))
    assert all(e < 1e-10 for e in err.values()), err
