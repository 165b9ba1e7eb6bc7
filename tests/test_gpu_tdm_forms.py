"""Forms of the tridiagonal solves against each other bit for bit: clusters of two and of four CTAs a wavenumber pair
against one block a pair, on the FP64 unit alone and shared with the integer pipes, staged in global memory, and
whatever the autotuner picks; cases of a batch that differ, each against itself alone."""
import numpy as np
import pytest

from simplebubblyflowsolver_gb300 import SYNC_NONE, SYNC_STATE, ic

from ._helpers import clone, new_state, set_env

pytestmark = pytest.mark.gpu

STATE = ("ux", "uy", "p", "psi0", "psi1", "vof")


@pytest.fixture(scope="module")
def libs():
    import oracle
    from simplebubblyflowsolver_gb300 import load_library
    return load_library(), oracle.Oracle()


def _start(libs, nx, ny, k=0):
    """a bubble in square cells, its place by k"""
    gpu, orc = libs
    h = max(2.0 / nx, 0.5 / ny)
    lx, ly = nx * h, ny * h
    r = min(0.25, 0.3 * ly, 0.3 * lx) * (1 - 0.07 * k)
    wl = ic.Workload("tdm", nx, ny, lx, ly, [(min(0.5, lx / 2) + 0.3 * k * h, ly * (0.5 + 0.11 * k) % ly, r)],
                     Re=35.0, We=10.0, Fr=1.0, denr=0.1, visr=0.1)
    set_env(wl)
    for lib in libs:
        lib.set_dt_coefs(wl.coef_dt_adv, wl.coef_dt_dif, wl.coef_dt_int)
    gpu.set_autotune(False)
    gpu.set_sync_mode(SYNC_STATE)
    return new_state(wl, orc)


def _same(a, b):
    for s in STATE:
        assert np.array_equal(a.field(s), b.field(s)), s


# warps a system 2 with FP64 alone, 2 with padding rows, 4 shared; 8192 rows: a block stages them in global memory
@pytest.mark.parametrize("nx,ny,warps", [(256, 128, 2), (200, 16, 2), (1000, 512, 4), (8192, 16, 4), (8192, 32, 4)])
def test_cluster_as_block(libs, nx, ny, warps):
    gpu = libs[0]
    st = _start(libs, nx, ny)
    runs = {}
    try:
        for on in (True, False):
            gpu.release()
            gpu.set_tdm_cluster(on)
            o = clone(st)
            dts = [gpu.integrate(o) for _ in range(2)]
            t = gpu.tiles()
            assert t["tdm_warps"] == warps and (t["tdm_modes"] == 0) == on, t
            runs[on] = (dts, o)
    finally:
        gpu.set_tdm_cluster(True)
        gpu.release()
    assert runs[True][0] == runs[False][0]
    _same(runs[True][1], runs[False][1])


# two warps a system: the pairs fill the SMs, so only the autotuner may take clusters
@pytest.mark.parametrize("ahead", [True, False])
@pytest.mark.parametrize("nx,ny", [(300, 1024), (256, 128)])
def test_autotuned_as_default(libs, nx, ny, ahead):
    """with the listed-faces form as well, whose lists every launch shape of the geometry has to start empty"""
    gpu = libs[0]
    st = _start(libs, nx, ny)
    a, b = clone(st), clone(st)
    try:
        gpu.set_geometry_ahead(ahead)
        for o, tune in ((a, False), (b, True)):
            gpu.release()
            gpu.set_autotune(tune)
            gpu.set_sync_mode(SYNC_NONE)
            o.dts = [gpu.integrate(o) for _ in range(4)]
            gpu.sync_to_host(o)
            gpu.set_sync_mode(SYNC_STATE)
            print(gpu.tiles())
    finally:
        gpu.set_geometry_ahead(True)
        gpu.set_autotune(False)
        gpu.set_sync_mode(SYNC_STATE)
        gpu.release()
    assert a.dts == b.dts
    _same(a, b)


# clusters of two in either; of four, shared only in the batch; blocks of two in the batch, shared; one warp a system;
# 8192 rows staged in global memory, shared only in the batch (the clusters off); transforms shared only in the batch,
# chunks of 4 rows in registers and plainly, of 5 plainly and shared; of 10 and 22 rows, groups of eight and the rest
@pytest.mark.parametrize("nx,ny,cases,cluster", [(256, 128, 3, True), (512, 256, 2, True), (256, 128, 8, True),
                                                 (125, 64, 33, True), (8192, 16, 2, True), (8192, 16, 2, False),
                                                 (100, 512, 8, True), (300, 512, 3, True), (1200, 64, 4, True),
                                                 (2700, 64, 2, True)])
def test_different_cases_in_a_batch_as_alone(libs, nx, ny, cases, cluster):
    gpu = libs[0]
    start = [_start(libs, nx, ny, k % 5) for k in range(cases)]
    alone = [clone(st) for st in start[:5]]
    batch = [clone(st) for st in start]
    try:
        gpu.set_tdm_cluster(cluster)
        gpu.release()
        dts = []
        for a in alone:
            dts.append([gpu.integrate(a) for _ in range(2)])
            warps = gpu.tiles()["tdm_warps"]
        got = [gpu.integrate_batch(batch) for _ in range(2)]
        assert gpu.tiles(0)["tdm_warps"] == warps
    finally:
        gpu.set_tdm_cluster(True)
        gpu.batch_release()
        gpu.release()
    for i, b in enumerate(batch):
        assert [g[i] for g in got] == dts[i % 5], i
        _same(b, alone[i % 5])
    assert not np.array_equal(alone[0].field("vof"), alone[1].field("vof"))
