"""decide_dt's advective limit, coef min(1, h / (|u| + small)), where the 1 is the least of its terms: slow flow in
cells wider than it travels in a unit of time, and an advective coefficient below the others'."""
import numpy as np
import pytest

from simplebubblyflowsolver_gb300 import ic
from simplebubblyflowsolver_gb300._abi import SolverState
from simplebubblyflowsolver_gb300.binding import SolverError

pytestmark = pytest.mark.gpu

COEFS = (0.25, 0.95, 0.95)


@pytest.fixture(scope="module")
def libs():
    import oracle
    from simplebubblyflowsolver_gb300 import load_library
    both = load_library(), oracle.Oracle()
    for lib in both:
        lib.set_dt_coefs(*COEFS)
    yield both
    wl = ic.single_bubble(64, 32)
    for lib in both:
        lib.set_dt_coefs(wl.coef_dt_adv, wl.coef_dt_dif, wl.coef_dt_int)


# a thread has a column's quotient, one the uy one: 256 threads a block, none without a quotient where nx = 256 or 512
@pytest.mark.parametrize("nx", [64, 255, 256, 257, 512])
def test_unit_bound(libs, nx):
    ny, h = 16, 4.0
    st = SolverState(nx, ny, nx * h, ny * h, Re=100.0, Fr=1.0, denr=0.5, visr=0.5, We=100.0)
    rng = np.random.default_rng(nx)
    for s in ("ux", "uy"):
        st.interior_rows(s)[...] = 0.1 * rng.uniform(-1, 1, st.interior_rows(s).shape)
        libs[1].update_boundaries(st, s)
    # the quotients are at least 4 / 0.1, the diffusive and capillary bounds 380 and 0.95
    for lib in libs:
        assert lib.decide_dt(st) == COEFS[0]


@pytest.mark.parametrize("nx", [64, 256, 512])
def test_non_finite_velocity_everywhere(libs, nx):
    gpu = libs[0]
    st = SolverState(nx, 16, nx * 4.0, 64.0, Re=100.0, Fr=1.0, denr=0.5, visr=0.5, We=100.0)
    for s in ("ux", "uy"):
        st.field(s)[...] = np.nan
    with pytest.raises(SolverError, match="non-finite"):
        gpu.decide_dt(st)
