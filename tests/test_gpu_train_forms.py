"""Training epochs in one launch (batches of up to 2048 rows): many steps in a launch as one by one, misaligned
feature rows as aligned ones, and the step against the gradient entry point's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def data():
    from simplebubblyflowsolver_gb300 import load_library
    from simplebubblyflowsolver_gb300 import learned_curvature as L
    x, y = L.dataset(1200, seed=5)
    n = x.shape[0]
    perm = np.random.default_rng(2).permutation(n).astype(np.int32)
    X = torch.from_numpy(x).cuda().to(torch.bfloat16).contiguous()
    return load_library(), L.init_params(3), X, torch.from_numpy(y).cuda(), torch.from_numpy(perm).cuda(), n


def _train(lib, p0, X, Y, idx, chunks, batch):
    lib.mlp_set_params(p0)
    loss = 0.0
    for off, rows in chunks:
        loss += lib.mlp_train_epoch(X.data_ptr(), Y.data_ptr(), idx.data_ptr() + 4 * off, rows, batch, 2e-3) * rows
    return lib.mlp_get_params().copy(), loss / sum(r for _, r in chunks)


# a tile short, one tile, ragged tiles, two tiles a block, and the first size of the separate launches
@pytest.mark.parametrize("batch", [50, 128, 1000, 1100, 2048, 2049])
def test_steps_in_one_launch_as_one_by_one(data, batch):
    lib, p0, X, Y, idx, n = data
    steps = min(n // batch, 5)
    a, la = _train(lib, p0, X, Y, idx, [(0, steps * batch)], batch)
    b, lb = _train(lib, p0, X, Y, idx, [(k * batch, batch) for k in range(steps)], batch)
    assert np.array_equal(a, b) and not np.array_equal(a, p0)
    assert abs(la - lb) <= 1e-12 * abs(la)


def test_more_steps_than_one_launch_takes(data):
    lib, p0, X, Y, idx, n = data
    a, _ = _train(lib, p0, X, Y, idx, [(0, 150 * 40)], 40)
    b, _ = _train(lib, p0, X, Y, idx, [(0, 70 * 40), (70 * 40, 80 * 40)], 40)
    assert np.array_equal(a, b)


def test_misaligned_rows(data):
    lib, p0, X, Y, idx, n = data
    raw = torch.zeros(X.numel() + 8, dtype=torch.bfloat16, device="cuda")
    odd = raw[1:1 + X.numel()].view_as(X)
    odd.copy_(X)
    assert odd.data_ptr() % 16
    a, _ = _train(lib, p0, X, Y, idx, [(0, 3000)], 1000)
    b, _ = _train(lib, p0, odd, Y, idx, [(0, 3000)], 1000)
    assert np.array_equal(a, b)


@pytest.mark.parametrize("batch", [100, 1000])
def test_first_step_is_adam_on_the_gradient(data, batch):
    lib, p0, X, Y, idx, n = data
    lib.mlp_set_params(p0)
    g, _ = lib.mlp_gradient(X.data_ptr(), Y.data_ptr(), idx.data_ptr(), batch)
    a, _ = _train(lib, p0, X, Y, idx, [(0, batch)], batch)
    # from zero moments the bias-corrected step is lr g / (|g| + eps) up to FP32 rounding of its few factors
    want = p0 - 2e-3 * g / (np.abs(g) + 1e-8)
    moved = a != p0
    assert moved.sum() > 0.5 * p0.size
    big = moved & (np.abs(g) > 1e-6)
    assert np.abs(a - want)[big].max() < 2e-3 * 1e-4 + 2 * np.spacing(np.abs(p0).max())
