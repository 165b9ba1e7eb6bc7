"""Training steps of both paths (the batches of an epoch in one launch, up to 2048 rows; separate launches above)
against Adam on the gradient entry point's gradients, every operation rounded to FP32 on the host: the same bits, over
several steps, so both paths form the same sums.  The two sums of Adam are fused multiply-adds on the GPU, of which
product the compiler decides: one choice has to fit all steps of all batches."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

F = np.float32
LR, B1, B2, EPS = F(2e-3), F(0.9), F(0.999), F(1e-8)


@pytest.fixture(scope="module")
def data():
    from simplebubblyflowsolver_gb300 import load_library
    from simplebubblyflowsolver_gb300 import learned_curvature as L
    x, y = L.dataset(1500, seed=7)
    perm = np.random.default_rng(3).permutation(x.shape[0]).astype(np.int32)
    X = torch.from_numpy(x).cuda().to(torch.bfloat16).contiguous()
    return load_library(), L.init_params(4), X, torch.from_numpy(y).cuda(), torch.from_numpy(perm).cuda()


def _fma(a, b, c):
    """a b + c rounded once: the product is exact in FP64, the sum rounded there to odd, which FP32's rounding undoes"""
    p, c = np.float64(a) * np.asarray(b, np.float64), np.asarray(c, np.float64)
    s = p + c
    t = s - p
    lost = (p - (s - t)) + (c - t)
    to_odd = (lost != 0) & (s.view(np.int64) % 2 == 0)
    return np.where(to_odd, np.nextafter(s, np.where(lost > 0, np.inf, -np.inf)), s).astype(F)


def _powf():
    f = C.CDLL("libm.so.6").powf
    f.argtypes, f.restype = [C.c_float, C.c_float], C.c_float
    return f


def _steps(data, batch, nsteps, first, second):
    """how many of the steps the host's Adam gives bit for bit, with the fused product of each sum"""
    lib, p0, X, Y, idx = data
    powf = _powf()
    moves = np.ones(p0.size, bool)
    w1 = np.arange(64 * 16)
    moves[:64 * 16] = w1 % 16 < 11
    lib.mlp_set_params(p0)
    p, m1, m2 = p0.astype(F).copy(), np.zeros(p0.size, F), np.zeros(p0.size, F)
    for t in range(1, nsteps + 1):
        at = idx.data_ptr() + 4 * batch * (t - 1)
        g, loss = lib.mlp_gradient(X.data_ptr(), Y.data_ptr(), at, batch)
        g = g.astype(F)
        trained = lib.mlp_train_epoch(X.data_ptr(), Y.data_ptr(), at, batch, batch, float(LR))
        assert trained == loss
        u, v = F(1) - B1, (F(1) - B2) * g
        a = _fma(B1, m1, u * g) if first else _fma(u, g, B1 * m1)
        b = _fma(B2, m2, v * g) if second else _fma(v, g, B2 * m2)
        c1, c2 = (F(1) / (F(1) - F(powf(float(q), float(t)))) for q in (B1, B2))
        new = p - (LR * (a * c1)) / (np.sqrt(b * c2) + EPS)
        p, m1, m2 = (np.where(moves, n, o) for n, o in ((new, p), (a, m1), (b, m2)))
        if not np.array_equal(lib.mlp_get_params(), p):
            return t - 1
    return nsteps


def test_both_paths_are_adam_bit_for_bit(data):
    steps = 4
    sizes = (2049, 50, 1000, 1100, 2048)  # separate launches, part of a tile, 8 tiles, two tiles a block, 16 tiles
    fits = {(first, second): [_steps(data, n, steps, first, second) for n in sizes]
            for first in (True, False) for second in (True, False)}
    assert [steps] * len(sizes) in fits.values(), fits
