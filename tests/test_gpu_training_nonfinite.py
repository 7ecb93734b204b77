"""Training with values that are not finite: sums that overflow are infinite,
as FP32 sums are, and samples outside a batch have no part in it."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_training import KEYS, f64, problem, shuffle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def F():
    import feddlib_gb300 as F
    return F


@pytest.mark.parametrize("H", [64, 16])
@pytest.mark.parametrize("n", [1, 20, 5001])
def test_infinite_sums(F, H, n):
    """A target of 1e25: its squared distance overflows, every gradient is
    still finite.  Targets of -3e38: b3's gradient overflows too."""
    X, ty, tg, m = problem(H, n, n)
    ty[n // 2] = 1e25
    tr = F.Trainer(H, X, ty, tg)
    tr.set_params(m)
    loss, g = tr.grad(wpsi=1.0, wgrad=0.7)
    _, go = O.mlp_loss({k: f64(v) for k, v in m.items()}, f64(X), f64(ty), f64(tg), 1.0, 0.7)
    assert loss == np.inf
    for k in KEYS:  # the bound of the finite case
        assert np.linalg.norm(f64(g[k]) - go[k]) <= 1e-4 * np.linalg.norm(go[k]), k
    assert abs(g["b3"] - go["b3"]) <= 1e-4 * abs(go["b3"])
    tr = F.Trainer(H, X, np.full(n, -3e38, dtype=np.float32), tg)
    tr.set_params(m)
    loss, g = tr.grad(wpsi=1.0, wgrad=0.7)
    assert loss == np.inf and g["b3"] == np.inf


@pytest.mark.parametrize("H", [64, 16])
@pytest.mark.parametrize("n,batch", [(40, 17), (6000, 5001)])
def test_samples_outside_the_batch(F, H, n, batch):
    """A step's last tile is filled up to 16 or 48 samples; a sample that is
    not finite but not in the batch changes nothing."""
    X, ty, tg, m = problem(H, n, 200 + n)
    seed = next(s for s in range(100) if 0 not in order_of(n, s)[:batch])
    got = []
    for bad in (None, np.nan, np.inf):
        x, y, g = X.copy(), ty.copy(), tg.copy()
        if bad is not None:
            x[0] = y[0] = g[0] = bad
        tr = F.Trainer(H, x, y, g)
        tr.set_params(m)
        got.append((tr.run(1, batch, 1e-3, wpsi=1.0, wgrad=0.7, seed=seed), tr.get_params()))
    assert np.isfinite(got[0][0])
    for loss, par in got[1:]:
        assert loss == got[0][0]
        assert all(np.array_equal(par[k], got[0][1][k]) for k in KEYS + ("b3",))


def order_of(n, seed):
    perm = list(range(n))
    shuffle(perm, seed, 0)
    return perm
