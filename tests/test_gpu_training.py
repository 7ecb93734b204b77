"""The surrogate's training kernels: the fused width-64 kernel's loss and
gradients at the edges of its 16-sample tiles and beyond one tile per CTA, and
training runs of both paths against a restatement of the seeded sample order
(sequential Fisher-Yates) and Adam on the oracle's FP64 gradients."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

KEYS = ("W1", "b1", "W2", "b2", "w3")


@pytest.fixture(scope="module")
def F():
    import feddlib_gb300 as F
    return F


def problem(H, n, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, 4)).astype(np.float32)
    ty = rng.standard_normal(n).astype(np.float32)
    tg = rng.standard_normal((n, 4)).astype(np.float32)
    m = {"W1": 0.5 * rng.standard_normal((H, 4)), "b1": 0.1 * rng.standard_normal(H),
         "W2": rng.standard_normal((H, H)) / np.sqrt(H), "b2": 0.1 * rng.standard_normal(H),
         "w3": rng.standard_normal(H) / np.sqrt(H), "b3": 0.05}
    return X, ty, tg, {k: np.asarray(v, dtype=np.float32) for k, v in m.items()}


def f64(a):
    return np.asarray(a, dtype=np.float64)


@pytest.mark.parametrize("n", [1, 15, 16, 17, 33, 500, 5001])
def test_fused_gradients(F, n):
    X, ty, tg, m = problem(64, n, n)
    tr = F.Trainer(64, X, ty, tg)
    tr.set_params(m)
    loss, g = tr.grad(wpsi=1.0, wgrad=0.7)
    lo, go = O.mlp_loss({k: f64(v) for k, v in m.items()}, f64(X), f64(ty), f64(tg), 1.0, 0.7)
    # the bounds of the general path's gradient test
    assert abs(loss - lo) <= 1e-5 * abs(lo)
    for k in KEYS:
        assert np.linalg.norm(g[k] - go[k]) <= 1e-4 * np.linalg.norm(go[k]), k
    assert abs(g["b3"] - go["b3"]) <= 1e-4 * max(1.0, abs(go["b3"]))


# one tile of 48 samples per SM instead of two rounds of 16: from 4,865 samples on 152 SMs
@pytest.mark.parametrize("n", [4865, 4895, 4896, 4897, 7296, 7297, 9740])
def test_fused_gradients_two_samples_per_thread(F, n):
    test_fused_gradients(F, n)


def shuffle(perm, seed, step):
    mask = (1 << 64) - 1
    s = (seed ^ (0x5851F42D4C957F2D * (step + 1))) & mask
    for i in range(len(perm) - 1, 0, -1):
        s = (s + 0x9E3779B97F4A7C15) & mask
        z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        j = (z ^ (z >> 31)) % (i + 1)
        perm[i], perm[j] = perm[j], perm[i]


@pytest.mark.parametrize("H", [64, 16])
@pytest.mark.parametrize("n,batch,calls", [(1, 1, [3]), (37, 10, [4, 0, 5]), (3000, 700, [9]), (64, 64, [2, 2])])
def test_runs_follow_the_seeded_order(F, H, n, batch, calls):
    X, ty, tg, m = problem(H, n, 100 + n)
    tr = F.Trainer(H, X, ty, tg)
    tr.set_params(m)
    p = {k: f64(v) for k, v in m.items()}
    m1, m2 = ({k: np.zeros_like(v) for k, v in p.items()} for _ in range(2))
    lr, seed, step, perm, cursor = 1e-3, 12345, 0, list(range(n)), n
    for steps in calls:
        last = tr.run(steps, batch, lr, wpsi=1.0, wgrad=0.7, seed=seed)
        for _ in range(steps):
            if cursor + batch > n:
                shuffle(perm, seed, step)
                cursor = 0
            q = perm[cursor:cursor + batch]
            cursor += batch
            step += 1
            lo, g = O.mlp_loss(p, f64(X)[q], f64(ty)[q], f64(tg)[q], 1.0, 0.7)
            for k in p:
                m1[k] = 0.9 * m1[k] + 0.1 * g[k]
                m2[k] = 0.999 * m2[k] + 0.001 * g[k] * g[k]
                p[k] = p[k] - lr * (m1[k] / (1 - 0.9 ** step)) / (np.sqrt(m2[k] / (1 - 0.999 ** step)) + 1e-8)
        if steps:
            assert abs(last - lo) <= 1e-4 * max(abs(lo), 1e-3)
    got = tr.get_params()
    # a wrong sample in one batch moves a parameter by about lr = 1e-3; FP32
    # gradients (1e-4 of their size) move an Adam step by less than 1e-4 lr
    for k in KEYS + ("b3",):
        assert np.abs(f64(got[k]) - p[k]).max() <= 0.05 * lr, k
