"""The Adam step of the training runs: its bias corrections 1 - beta^t, and the
loss that a run of eight steps of 65,536 samples returns, against 64 bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def F():
    import feddlib_gb300 as F
    return F


@pytest.mark.parametrize("H", [64, 16])
def test_step_length(F, H):
    """Targets of 1e6 at a network that is zero: b3's gradient is the same in
    every step to 1e-7, so each Adam step moves b3 by lr.  The quotient of the
    corrected moments is some ten FP32 roundings (three per moment, a
    correction, two divisions, a root, the product and the update), 6e-8 each:
    1e-6 is above their sum."""
    n, lr = 16, 2.0 ** -10
    tr = F.Trainer(H, np.zeros((n, 4)), np.full(n, 1e6), np.zeros((n, 4)))
    tr.set_params({"W1": np.zeros((H, 4)), "b1": np.zeros(H), "W2": np.zeros((H, H)), "b2": np.zeros(H),
                   "w3": np.zeros(H), "b3": 0.0})
    for step in range(1, 9):
        tr.run(1, n, lr, wpsi=1.0, wgrad=0.0, seed=3)
        assert abs(tr.get_params()["b3"] / (step * lr) - 1.0) < 1e-6, step


def fibre_samples(n, seed):
    """Normalised fibre invariants max(I4 - 1, 0)^2, the two-fibre law's energy
    and its gradient: the data the surrogate is trained on."""
    rng = np.random.default_rng(seed)
    e = np.maximum(rng.normal(0.05, 0.08, (n, 2)), 0.0)
    z = e * e
    s = 1.0 / np.sqrt((z * z).mean())
    psi = (np.exp(z) - 1.0).sum(1)
    x, tg = np.zeros((n, 4)), np.zeros((n, 4))
    x[:, 2:] = z * s
    tg[:, 2:] = np.exp(z) / (s * psi.max())
    par = {"W1": 0.5 * rng.standard_normal((64, 4)), "b1": np.zeros(64), "W2": rng.standard_normal((64, 64)) / 8.0,
           "b2": np.zeros(64), "w3": rng.standard_normal(64) / 8.0, "b3": 0.0}
    f = lambda a: np.asarray(a, dtype=np.float32)
    return f(x), f(psi / psi.max()), f(tg), {k: f(v) for k, v in par.items()}


def run_fp64(x, ty, tg, par, steps, lr):
    """Full-batch Adam steps in FP64; the last step's loss."""
    import torch
    t = lambda a: torch.tensor(np.asarray(a, dtype=np.float64), device="cuda")
    x, ty, tg = t(x), t(ty), t(tg)
    P = {k: t(v).requires_grad_() for k, v in par.items()}
    m1, m2 = ({k: torch.zeros_like(v) for k, v in P.items()} for _ in range(2))
    lr, b1, b2 = (float(np.float32(v)) for v in (lr, 0.9, 0.999))
    for step in range(1, steps + 1):
        z1 = x @ P["W1"].T + P["b1"]
        z2 = torch.nn.functional.softplus(z1, threshold=1e9) @ P["W2"].T + P["b2"]
        y = torch.nn.functional.softplus(z2, threshold=1e9) @ P["w3"] + P["b3"]
        g = (((P["w3"] * torch.sigmoid(z2)) @ P["W2"]) * torch.sigmoid(z1)) @ P["W1"]
        loss = ((y - ty) ** 2).mean() + ((g - tg) ** 2).sum(1).mean()
        grads = torch.autograd.grad(loss, list(P.values()))
        with torch.no_grad():
            for (k, v), gr in zip(P.items(), grads):
                m1[k].mul_(b1).add_(gr, alpha=1.0 - b1)
                m2[k].mul_(b2).add_(gr * gr, alpha=1.0 - b2)
                v -= lr * (m1[k] / (1.0 - b1 ** step)) / ((m2[k] / (1.0 - b2 ** step)).sqrt() + 1e-8)
    return float(loss.detach())


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_loss_after_eight_steps(F, seed):
    """Every parameter's moves carry the same error of the corrections, so it
    adds up in the loss.  Eight steps with one FP32 rounding (1.2e-7) of a
    common factor each: 1e-6."""
    x, ty, tg, par = fibre_samples(65_536, seed)
    tr = F.Trainer(64, x, ty, tg)
    tr.set_params(par)
    loss = tr.run(8, 65_536, 3e-3, seed=seed)
    exact = run_fp64(x, ty, tg, par, 8, 3e-3)
    assert abs(loss - exact) <= 1e-6 * exact
