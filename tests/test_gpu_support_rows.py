"""The loss passes skip the row tiles without support: supports that are
empty, one pixel in a corner, rows at the tile edges, scattered over the
field, full, and with values other than 0 and 1 (only > 0 counts), each in
its own individual of one call.

The gradient is compared with 64-bit arithmetic: transforms of 2 log2 n
radix-2 stages round to about 2 log2(n) 2^-24 of the norm twice (1.3e-6 at
2048), the loss term's derivative adds |F| - A, which the random densities
here keep at the size of |F|: 1e-5 of the norm."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import spring_oracle as o
from s_spi_spring_gb300 import _lib, synthetic
from s_spi_spring_gb300.refine import FarFieldLoss, population_tensors, refine

pytestmark = pytest.mark.gpu
DEV = "cuda"


def setup(n, seed=3):
    rng = np.random.default_rng(seed)
    I, _, _ = synthetic.polygon_pattern(seed=seed, n=n, diameter=n * 0.23, photons=1e7, stop_radius=max(1, n // 64))
    A = _lib.prepare_pattern(I, (-1, -1), True)
    S = np.zeros((6, n, n), np.int32)
    S[1, n - 1, 0] = 1
    S[2, [0, 3, 4, n // 2, n - 4], :] = 1
    S[3] = rng.integers(0, 60, (n, n)) == 0
    S[4] = 1
    S[5, n // 3:n // 2, n // 4:n // 2] = rng.integers(-2, 4, (n // 2 - n // 3, n // 2 - n // 4))
    dens = (rng.standard_normal(S.shape) + 1j * rng.standard_normal(S.shape)).astype(np.complex64)
    dens[4] *= np.float32(np.sqrt((A[A > 0] ** 2).mean()) / n)
    e = _lib.Engine(n, 0)
    e.set_amplitudes(A)
    return e, A, dens, S


@pytest.mark.parametrize("n", [64, 100, 256, 384, 512, 768, 1024, 2048])
def test_gradient_through_any_support(n):
    e, A, dens, S = setup(n)
    d = torch.tensor(dens, device=DEV, requires_grad=True)
    L = FarFieldLoss.apply(d, torch.tensor(S, device=DEV), e, "amplitude", 0.0)
    w = torch.tensor([1.0, 2.0, 0.5, 1.0, 1.0, 3.0], device=DEV, dtype=torch.float64)
    (L * w).sum().backward()
    got, loss = d.grad.cpu().numpy(), L.detach().cpu().numpy()
    for i in range(len(S)):
        rl, rg = o.farfield_loss_grad(dens[i].astype(complex), (S[i] > 0).astype(int), A, "amplitude", 0.0)
        assert abs(loss[i] - rl) <= 1e-5 * rl, i
        assert np.all(got[i][S[i] <= 0] == 0), i
        norm = np.linalg.norm(rg)
        assert np.linalg.norm(got[i] - float(w[i]) * rg) <= 1e-5 * float(w[i]) * norm, i


@pytest.mark.parametrize("n", [256, 1024])
def test_not_finite_reaches_every_pixel(n):
    """As 0 times NaN did in the dense passes, and only in its own item."""
    e, A, dens, S = setup(n)
    dens[5, n // 3:n // 2, n // 4:n // 2] = np.nan
    d = torch.tensor(dens, device=DEV, requires_grad=True)
    L = FarFieldLoss.apply(d, torch.tensor(S, device=DEV), e, "poisson", 1e-3)
    L.sum().backward()
    assert np.isnan(L.detach().cpu().numpy()[5])
    assert torch.isnan(d.grad[5].real).all()
    assert torch.isfinite(torch.view_as_real(d.grad[:5])).all()


@pytest.mark.parametrize("n", [64, 100, 256, 384, 512, 768, 1024, 2048])
def test_run_equals_single_steps(n):
    """spe_adam_run from uninitialised moments against spe_adam_step from
    zeroed ones: the same bits, and nothing written outside the support."""
    e, A, dens, S = setup(n)
    P, steps = len(S), 4
    e.upload(0, dens, S)
    losses = refine(e, 0, P, steps=steps, lr=1e-2, loss="amplitude", device=torch.device(DEV, 0))
    got, _ = e.download(0, P)
    d, s = torch.tensor(dens, device=DEV), torch.tensor(S, device=DEV)
    m, v = torch.zeros_like(d), torch.zeros_like(d)
    one = torch.empty(steps, P, dtype=torch.float64, device=DEV)
    torch.cuda.synchronize()
    for t in range(steps):
        e.adam_step(d.data_ptr(), s.data_ptr(), m.data_ptr(), v.data_ptr(), P, _lib.SPE_LOSS_AMPLITUDE, 1e-6, 1e-2,
                    step=t + 1, loss_ptr=one[t].data_ptr())
    e.synchronize()
    assert losses == one.sum(dim=1).tolist()
    assert np.array_equal(got.view(np.uint32), d.cpu().numpy().view(np.uint32))
    assert np.array_equal(got[S <= 0].view(np.uint32), dens[S <= 0].view(np.uint32))
    # steps with moments outside the support: they decay, the density moves
    m.fill_(1.0)
    v.fill_(1.0 + 1.0j)
    before = d.clone()
    e.adam_step(d.data_ptr(), s.data_ptr(), m.data_ptr(), v.data_ptr(), P, _lib.SPE_LOSS_AMPLITUDE, 1e-6, 1e-2, step=1)
    e.synchronize()
    out = s <= 0
    assert torch.allclose(m[out].real, torch.tensor(0.9, device=DEV), rtol=1e-6)
    step = 1e-2 / (1 - 0.9) * 0.9 / (np.sqrt(0.999) / np.sqrt(1 - 0.999) + 1e-8)
    # |density| < 8, so its float step of 2^-22 bounds the rounding
    assert torch.allclose((before - d)[out].real, torch.tensor(step, device=DEV, dtype=torch.float32), rtol=1e-5,
                          atol=5e-7)
