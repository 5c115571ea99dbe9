"""What lies between the two halves of the loss's gradient.

spe_loss_grad_cols leaves the column-transformed gradient, whole and
row-major, and spe_grad_rows finishes it with no engine memory of its own:
on an engine without a population, and for more items than the engine holds.
spe_loss_forward / spe_loss_backward keep theirs in the caller's buffers.  All
give spe_loss_grad's gradient bit for bit.  Supports as in
test_gpu_support_rows.py: empty, one pixel, tile edges, scattered, full,
values other than 0 and 1.

The half is compared with 64-bit arithmetic; its bound is that of the
gradient there (1e-5 of the norm: two transforms' rounding and that of the
loss term, without the last row transform)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from s_spi_spring_gb300 import _lib
from s_spi_spring_gb300.refine import farfield_loss
from test_gpu_support_rows import setup

pytestmark = pytest.mark.gpu
DEV = "cuda"
SIDES = [64, 100, 256, 384, 512, 768, 1024, 2048]


def bits(t):
    return torch.view_as_real(t).view(torch.int32)


def bind(e):
    e.set_stream(torch.cuda.current_stream().cuda_stream or 1)


@pytest.mark.parametrize("n", SIDES)
def test_halves(n):
    e, A, dens, S = setup(n)
    P = len(S)
    d, s = torch.tensor(dens, device=DEV), torch.tensor(S, device=DEV)
    scale = torch.tensor([1.0, 2.0, 0.5, 1.0, 0.0, 3.0], device=DEV)
    full, half, out = (torch.full_like(d, 7.0) for _ in range(3))
    loss = torch.empty(2, P, dtype=torch.float64, device=DEV)
    bind(e)
    e.loss_grad(d.data_ptr(), s.data_ptr(), P, 0, 0.0, loss[0].data_ptr(), full.data_ptr(), scale.data_ptr())
    for k in range(P):  # one item a call, into one buffer
        e.loss_grad_cols(d[k].data_ptr(), s[k].data_ptr(), 1, half[k].data_ptr(), 0, 0.0, loss[1, k].data_ptr())
    f = _lib.Engine(n, 0)
    f.set_amplitudes(A)
    bind(f)
    f.grad_rows(half.data_ptr(), s.data_ptr(), P, out.data_ptr(), scale.data_ptr())
    torch.cuda.synchronize()
    assert f.capacity == 0
    assert torch.equal(loss[0], loss[1]) and torch.equal(bits(out), bits(full))
    for k in range(P):
        F = np.fft.ifft2(np.where(S[k] > 0, dens[k].astype(complex), 0)) * n * n
        m = np.abs(F)
        g = np.where((A >= 0) & (m > 0), 2 * (m - A) / np.where(m > 0, m, 1), 0) * F
        want = np.fft.fft(g, axis=0)
        err = np.linalg.norm(half[k].cpu().numpy() - want)
        assert err <= 1e-5 * np.linalg.norm(want) + 1e-30, k
    # one more item than twice the capacity
    f.loss_grad_cols(d.data_ptr(), s.data_ptr(), 1, half.data_ptr(), 0, 0.0)
    assert f.capacity == 1
    f.grad_rows(half.data_ptr(), s.data_ptr(), 3, half.data_ptr(), scale.data_ptr())
    torch.cuda.synchronize()
    assert torch.equal(bits(half[:3]), bits(full[:3]))


@pytest.mark.parametrize("n", SIDES)
def test_kept(n):
    e, A, dens, S = setup(n, seed=8)
    P = len(S)
    d, s = torch.tensor(dens, device=DEV), torch.tensor(S, device=DEV)
    scale = torch.tensor([1.0, 2.0, 0.5, 1.0, 0.0, 3.0], device=DEV)
    kept, full = torch.full_like(d, 7.0), torch.empty_like(d)
    marks = torch.full((P * (n + 4),), 255, dtype=torch.uint8, device=DEV)
    raw = torch.full((P * n * n + 1,), 7.0, dtype=torch.complex64, device=DEV)
    apart = raw[1:].view(P, n, n)  # 8 bytes past a 16-byte boundary
    loss = torch.empty(2, P, dtype=torch.float64, device=DEV)
    bind(e)
    e.loss_grad(d.data_ptr(), s.data_ptr(), P, 1, 1e-3, loss[0].data_ptr(), full.data_ptr(), scale.data_ptr())
    e.loss_forward(d.data_ptr(), s.data_ptr(), P, kept.data_ptr(), marks.data_ptr(), 1, 1e-3, loss[1].data_ptr())
    e.loss_backward(kept.data_ptr(), marks.data_ptr(), s.data_ptr(), P, apart.data_ptr(), scale.data_ptr())
    e.loss_backward(kept.data_ptr(), marks.data_ptr(), s.data_ptr(), P, kept.data_ptr(), scale.data_ptr())
    torch.cuda.synchronize()
    assert torch.equal(loss[0], loss[1])
    assert torch.equal(bits(kept), bits(full)) and torch.equal(bits(apart), bits(full))
    for bad in ((0, marks.data_ptr()), (kept.data_ptr(), 0), (d.data_ptr(), marks.data_ptr()),
                (kept.data_ptr(), marks.data_ptr() + 1)):
        with pytest.raises(RuntimeError):
            e.loss_forward(d.data_ptr(), s.data_ptr(), P, *bad, 1, 1e-3)


@pytest.mark.parametrize("n", [100, 256, 1024])
def test_no_support_and_a_loss_without_bound(n):
    """The Poisson term at |F|^2 + eps = 0: its derivative is not finite, and
    0 times it is not a number, at every pixel of the individual without
    support and of no other."""
    e, A, dens, S = setup(n)
    d = torch.tensor(dens, device=DEV, requires_grad=True)
    s = torch.tensor(S, device=DEV)
    farfield_loss(d, s, e, "poisson", 0.0).sum().backward()
    full, half = torch.empty_like(d), torch.empty_like(d)
    e.loss_grad(d.data_ptr(), s.data_ptr(), len(S), 1, 0.0, 0, full.data_ptr())
    e.loss_grad_cols(d.data_ptr(), s.data_ptr(), len(S), half.data_ptr(), 1, 0.0)
    e.grad_rows(half.data_ptr(), s.data_ptr(), len(S), half.data_ptr())
    torch.cuda.synchronize()
    for g in (d.grad, full, half):
        assert torch.isnan(torch.view_as_real(g[0])).all()
        assert torch.isfinite(torch.view_as_real(g[1:])).all()
