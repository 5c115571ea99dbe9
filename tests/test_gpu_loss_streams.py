"""An error-reduction call on the engine's own stream and, while it runs, the
far-field loss of tensors of the user's own on torch's stream: both give what
they give alone, bit for bit (they share no array of the engine)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from s_spi_spring_gb300 import _lib, synthetic
from s_spi_spring_gb300.refine import farfield_loss

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,P", [(256, 64), (512, 24), (1024, 8), (100, 64)])
def test_loss_beside_er(n, P):
    I, _, _ = synthetic.polygon_pattern(seed=4, n=n, diameter=n * 0.23, photons=1e9, stop_radius=2)
    dens, S = synthetic.start_population(n, 2, n * 0.25, seed=5)
    dens, S = np.concatenate([dens] * (P // 2)), np.concatenate([S] * (P // 2))
    e = _lib.Engine(n, 0)
    e.set_amplitudes(_lib.prepare_pattern(I, (-1, -1), True))
    e.reserve(P)
    rho = torch.tensor(np.roll(dens, n // 2, axis=1), device="cuda", requires_grad=True)  # other rows
    supp = torch.tensor(np.roll(S, n // 2, axis=1), device="cuda")

    def er():
        e.set_stream(0)
        e.er(0, P, 30, 0.0)

    def loss():
        rho.grad = None
        L = farfield_loss(rho, supp, e, "poisson", 1e-3)
        L.sum().backward()
        return L.detach(), rho.grad

    e.upload(0, dens, S)
    er()
    want_d, _ = e.download(0, P)
    want_l, want_g = (t.clone() for t in loss())
    torch.cuda.synchronize()
    for _ in range(5):
        e.set_stream(0)
        e.upload(0, dens, S)
        er()
        for _ in range(4):
            got_l, got_g = loss()
        torch.cuda.synchronize()
        e.set_stream(0)
        got_d, _ = e.download(0, P)
        assert np.array_equal(got_d.view(np.uint32), want_d.view(np.uint32))
        assert torch.equal(got_l, want_l) and torch.equal(torch.view_as_real(got_g), torch.view_as_real(want_g))
