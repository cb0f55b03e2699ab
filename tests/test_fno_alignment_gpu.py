"""Network parameters that start on an 8-byte boundary (a slice of a larger
array): complex weights are read in pairs only where the boundary is 16 bytes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("modes", [4, 12])
def test_parameters_and_gradients_on_an_8_byte_boundary(modes):
    """The same values at both boundaries.  Output bit for bit; gradients to the
    order of their float32 sums over the 468 z lines of the batch (a warp each),
    whose terms' magnitudes add up to a few times the largest entry: 468 x 6e-8 x 4."""
    from bdda_b200 import runtime, warmstart
    n, L = (13, 12, 14), 3
    rng = np.random.default_rng(5)
    address = np.sort(rng.choice(int(np.prod(n)), int(0.6 * np.prod(n)), replace=False))
    rows = 3 * address.size
    cplx = lambda *s: torch.from_numpy(rng.standard_normal(s) + 1j * rng.standard_normal(s)).cuda()
    diag, B, X, er = cplx(rows) + 4.0, cplx(rows, L), cplx(rows, L), np.array([2.1 + 0.1j, 2.2, 2.0])
    occ = runtime.Occupancy(runtime.Plan(n), address)
    out = []
    for at in (0, 2):
        m = warmstart.WarmStartFNO(layers=2, modes=modes, seed=3)
        params, grads = (torch.zeros(m.n_params + 4, device="cuda") for _ in range(2))
        params[at:at + m.n_params] = m.params
        m.params, m.grads = params[at:at + m.n_params], grads[at:at + m.n_params]
        assert m.params.data_ptr() % 16 == 4 * at
        y = m.predict(n, occ, diag, B, er).clone()
        loss = m.loss_and_grad(n, occ, diag, B, er, X)
        out.append((y, loss, m.grads.clone(), float(grads[:at].abs().sum() + grads[at + m.n_params:].abs().sum())))
    (y, loss, g, _), (y8, loss8, g8, outside) = out
    assert torch.equal(y, y8) and abs(loss8 - loss) <= 1e-12 * loss and outside == 0.0
    assert float((g8 - g).abs().max()) <= 1e-4 * float(g.abs().max())
