"""The network's kernels at the edges of their tiles: modes 2 to 32, axes that
are no multiple of the 16-row, 12-row and 32-cell tiles, sample counts around
the 16-sample tile, the most modes and the longest axis, against the float64 CPU oracle (features, output, loss,
every parameter's gradient)."""
import numpy as np
import pytest
import torch

from oracle import fno_oracle as F

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-30))


@pytest.mark.parametrize("n,L,modes,layers", [((2, 3, 2), 1, 2, 1), ((6, 9, 17), 16, 6, 3), ((12, 14, 33), 17, 12, 2),
                                              ((25, 13, 16), 2, 12, 1), ((15, 16, 49), 3, 14, 2),
                                              ((32, 32, 32), 1, 32, 1), ((4, 3, 512), 1, 2, 2)])
def test_shapes_against_the_oracle(n, L, modes, layers):
    """FP32 sums of at most a few thousand terms: the bounds of the other
    network test (features 1e-6, output and loss 1e-4, gradients 2e-3 of the
    block's largest entry)."""
    from bdda_b200.runtime import Occupancy, Plan
    from bdda_b200.warmstart import WarmStartFNO, chi_of
    rng = np.random.default_rng(sum(n) + L)
    ncell = int(np.prod(n))
    address = np.sort(rng.choice(ncell, max(1, int(0.6 * ncell)), replace=False))
    N = address.size
    diag = rng.uniform(2, 5, 3 * N) + 1j * rng.uniform(-1, 1, 3 * N)
    B = rng.standard_normal((3 * N, L)) + 1j * rng.standard_normal((3 * N, L))
    X = B / diag[:, None] * (1 + 0.3 * rng.standard_normal((3 * N, L)))
    eps = np.array([2.3 + 0.1j, 2.5 + 0.05j, 2.1 + 0.2j])
    cell_map = np.full(ncell, -1, np.int64)
    cell_map[address] = np.arange(N)
    model = WarmStartFNO(layers=layers, modes=modes, seed=3)
    g = torch.Generator(device="cpu").manual_seed(5)
    model.params.copy_((torch.randn(model.n_params, generator=g) * 0.15).to(model.device))
    d, b, x = (torch.as_tensor(v, device=model.device) for v in (diag, B, X))
    occ = Occupancy(Plan(n), address)
    loss_gpu = model.loss_and_grad(n, occ, d, b, eps, x)
    work = model._workspace(L, n)
    x_gpu = model.buffer(work, L, n, 0, L * ncell * 13).cpu().numpy().reshape(L, ncell, 13)
    y_gpu = model.buffer(work, L, n, 1, L * ncell * 6).cpu().numpy()
    x_ref, scale, J = F.features(cell_map, N, diag, B, chi_of(eps))
    assert _rel(x_gpu, x_ref) < 1e-6
    params = F.unflatten(model.params.cpu().numpy(), layers, modes)
    xt = torch.tensor(x_gpu.astype(np.float64).reshape((L,) + tuple(n) + (13,)))
    y = F.forward(params, xt, n, layers, modes)
    assert _rel(y_gpu.reshape(y.shape), y.detach().numpy()) < 1e-4
    t = F.target(cell_map, N, J, X, scale).reshape((L,) + tuple(n) + (6,))
    loss = F.loss(y, torch.tensor(t), torch.tensor((cell_map >= 0).reshape(n).astype(np.float64)))
    assert abs(loss_gpu - loss.item()) < 1e-4 * loss.item()
    loss.backward()
    g_gpu, off = model.grads.cpu().numpy(), 0
    for name, shape in F.param_layout(layers, modes):
        k = int(np.prod(shape))
        assert _rel(g_gpu[off:off + k], params[name].grad.numpy().ravel()) < 2e-3, name
        off += k
    # inference leaves the same output and the warm start adds it to the Jacobi guess
    X0 = model.predict(n, occ, d, b, eps).cpu().numpy()
    yo = y_gpu.reshape(L, ncell, 6)[:, address, :]
    corr = (yo[..., 0::2] + 1j * yo[..., 1::2]).transpose(1, 2, 0).reshape(3 * N, L)
    assert _rel(X0, J + corr * scale[None, :]) < 1e-6
