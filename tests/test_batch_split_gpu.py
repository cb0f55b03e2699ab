"""A batch that fits is split once and keeps torch's cached memory."""
import numpy as np
import pytest
import torch

from oracle import dda_oracle as O

pytestmark = pytest.mark.gpu


def test_a_batch_that_fits_is_split_once(monkeypatch):
    from bl_krylov import bl_krylov as bk
    from mvp_fft import mvp_fft
    n, lf, k = (9, 8, 11), 0.03, 10.0
    rng = np.random.default_rng(0)
    address = np.sort(rng.choice(792, 500, replace=False))
    _, _, diag = O.polarizability(np.array([1.5 + 0.01j, 1.55 + 0.01j, 1.45 + 0.02j]), 1.33, lf, k, 500)
    til = mvp_fft.fft_init(n, 3, lf, k)
    B = rng.standard_normal((1500, 8)) + 1j * rng.standard_normal((1500, 8))
    splits, given, real = [], [], bk._batch_groups
    monkeypatch.setattr(bk, "_batch_groups", lambda *a: splits.append(1) or real(*a))
    monkeypatch.setattr(torch.cuda, "empty_cache", lambda: given.append(1))
    out = bk.bl_bicgstab_jacobi_mvp_fft_batch([(n, address, til, diag, B)] * 4, 1e-6, 40)
    assert len(splits) == 1 and not given and all(err < 1e-6 for _, _, err in out)
