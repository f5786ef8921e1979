"""Weight gradients of all layers in one launch, or in groups of layers where their split partials exceed
the buffer: a large batch's gradient is the mean of its quarters' (quarters scale the loss gradient by a
power of two, so every BF16 value is the same and only the FP32 sums over splits differ)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,n_hidden,n", [(512, 8, 32768), (128, 1, 256), (256, 4, 8192)])
@pytest.mark.parametrize("gemm", [1, 0])
def test_gradient_of_a_batch_is_the_mean_of_its_quarters(hidden, n_hidden, n, gemm):
    import torch

    from pystarc_b200.surrogate import MLPEnsemble

    ens = MLPEnsemble(n_members=1, hidden=hidden, n_hidden=n_hidden, seed=3)
    ens.set_gemm(gemm)
    g = torch.Generator(device="cuda").manual_seed(4)
    X = torch.randn(n, 13, generator=g, device="cuda")
    T = torch.randn(n, 6, generator=g, device="cuda")
    loss, whole = ens.grad(0, X, T)
    q = n // 4
    parts = [ens.grad(0, X[i * q:(i + 1) * q], T[i * q:(i + 1) * q]) for i in range(4)]
    mean = sum(p[1].double() for p in parts) / 4
    # FP32 sums of at most 64 partials in two orders: 64 x 6e-8 of the terms' size, which cancel by up to 10
    err = float((whole.double() - mean).norm() / mean.norm())
    assert err < 4e-5, err
    assert np.isclose(loss, np.mean([p[0] for p in parts]), rtol=1e-5)
    ens.close()
