"""Colours of degree 4, the widest rows, at the edges of a block of 128 rows."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 1000])
def test_colours_and_gradients(n):
    """Against 64 bits: 25 terms of at most about 12, each with five roundings,
    are 9e-5 apart at the very most."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gstex_cuda_gb300 as G
    g = torch.Generator().manual_seed(n)
    dirs, co, v = (torch.randn(*s, generator=g) for s in ((n, 3), (n, 25, 3), (n, 3)))
    want = oracle.sh_forward(4, 4, dirs.double().numpy(), co.double().numpy(), prec="f64")
    got = G.cuda.compute_sh_forward(n, 4, 4, dirs.to(DEV), co.to(DEV)).cpu().numpy()
    assert np.abs(got - want).max() <= 1e-4
    # the gradient is the basis times v, and the colours are linear in the basis
    basis = G.cuda.compute_sh_backward(n, 4, 4, dirs.to(DEV), v.to(DEV)).cpu().double() / v[:, None].double()
    assert float(((basis * co).sum(1) - torch.from_numpy(np.asarray(want))).abs().max()) <= 1e-4
