"""SH kernels that move coefficient rows through shared memory against the
kernels that read them in place (which serve fewer bases in use than stored):
the same operations, so the same bits, at the edges of a block of 128 rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000])
@pytest.mark.parametrize("deg", [1, 2, 3])
def test_rows_match_in_place(n, deg):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gstex_cuda_gb300 as G
    g = torch.Generator().manual_seed(n + deg)
    nb = (deg + 1) ** 2
    dirs = torch.randn(n, 3, generator=g).to(DEV)
    co = torch.randn(n, nb, 3, generator=g).to(DEV)
    wide = torch.zeros(n, 25, 3, device=DEV)
    wide[:, :nb] = co
    v = torch.randn(n, 3, generator=g).to(DEV)
    assert torch.equal(G.cuda.compute_sh_forward(n, deg, deg, dirs, co),
                       G.cuda.compute_sh_forward(n, 4, deg, dirs, wide))
    full = G.cuda.compute_sh_backward(n, 4, deg, dirs, v)
    assert torch.equal(G.cuda.compute_sh_backward(n, deg, deg, dirs, v), full[:, :nb])
    assert float(full[:, nb:].abs().sum()) == 0.0
