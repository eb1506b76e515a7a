"""The FMM kernels of large grids (k_l2p_wide, 32-target M2L items) against the
forms of small ones: the fused far field ends in k_l2p, the tensor-core M2L
replaces the resident one.

Tolerances: either form is held to 2e-5 of the FP64 restatement, so the two are
within 4e-5 of each other; the split-BF16 M2L adds its 3.3e-5.
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

# whole and ragged boxes, an odd number of box rows, 1 to 4 layers, both leaf sides
DIMS = [(512, 496, 3, 4, 8), (509, 517, 1, 3, 4), (700, 300, 2, 2, 8), (1101, 262, 3, 4, 4), (352, 352, 4, 1, 8),
        (513, 512, 3, 5, 8)]


@pytest.mark.parametrize("X,Y,Z,P,s", DIMS)
def test_large_grid_kernels_match(cuda, lib, X, Y, Z, P, s):
    import mmsb200
    torch = cuda
    rho = torch.randn(Z, Y, X, device="cuda", generator=torch.Generator("cuda").manual_seed(X))
    out = []
    for kw in (dict(), dict(far_mode=mmsb200.FAR_FUSED) if P <= 4 else dict(m2l_mode=mmsb200.M2L_TENSOR)):
        with mmsb200.Context(mmsb200.Grid(X, Y, Z, 5e-9, 4e-9, 6e-9), mmsb200.make_params(),
                             mmsb200.make_solver(mmsb200.SOLVER_FMM, P, s, **kw)) as ctx:
            phi = torch.empty_like(rho)
            ctx.potential_dev(rho, phi)
            ctx.sync()
            out.append(phi.double().cpu().numpy())
    assert np.isfinite(out[0]).all()
    assert rel_l2(out[0], out[1]) < (4e-5 if P <= 4 else 7.3e-5)
