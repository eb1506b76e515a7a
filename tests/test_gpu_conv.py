"""GPU parity of the exact potential's convolution against the FP64 pair sum of
the oracle, at the sizes where its plans, groups and layouts change.

Tolerance: the convolution runs in FP64 and rounds phi to FP32 once, so each
value is within 2^-24 of the FP64 sum of the same charges and so is the
relative L2 norm; 6.1e-8 = 1.02 * 2^-24 leaves room for the FP64 rounding.
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

# both sides of every transform length's last cell count (2 X - 1 <= n: 8 | 9,
# 16 | 17, 24 | 25, ...) along x and along y, odd rows (a lone last row), every
# number of layers, ragged pairs per CTA
SIDES = (8, 9, 16, 17, 24, 25, 32, 33, 40, 41, 48, 49, 64, 65, 80, 81, 96, 97, 128, 129, 160, 161, 192, 193, 256, 257,
         320, 321, 384, 385, 512, 513, 768, 769, 1024, 1025)
DIMS = ([(n, 300 // n + 3, 3) for n in SIDES] + [(300 // n + 3, n, 2) for n in SIDES] +
        [(19, 14, z) for z in range(1, 9)] + [(2048, 1, 1), (1, 2048, 1), (86, 3, 1), (3, 86, 1)])


@pytest.mark.parametrize("dims", DIMS)
def test_convolution_matches_the_fp64_sum(cuda, lib, oracle_mod, dims):
    import mmsb200
    torch = cuda
    d = (5e-9, 4e-9, 6e-9)
    X, Y, Z = dims
    rho_h = (np.random.default_rng(X * 7919 + Y * 31 + Z).standard_normal((Z, Y, X)) * 1e14).astype(np.float32)
    rho = torch.from_numpy(rho_h).cuda()
    phi = torch.full_like(rho, float("nan"))
    with mmsb200.Context(mmsb200.Grid(X, Y, Z, *d), mmsb200.make_params(),
                         mmsb200.make_solver(mmsb200.SOLVER_DIRECT)) as ctx:
        ctx.potential_dev(rho, phi)
        first = phi.clone()
        ctx.potential_dev(rho, phi)  # the column store is reused
        ctx.sync()
    assert torch.equal(first, phi)
    ref = oracle_mod.potential_direct(oracle_mod.Grid(X, Y, Z, *d), rho_h.astype(np.float64))
    assert rel_l2(phi.cpu().numpy(), ref) <= 6.1e-8


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_convolution_spreads_a_non_finite_charge(cuda, lib, value):
    """as in the pair sum, a charge that is not finite leaves no finite potential"""
    import mmsb200
    torch = cuda
    rho = torch.ones((3, 20, 24), device="cuda")
    rho[1, 5, 7] = value
    phi = torch.zeros_like(rho)
    with mmsb200.Context(mmsb200.Grid(24, 20, 3, 5e-9, 5e-9, 5e-9)) as ctx:
        ctx.potential_dev(rho, phi)
        ctx.sync()
    assert not torch.isfinite(phi).any()
