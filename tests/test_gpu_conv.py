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
# (grids of more than 5000 cells: smaller ones are summed in one launch)
DIMS = ([(n, 5001 // (3 * n) + 1, 3) for n in SIDES] + [(5001 // (2 * n) + 1, n, 2) for n in SIDES] +
        [(71, 71, 1), (51, 50, 2)] + [(41, 5000 // (41 * z) + 1, z) for z in range(3, 9)] +
        [(2048, 3, 1), (3, 2048, 1)])


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
    for X, Y in ((24, 20), (60, 50)):  # in one launch, and as a convolution
        rho = torch.ones((3, Y, X), device="cuda")
        rho[1, 5, 7] = value
        phi = torch.zeros_like(rho)
        with mmsb200.Context(mmsb200.Grid(X, Y, 3, 5e-9, 5e-9, 5e-9)) as ctx:
            ctx.potential_dev(rho, phi)
            ctx.sync()
        assert not torch.isfinite(phi).any()


SMALL = [(1, 1, 1), (1, 1, 7), (2, 1, 1), (3, 2, 1), (4, 5, 3), (5, 4, 3), (7, 9, 2), (16, 16, 3), (17, 20, 3),
         (31, 11, 3), (341, 1, 3), (1, 341, 3), (342, 1, 3), (33, 50, 3), (100, 1, 50), (5, 100, 5), (4999, 1, 1),
         (2, 512, 1), (2, 513, 1), (40, 41, 3)]


@pytest.mark.parametrize("dims", SMALL)
def test_small_grids_in_one_launch(cuda, lib, oracle_mod, dims):
    """Potential, field and one RK4 step of grids around the one-launch sum's
    limits (1024 and 5000 cells, 512 rows, 2048 wide), ragged widths.  The
    direct sum's tolerance (FP32 table, FP32 row sums): phi rel-L2 2e-6; the
    charge has the divergence kernel's bits; the step 1e-4 deg."""
    import mmsb200
    from conftest import max_angle_deg
    torch = cuda
    X, Y, Z = dims
    d = (5e-9, 4e-9, 6e-9)
    og = oracle_mod.Grid(X, Y, Z, *d)
    rng = np.random.default_rng(X + 37 * Y + 1009 * Z)
    v = rng.standard_normal((Z, Y, X, 3))
    M = v / np.linalg.norm(v, axis=-1, keepdims=True) * 8.6e5
    Mf = torch.from_numpy(M.astype(np.float32)).cuda()
    if X > 2048:
        with pytest.raises(mmsb200.MmsError):
            mmsb200.Context(mmsb200.Grid(X, Y, Z, *d))
        return
    with mmsb200.Context(mmsb200.Grid(X, Y, Z, *d)) as ctx:
        rho = torch.empty((Z, Y, X), device="cuda")
        q, phi = torch.full_like(rho, float("nan")), torch.full_like(rho, float("nan"))
        H = torch.empty((Z, Y, X, 3), device="cuda")
        ctx.divergence_dev(Mf, rho)
        ctx.hfield_dev(Mf, H, q, phi)
        phi2 = torch.full_like(rho, float("nan"))
        ctx.potential_dev(rho, phi2)
        ctx.state_set(np.ones((Z, Y, X), np.uint8), M)
        ctx.run_fixed(1e-13, 1)
        M1, _ = ctx.state_get()
    assert torch.equal(q, rho) and torch.equal(phi, phi2)
    ref = oracle_mod.potential_direct(og, rho.cpu().numpy().astype(np.float64))
    assert np.linalg.norm(phi.cpu().numpy() - ref) <= 2e-6 * np.linalg.norm(ref)
    Mo = oracle_mod.rk4_run(og, oracle_mod.Params(), np.ones((Z, Y, X), np.uint8), M, 1e-13, 1)
    assert max_angle_deg(M1, Mo) < 1e-4


# the column CTAs hold all layers of a column in 200 KB of shared memory: on both
# sides of that limit, the second of each pair takes the pair sum
@pytest.mark.parametrize("dims,conv", [((3, 1024, 3), True), ((3, 1025, 3), False), ((3, 768, 6), True),
                                       ((3, 769, 6), False), ((3, 512, 8), True), ((3, 513, 8), False),
                                       ((1025, 3, 3), True), ((71, 9, 8), True), ((71, 8, 9), False)])
def test_grids_at_the_column_limit(cuda, lib, oracle_mod, dims, conv):
    """the convolution's tolerance where it serves, else the pair sum's (2e-6)"""
    import mmsb200
    torch = cuda
    d = (5e-9, 4e-9, 6e-9)
    X, Y, Z = dims
    rho_h = (np.random.default_rng(X + 31 * Y + Z).standard_normal((Z, Y, X)) * 1e14).astype(np.float32)
    rho = torch.from_numpy(rho_h).cuda()
    phi = torch.full_like(rho, float("nan"))
    with mmsb200.Context(mmsb200.Grid(X, Y, Z, *d)) as ctx:
        ctx.potential_dev(rho, phi)
        ctx.sync()
        before = ctx.kernel_launches
        ctx.potential_dev(rho, phi)
        assert ctx.kernel_launches - before == (3 if conv else 1)
        ctx.sync()
    ref = oracle_mod.potential_direct(oracle_mod.Grid(X, Y, Z, *d), rho_h.astype(np.float64))
    assert rel_l2(phi.cpu().numpy(), ref) <= (6.1e-8 if conv else 2e-6)
