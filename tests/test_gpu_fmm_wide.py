"""The FMM's wide leaf kernels (k_p2m_wide, k_l2p_wide; grids of 240 columns of
32 x 16 cells or more) against the kernels of small grids, the exact sum, and
stepped.

Charges that fill one box of level l alone have, inside it, the same tree, lists
and operators as a grid of that box's size: a small context, which runs k_p2m_row
and k_l2p, gives the same potential to rounding, at any order (no truncation
between the two).  Tolerance: either is held to 2e-5 of the FP64 restatement,
4e-5 together; the split-BF16 M2L (P >= 8, and P >= 6 at leaf side 4) adds
3.3e-5 to each side.
"""
import numpy as np
import pytest

from conftest import max_angle_deg, rel_l2

pytestmark = pytest.mark.gpu

# order, leaf side, layers; weights staged and read as they go (C NR beyond 10,240),
# expansions above and below 32, the row P2M beside the wide L2P (NR > 32 and C > 256),
# both near fields, extra warps for the locals of few layers, up to 16 layers
DIMS = [(512, 496, 3, 4, 8), (509, 517, 1, 3, 4), (512, 256, 3, 6, 8), (400, 400, 2, 8, 4), (352, 352, 3, 9, 8),
        (352, 352, 4, 5, 8), (352, 352, 6, 5, 8), (352, 352, 8, 4, 8), (349, 363, 16, 2, 8), (352, 352, 16, 4, 4),
        (512, 320, 1, 1, 8), (357, 352, 3, 7, 4), (512, 250, 5, 3, 4), (256, 500, 2, 8, 8), (400, 390, 1, 5, 4)]


def _ctx(X, Y, Z, P, s, **kw):
    import mmsb200
    return mmsb200.Context(mmsb200.Grid(X, Y, Z, 5e-9, 5e-9, 5e-9), mmsb200.make_params(),
                           mmsb200.make_solver(mmsb200.SOLVER_FMM, P, s, **kw))


@pytest.mark.parametrize("X,Y,Z,P,s", DIMS)
def test_wide_kernels_match_small_grids_box_by_box(cuda, lib, X, Y, Z, P, s):
    torch = cuda
    assert -(-X // 32) * -(-Y // 16) >= 240
    rho = torch.randn(Z, Y, X, device="cuda", generator=torch.Generator("cuda").manual_seed(X + P))
    part, phi = torch.zeros_like(rho), torch.empty_like(rho)
    side = 16 * s  # 16 x 16 leaf boxes: levels 2 .. 4 of its own
    tc = P >= 8 or (P >= 6 and s <= 4)
    tol = 4e-5 + (6.6e-5 if tc else 0.0)
    with _ctx(X, Y, Z, P, s) as ctx:
        xs, ys = (sorted({0, n // side // 2 * side, (n - 1) // side * side}) for n in (X, Y))
        for y0 in ys:
            for x0 in xs:
                h, w = min(side, Y - y0), min(side, X - x0)
                if max(h, w) <= 8 * s:  # (a smaller tree)
                    continue
                at = (slice(None), slice(y0, y0 + h), slice(x0, x0 + w))
                part.zero_()
                part[at] = rho[at]
                ctx.potential_dev(part, phi)
                ctx.sync()
                small_rho = rho[at].contiguous()
                small = torch.full_like(small_rho, float("nan"))
                with _ctx(w, h, Z, P, s) as c2:
                    c2.potential_dev(small_rho, small)
                    c2.sync()
                assert rel_l2(phi[at].cpu().numpy(), small.cpu().numpy()) < tol, (x0, y0)


# Error against the exact sum of the films below with the row kernels (k_p2m_row and
# k_l2p at these sizes, measured with them before the wide ones were there): truncation
# all but alone
ROW_KERNELS = {(512, 496, 3, 4, 8): 1.10503e-03, (509, 517, 1, 3, 4): 3.93478e-03, (512, 256, 3, 6, 8): 1.13114e-04,
               (400, 400, 2, 8, 4): 1.08643e-05, (352, 352, 3, 9, 8): 1.47816e-05, (352, 352, 4, 5, 8): 3.79093e-04,
               (512, 320, 1, 1, 8): 4.03738e-02, (357, 352, 3, 7, 4): 4.77326e-05, (256, 500, 2, 8, 8): 1.27083e-05,
               (400, 390, 1, 5, 4): 3.54661e-04}


@pytest.mark.parametrize("dims", list(ROW_KERNELS))
def test_wide_kernels_against_the_exact_sum(cuda, lib, dims):
    """within 0.1 % of the row kernels' error: another order of the FP32 sums
    changes it by less, the least accurate thing left out by far more"""
    import mmsb200
    X, Y, Z, P, s = dims
    torch = cuda
    M = torch.randn(Z, Y, X, 3, device="cuda", generator=torch.Generator("cuda").manual_seed(Y + P))
    M *= 8.6e5 / M.norm(dim=-1, keepdim=True)
    if Z >= 3:
        M[0] = 0
        M[-1] = 0
    rho = torch.empty(Z, Y, X, device="cuda")
    phi, ref = torch.empty_like(rho), torch.empty_like(rho)
    with _ctx(X, Y, Z, P, s) as ctx, mmsb200.Context(mmsb200.Grid(X, Y, Z, 5e-9, 5e-9, 5e-9)) as exact:
        ctx.divergence_dev(M, rho)
        ctx.potential_dev(rho, phi)
        ctx.sync()
        exact.potential_dev(rho, ref)
        exact.sync()
    assert rel_l2(phi.cpu().numpy(), ref.cpu().numpy()) <= 1.001 * ROW_KERNELS[dims]


@pytest.mark.parametrize("X,Y,Z,s", [(1024, 1024, 3, 8), (1024, 512, 2, 4)])
def test_wide_sums_are_no_less_exact_than_those_of_small_grids(cuda, lib, X, Y, Z, s):
    """The same boxes' potentials at P = 9 against the exact sum: both sides have
    the same truncation e and M2L, and rounding errors of some 2^-23 = 1.2e-7 of
    the potential.  Of N cells, the squares of the two relative errors differ by
    the difference of the rounding's squares and, by chance, by 2 e 1.2e-7 /
    sqrt(N); bound: three times that."""
    import mmsb200
    torch = cuda
    side = 16 * s
    rho = torch.randn(Z, Y, X, device="cuda", generator=torch.Generator("cuda").manual_seed(X + s))
    part, phi = torch.zeros_like(rho), torch.empty_like(rho)
    wide = small = norm = 0.0
    kw = dict(m2l_mode=mmsb200.M2L_SIMT)
    with _ctx(X, Y, Z, 9, s, **kw) as ctx, _ctx(side, side, Z, 9, s, **kw) as c2, \
            mmsb200.Context(mmsb200.Grid(side, side, Z, 5e-9, 5e-9, 5e-9)) as exact:
        for y0 in range(0, Y, side):
            for x0 in range(0, X, side):
                at = (slice(None), slice(y0, y0 + side), slice(x0, x0 + side))
                part.zero_()
                part[at] = rho[at]
                q = rho[at].contiguous()
                ps, ref = torch.empty_like(q), torch.empty_like(q)
                for c, r, p in ((ctx, part, phi), (c2, q, ps), (exact, q, ref)):
                    c.potential_dev(r, p)
                    c.sync()
                ref = ref.double()
                wide += float(((phi[at].double() - ref) ** 2).sum())
                small += float(((ps.double() - ref) ** 2).sum())
                norm += float((ref ** 2).sum())
    chance = 2 * (small / norm) ** 0.5 * 2.0 ** -23 / (X * Y * Z) ** 0.5
    print(f"P = 9, leaf {s}: wide {(wide / norm) ** 0.5:.4e}, small {(small / norm) ** 0.5:.4e}, squares differ by "
          f"{(wide - small) / norm / chance:.2f} of the chance")
    assert (wide - small) / norm <= 3 * chance


STEPS = [(512, 496, 3, 4, 8), (509, 517, 1, 3, 4), (352, 352, 4, 5, 8), (352, 352, 8, 4, 8), (352, 352, 6, 5, 8),
         (700, 300, 2, 2, 4), (400, 390, 2, 5, 4)]


@pytest.mark.parametrize("X,Y,Z,P,s", STEPS)
def test_wide_grids_step_with_the_divergence_formed_on_the_way(cuda, lib, X, Y, Z, P, s):
    """Steps form the charges, store them and write their BF16 split in the wide
    P2M; the fused far field and the tensor-core M2L step with a divergence
    kernel of its own.  Bound: the two potentials are within 7.3e-5; a cell's
    demag field, up to 1e7 A/m in a random state, turns M by gamma dt H = 0.4 rad
    in two steps of 1e-13 s, so by 3e-5 rad = 1.7e-3 deg between the two.  (A
    stale charge or split turns it by degrees.)"""
    import mmsb200
    rng = np.random.default_rng(X + Z)
    mat = np.repeat(np.repeat(rng.random((Z, -(-Y // 4), -(-X // 4))) < 0.7, 4, 1), 4, 2)[:, :Y, :X].astype(np.uint8)
    M = rng.standard_normal((Z, Y, X, 3))
    M *= 8.6e5 / np.linalg.norm(M, axis=-1, keepdims=True) * mat[..., None]
    out = []
    for kw in (dict(), dict(far_mode=mmsb200.FAR_FUSED) if P <= 4 else dict(m2l_mode=mmsb200.M2L_TENSOR)):
        with _ctx(X, Y, Z, P, s, **kw) as ctx:
            ctx.state_set(mat, M)
            ctx.run_fixed(1e-13, 2)
            out.append(ctx.state_get()[0])
    assert max_angle_deg(out[0], M, mat) > 0.1
    assert max_angle_deg(out[0], out[1], mat) < 1.7e-3
