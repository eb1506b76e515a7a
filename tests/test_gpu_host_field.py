"""mms_hfield_host on pageable, pinned and missing arrays, on both sides of the
staged size (32,768 cells): the bits of mms_hfield_dev."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (16, 16, 3), (128, 128, 2), (105, 105, 3)])
@pytest.mark.parametrize("solver", [(0, 4), (1, 3)])
def test_host_field_keeps_the_bits(cuda, lib, dims, solver):
    import mmsb200
    torch = cuda
    X, Y, Z = dims
    if solver[0] and X < 16:
        pytest.skip("no tree")
    with mmsb200.Context(mmsb200.Grid(X, Y, Z, 5e-9, 4e-9, 6e-9), mmsb200.make_params(external=True),
                         mmsb200.make_solver(*solver)) as ctx:
        M = torch.randn(Z, Y, X, 3, generator=torch.Generator().manual_seed(X))
        Md = M.cuda()
        H, q, phi = torch.empty_like(Md), torch.empty(dims[::-1], device="cuda"), torch.empty(dims[::-1], device="cuda")
        torch.cuda.synchronize()
        ctx.hfield_dev(Md, H, q, phi, 1e-10)
        ctx.sync()
        ref = [a.cpu().numpy() for a in (H, q, phi)]
        for pin in (False, True, None):  # None: M pinned alone
            new = lambda shape, p: torch.zeros(shape, pin_memory=bool(p))  # noqa: E731
            m = M.pin_memory() if pin is not False else M
            out = [new(a.shape, pin) for a in ref]
            mmsb200._check(lib.mms_hfield_host(ctx.h, m.data_ptr(), *[o.data_ptr() for o in out], 1e-10))
            for o, a in zip(out, ref):
                assert np.array_equal(o.numpy(), a)
        h = torch.zeros(ref[0].shape)
        mmsb200._check(lib.mms_hfield_host(ctx.h, M.data_ptr(), h.data_ptr(), None, None, 1e-10))
        assert np.array_equal(h.numpy(), ref[0])
