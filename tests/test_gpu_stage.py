"""The RK4 stages' external field: a stage reads H_ext from the slot that the
stage before it, a new state, a restored time or new parameters filled.

Every way to the same state and time gives the same bits, so no tolerance.
Sizes on both sides of the eager loads' limit (75,776 cells), and no whole CTA.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

T1 = dict(hext_t=[0.0, 2.5e-13, 4e-13, 1e-12], hext_b=[[-0.05, 0.0, 0.01], [0.05, 0.02, 0.0], [0.3, 0.0, 0.0], [0, 0, 0]])
T2 = dict(hext_t=[1e-13], hext_b=[[0.0, 0.4, 0.0]])


@pytest.mark.parametrize("dims", [(1, 1, 1), (17, 15, 3), (148, 256, 2), (149, 256, 2)])
@pytest.mark.parametrize("ref_time", [False, True])
def test_stage_fields_by_every_way(cuda, lib, dims, ref_time):
    import mmsb200
    X, Y, Z = dims
    rng = np.random.default_rng(X)
    mat = (rng.random((Z, Y, X)) < 0.7).astype(np.uint8)
    mat.flat[0] = 1
    M = rng.normal(size=(Z, Y, X, 3))
    M *= 8.6e5 / np.linalg.norm(M, axis=-1, keepdims=True) * mat[..., None]

    def context(tab):
        return mmsb200.Context(mmsb200.Grid(X, Y, Z, 5e-9, 5e-9, 5e-9),
                               mmsb200.make_params(external=True, ref_stage_time=ref_time, **tab),
                               mmsb200.make_solver(mmsb200.SOLVER_DIRECT))

    def plain(tab, m, t, n):
        """n steps without the graph, from a new state before each step"""
        for _ in range(n):
            c = context(tab)
            c.state_set(mat, m, t)
            c.run_fixed(1e-13, 1, use_graph=False)
            m, t = c.state_get()
            c.close()
        return m, t

    c = context(T1)
    c.state_set(mat, M)
    c.run_fixed(1e-13, 5)
    a, t = c.state_get()
    if not ref_time:  # (there a step's first stage is at the time before the step before it)
        b, tb = plain(T1, M, 0.0, 5)
        assert t == tb and np.array_equal(a, b)
    # new parameters in mid-run, then back; against a new context's state
    c.set_params(mmsb200.make_params(external=True, ref_stage_time=ref_time, **T2))
    c.run_fixed(1e-13, 1)
    a2, t2 = c.state_get()
    b2, _ = plain(T2, a, t, 1)  # one field at all times
    assert np.array_equal(a2, b2)
    c.state_set(mat, a2, t2)
    c.set_params(mmsb200.make_params(external=True, ref_stage_time=ref_time, **T1))
    c.run_fixed(1e-13, 1)
    a3, _ = c.state_get()
    b3, _ = plain(T1, a2, t2, 1)
    assert np.array_equal(a3, b3)
    c.close()
