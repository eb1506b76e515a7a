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


@pytest.mark.parametrize("mode,ref_time", [(0, False), (1, False), (1, True)])
def test_march_restores_the_field_of_its_time(cuda, lib, mode, ref_time):
    """The adaptive march under a steep field table, with rejections (and, in
    mode 1, the rollback before every pair of half steps), against its own
    accepted steps taken one after the other without any rollback.  A step's
    first field at a stale time turns M by 6e-6 or more.  Bound 1e-7 of Ms: the
    times differ by rounding, so a potential's value may round the other way, 1e-10
    of Ms a field evaluation, some hundreds of them."""
    import mmsb200
    X, Y, Z = 7, 5, 3
    mat = np.ones((Z, Y, X), np.uint8)
    M = np.empty((Z, Y, X, 3))
    M[:] = 8.6e5 * np.array([-1.0, 0.1, 0.05]) / np.linalg.norm([-1.0, 0.1, 0.05])

    def context():
        return mmsb200.Context(mmsb200.Grid(X, Y, Z, 5e-9, 5e-9, 5e-9),
                               mmsb200.make_params(external=True, ref_stage_time=ref_time, **T1),
                               mmsb200.make_solver(mmsb200.SOLVER_DIRECT))

    rejected = []
    with context() as c:
        c.state_set(mat, M)
        final, dt0 = (3e-14, 1e-13) if mode == 0 else (1.2e-12, 4e-13)
        rows, st = c.march(final, dt0, mode=mode, rtol=1e-6, torque_stop=1e-9 if mode == 0 else 0.0,
                           callback=lambda rej, r: rejected.append(rej) and False)
        a, t = c.state_get()
    assert st == mmsb200.MMS_OK and 3 <= len(rows) <= 100 and sum(rejected) >= 2
    with context() as c:
        c.state_set(mat, M)
        at = 0.0
        for row in rows:
            n = 1 if mode == 0 else 2
            c.run_fixed((row[1] - at) / n, n, use_graph=False)
            at = row[1]
        b, tb = c.state_get()
    assert abs(t - tb) <= 1e-12 * t
    assert np.abs(a - M).max() > 5e-4 * 8.6e5
    assert np.abs(a - b).max() <= 1e-7 * 8.6e5


def test_reference_stage_times_over_several_steps(cuda, lib, oracle_mod):
    """five captured steps with the reference's stage times under the steep
    table, against the FP64 oracle's (the RK4 tests' bound, 1e-4 deg)"""
    import mmsb200
    from conftest import max_angle_deg
    X, Y, Z = 17, 15, 3
    rng = np.random.default_rng(3)
    mat = np.ones((Z, Y, X), np.uint8)
    M = rng.normal(size=(Z, Y, X, 3))
    M *= 8.6e5 / np.linalg.norm(M, axis=-1, keepdims=True)
    with mmsb200.Context(mmsb200.Grid(X, Y, Z, 5e-9, 5e-9, 5e-9),
                         mmsb200.make_params(external=True, ref_stage_time=True, **T1)) as c:
        c.state_set(mat, M)
        c.run_fixed(1e-13, 5)
        a, _ = c.state_get()
    p = oracle_mod.Params(external=True, ref_stage_time=True, **T1)
    ref = oracle_mod.rk4_run(oracle_mod.Grid(X, Y, Z, 5e-9, 5e-9, 5e-9), p, mat, M, 1e-13, 5)
    other = oracle_mod.rk4_run(oracle_mod.Grid(X, Y, Z, 5e-9, 5e-9, 5e-9),
                               oracle_mod.Params(external=True, **T1), mat, M, 1e-13, 5)
    assert max_angle_deg(other, ref) > 1e-2  # (the stage times show)
    assert max_angle_deg(a, ref) < 1e-4
