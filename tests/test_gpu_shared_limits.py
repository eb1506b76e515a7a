"""A kernel's dynamic shared-memory limit is one for the process: contexts of
different needs, created by several threads at once or one after the other,
leave each other's launches valid.

A limit that is too small is refused by the launch on the host (an error
status), so a lost update shows as an MmsError.
"""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

THREADS = """
import sys, threading
sys.path.insert(0, sys.argv[1])
import numpy as np
import mmsb200
# two layer counts a transform length, both beyond 48 KB a CTA
for Y, layers in ((200, (8, 6)), (300, (8, 5)), (500, (8, 3)), (700, (7, 3)), (1000, (5, 2))):
    gate, failed = threading.Barrier(12), []

    def work(Z):
        try:
            gate.wait()
            with mmsb200.Context(mmsb200.Grid(5001 // Y + 2, Y, Z, 5e-9, 5e-9, 5e-9)) as c:
                gate.wait()
                rho = np.ones((Z, Y, c.grid.xdim), np.float32)
                phi = np.empty_like(rho)
                mmsb200._check(mmsb200.load().mms_potential_host(c.h, rho.ctypes.data, phi.ctypes.data))
        except mmsb200.MmsError as e:
            failed.append((Y, Z, str(e)))
            gate.abort()
        except threading.BrokenBarrierError:
            pass

    threads = [threading.Thread(target=work, args=(layers[i % 2],)) for i in range(12)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not failed, failed
print("done")
"""


def test_contexts_created_by_several_threads(cuda, lib):
    """every kernel's first limit is set by two needs at once, in a new process"""
    r = subprocess.run([sys.executable, "-c", THREADS, ROOT + "/mms-gpu_b200"], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr


@pytest.mark.parametrize("kw", [dict(), dict(m2l_mode=1), dict(near_mode=1)])
@pytest.mark.parametrize("first,second", [((9, 8, 3), (8, 8, 3)), ((9, 4, 3), (8, 4, 3)), ((9, 8, 2), (9, 8, 1)),
                                          ((8, 8, 8), (7, 8, 8)), ((3, 8, 16), (3, 8, 15))])
def test_a_smaller_plan_leaves_a_larger_one_its_kernels(cuda, lib, first, second, kw):
    """two FMM contexts (order, leaf side, layers) live together: the second
    one needs less shared memory of the same kernels, and the first one's
    potential is that from before"""
    import mmsb200
    torch = cuda

    def context(P, leaf, Z):
        return mmsb200.Context(mmsb200.Grid(64, 64, Z, 5e-9, 5e-9, 5e-9), mmsb200.make_params(),
                               mmsb200.make_solver(mmsb200.SOLVER_FMM, P, leaf, **kw))

    rho = torch.randn(first[2], 64, 64, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    before, after = torch.empty_like(rho), torch.empty_like(rho)
    with context(*first) as a:
        a.potential_dev(rho, before)
        a.sync()
        with context(*second):
            a.potential_dev(rho, after)
            a.sync()
    assert torch.equal(before, after)
