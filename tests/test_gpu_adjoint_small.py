"""First-order FP64 gradients: a small mesh's reverse flux kernels compute on the FP64 unit, a
large one's on the integer pipes, with the same bits. The small mesh is differentiated alone and
as an instance of a batch that is large enough for the other form."""
import os

import numpy as np
import pytest

from cfd2d import cases, meshgen as mg

pytestmark = pytest.mark.gpu

KINDS = ("BOUND_INLET", "BOUND_OUTLET", "BOUND_WALL_SLIP", "BOUND_INLET")


def _gradient(s, U, w):
    s.set_state(U)
    s.set_objective(1, w)
    s.forward(4, 2)
    return s.backward()[0]


@pytest.mark.parametrize("n", [2, 3, 7, 12])
@pytest.mark.parametrize("flux,store", [("HLLC", None), ("HLLC", "ALL"), ("LAX", None)])
def test_first_order_gradient_of_small_and_large_form_equal(capi, tmp_path, n, flux, store):
    made = []
    for k, size in enumerate((n, 96)):  # 27,840 edges with the second
        t, m, U0, w, _ = cases.vortex_adjoint(size, steps=4, mach=0.4, beta=1.0, flux=flux, recon="NONE", cfl=0.2,
                                              bnd_kinds=KINDS, seed=5 + k, box=((2.0, 10.0), (2.5, 7.5)))
        t.adjoint_store = store
        path = os.path.join(str(tmp_path), "task%d.xml" % k)
        with open(path, "w") as f:
            f.write(mg.write_task_xml(t))
        made.append((path, m, U0, w))
    alone = capi.Solver(made[0][0], mesh=made[0][1])
    g = _gradient(alone, made[0][2], made[0][3])
    both = capi.Batch([p for p, *_ in made], meshes=[m for _, m, *_ in made])
    gb = _gradient(both, np.concatenate([U for _, _, U, _ in made], axis=1), np.concatenate([w for *_, w in made]))
    assert np.isfinite(g).all() and np.abs(g).max() > 0.0
    part = np.ascontiguousarray(gb[:, :g.shape[1]])
    assert np.array_equal(g.view(np.int64), part.view(np.int64))
