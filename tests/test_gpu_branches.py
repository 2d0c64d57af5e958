"""Paths of the kernels and of the host that the workloads' own sizes do not reach: many Krylov
vectors, edge counts that end in mid-warp, steps taken in graphs of eight."""
import numpy as np
import pytest

from cfd2d import cases
from test_gpu_adjoint import KINDS
from test_gpu_implicit import RTOL, close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gm", [(48, 48, 1e-10), (64, 64, 1e-12), (40, 60, 1e-10)], ids=["k48", "k64", "k40_restart"])
def test_implicit_many_krylov_vectors_match_oracle(capi, oracle, tmp_path, gm):
    """45 or more columns: inner products past the first kernel's twelve (three further kernels),
    two rows per lane in the back substitution."""
    t, m, U0 = cases.vortex_implicit(16, flux="LAX", beta=1.0, tau=0.5)
    t.gmres = gm
    s = capi.Solver(cases.write_implicit_task(t, m, str(tmp_path)), mesh=m)
    s.set_state(U0)
    s.step(1)
    o = oracle.implicit_from_task(t, m, U0=U0)
    o.step(1)
    st, oi = s.implicit_stats(), o.info()
    assert oi["iters"] > 40
    assert (st["iters"], st["status"]) == (oi["iters"], oi["status"])
    assert close(s.state(), o.state()[0]) < RTOL


@pytest.mark.parametrize("n", [2, 3, 5])
def test_implicit_godunov_edge_tails(capi, oracle, tmp_path, n):
    t, m, U0 = cases.vortex_implicit(n, flux="GODUNOV", beta=1.0)
    s = capi.Solver(cases.write_implicit_task(t, m, str(tmp_path)), mesh=m)
    s.set_state(U0)
    s.step(2)
    o = oracle.implicit_from_task(t, m, U0=U0)
    o.step(2)
    st, oi = s.implicit_stats(), o.info()
    assert (st["iters"], st["status"]) == (oi["iters"], oi["status"])
    assert close(s.state(), o.state()[0]) < RTOL


@pytest.mark.parametrize("n", [3, 5, 7])
@pytest.mark.parametrize("flux,recon,store", [("LAX", "LINEAR", None), ("LAX", "MINMOD", None), ("HLLC", "LINEAR", "ALL"),
                                              ("HLLC", "MINMOD", None)])
def test_adjoint_edge_tails(capi, tmp_path, n, flux, recon, store):
    """A mesh whose interior edges end in mid-warp, alone and as the second instance of a batch,
    where its edges lie in other lanes: the same gradient bit for bit."""
    made = []
    for k, size in enumerate((9, n)):
        t, m, U0, w, _ = cases.vortex_adjoint(size, steps=4, flux=flux, recon=recon, beta=1.0, cfl=0.2, bnd_kinds=KINDS,
                                              seed=4 + k, box=((0.0, 10.0), (0.0, 10.0)))
        t.adjoint_store = store
        d = tmp_path / str(k)
        d.mkdir()
        made.append((cases.write_task(t, m, str(d)), m, U0, w))

    def gradient(s, U, w):
        s.set_state(U)
        s.set_objective(0, w, 0.9)
        s.forward(4, 3)
        return s.backward()[0]

    path, m, U0, w = made[1]
    g = gradient(capi.Solver(path, mesh=m), U0, w)
    both = capi.Batch([q[0] for q in made], meshes=[q[1] for q in made])
    gb = gradient(both, np.concatenate([q[2] for q in made], axis=1), np.concatenate([q[3] for q in made]))
    assert np.all(np.isfinite(g)) and np.abs(g).max() > 0.0
    part = np.ascontiguousarray(gb[:, gb.shape[1] - g.shape[1]:])
    assert np.array_equal(g.view(np.int64), part.view(np.int64))


@pytest.mark.parametrize("precision", [None, "MIXED"])
@pytest.mark.parametrize("steady", [0, 1])
def test_steps_at_once_equal_single_steps(capi, tmp_path, precision, steady):
    t, m, U0 = cases.vortex(9, flux="HLLC", recon="MINMOD", scheme="SSPRK3", steady=steady, precision=precision)
    path = cases.write_task(t, m, str(tmp_path))
    a, b = capi.Solver(path, mesh=m), capi.Solver(path, mesh=m)
    for s in (a, b):
        s.set_state(U0, reset_time_step=True)
    for n in (7, 8, 9, 16, 21, 3):  # the first eight in single steps, later ones by graphs of eight
        a.step(n)
        for _ in range(n):
            b.step(1)
        assert np.array_equal(a.state().view(np.int64), b.state().view(np.int64))
        i, j = a.get_info(), b.get_info()
        assert (i.step, i.time, i.tau) == (j.step, j.time, j.tau)
    assert np.array_equal(a.time_step().view(np.int64), b.time_step().view(np.int64))
