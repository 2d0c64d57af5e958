"""The FP64 flux kernels that give an edge one lane per Gauss point: meshes whose edge counts end
in the middle of a warp, against the oracle (bit for bit; GODUNOV within 1e-12, x^a)."""
import numpy as np
import pytest

from cfd2d import capi, cases
from conftest import PKG  # noqa: F401

pytestmark = pytest.mark.gpu


def _same(flux, a, b):
    if flux == "GODUNOV":
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
    else:
        assert np.array_equal(a.view(np.int64), b.view(np.int64))


@pytest.mark.parametrize("n", [1, 2, 3, 5, 7])
@pytest.mark.parametrize("flux,recon", [("HLLC", "MINMOD"), ("ROE", "LINEAR"), ("LAX", "MINMOD"), ("GODUNOV", "LINEAR")])
def test_explicit_edge_tails(oracle, tmp_path, n, flux, recon):
    t, m, U0 = cases.vortex(n, flux=flux, recon=recon, scheme="HEUN", cfl=0.2, beta=1.0)
    s = capi.Solver(cases.write_task(t, m, str(tmp_path)), mesh=m)
    s.set_state(U0, reset_time_step=True)
    s.step(3)
    o = oracle.solver_from_task(t, m, U0=U0, flux=flux, recon=recon, scheme="HEUN")
    o.step(3)
    _same(flux, s.state(), o.state()[0])
    s.close()


@pytest.mark.parametrize("n", [2, 3, 4, 7])
@pytest.mark.parametrize("flux", ["LAX", "GODUNOV"])
@pytest.mark.parametrize("gp_edge", [2, 3])
def test_rkdg_edge_tails(oracle, tmp_path, n, flux, gp_edge):
    t, m, pm, U0 = cases.rkdg_vortex(n, flux=flux, gp_edge=gp_edge, beta=1.0)
    s = capi.Solver(cases.write_rkdg_task(t, pm, str(tmp_path)))  # the mesh part, as the oracle has it
    s.set_dg_coeffs(U0)
    s.step(2)
    o = oracle.OracleDG(t, pm)
    o.set_coeffs(U0)
    o.step(2)
    _same(flux, s.dg_coeffs(), o.state()["U"])
    s.close()


@pytest.mark.parametrize("n", [2, 3, 5])
def test_implicit_edge_tails(oracle, tmp_path, n):
    t, m, U0 = cases.vortex_implicit(n, flux="LAX", beta=1.0)
    s = capi.Solver(cases.write_implicit_task(t, m, str(tmp_path)), mesh=m)
    s.set_state(U0)
    o = oracle.implicit_from_task(t, m, U0=U0)
    for a, b in zip(s.implicit_system(), o.system()):
        assert np.array_equal(np.asarray(a).ravel().view(np.int64), np.asarray(b).ravel().view(np.int64))
    s.close()
