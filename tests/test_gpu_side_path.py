"""The explicit path's residual kernels (side_kernels.cuh) against the oracle where a block or
warp is not full, where every boundary branch and the limiter's cases occur, and for every
form the entry point takes (triangles, exact face vectors, global time step, batches)."""
import numpy as np
import pytest

from bes_gb300 import lib, meshgen
from oracle import pyoracle
from tests._gpu import context, rel_err

pytestmark = pytest.mark.gpu

MESHES = {
    "6": lambda: meshgen.bump_channel(1, 1, 1, 0.0),
    "30": lambda: meshgen.bump_channel(5, 1, 1, 0.04),
    "162": lambda: meshgen.bump_channel(9, 3, 1, 0.08),
    "tri": lambda: meshgen.bump_channel_2d(13, 5, 0.08),
    "box": lambda: meshgen.gaussian_box(6, 3, 4, 1.05),
}


def _wavy(mesh, mach, seed, amp):
    r = np.random.default_rng(seed)
    n = mesh.n_cells
    rho = 1.0 + amp * r.uniform(-1, 1, n)
    p = (1.0 + amp * r.uniform(-1, 1, n)) / 1.4
    u = np.array([mach[d] + amp * r.uniform(-1, 1, n) for d in range(3)])
    if mesh.dim == 2:
        u[2] = 0.0
    return np.stack([rho, rho * u[0], rho * u[1], rho * u[2],
                     p / 0.4 + 0.5 * rho * (u * u).sum(0)], 1)


@pytest.mark.parametrize("name", list(MESHES))
@pytest.mark.parametrize("mach", [(0.5, 0.02, 0.03), (1.6, 0.1, 0.0), (-0.3, 0.0, 0.1),
                                  (0.0, 0.0, 0.0)])
@pytest.mark.parametrize("amp", [0.0, 1e-6, 0.1])
@pytest.mark.parametrize("exact,local", [(0, 1), (1, 0)])
def test_iterations_match_oracle(name, mach, amp, exact, local):
    mesh = MESHES[name]()
    if mesh.dim == 2:
        mach = (mach[0], mach[1], 0.0)
    U0 = _wavy(mesh, mach, 3, amp)
    ctx = context(mesh, solver_type=0, local_time_step=local, courant_num=0.5,
                  freestream_mach=mach, muscl_face_vector=exact)
    ctx.set_state(U0)
    h = ctx.explicit_iterations(3)
    U = ctx.get_state()
    ctx.close()

    def oracle(U):
        O = pyoracle.Oracle(mesh, cfl=0.5, mach=mach, local_dt=local, muscl_exact=exact)
        O.set_state(U)
        return O.explicit_run(3), O.get_state()

    ho, Uo = oracle(U0)
    # rounding: a few hundred ulp (1.1e-16) of the residual, plus of the face fluxes times areas
    # that cancel in it (up to about five per unit area, four faces, a dozen roundings each)
    area = lib.host_geometry(mesh)["face_area"].max()
    bound = 1e-12 * np.abs(ho).max() + 1e-13 * area
    # The freestream boundary is discontinuous at zero normal velocity (inlet or outlet): where
    # that velocity is rounding noise, the oracle's own answer moves by more than the bound when
    # its input moves by one ulp, and the comparison says nothing.
    ulp = np.random.default_rng(0).choice([-2.2e-16, 2.2e-16], U0.shape)
    if np.abs(oracle(U0 * (1.0 + ulp))[0] - ho).max() > bound:
        pytest.skip("the oracle's own residuals move by more than the bound")
    assert np.abs(h - ho).max() <= bound
    assert rel_err(U, Uo) <= 1e-12


def test_batch_equals_single_contexts():
    mesh = MESHES["162"]()
    machs = np.array([[0.4, 0.0, 0.02], [0.8, 0.03, 0.0], [1.3, 0.0, 0.0]])
    opts = dict(solver_type=0, local_time_step=0, courant_num=0.5, muscl_face_vector=1)
    ctx = lib.Context(mesh, lib.default_options(freestream_mach=tuple(machs[0]), **opts), machs=machs)
    U0 = np.stack([_wavy(mesh, m, k, 0.05) for k, m in enumerate(machs)])
    ctx.set_state(U0)
    h, U = ctx.explicit_iterations(4), ctx.get_state()
    ctx.close()
    for k, m in enumerate(machs):
        one = context(mesh, freestream_mach=tuple(m), **opts)
        one.set_state(U0[k])
        assert np.array_equal(one.explicit_iterations(4), h[:, k])
        assert np.array_equal(one.get_state(), U[k])
        one.close()
