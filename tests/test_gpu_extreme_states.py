"""Explicit iterations on states at the edge of what the scheme takes (GPU), against the oracle."""
import numpy as np
import pytest

from bes_gb300 import lib, meshgen
from oracle import pyoracle
from tests._gpu import context, rel_err

pytestmark = pytest.mark.gpu


def _uniform(mesh, mach):
    n = mesh.n_cells
    U = np.zeros((n, 5))
    U[:, 0] = 1.0
    U[:, 1:4] = mach
    U[:, 4] = 1.0 / (1.4 * 0.4) + 0.5 * np.dot(mach, mach)
    return U


def _compare(mesh, U0, mach, local, exact, steps, cfl):
    ctx = context(mesh, solver_type=0, local_time_step=local, courant_num=cfl, freestream_mach=mach,
                  muscl_face_vector=exact)
    ctx.set_state(U0)
    h = ctx.explicit_iterations(steps)
    U = ctx.get_state()
    ctx.close()
    O = pyoracle.Oracle(mesh, cfl=cfl, mach=mach, local_dt=local, muscl_exact=exact)
    O.set_state(U0)
    ho, Uo = O.explicit_run(steps), O.get_state()
    assert np.isfinite(ho).all() and np.isfinite(Uo).all()
    # the bound of test_gpu_side_path.py: a few hundred ulp of the residual, plus of the face fluxes
    # times areas that cancel in it
    bound = 1e-12 * np.abs(ho).max() + 1e-13 * lib.host_geometry(mesh)["face_area"].max()
    assert np.abs(h - ho).max() <= bound
    assert rel_err(U, Uo) <= 1e-12


@pytest.mark.parametrize("mesh", [meshgen.bump_channel(9, 3, 1, 0.08), meshgen.bump_channel_2d(13, 5, 0.08)])
@pytest.mark.parametrize("local", [1, 0])
@pytest.mark.parametrize("exact", [0, 1])
def test_cell_without_pressure(mesh, local, exact):
    """(rho, u, p) = (1, 0.5, 0) in one cell: its sound speed is 0, its time step finite."""
    mach = (0.5, 0.0, 0.0)
    U0 = _uniform(mesh, mach)
    U0[mesh.n_cells // 2, 4] = 0.5 * 0.5 ** 2
    _compare(mesh, U0, mach, local, exact, 3, 0.5)


@pytest.mark.parametrize("mesh,cell,low", [(meshgen.bump_channel(5, 1, 1, 0.04), 1, 0.004),
                                           (meshgen.bump_channel(9, 3, 1, 0.08), 100, 0.02),
                                           (meshgen.bump_channel_2d(13, 5, 0.08), 10, 0.02)])
def test_density_below_zero_at_a_wall_face(mesh, cell, low):
    """A light cell at a wall: the density extrapolated to the wall's face (no face values limit it)
    is negative, the pressure there is not, and the wall's flux takes the pressure only."""
    mach = (0.5, 0.0, 0.0)
    U0 = _uniform(mesh, mach)
    U0[cell, 4] += 0.5 * (low - 1.0) * 0.5 ** 2
    U0[cell, :4] *= low
    O = pyoracle.Oracle(mesh, cfl=0.05, mach=mach, local_dt=1, muscl_exact=1)
    O.set_state(U0)
    below = O.operators(0.05)["face_UL"][:, 0] < 0
    assert below.any() and (lib.host_geometry(mesh)["face_type"][below] == 1).all()
    _compare(mesh, U0, mach, 1, 1, 1, 0.05)
