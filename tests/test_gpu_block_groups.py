"""The block storage in groups of 32 rows where the last group is not full (GPU): 6, 30, 32, 34, 64,
66, 96 and 162 cells, every precision and preconditioner, both forms of the linear solve.

The FP64 blocks are the oracle's (1e-12, as in test_gpu_implicit.py).  The step of each precision
solves its own system: with the blocks that the library assembled (rounded to the 16-bit form
here for precision 2) the residual of the update is at most twice the linear tolerance (the
Krylov basis is orthogonal to a quarter, so the solver's estimate is within that factor)."""
import numpy as np
import pytest

from bes_gb300 import build as nbuild
from bes_gb300 import lib, meshgen
from oracle import pyoracle

pytestmark = pytest.mark.gpu

MESHES = {
    6: lambda: meshgen.bump_channel(1, 1, 1, 0.0),
    30: lambda: meshgen.bump_channel_2d(5, 3, 0.08),
    32: lambda: meshgen.bump_channel_2d(4, 4, 0.08),
    34: lambda: meshgen.bump_channel_2d(17, 1, 0.08),
    64: lambda: meshgen.bump_channel_2d(8, 4, 0.08),
    66: lambda: meshgen.bump_channel(11, 1, 1, 0.08),
    96: lambda: meshgen.bump_channel(4, 2, 2, 0.08),
    162: lambda: meshgen.bump_channel(9, 3, 1, 0.08),
}
CFL, MACH = 30.0, (0.6, 0.02, 0.0)


def _packed(blocks):
    """The entries as the 16-bit form holds them: halves of the block over its power of two."""
    mx = np.abs(blocks.astype(np.float32)).max(axis=(1, 2))
    scale = np.where(mx > 0, 2.0 ** np.ceil(np.log2(np.where(mx > 0, mx, 1.0))), 1.0)[:, None, None]
    return (blocks / scale).astype(np.float16).astype(np.float64) * scale


@pytest.mark.parametrize("cells", list(MESHES))
@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("linear", [0, 1])
@pytest.mark.parametrize("sweep_kernel", [0, 1])
def test_step_solves_the_assembled_system(cells, precision, linear, sweep_kernel):
    nbuild.build()
    mesh = MESHES[cells]()
    assert mesh.n_cells == cells
    tol = 1e-8 if precision == 0 else 1e-3
    mach = MACH if mesh.dim == 3 else MACH[:2] + (0.0,)
    ctx = lib.Context(mesh, lib.default_options(
        solver_type=1, local_time_step=1, courant_num=CFL, linear_solver=linear, linear_solver_tol=tol,
        linear_solver_max_iter=300, gmres_restart=30, precision=precision, sweep_kernel=sweep_kernel,
        freestream_mach=mach))
    exp = pyoracle.Oracle(mesh, solver=1, local_dt=1, cfl=CFL, mach=mach).implicit_assemble(CFL)
    got = ctx.implicit_assemble(CFL)
    if precision == 0:
        assert np.linalg.norm(got["blocks"] - exp["vals"]) <= 1e-12 * np.linalg.norm(exp["vals"])
    U0 = ctx.get_state()
    ctx.implicit_steps(1)
    dU = ctx.get_state() - U0
    blocks = _packed(got["blocks"]) if precision == 2 else got["blocks"]
    r = got["rhs"].copy()
    for i in range(cells):
        for k in range(exp["rowptr"][i], exp["rowptr"][i + 1]):
            r[i] -= blocks[k] @ dU[exp["col"][k]]
    assert np.linalg.norm(r) <= 2.0 * tol * np.linalg.norm(got["rhs"])
    ctx.close()
