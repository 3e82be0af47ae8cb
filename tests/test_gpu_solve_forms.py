"""The linear solves in one persistent launch against the step graph's own solve
(SWEEP_KERNEL = PER_COLOUR): every phase computes the same values in the same order, so the
steps are equal bit for bit.  Sizes where a warp, a virtual block or a 16-byte granule of the
vectors is not full (6 to 6,912 cells), restarts, second Gram-Schmidt passes (6 cells), batches
with a frozen condition, and the iteration limit."""
import numpy as np
import pytest

from bes_gb300 import build as nbuild
from bes_gb300 import lib, meshgen

pytestmark = pytest.mark.gpu

MESHES = {
    "6": lambda: meshgen.bump_channel(1, 1, 1, 0.0),
    "162": lambda: meshgen.bump_channel(9, 3, 1, 0.08),
    "tri": lambda: meshgen.bump_channel_2d(13, 5, 0.08),
    "6912": lambda: meshgen.bump_channel(24, 8, 6, 0.08),
}
MACHS = np.array([[0.5, 0.02, 0.0], [0.84, 0.0, 0.0], [0.7, 0.03, 0.0]])


def _steps(mesh, machs, sweep_kernel, frozen, **kw):
    o = dict(solver_type=1, local_time_step=1, courant_num=30.0, linear_solver_tol=1e-3,
             linear_solver_max_iter=200, gmres_restart=12, sweep_kernel=sweep_kernel,
             freestream_mach=tuple(machs[0]))
    o.update(kw)
    ctx = lib.Context(mesh, lib.default_options(**o), machs=machs if len(machs) > 1 else None)
    h = [ctx.implicit_steps(2)]
    if frozen:
        ctx.set_active([1, 0, 1])
    h.append(ctx.implicit_steps(2))
    out = (np.concatenate(h), ctx.get_state(), ctx.implicit_stats(), ctx.counters()["gram_schmidt_second_passes"],
           ctx.tuning())
    ctx.close()
    return out


@pytest.mark.parametrize("name", list(MESHES))
@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("linear", [0, 1])
@pytest.mark.parametrize("n_cond", [1, 3])
def test_persistent_solve_equals_graph_solve(name, precision, linear, n_cond):
    nbuild.build()
    mesh = MESHES[name]()
    a = _steps(mesh, MACHS[:n_cond], 0, n_cond > 1, precision=precision, linear_solver=linear)
    b = _steps(mesh, MACHS[:n_cond], 1, n_cond > 1, precision=precision, linear_solver=linear)
    if mesh.n_cells * n_cond <= 7000:  # larger ones may be the graph's on both sides
        assert "one persistent launch" in a[4]
    assert "persistent" not in b[4]
    assert np.array_equal(a[0], b[0])
    assert np.array_equal(a[1], b[1])
    assert a[2] == b[2] and a[3] == b[3]


@pytest.mark.parametrize("limit", [1, 5, 12, 13])
def test_iteration_limit_and_guard(limit):
    nbuild.build()
    mesh = MESHES["162"]()
    kw = dict(precision=2, linear_solver=1, linear_solver_max_iter=limit, linear_solver_tol=1e-6)
    a, b = (_steps(mesh, MACHS[:1], k, False, **kw) for k in (0, 1))
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    ctx = lib.Context(mesh, lib.default_options(solver_type=1, local_time_step=1, courant_num=30.0,
                                                linear_solver=1, linear_solver_tol=1e-6,
                                                linear_solver_max_iter=200, gmres_restart=4,
                                                freestream_mach=(0.5, 0.0, 0.0)))
    ctx.set_linear_guard(1)
    with pytest.raises(lib.BesError) as e:
        ctx.implicit_steps(1)
    assert e.value.code == 7
    ctx.set_linear_guard(0)
    ctx.implicit_steps(1)
    ctx.close()
