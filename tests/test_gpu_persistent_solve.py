"""The one-launch linear solve (GPU): rows wait for entries that other blocks write."""
import numpy as np
import pytest

from bes_gb300 import meshgen
from tests._gpu import context

pytestmark = pytest.mark.gpu

OPTS = dict(solver_type=1, local_time_step=1, courant_num=30.0, linear_solver_tol=1e-3,
            linear_solver_max_iter=200, gmres_restart=12, freestream_mach=(0.5, 0.02, 0.0))


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("linear", [0, 1])
def test_repeated_solves_are_equal(precision, linear):
    """The order in which rows find their neighbours changes from run to run, the bits do not."""
    ctx = context(meshgen.bump_channel(24, 8, 6, 0.08), precision=precision, linear_solver=linear, **OPTS)
    U0 = ctx.get_state()
    runs = []
    for _ in range(12):
        ctx.set_state(U0)
        runs.append((ctx.implicit_steps(2), ctx.get_state()))
    assert "one persistent launch" in ctx.tuning()
    ctx.close()
    for h, U in runs[1:]:
        assert np.array_equal(h, runs[0][0]) and np.array_equal(U, runs[0][1])
