"""The one-launch linear solve (GPU): rows wait for entries that other blocks write, and a failure (made
on the host) leaves the context usable."""
import numpy as np
import pytest

from bes_gb300 import lib, meshgen
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


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("sweep_kernel", [0, 2])
@pytest.mark.parametrize("n_cond", [1, 3])
def test_step_whose_wait_gave_up_is_not_applied(precision, sweep_kernel, n_cond):
    """The second step fails: the state stays the first step's, and the next step is the second."""
    mesh = meshgen.bump_channel(9, 3, 1, 0.08)
    machs = np.array([[0.5, 0.02, 0.0], [0.7, 0.0, 0.0], [0.6, 0.0, 0.03]])[:n_cond]

    def ctx():
        o = lib.default_options(precision=precision, linear_solver=1, sweep_kernel=sweep_kernel, **OPTS)
        return lib.Context(mesh, o, machs=machs if n_cond > 1 else None)

    plain = ctx()
    plain.implicit_steps(1)
    U1 = plain.get_state()
    h2, U2 = plain.implicit_steps(1), plain.get_state()
    plain.close()
    c = ctx()
    c.implicit_steps(1)
    c.inject_failure(lib.FAIL_WAIT)
    with pytest.raises(lib.BesError) as e:
        c.implicit_steps(1)
    assert e.value.code == 7
    assert np.array_equal(c.get_state(), U1)
    assert np.array_equal(c.implicit_steps(1), h2)
    assert np.array_equal(c.get_state(), U2)
    c.close()


def _three_steps(failure, at, precision, linear, profile=False):
    """Three steps with a failure injected before step `at`; histories, state and the tuning text."""
    c = context(meshgen.bump_channel(9, 3, 1, 0.08), precision=precision, linear_solver=linear, **OPTS)
    c.profile(profile)
    h = []
    for k in range(3):
        if k == at:
            c.inject_failure(failure)
        try:
            h.append(c.implicit_steps(1))
        except lib.BesError as e:
            assert e.code == 7 and failure == lib.FAIL_WAIT and k == at
            h.append(c.implicit_steps(1))
    U, text = c.get_state(), c.tuning()
    c.close()
    return np.concatenate(h), U, text


@pytest.mark.parametrize("failure,at", [(lib.FAIL_SOLVE_CAPTURE, 0), (lib.FAIL_WAIT, 1)])
@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("linear", [0, 1])
def test_refused_solve_falls_back_to_the_graph(failure, at, precision, linear):
    """Refused when the step graph is made, or given up in a step: the steps are those of a
    context in which nothing failed, and the persistent form is not taken again."""
    h, U, text = _three_steps(0, -1, precision, linear)
    assert "taken: the step graph's solve" not in text
    hf, Uf, textf = _three_steps(failure, at, precision, linear, profile=failure == lib.FAIL_WAIT)
    assert textf.count("taken: the step graph's solve") == 1
    assert np.array_equal(hf, h) and np.array_equal(Uf, U)


@pytest.mark.parametrize("precision", [0, 1, 2])
def test_no_memory_for_the_solve(precision):
    """The graph's solve, with every colour-sweep form in the running (the allocation's error, left
    for the next check, took the first form out of it)."""
    h, U, _ = _three_steps(0, -1, precision, 1)
    hf, Uf, text = _three_steps(lib.FAIL_SOLVE_ALLOC, 0, precision, 1)
    assert "one persistent launch" not in text and "one launch per colour failed" not in text
    assert np.array_equal(hf, h) and np.array_equal(Uf, U)
