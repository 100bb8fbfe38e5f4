"""2D programs of different sizes stepped side by side: from two host threads,
and alternately through cached graphs.  The step kernel's shared memory depends
on the program, so one program's launches must not depend on what another's
set."""

from __future__ import annotations

import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from beamz_b200 import plan as P  # noqa: E402
from beamz_b200 import runtime as R  # noqa: E402
from tests.scenarios import random_initial_fields, scenario_2d  # noqa: E402

pytestmark = pytest.mark.gpu

# One instance of the step kernel (TM, CPML, one coefficient per site of E only,
# tiles of up to 32 rows), with as much and as little shared memory as it takes.
SIZES = (((180, 190), 20, 8), ((20, 30), 2, 2))


def _program(size, graphs):
    grid, pml, steps = size
    spec = scenario_2d(grid=grid, pml_cells=pml, seed=steps, nsteps=40)
    return spec, R.compile_program(spec, graphs=graphs), steps


def _run(prog, fields, steps, calls, stream):
    with torch.cuda.stream(stream):
        st = R.initial_state(prog, fields=fields)
        for _ in range(calls):
            R.run_steps(st, prog, steps)
        return st.numpy()


def _assert_same(got, want):
    for c in P.active_components(2, "tm"):
        np.testing.assert_array_equal(got[c], want[c], err_msg=c)
    for k in ("psi_h", "psi_e"):
        for x, y in zip(got[k], want[k]):
            np.testing.assert_array_equal(x, y, err_msg=k)
    np.testing.assert_array_equal(got["dft_re"], want["dft_re"])


def test_two_threads_step_programs_of_different_sizes():
    calls = 400
    made = [_program(size, graphs=False) for size in SIZES]
    fields = [random_initial_fields(spec, seed=5) for spec, _, _ in made]
    want = [_run(p, f, n, calls, torch.cuda.Stream()) for (_, p, n), f in zip(made, fields)]
    got, errors = [None] * 2, []
    start = threading.Barrier(2)

    def work(i):
        try:
            stream = torch.cuda.Stream()
            start.wait()
            got[i] = _run(made[i][1], fields[i], made[i][2], calls, stream)
        except Exception as exc:  # reported by the test's own thread
            errors.append(exc)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for g, w in zip(got, want):
        _assert_same(g, w)


def test_cached_graphs_of_different_sizes_alternate():
    made = [_program(size, graphs=True) for size in SIZES]
    fields = [random_initial_fields(spec, seed=6) for spec, _, _ in made]
    want = [_run(_program(size, False)[1], f, size[2], 6, torch.cuda.Stream()) for size, f in zip(SIZES, fields)]
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        states = [R.initial_state(p, fields=f) for (_, p, _), f in zip(made, fields)]
        for _ in range(6):
            for (_, p, n), st in zip(made, states):
                R.run_steps(st, p, n)
        got = [st.numpy() for st in states]
    for g, w in zip(got, want):
        _assert_same(g, w)
