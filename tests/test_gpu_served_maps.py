"""Served mixed p = 7 requests, whose kernel finds the tensor maps of its
members in device tables that are rewritten in place whenever a member comes or
goes: each result has the bits of a handle of its own."""
import time

import numpy as np
import pytest

import sdg_b200 as sdg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


def test_results_across_membership_changes():
    p = 7
    ops = sdg.read_operators(p)
    boxes = [(2, 3, 2), (5, 4, 3), (3, 3, 3), (6, 2, 5), (4, 4, 4)]
    want, jobs = {}, []
    for k in range(24):
        box, nstep = boxes[k % len(boxes)], 3 + 5 * (k % 7)
        mesh = sdg.mesh_setup(*box, p, ops.x1D)
        fields = sdg.init_fields(mesh, ic_kind=1, seed=50 + k, vel_kind=1)
        dt = 0.1 / max(box) / (p + 1) ** 2
        h = sdg.Handle(ops, mesh, sdg.FLAG_MIXED)
        h.set_state(*(f.copy(order="F") for f in fields))
        h.rk3_steps(dt, nstep)
        want[k] = h.get_field()
        h.close()
        jobs.append((k, box, fields, dt, nstep))
    srv = sdg.Server()
    ids = {}
    for wave in range(3):
        # Members of one wave leave at different chunks while others join.
        for k, box, fields, dt, nstep in jobs[8 * wave: 8 * wave + 8]:
            ids[k] = srv.submit(*box, p, ops, *fields, dt, nstep, mixed=True)
        time.sleep(0.02)
    end = time.time() + 120
    while time.time() < end:
        states = {k: srv.poll(i)[0] for k, i in ids.items()}
        if all(s in (sdg.SERVE_DONE, sdg.SERVE_FAILED) for s in states.values()):
            break
        time.sleep(0.01)
    assert all(s == sdg.SERVE_DONE for s in states.values()), states
    for k, i in ids.items():
        assert np.array_equal(srv.result(i), want[k]), k
    srv.close()
