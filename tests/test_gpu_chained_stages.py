"""The step graphs' stage kernels start while the stage before them still runs
(programmatic dependent launches); stage calls of their own do not.  Both give
the same bits at every order and form, on meshes that leave several blocks on an
SM and whose neighbours share memory sectors (odd orders' element sizes)."""
import numpy as np
import pytest

import sdg_b200 as sdg

pytestmark = pytest.mark.gpu

FORMS = ([(p, f) for p in range(1, 9) for f in (0, sdg.FLAG_EXACT, sdg.FLAG_MIXED)] +
         [(p, 0) for p in (9, 10, 12, 15)] + [(p, sdg.FLAG_EXACT) for p in (11, 13)])


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


@pytest.mark.parametrize("p,flags", FORMS)
def test_steps_equal_single_stages(p, flags):
    ops = sdg.read_operators(p)
    for dims in [(5, 3, 2), (17, 13, 11) if p < 9 else (11, 9, 7)]:
        mesh = sdg.mesh_setup(*dims, p, ops.x1D)
        fields = sdg.init_fields(mesh, ic_kind=1, seed=6, vel_kind=1)
        dt, steps = 0.1 / max(dims) / (p + 1) ** 2, 26
        h = sdg.Handle(ops, mesh, flags)
        h.set_state(*fields)
        h.rk3_steps(dt, steps)
        chained = h.get_field()
        h.set_state(*fields)
        for _ in range(steps):
            for stage in (1, 2, 3):
                h.rk3_stage(stage, dt)
        assert np.array_equal(chained, h.get_field()), dims
        h.close()
