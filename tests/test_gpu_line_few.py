"""Element counts around which the automatic variant changes between the line
kernel and the ones before it (148 SMs): chained steps, stage calls of their
own, host-buffer calls and the tendency give the block kernel's bits on both
sides."""
import numpy as np
import pytest

import sdg_b200 as sdg

pytestmark = pytest.mark.gpu

# (p, flags, boxes): p = 1 at 17, 30, 32 and 64 elements an SM; p = 9 to 12 at one
# and two; p = 10 also at three and a half and four.
CASES = [(1, 0, [(37, 17, 4), (2517, 1, 1), (37, 32, 4), (37, 43, 3)]),
         (1, sdg.FLAG_MIXED, [(37, 30, 4), (53, 28, 3), (37, 32, 8), (41, 33, 7)]),
         (9, 0, [(37, 4, 2), (33, 9, 1)]), (11, 0, [(37, 2, 2), (149, 1, 1)]),
         (12, 0, [(37, 2, 2), (149, 1, 1)]),
         (10, 0, [(37, 4, 2), (33, 9, 1), (37, 7, 2), (173, 3, 1), (37, 4, 4), (593, 1, 1)])]


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


@pytest.mark.parametrize("p,flags,boxes", CASES)
def test_both_sides_of_the_line(p, flags, boxes):
    ops = sdg.read_operators(p)
    for dims in boxes:
        mesh = sdg.mesh_setup(*dims, p, ops.x1D)
        q, u, v, w = sdg.init_fields(mesh, ic_kind=1, seed=8, vel_kind=1)
        dt, n = 0.1 / max(dims) / (p + 1) ** 2, mesh.Ne
        res = []
        for variant in (sdg.VARIANT_BLOCK, sdg.VARIANT_AUTO):
            h = sdg.Handle(ops, mesh, flags)
            h.set_kernel_variant(variant)
            tend = h.cal_tend(q, u, v, w)[:, :n]
            h.set_state(q, u, v, w)
            h.rk3_steps(dt, 2)
            steps = h.get_field()
            h.set_state(q, u, v, w)
            for stage in (1, 2, 3) * 2:
                h.rk3_stage(stage, dt)
            stages = h.get_field()
            host = h.rk3_steps_host(q[:, :n].copy(order="F"), dt, 2)
            res.append((tend, steps, stages, host))
            h.close()
        assert np.array_equal(res[0][0], res[1][0]), dims
        for got in (res[0][2], res[0][3], *res[1][1:]):
            assert np.array_equal(got, res[0][1]), dims
