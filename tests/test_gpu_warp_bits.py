"""The warp-per-element kernel of the fast FP64 form at p = 7 computes every node
in the operations and order of the one-tile-per-block kernel: the same bits.  The
block kernel is the one that runs where Lift_mat does not factorise, so the two
meet on a Lift_mat that does, and on the same one with an entry of the -z face
changed while w is zero (that face's flux, and with it the change, is zero)."""
import numpy as np
import pytest

import sdg_b200 as sdg

pytestmark = pytest.mark.gpu

P = 7


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


def lifts():
    """Operators with a Lift_mat that is one factor a face, and with the change."""
    ops = sdg.read_operators(P)
    axis = (1, 0, 1, 0, 2, 2)  # normal of faces -y, +x, +y, -x, -z, +z
    lift = np.zeros_like(ops.Lift_mat)
    for f in range(6):
        at = [0, 0, 0]
        at[axis[f]] = slice(None)
        shape = [1, 1, 1]
        shape[axis[f]] = ops.Nq
        lift[..., f] = ops.Lift_mat[(*at, f)].reshape(shape)
    changed = lift.copy(order="F")
    changed[3, 4, 0, 4] *= 1.0 + 1e-3
    return [ops._replace(Lift_mat=x) for x in (lift, changed)]


@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 2, 2), (37, 4, 2), (9, 8, 7), (13, 11, 9)])
def test_bits_of_the_block_kernel(dims):
    pair = lifts()
    mesh = sdg.mesh_setup(*dims, P, pair[0].x1D)
    q, u, v, w = sdg.init_fields(mesh, ic_kind=1, seed=5, vel_kind=1)
    w[:] = 0.0
    dt = 0.1 / max(dims) / (P + 1) ** 2
    res = []
    for ops in pair:
        h = sdg.Handle(ops, mesh, 0)
        tend = h.cal_tend(q, u, v, w)[:, : mesh.Ne]
        h.set_state(q, u, v, w)
        h.rk3_steps(dt, 3)
        res.append((tend, h.get_field()))
        h.close()
    assert np.array_equal(res[0][0], res[1][0])
    assert np.array_equal(res[0][1], res[1][1])
