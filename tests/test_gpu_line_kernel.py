"""The line kernel (sdg_tend_line.cuh) against the one-tile-per-block kernel,
whose bits it reproduces: single elements, fewer elements than blocks, full
tiles with a remainder, halo and direct neighbours, batches."""
import numpy as np
import pytest

import sdg_b200 as sdg

pytestmark = pytest.mark.gpu

GENERAL = sdg.FLAG_EXACT | sdg.FLAG_ORDER_GENERAL
# (p, flags): the orders and forms at which the automatic variant takes it.
FORMS = ([(1, 0), (1, sdg.FLAG_MIXED)] + [(p, 0) for p in range(9, 16)] +
         [(p, sdg.FLAG_EXACT) for p in (11, 12, 13)] + [(11, GENERAL)])


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


@pytest.mark.parametrize("p,flags", FORMS)
def test_bits_of_the_block_kernel(p, flags):
    ops = sdg.read_operators(p)
    # One element; some; more than one round of tiles of 1, 2 or 3 elements on
    # 148 SMs with a remainder (p = 1: of 32 and 48).
    large = [(37, 25, 20), (41, 29, 25)] if p == 1 else [(23, 13, 1), (149, 6, 1)]
    for dims in [(1, 1, 1), (3, 2, 3)] + large:
        mesh = sdg.mesh_setup(*dims, p, ops.x1D)
        q, u, v, w = sdg.init_fields(mesh, ic_kind=1, seed=4, vel_kind=1)
        dt = 0.1 / max(dims) / (p + 1) ** 2
        res = []
        for variant in (sdg.VARIANT_AUTO, sdg.VARIANT_BLOCK):
            h = sdg.Handle(ops, mesh, flags)
            h.set_kernel_variant(variant)
            tend = h.cal_tend(q, u, v, w)[:, : mesh.Ne]
            h.set_state(q, u, v, w)
            h.rk3_steps(dt, 2)
            res.append((tend, h.get_field()))
            h.close()
        assert np.array_equal(res[0][0], res[1][0]), dims
        assert np.array_equal(res[0][1], res[1][1]), dims
        b = sdg.Batch(flags)
        small = sdg.mesh_setup(2, 1, 2, p, ops.x1D)
        b.add(2, 1, 2, p, ops, *sdg.init_fields(small, ic_kind=1, seed=3, vel_kind=1), 1e-4)
        i = b.add(*dims, p, ops, q, u, v, w, dt)
        b.commit(autotune=False)
        b.run(2)
        assert np.array_equal(b.get(i), res[0][1]), dims
        b.close()
