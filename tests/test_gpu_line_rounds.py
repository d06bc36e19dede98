"""The line kernel over many rounds of tiles per block (p = 1: the barriers'
phases wrap with nothing but the copies between them), single and batched,
FP64 and mixed: the bits of the one-tile-per-block kernel."""
import numpy as np
import pytest

import sdg_b200 as sdg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


@pytest.mark.parametrize("flags", [0, sdg.FLAG_MIXED])
def test_many_rounds_of_tiles(flags):
    # 592 blocks of tiles of 32 (FP64) or 48 elements: 12 to 20 rounds.
    p, dims, steps = 1, (73, 72, 70), 20
    ops = sdg.read_operators(p)
    mesh = sdg.mesh_setup(*dims, p, ops.x1D)
    q, u, v, w = sdg.init_fields(mesh, ic_kind=1, seed=4, vel_kind=1)
    dt = 0.1 / max(dims) / (p + 1) ** 2
    res = []
    for variant in (sdg.VARIANT_AUTO, sdg.VARIANT_BLOCK):
        h = sdg.Handle(ops, mesh, flags)
        h.set_kernel_variant(variant)
        h.set_state(q, u, v, w)
        h.rk3_steps(dt, steps)
        res.append(h.get_field())
        h.close()
    assert np.array_equal(res[0], res[1])
    b = sdg.Batch(flags)
    small = sdg.mesh_setup(3, 2, 2, p, ops.x1D)
    fs = sdg.init_fields(small, ic_kind=1, seed=3, vel_kind=1)
    for _ in range(3):
        b.add(3, 2, 2, p, ops, *fs, 1e-4)
    i = b.add(*dims, p, ops, q, u, v, w, dt)
    b.commit(autotune=False)
    b.run(steps)
    assert np.array_equal(b.get(i), res[0])
    b.close()
