"""Several handles stepped in turn without waiting, whose kernels share the GPU:
each ends with the bits of a handle alone, at sizes at which their launches
overlap."""
import numpy as np
import pytest

import sdg_b200 as sdg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


@pytest.mark.parametrize("p,flags,box", [
    (1, 0, (17, 14, 17)), (1, sdg.FLAG_MIXED, (20, 20, 20)), (7, 0, (3, 4, 5)), (7, 0, (5, 5, 5)),
    (7, 0, (9, 9, 8)), (7, sdg.FLAG_MIXED, (7, 7, 7)), (7, sdg.FLAG_MIXED, (24, 20, 20)),
    (2, 0, (36, 30, 25)), (4, sdg.FLAG_MIXED, (18, 17, 15)), (10, 0, (5, 5, 5))])
def test_side_by_side(p, flags, box):
    ops = sdg.read_operators(p)
    mesh = sdg.mesh_setup(*box, p, ops.x1D)
    dt = 0.1 / max(box) / (p + 1) ** 2
    fields = [sdg.init_fields(mesh, ic_kind=1, seed=s, vel_kind=1) for s in (1, 2, 3)]

    def handle(f):
        h = sdg.Handle(ops, mesh, flags)
        h.set_state(*f)
        return h

    want = []
    for f in fields:
        h = handle(f)
        h.set_kernel_variant(sdg.VARIANT_BLOCK)
        h.rk3_steps(dt, 6)
        want.append(h.get_field())
        h.close()
    hs = [handle(f) for f in fields]
    for _ in range(3):
        for h in hs:
            h.rk3_steps(dt, 2)
    for h, w in zip(hs, want):
        assert np.array_equal(h.get_field(), w)
        h.close()
