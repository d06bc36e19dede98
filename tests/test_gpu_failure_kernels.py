"""Failure detection in the line and warp-per-element kernels, as in
test_gpu_failure.py: a tile left without copies makes its wait run out at a small
poll limit, the block drains what is in flight and leaves, and the next
synchronising call reports it; the handle works again afterwards.  Tiles of a
block's first and of a later round, single and batched."""
import numpy as np
import pytest

import sdg_b200 as sdg

pytestmark = pytest.mark.gpu

MIXED, EXACT = sdg.FLAG_MIXED, sdg.FLAG_EXACT
# (p, flags, box, tiles to skip), on 148 SMs.
LINE = [(1, 0, (40, 32, 25), (5, 700)), (1, MIXED, (40, 32, 25), (5, 600)),
        (9, 0, (13, 12, 11), (5, 500)), (11, 0, (9, 8, 7), (3, 200)),
        (12, EXACT, (9, 8, 7), (3, 200)), (15, 0, (9, 9, 8), (0, 500))]
WARP = [(7, 0, (4, 4, 4), (0, 40)), (7, 0, (7, 6, 6), (5, 30)), (7, 0, (13, 12, 11), (3, 200)),
        (7, MIXED, (8, 8, 7), (0, 100)), (7, MIXED, (22, 22, 20), (3, 500))]
# Forms that only single stages take: two elements a tile, three, four (two rounds).
STAGES = [(7, 0, (7, 6, 6), (5, 100)), (7, 0, (8, 7, 7), (2, 100)), (7, 0, (12, 12, 8), (3, 200)),
          (9, 0, (9, 8, 7), (3, 200)), (1, 0, (20, 20, 16), (3, 150))]


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


def block_result(ops, mesh, flags, fields, dt, steps):
    h = sdg.Handle(ops, mesh, flags)
    h.set_kernel_variant(sdg.VARIANT_BLOCK)
    h.set_state(*fields)
    h.rk3_steps(dt, steps)
    got = h.get_field()
    h.close()
    return got


@pytest.mark.parametrize("p,flags,box,tiles", LINE + WARP)
def test_handle(p, flags, box, tiles):
    ops = sdg.read_operators(p)
    mesh = sdg.mesh_setup(*box, p, ops.x1D)
    fields = sdg.init_fields(mesh, ic_kind=1, seed=3, vel_kind=1)
    dt = 0.1 / max(box) / (p + 1) ** 2
    h = sdg.Handle(ops, mesh, flags)
    for tile in tiles:
        h.set_state(*fields)
        h.inject_wait_timeout(tile, spins=2048)
        h.rk3_steps(dt, 1)
        with pytest.raises(sdg.SdgError) as e:
            h.synchronize()
        assert e.value.code == sdg.SDG_ERR_CUDA and "timed out" in str(e.value)
        h.synchronize()                  # the status word was cleared
        h.inject_wait_timeout(-1)
        h.set_state(*fields)
        h.rk3_steps(dt, 2)
        assert np.array_equal(h.get_field(), block_result(ops, mesh, flags, fields, dt, 2)), tile
    h.close()


@pytest.mark.parametrize("p,flags,box,tiles", STAGES)
def test_single_stage(p, flags, box, tiles):
    ops = sdg.read_operators(p)
    mesh = sdg.mesh_setup(*box, p, ops.x1D)
    fields = sdg.init_fields(mesh, ic_kind=1, seed=3, vel_kind=1)
    dt = 0.1 / max(box) / (p + 1) ** 2
    h = sdg.Handle(ops, mesh, flags)
    for tile in tiles:
        h.set_state(*fields)
        h.inject_wait_timeout(tile, spins=2048)
        h.rk3_stage(1, dt)
        with pytest.raises(sdg.SdgError) as e:
            h.synchronize()
        assert e.value.code == sdg.SDG_ERR_CUDA and "timed out" in str(e.value)
        h.inject_wait_timeout(-1)
        h.set_state(*fields)
        for stage in (1, 2, 3):
            h.rk3_stage(stage, dt)
        assert np.array_equal(h.get_field(), block_result(ops, mesh, flags, fields, dt, 1)), tile
    h.close()


@pytest.mark.parametrize("p,flags,box,tiles", [
    (1, 0, (40, 32, 25), (5, 700)), (1, MIXED, (40, 32, 25), (5, 600)),
    (9, 0, (9, 9, 8), (5, 300)), (12, EXACT, (9, 8, 7), (3, 200)),
    (7, 0, (13, 12, 11), (3, 200)), (7, MIXED, (16, 16, 11), (3, 200))])
def test_batch(p, flags, box, tiles):
    ops = sdg.read_operators(p)
    small = (3, 2, 2)
    cases = []
    for k, bx in enumerate((small, box)):
        mesh = sdg.mesh_setup(*bx, p, ops.x1D)
        cases.append((bx, mesh, sdg.init_fields(mesh, ic_kind=1, seed=3 + k, vel_kind=1),
                      0.1 / max(bx) / (p + 1) ** 2))

    def make():
        b = sdg.Batch(flags)
        for bx, _, f, dt in cases:
            b.add(*bx, p, ops, *f, dt)
        b.commit(autotune=False)
        return b

    b = make()
    for tile in tiles:
        b.inject_wait_timeout(tile, spins=2048)
        with pytest.raises(sdg.SdgError) as e:
            b.run(1)
        assert e.value.code == sdg.SDG_ERR_CUDA and "timed out" in str(e.value)
        b.inject_wait_timeout(-1)
        b.run(1)                         # runs clean again (its state is now stale)
    b.close()
    b = make()
    b.run(2)
    for i, (bx, mesh, f, dt) in enumerate(cases):
        assert np.array_equal(b.get(i), block_result(ops, mesh, flags, f, dt, 2)), bx
    b.close()
