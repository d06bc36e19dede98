"""Kernel variants at p = 7, where the automatic one is a warp-per-element kernel:
the block kernels run when they are asked for (they have no waits, so a skipped
copy does not time out), and all give the same bits, single and in a batch."""
import numpy as np
import pytest

import sdg_b200 as sdg

pytestmark = pytest.mark.gpu

P = 7


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


def run(ops, mesh, flags, fields, dt, variant, skip_tile=-1):
    h = sdg.Handle(ops, mesh, flags)
    h.set_kernel_variant(variant)
    h.set_state(*fields)
    if skip_tile >= 0:
        h.inject_wait_timeout(skip_tile, spins=1024)
    h.rk3_steps(dt, 2)
    h.synchronize()
    for stage in (1, 2, 3):
        h.rk3_stage(stage, dt)
    got = h.get_field()
    h.close()
    return got


@pytest.mark.parametrize("flags", [0, sdg.FLAG_MIXED])
@pytest.mark.parametrize("dims", [(1, 1, 1), (4, 3, 5), (37, 4, 1), (37, 20, 1), (19, 39, 1),
                                  (12, 12, 11)])
def test_same_bits(flags, dims):
    ops = sdg.read_operators(P)
    mesh = sdg.mesh_setup(*dims, P, ops.x1D)
    fields = sdg.init_fields(mesh, ic_kind=1, seed=9, vel_kind=1)
    dt = 0.1 / max(dims) / (P + 1) ** 2
    want = run(ops, mesh, flags, fields, dt, sdg.VARIANT_AUTO)
    for variant in (sdg.VARIANT_BLOCK, sdg.VARIANT_BLOCK8):
        assert np.array_equal(run(ops, mesh, flags, fields, dt, variant, 0), want), variant
    for variant in (sdg.VARIANT_PIPE, sdg.VARIANT_SPLIT):
        assert np.array_equal(run(ops, mesh, flags, fields, dt, variant), want), variant


@pytest.mark.parametrize("flags", [0, sdg.FLAG_MIXED])
@pytest.mark.parametrize("name,variant", [("block", sdg.VARIANT_BLOCK),
                                          ("blockocc", sdg.VARIANT_BLOCK8),
                                          ("pipe", sdg.VARIANT_PIPE)])
def test_forced_in_a_batch(flags, name, variant, monkeypatch):
    monkeypatch.setenv("SDG_KERNEL", name)
    ops = sdg.read_operators(P)
    b = sdg.Batch(flags)
    boxes, ids = [(3, 2, 4), (5, 4, 3)], []
    for k, box in enumerate(boxes):
        mesh = sdg.mesh_setup(*box, P, ops.x1D)
        ids.append(b.add(*box, P, ops, *sdg.init_fields(mesh, ic_kind=1, seed=k, vel_kind=1),
                         1e-4))
    b.commit()
    assert [g["variant"] for g in b.info()["groups"]] == [variant]
    b.run(3)
    monkeypatch.delenv("SDG_KERNEL")
    for k, (box, i) in enumerate(zip(boxes, ids)):
        mesh = sdg.mesh_setup(*box, P, ops.x1D)
        h = sdg.Handle(ops, mesh, flags)
        h.set_state(*sdg.init_fields(mesh, ic_kind=1, seed=k, vel_kind=1))
        h.rk3_steps(1e-4, 3)
        assert np.array_equal(b.get(i), h.get_field())
        h.close()
    b.close()
