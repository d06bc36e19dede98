"""The warp-per-element kernels (p = 7: fast FP64, sdg_tend_warp.cuh, and the
mixed form, sdg_tend_warp32.cuh) where their tiling can go wrong: one element,
the element counts around the changes of form (148, 149, 444 and 445 elements
on 148 SMs; mixed 740 and 741), partial last tiles, halo and direct neighbours,
and arrays that are not 16-byte aligned."""
import numpy as np
import pytest

import orc
import sdg_b200 as sdg
from conftest import rel_maxnorm

pytestmark = pytest.mark.gpu

TOL = 1e-12   # the fast FP64 form's bar against the oracle
P = 7


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 2, 2), (37, 2, 2), (149, 1, 1), (12, 37, 1),
                                  (89, 5, 1), (61, 17, 1)])
def test_sizes_and_alignment(dims):
    import torch
    ops = sdg.read_operators(P)
    mesh = sdg.mesh_setup(*dims, P, ops.x1D)
    omesh = orc.mesh_setup(*dims, P, ops.x1D)
    q, u, v, w = sdg.init_fields(mesh, ic_kind=1, seed=9, vel_kind=1)
    h = sdg.Handle(ops, mesh, 0)
    ref = orc.cal_tend(orc.OPT1, q, u, v, w, ops, omesh)[:, : mesh.Ne]

    # The tendency reads its halo: aligned arrays (bulk copies), then arrays
    # that start at an odd word (plain loads): the same bits.
    n, full = mesh.Np * mesh.Ne, mesh.Np * mesh.NeA
    got = []
    for shift in (0, 1):
        arrs = [torch.zeros(full + shift, dtype=torch.float64, device="cuda")[shift:]
                for _ in range(5)]
        for a, f in zip(arrs[1:], (q, u, v, w)):
            a.copy_(torch.from_numpy(f.reshape(-1, order="F").copy()))
        torch.cuda.synchronize()
        h.cal_tend_dev(*arrs)
        h.synchronize()
        got.append(arrs[0][:n].cpu().numpy().reshape(mesh.Np, mesh.Ne, order="F"))
    assert rel_maxnorm(got[0], ref) <= TOL
    assert np.array_equal(got[0], got[1])

    # RK steps read their periodic neighbours directly.
    dt = 0.1 / max(dims) / (P + 1) ** 2
    h.set_state(q, u, v, w)
    h.rk3_steps(dt, 2)
    qo = q.copy(order="F")
    orc.run_rk3(orc.OPT1, qo, u, v, w, ops, omesh, dt, 2)
    single = h.get_field()
    h.close()
    assert rel_maxnorm(single, qo[:, : mesh.Ne]) <= TOL

    # A batch of this box and a smaller one (tiles of both in one launch).
    b = sdg.Batch(0)
    small = sdg.mesh_setup(2, 2, 1, P, ops.x1D)
    b.add(2, 2, 1, P, ops, *sdg.init_fields(small, ic_kind=1, seed=3, vel_kind=1), 1e-4)
    i = b.add(*dims, P, ops, q, u, v, w, dt)
    b.commit()
    b.run(2)
    assert np.array_equal(b.get(i), single)
    b.close()


@pytest.mark.parametrize("dims", [(1, 1, 1), (5, 3, 1), (37, 20, 1), (19, 39, 1), (149, 11, 1)])
def test_mixed_sizes(dims):
    ops = sdg.read_operators(P)
    mesh = sdg.mesh_setup(*dims, P, ops.x1D)
    omesh = orc.mesh_setup(*dims, P, ops.x1D)
    q, u, v, w = sdg.init_fields(mesh, ic_kind=1, seed=9, vel_kind=1)
    dt = 0.1 / max(dims) / (P + 1) ** 2
    h = sdg.Handle(ops, mesh, sdg.FLAG_MIXED)
    h.set_state(q, u, v, w)
    h.rk3_steps(dt, 3)
    single = h.get_field()
    h.close()
    qo = q.copy(order="F")
    orc.run_rk3(orc.OPT1, qo, u, v, w, ops, omesh, dt, 3)
    ref = qo[:, : mesh.Ne]
    assert np.linalg.norm(single - ref) <= 1e-5 * np.linalg.norm(ref)   # the mixed form's bar

    # The batch always runs one warp per element: the same bits.
    b = sdg.Batch(sdg.FLAG_MIXED)
    i = b.add(*dims, P, ops, q, u, v, w, dt)
    b.commit()
    b.run(3)
    assert np.array_equal(b.get(i), single)
    b.close()
