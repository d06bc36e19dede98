"""sdg_batch_info lists the tuned time of every kernel the autotuner timed, the
line kernel's too: the chosen variant of each group has one."""
import pytest

import sdg_b200 as sdg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


@pytest.mark.parametrize("flags", [0, sdg.FLAG_MIXED, sdg.FLAG_EXACT])
def test_every_chosen_kernel_has_a_time(flags):
    b = sdg.Batch(flags)
    for p in (1, 3, 7, 9, 11):
        ops = sdg.read_operators(p)
        mesh = sdg.mesh_setup(6, 5, 4, p, ops.x1D)
        b.add(6, 5, 4, p, ops, *sdg.init_fields(mesh, ic_kind=1, seed=p, vel_kind=1), 1e-5)
    b.commit()
    key = {1: "ms_block", 2: "ms_pipe", 3: "ms_block8", 4: "ms_split", 6: "ms_line"}
    groups = b.info()["groups"]
    b.close()
    assert [g["p"] for g in groups] == [1, 3, 7, 9, 11]
    for g in groups:
        times = {k: g[k] for k in key.values()}
        assert times[key[g["variant"]]] > 0.0, g
        line = g["p"] in {0: (1, 9, 11), sdg.FLAG_MIXED: (1,), sdg.FLAG_EXACT: (11,)}[flags]
        assert (g["ms_line"] > 0.0) == line, g
