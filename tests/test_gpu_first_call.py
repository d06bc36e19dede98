"""A process whose first call is a captured one: rk3_steps on meshes of the
sizes at which an order's automatic variant changes kernels.  Every kernel the
mesh takes is set up by the call without elements that precedes the capture."""
import os
import subprocess
import sys

import pytest

import sdg_b200 as sdg

pytestmark = pytest.mark.gpu

PROGRAM = """
import sys
sys.path.insert(0, sys.argv[1])
import numpy as np
import sdg_b200 as sdg
p, flags, dims = int(sys.argv[2]), int(sys.argv[3]), tuple(map(int, sys.argv[4].split(",")))
ops = sdg.read_operators(p)
mesh = sdg.mesh_setup(*dims, p, ops.x1D)
fields = sdg.init_fields(mesh, ic_kind=1, seed=2, vel_kind=1)
res = []
for variant in (sdg.VARIANT_AUTO, sdg.VARIANT_BLOCK):
    h = sdg.Handle(ops, mesh, flags)
    h.set_kernel_variant(variant)
    h.set_state(*fields)
    h.rk3_steps(1e-5, 25)
    res.append(h.get_field())
    h.close()
assert np.array_equal(*res)
"""


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


@pytest.mark.parametrize("dims", [(3, 2, 2), (11, 9, 7)])
@pytest.mark.parametrize("p,flags", [(15, 0), (11, sdg.FLAG_EXACT), (13, sdg.FLAG_EXACT), (1, 0),
                                     (1, sdg.FLAG_MIXED), (10, 0)])
def test_first_call_is_captured(p, flags, dims):
    root = os.path.dirname(os.path.dirname(os.path.abspath(sdg.__file__)))
    subprocess.run([sys.executable, "-c", PROGRAM, root, str(p), str(flags),
                    ",".join(map(str, dims))], check=True, timeout=300)
