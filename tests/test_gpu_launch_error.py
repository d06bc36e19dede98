"""A launch that fails (into a stream capture that another call has invalidated)
is reported by its own call and by no later one."""
import pytest

import sdg_b200 as sdg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


@pytest.mark.parametrize("p,flags", [(4, 0), (7, 0), (10, 0), (3, sdg.FLAG_EXACT)])
def test_failed_launch_is_reported_once(p, flags):
    import torch
    ops = sdg.read_operators(p)
    mesh = sdg.mesh_setup(3, 2, 3, p, ops.x1D)
    h = sdg.Handle(ops, mesh, flags)
    arrs = [torch.ones(mesh.Np * mesh.NeA, dtype=torch.float64, device="cuda")
            for _ in range(5)]
    h.cal_tend_dev(*arrs)
    h.synchronize()
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        g.capture_begin(capture_error_mode="thread_local")
        with pytest.raises(RuntimeError):
            s.synchronize()                       # not allowed in a capture: ends it
        with pytest.raises(sdg.SdgError) as e:
            h.cal_tend_dev(*arrs, s.cuda_stream)
        assert e.value.code == sdg.SDG_ERR_CUDA
        with pytest.raises(RuntimeError):
            g.capture_end()
    h.update_halo_dev(arrs[1])                    # a valid call on another stream
    h.cal_tend_dev(*arrs)
    h.synchronize()
    h.close()
