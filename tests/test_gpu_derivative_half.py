"""The derivative operators whose y-lines bypass shared memory, against the
other kernel of the same arithmetic (which a call whose output shares memory
with its input takes): the same bits, at unit counts around a block's."""
import pytest

import sdg_b200 as sdg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


@pytest.mark.parametrize("p", [1, 2, 4, 5, 6, 7, 8, 14, 15])
@pytest.mark.parametrize("ne", [1, 3, 37, 150])
def test_same_bits_as_with_shared_memory(p, ne):
    import torch
    D = sdg.read_operators(p).D1D
    np_ = (p + 1) ** 3
    g = torch.Generator(device="cuda").manual_seed(p)
    for nvar in (0, 5):
        n = ne * np_ * max(1, nvar)
        ins = [torch.randn(n, generator=g, device="cuda", dtype=torch.float64) for _ in range(3)]
        outs = [torch.zeros(n, device="cuda", dtype=torch.float64) for _ in range(3)]
        # In place (each output over the input of its own direction).
        same = [x.clone() for x in ins]
        if nvar:
            sdg.divlike_dirXYZ_var_dev(D, nvar, ne, *ins, *outs)
            sdg.divlike_dirXYZ_var_dev(D, nvar, ne, *same, *same)
        else:
            other = [torch.zeros_like(ins[0]) for _ in range(2)]
            sdg.gradlike_dirXYZ_dev(D, ne, ins[0], *outs)
            sdg.gradlike_dirXYZ_dev(D, ne, same[0], same[0], *other)
            same = [same[0], *other]
        torch.cuda.synchronize()
        for a, b in zip(outs, same):
            assert torch.equal(a, b), (p, ne, nvar)
