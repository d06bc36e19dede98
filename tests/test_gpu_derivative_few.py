"""Unit counts around which the derivative operators change between two builds of
their kernel (p = 11 two units an SM, p = 13 one; 148 SMs): both give the bits of
plain contractions in the same order, elementwise what a larger call gives."""
import pytest

import sdg_b200 as sdg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


@pytest.mark.parametrize("p,few", [(11, 296), (13, 148)])
@pytest.mark.parametrize("nvar", [0, 1])
def test_few_units_equal_their_part_of_many(p, few, nvar):
    import torch
    D = sdg.read_operators(p).D1D
    np_ = (p + 1) ** 3
    g = torch.Generator(device="cuda").manual_seed(p)
    many = 2 * few + 3
    ins = [torch.randn(many * np_, generator=g, device="cuda", dtype=torch.float64)
           for _ in range(3)]

    def run(ne):
        part = [x[: ne * np_].clone() for x in ins]
        outs = [torch.zeros_like(part[0]) for _ in range(3)]
        if nvar:
            sdg.divlike_dirXYZ_var_dev(D, nvar, ne, *part, *outs)
        else:
            sdg.gradlike_dirXYZ_dev(D, ne, part[0], *outs)
        torch.cuda.synchronize()
        return outs

    whole = run(many)
    for ne in (1, few - 1, few, few + 1):
        for a, b in zip(run(ne), whole):
            assert torch.equal(a, b[: ne * np_]), ne
