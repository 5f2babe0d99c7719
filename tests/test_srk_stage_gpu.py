"""The fused stage pass of the SRK step at the widths its dispatch takes apart: NX a multiple
of four (16-byte accesses) and only of two (8-byte accesses in float), an x-extent of one
partial block, of exactly one and of one and a remainder, and one with rows left over in y,
against the oracle with the bounds of test_srk_gpu."""
import pytest

from test_srk_gpu import _srk_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nx,ny", [(54, 18), (64, 16), (128, 12), (162, 8)])
def test_stage_pass_widths(nx, ny, precision):
    _srk_case("ARS_343", 1, precision, nx, ny, 9)


@pytest.mark.parametrize("precision", [0, 1])
def test_stage_pass_without_stabilisation(precision):
    _srk_case("ARS_343", 0, precision, 54, 18, 9)
