"""3-D grids around 80 points per axis, where the FFT passes take over from the
plain transforms, with the checks and bars of the repulsion modes' test."""
import pytest

import test_repulsion_modes as modes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ng", [(3000, 76), (3000, 78), (3000, 80), (20000, 96)])
def test_large_3d_grids_against_oracle(n, ng):
    modes.test_modes_against_oracle(3, n, ng)
