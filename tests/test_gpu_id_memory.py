"""The decomposition by phases holds no more device memory than the row compression of the
column-by-column QR: after two factorizations (the second sizes the workspace by what the
first asked for) a handle's workspace is no larger with the one than with the other.
"""
import numpy as np
import pytest

import hifde3d_b200 as hb
from hifde3d_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,part", [(51, hb.PARTITION_CLIPPED), (63, hb.PARTITION_REFERENCE)])
def test_workspace_no_larger_than_column_by_column(N, part):
    coef = synth.face_coefficients_lognormal(N, 3)
    held = {}
    for phases in (0, 40):
        f = hb.HIFFactor(N, 4, 1e-6, part)
        f.set_option(hb.OPT_ID_MAX_PHASES, phases)
        hb.SetupStencilFaces(f, N, 1.0 / (N + 1), *coef, np.zeros((N + 2,) * 3))
        f.Factor()
        f.Factor()
        assert (f.id_stats()["faces"] > 0) == (phases > 0)
        held[phases] = f.memory()["workspace_bytes"]
        f.close()
    assert held[40] <= held[0]
