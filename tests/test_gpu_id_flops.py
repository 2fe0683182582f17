"""The flops that the profile counts for the column-by-column interpolative decompositions:
4 m n^2 - 4/3 n^3 for a face of m rows and n <= 64 columns, and the same of its triangular
factor (m = n) for a wider one, whose row compression is counted as what it consists of.
Integers up to the division, so equal to the last bits.
"""
import numpy as np
import pytest

import hifde3d_b200 as hb
from hifde3d_b200 import synth

pytestmark = pytest.mark.gpu


def test_id_flops_column_by_column():
    N, P = 31, 4
    f = hb.HIFFactor(N, P, 1e-6)
    f.set_option(hb.OPT_ID_MAX_PHASES, 0)
    coef = synth.face_coefficients_lognormal(N, 3)
    hb.SetupStencilFaces(f, N, 1.0 / (N + 1), *coef, np.zeros((N + 2,) * 3))
    f.set_option(hb.OPT_PROFILE, 1)
    f.Factor()
    counted = f.kernel_stats()["id"]["flops"]
    phase = f.dof_levels()
    f.set_option(hb.OPT_PROFILE, 0)
    expect, narrow, wide = 0.0, 0, 0
    for lev in range(f.num_levels() - 1):
        mask = (phase > 2 * lev).astype(np.uint8)  # left after the level's cells
        c = (N + 1) // (P << lev)
        faces = 0
        for cell in np.ndindex(c, c, c):
            for face in (hb.TOP, hb.FRONT, hb.LEFT):
                rows, cols = hb.partition_face(N, P, lev, cell, face, mask)
                m, n = rows.size, cols.size
                if n == 0:
                    continue
                faces += 1
                if n > 64:
                    m, wide = n, wide + 1
                else:
                    narrow += 1
                expect += 4.0 * m * n * n - 4.0 / 3.0 * n * n * n
        assert faces == f.num_blocks(lev, 1)
    f.close()
    assert narrow > 0 and wide > 0
    assert abs(counted - expect) < 1e-12 * expect
