"""Faces that the decomposition by phases does not take (FP64 interpolative decomposition
of faces wider than 64 columns): they are assembled again and decomposed column by
column, the other faces of the level by phases.

The reasons are each met once: more phases than HIF_OPT_ID_MAX_PHASES allows (all faces
of a level, or some of them), and kept columns that are not a prefix of the pivot order
(two tied norms on either side of the rank test). A face whose rest is exactly zero is
taken. Skeletons are those of the column-by-column QR; where every face takes that route
the factor is the same bit for bit, and elsewhere the two agree as the parity tests ask
(1e-9), for W differs by n u / eps.
"""
import numpy as np
import pytest

import hifde3d_b200 as hb
from hifde3d_b200 import synth

pytestmark = pytest.mark.gpu


def build(N, P, eps, part, coef, V, options=()):
    f = hb.HIFFactor(N, P, eps, part)
    for o, v in options:
        f.set_option(o, v)
    hb.SetupStencilFaces(f, N, 1.0 / (N + 1), *coef, V)
    f.Factor()
    return f


def skeletons(f):
    return [f.block(lev, 1, b)["skel"].tolist() for lev in range(f.num_levels() - 1)
            for b in range(f.num_blocks(lev, 1))]


def inverse(f):
    return f.Apply(synth.dof_vector(f.N(), 1), True)


COLUMNS = [(hb.OPT_ID_MAX_PHASES, 0)]


def test_no_face_goes_back_on_ordinary_fields():
    N = 31
    V = np.full((N + 2,) * 3, 1e-2)
    for coef, eps in [(synth.face_coefficients_grf(N, 2, ell=1.0 / 8, sigma=1.0), 1e-6),
                      (synth.face_coefficients_blocks(N, 1), 1e-8)]:
        f = build(N, 4, eps, hb.PARTITION_REFERENCE, coef, V)
        s = f.id_stats()
        assert s["faces"] > 0 and s["phases"] > 0 and s["column_by_column"] == 0
        f.close()


@pytest.mark.parametrize("N,part", [(31, hb.PARTITION_REFERENCE), (27, hb.PARTITION_CLIPPED)])
def test_more_phases_than_allowed(N, part):
    coef = synth.face_coefficients_lognormal(N, 3)
    V = np.zeros((N + 2,) * 3)
    eps = 1e-6
    ref = build(N, 4, eps, part, coef, V, COLUMNS)
    assert ref.id_stats() == {"phases": 0, "faces": 0, "column_by_column": 0}
    sk, x = skeletons(ref), inverse(ref)
    ref.close()
    seen = []
    for limit in range(1, 40):
        f = build(N, 4, eps, part, coef, V, [(hb.OPT_ID_MAX_PHASES, limit)])
        s = f.id_stats()
        seen.append(s["column_by_column"])
        assert skeletons(f) == sk
        y = inverse(f)
        if s["column_by_column"] == s["faces"]:
            np.testing.assert_array_equal(y, x)
        assert np.linalg.norm(y - x) < 1e-9 * np.linalg.norm(x)
        faces = s["faces"]
        f.close()
        if seen[-1] == 0:
            break
    assert seen[0] == faces and seen[-1] == 0
    if part == hb.PARTITION_CLIPPED:  # ragged faces: some need more phases than others
        assert any(0 < b < faces for b in seen)


def test_option_order():
    """The group option selects the column-by-column QR, the phase option the phases
    again; what either refuses leaves the choice as it was."""
    N = 31
    coef = synth.face_coefficients_grf(N, 2, ell=1.0 / 8, sigma=1.0)
    f = hb.HIFFactor(N, 4, 1e-6)
    hb.SetupStencilFaces(f, N, 1.0 / (N + 1), *coef, np.zeros((N + 2,) * 3))
    for opt, value, by_phases in [(hb.OPT_ID_GROUP_MIN_N, 512, False),
                                  (hb.OPT_ID_MAX_PHASES, 40, True),
                                  (hb.OPT_ID_MAX_PHASES, 0, False)]:
        f.set_option(opt, value)
        f.Factor()
        assert (f.id_stats()["faces"] > 0) == by_phases
    for opt, value in [(hb.OPT_ID_MAX_PHASES, -1), (hb.OPT_ID_GROUP_MIN_N, 1)]:
        with pytest.raises(hb.HIFError) as e:
            f.set_option(opt, value)
        assert e.value.code == hb.HIF_ERR_ARG
    f.close()


def test_kept_columns_not_a_prefix():
    """Slabs of equal coefficients, cut off from one another: a face across two of them has
    its columns in mirrored, mutually orthogonal pairs of one norm, so R's diagonal is not
    monotone in its last bits, and a rank test between the two entries of a pair keeps the
    second and not the first. P = 16: the wide faces come first, and their blocks do not
    depend on eps."""
    N, P = 31, 16
    coef = [np.ones((N + 2,) * 3) for _ in range(3)]
    for j in (0, 7, 8, 15, 16, 23, 24, 31):
        coef[1][:, j, :] = 0.0
    V = np.ones((N + 2,) * 3)
    f = build(N, P, 1e-10, hb.PARTITION_REFERENCE, coef, V)
    rd = [np.abs(f.pivots(0, b)[1]) for b in range(f.num_blocks(0, 1))]
    assert f.id_stats()["faces"] == len(rd) and rd[0].size == 225
    f.close()
    found = []
    for r in rd:
        for i in np.nonzero(r[:-1] < r[1:])[0]:
            e = r[i] / r[0]
            if e > 1e-9 and r[i] <= r[0] * e < r[i + 1]:
                found.append(float(e))
    assert found
    eps = max(found)
    out = []
    for options in ((), COLUMNS):
        g = build(N, P, eps, hb.PARTITION_REFERENCE, coef, V, options)
        out.append((g.id_stats(), inverse(g)))
        g.close()
    assert 0 < out[0][0]["column_by_column"] <= out[0][0]["faces"]
    # the rank tests of the two routes see norms that differ in their last bits: the
    # skeletons may differ by the tied column, the factors by what eps leaves out
    assert np.linalg.norm(out[0][1] - out[1][1]) < 1e2 * eps * np.linalg.norm(out[1][1])


def test_exactly_zero_rest():
    """DOFs cut off from all others have zero columns in their faces' blocks: the rest of
    such a face is exactly zero once its other columns are picked."""
    N = 31
    coef = [a.copy() for a in synth.face_coefficients_grf(N, 2, ell=1.0 / 8, sigma=1.0)]
    for a in coef:
        a[18:26, 12:20, 12:20] = 0.0
    V = np.ones((N + 2,) * 3)
    out = []
    for options in ((), COLUMNS):
        f = build(N, 4, 1e-6, hb.PARTITION_REFERENCE, coef, V, options)
        out.append((skeletons(f), inverse(f), f.id_stats()))
        f.close()
    assert out[0][2]["faces"] > 0 and out[0][2]["column_by_column"] == 0
    assert [set(s) for s in out[0][0]] == [set(s) for s in out[1][0]]
    assert np.linalg.norm(out[0][1] - out[1][1]) < 1e-9 * np.linalg.norm(out[1][1])
