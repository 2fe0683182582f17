"""Pivoted QR of the wide faces by phases (FP64 interpolative decomposition) against
the oracle's geqp3 on the same operator.

Sizes where the scheme can go wrong: faces just above its width limit and ragged ones
(clipped partitions), a rank of a few columns (eps = 0.3: one phase decides it), a rank
near the width (eps = 1e-11: every phase contributes), a contrast of 10^6,
and the non-symmetric operator.

Tolerances. R carries a backward error of a few u = 1.1e-16 times ||M||, so the
interpolation matrix W = R11^{-1} R12 carries about n u / eps of both sides: with n <=
225 columns, eps >= 1e-11 and the entries of W of order one, 10 n u / eps relative
bounds their difference (capped below by 1e-12, above by 0.5). Pivots are compared up to
the rank; a tie of two norms within rounding has not been met in these fields.
"""
import numpy as np
import pytest

import hifde3d_b200 as hb
from hifde3d_b200 import synth
from oracle import hif_oracle as ho

pytestmark = pytest.mark.gpu

U = 1.1e-16


@pytest.mark.parametrize("N,part,field,eps", [
    (31, "reference", "grf", 0.3),
    (31, "reference", "grf", 1e-6),
    (31, "reference", "grf", 1e-11),
    (31, "reference", "blocks", 1e-8),
    (31, "reference", "node", 1e-6),
    (19, "clipped", "lognormal", 1e-6),
    (27, "clipped", "lognormal", 1e-4),
])
def test_wide_faces_match_oracle(N, part, field, eps):
    NC = N + 1
    f = hb.HIFFactor(N, 4, eps,
                     hb.PARTITION_CLIPPED if part == "clipped" else hb.PARTITION_REFERENCE)
    if field == "node":
        A, V = synth.node_lognormal(N, 1, sigma=0.5, vscale=0.1)
        op = ho.setup_stencil(N, 1.0 / NC, A, V)
        hb.SetupStencil(f, N, 1.0 / NC, A, V)
    else:
        V = np.full((NC + 1,) * 3, 1e-2 if field == "blocks" else 0.0)
        if field == "grf":
            a = synth.face_coefficients_grf(N, 2, ell=1.0 / 8, sigma=1.0)
        elif field == "blocks":
            a = synth.face_coefficients_blocks(N, 1)
        else:
            a = synth.face_coefficients_lognormal(N, 3)
        op = ho.setup_stencil_faces(N, 1.0 / NC, *a, V)
        hb.SetupStencilFaces(f, N, 1.0 / NC, *a, V)
    fo = ho.HIFOracle(N, 4, eps, partition=part)
    fo.set_matrix(op)
    fo.initialize()
    fo.factor()
    f.Factor()
    wide = 0
    for lev in range(fo.L - 1):
        for b, ob in enumerate(fo.skel_levels[lev]):
            ours = f.block(lev, 1, b, matrices=True)
            n = ob.global_inds.size
            np.testing.assert_array_equal(ours["global"], ob.global_inds)
            assert set(ours["skel"].tolist()) == set(ob.skel.tolist()), (lev, b)
            if n <= 64:
                continue
            wide += 1
            k = ours["skel"].size
            jp, rd = f.pivots(lev, b)
            np.testing.assert_array_equal(jp[:k], ours["skel"])
            assert sorted(jp.tolist()) == list(range(n))
            assert np.all(np.abs(rd[:k]) > eps * abs(rd[0]))
            assert not np.any(np.abs(rd[k:]) > eps * abs(rd[0]))
            # pivots in the same order, W by redundant column
            np.testing.assert_array_equal(ours["skel"], ob.skel)
            if 0 < k < n:
                col = {int(c): q for q, c in enumerate(ob.red)}
                W = ob.W[:, [col[int(c)] for c in ours["red"]]]
                err = np.linalg.norm(ours["W"] - W) / np.linalg.norm(W)
                assert err < min(0.5, max(1e-12, 10 * n * U / eps)), (lev, b, err)
    assert wide > 0
    f.close()


@pytest.mark.parametrize("prec,eps", [(hb.PRECISION_FP64, 1e-6), (hb.PRECISION_MIXED, 1e-8)])
def test_phases_match_column_by_column(prec, eps):
    """The widest faces (n = 96: up to about 1600 columns, split over a cluster of CTAs)
    by phases against the column-by-column QR of the same faces, selected by
    HIF_OPT_ID_GROUP_MIN_N: the same skeletons and, with them, the same operator to the
    bar of the parity tests (1e-9; in mixed precision the two factors differ by rounding
    in what the int8 slices truncate: the mixed factor's own 1e-5)."""
    n = 96
    N = n - 1
    a = synth.face_coefficients_lognormal(N, 5)
    V = np.zeros((n + 1,) * 3)
    u = synth.dof_vector(N, 1)
    out, skel = [], []
    for group in (0, 512):
        f = hb.HIFFactor(N, 4, eps, hb.PARTITION_CLIPPED)
        f.set_option(hb.OPT_PRECISION, prec)
        if group:
            f.set_option(hb.OPT_ID_GROUP_MIN_N, group)
        hb.SetupStencilFaces(f, N, 1.0 / n, *a, V)
        f.Factor()
        out.append(f.Apply(u.copy(), True))
        widest = 0
        sk = []
        for lev in range(2, f.num_levels() - 1):
            for b in range(f.num_blocks(lev, 1)):
                blk = f.block(lev, 1, b)
                widest = max(widest, blk["global"].size)
                sk.append(set(blk["skel"].tolist()))
        assert widest > 832
        skel.append(sk)
        f.close()
    if prec == hb.PRECISION_FP64:
        assert skel[0] == skel[1]
    bar = 1e-9 if prec == hb.PRECISION_FP64 else 1e-5
    assert np.linalg.norm(out[0] - out[1]) < bar * np.linalg.norm(out[1])
