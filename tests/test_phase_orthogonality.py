"""The limit on |E|, E = Q1^T Q1 - I, up to which a face is decomposed by phases.

The phases keep E to first order: R11 = (I + U) R1 with U the upper triangle of E and half
its diagonal, and the projection Q1 (I - E) Q1^T. What they drop is E^2, times the phase's
first pivot p, the size of its rows. With entries of random sign bounded by the limit,
||E|| and ||U|| stay below 2 sqrt(k) times it, so the dropped terms stay below
4 k p limit^2: within the 4 k u |R_00| that a Householder QR's own error may reach
(u = 1.1e-16) when p limit^2 <= u |R_00|.
"""
import os
import re

import numpy as np
import pytest

HEADER = os.path.join(os.path.dirname(__file__), "..", "hifde3d_b200", "csrc", "hif_kernels.cuh")
U = 1.1e-16


def limit(ratio):
    """of a phase whose first pivot is ratio |R_00|"""
    with open(HEADER) as fh:
        m = re.search(r"constexpr double kPqrMaxE = (\S+), kPqrCapE = (\S+);", fh.read())
    return min(float(m.group(1)) / np.sqrt(ratio), float(m.group(2)))


@pytest.mark.parametrize("ratio", [1.0, 1e-3, 1e-6, 1e-9])
@pytest.mark.parametrize("k", [32, 256])  # 256: the pivots of one phase at most
def test_dropped_terms_at_the_limit(k, ratio):
    rng = np.random.default_rng(k)
    lim = limit(ratio)
    E = np.triu(rng.uniform(-lim, lim, (k, k)))
    E = E + np.triu(E, 1).T
    up = np.triu(E, 1) + 0.5 * np.diag(np.diag(E))
    # (I + U)^T (I + U) = I + E + U^T U
    assert ratio * np.linalg.norm(up.T @ up, 2) < 4 * k * U
    # Q1 = Q (I + E)^{1/2}: Q1 (I - E) Q1^T = Q (I - E^2) Q^T
    assert ratio * np.linalg.norm(E @ E, 2) < 4 * k * U
