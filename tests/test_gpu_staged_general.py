"""The staged solve against the general kernel on the same ray pairs: a model of several lines with
its frequencies in reverse order takes the general kernel.

Bar: 1e-9 of each element of u.  The two take the same single-precision physics, and their rows
differ by their roundings, 2^-45 and 2^-46 a row over some hundred rows, with room for rows that
amplify a hundredfold; one single-precision rounding that differs is 6e-8."""
from dataclasses import replace

import numpy as np
import pytest

import helpers as H
from magritte_gb300 import _abi
from magritte_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


def in_reverse(a):
    b = dict(a, nu=np.ascontiguousarray(np.asarray(a["nu"]).reshape(a["npoints"], -1)[:, ::-1]))
    for k in ("corr_line", "corr_lspec", "corr_k", "corr_z", "in_line_integral"):
        b[k] = np.ascontiguousarray(a[k][::-1])
    return b


def assert_same_u(a, bar=1e-9, precisions=("split",)):
    dev, general = _abi.DeviceModel(a), _abi.DeviceModel(in_reverse(a))
    try:
        for precision in precisions:
            u = dev.formal_solve_fo2(precision, want_u=True)["u"]
            g = general.formal_solve_fo2(precision, want_u=True)["u"][:, :, ::-1]
            assert H.max_rel(u, g) < bar, precision
    finally:
        dev.close()
        general.close()


@pytest.mark.parametrize("reach,seed", [(1.5, 0), (2.0, 1), (3.0, 2), (10.0, 3)])
def test_edge_of_a_lines_reach(gpu_lib, reach, seed):
    """max_distance_opacity_contribution widths: at 1.5 to 3 a pair whose line is dropped at the
    edge of its reach shows in u, and with 1e8 pairs some ten lie at the edge's rounding."""
    raw = S.batch_model(npoints=4000, nside=2, nlev=5, nquads=31, seed=seed)
    assert_same_u(H.setup(raw, max_distance_opacity_contribution=reach))


def test_boundary_intensities_fp64(gpu_lib):
    """A transparent model at rest: u is the mean of the boundary intensities the two halves start
    from.  At most three rows a half, each with four roundings of 2^-53 in either kernel, and the
    combination's: below 6e-15.  Intensities formed in double-float are off by up to 3e-14 (mean
    3e-15), and by 6e-8 where their exponent rounds to another float."""
    raw = S.batch_model(npoints=65, nside=2, nlev=5, nquads=31)
    raw = replace(raw, abundance=raw.abundance * np.array([1.0e-20, 1.0]), velocity=np.zeros_like(raw.velocity))
    assert_same_u(H.setup(raw), 6e-15, ("fp64",))
