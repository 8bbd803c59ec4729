"""The staged solve (lines apart: rays traced once into memory, one line's data per tile) against
the general kernel and the oracle, where its tiles end: whole lines per chunk, chunks cut inside
a line, one pair of rays per warp and several, models it does not serve, and pixel rays longer
than the imager's guess.

Bars: J and the ALO diagonal within 1e-5 of the oracle, as every formal solve here.  With its
frequencies in another order a model of several lines takes the general kernel, whose
single-precision physics is the same, so only the eliminations' rounding may differ: 1e-9 covers the roughly 100 rows of a ray at 2^-45 each in
split precision (double-float rows) with room for rows that amplify a hundredfold, and one
differing FP32 rounding in a thick pair would exceed it."""
from dataclasses import replace

import numpy as np
import pytest

import helpers as H
import oracle as O
from magritte_gb300 import _abi
from magritte_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _oracle_with_correctly_rounded_erf():
    O.set_erf_mode(1)
    yield
    O.set_erf_mode(0)


def overlapping(raw):
    """The second line moved onto the first one's wing: the general kernel's model."""
    ld = raw.linedata[0]
    f = np.array(ld.frequency, np.float64)
    f[1] = f[0] * (1.0 + 2.0e-6)
    return replace(raw, linedata=[replace(ld, frequency_given=f)])


def reversed_frequencies(a):
    b = dict(a, nu=np.ascontiguousarray(np.asarray(a["nu"]).reshape(a["npoints"], -1)[:, ::-1]))
    for k in ("corr_line", "corr_lspec", "corr_k", "corr_z", "in_line_integral"):
        b[k] = np.ascontiguousarray(a[k][::-1])
    return b


@pytest.mark.parametrize("nlev,nquads,approx", [
    (2, 5, "None"), (2, 31, "CloseLines"), (2, 32, "CloseLines"), (2, 33, "CloseLines"), (2, 50, "OneLine"),
    (3, 16, "CloseLines"), (3, 17, "OneLine"), (4, 11, "CloseLines"), (6, 5, "CloseLines"), (3, 7, "None"),
    (3, 7, "overlapping"),
])
def test_solve_matches_general_kernel_and_oracle(gpu_lib, nlev, nquads, approx):
    raw = S.grid_sphere(n=9, nside=1, nquads=nquads, nlev=nlev)
    if approx == "overlapping":
        raw, approx = overlapping(raw), "CloseLines"
    a = H.setup(raw, approx=approx)
    ref = O.Oracle(a).formal_solve_fo2()
    has = ref["lambda_has"].astype(bool)
    dev, general = _abi.DeviceModel(a), _abi.DeviceModel(reversed_frequencies(a))
    try:
        for precision in ("fp64", "split"):
            out = dev.formal_solve_fo2(precision, want_u=True)
            assert H.max_rel(out["J"], ref["J"]) < 1e-5, precision
            assert H.max_rel(out["lambda_diag"][has], ref["lambda_diag"][has]) < 1e-5, precision
            u = general.formal_solve_fo2(precision, want_u=True)["u"][:, :, ::-1]
            assert H.max_rel(out["u"], u) < 1e-9, precision
    finally:
        dev.close()
        general.close()


def rod(n=31):
    """A rod along z, 5 x 5 x n points: every ray of the solve leaves it sideways within a few
    steps, a line of sight along it takes n."""
    keep = np.zeros((n, n, n), bool)
    c = n // 2
    keep[c - 2:c + 3, c - 2:c + 3, :] = True
    raw = S.grid_sphere(n=9, nside=1, nquads=5, nlev=3)
    pts, nbs, counts, full = S.grid_neighbors(keep)
    P, b = len(pts), np.nonzero(~full)[0].astype(np.uint32)
    rng = np.random.default_rng(0)
    return replace(
        raw, name="rod", position=pts * 1.0e12, velocity=rng.normal(0.0, 1.0e3, size=(P, 3)) / S.CC, neighbors=nbs,
        n_neighbors=counts, boundary2point=b, boundary_condition=np.full(len(b), S.BC_CMB, np.int32),
        boundary_temperature=np.full(len(b), S.T_CMB), abundance=np.repeat(raw.abundance[:1], P, axis=0),
        temperature=rng.uniform(20.0, 100.0, size=P), vturb2=np.full(P, raw.vturb2[0]))


@pytest.mark.parametrize("model,nfreqs,direction", [
    ("sphere", 1, (0.48, 0.36, 0.8)), ("sphere", 31, (0.48, 0.36, 0.8)), ("sphere", 33, (0.0, 0.0, 1.0)),
    ("sphere", 65, (0.48, 0.36, 0.8)), ("rod", 9, (0.0, 0.0, 1.0)), ("rod", 9, (0.48, 0.36, 0.8)),
])
def test_image_matches_oracle(gpu_lib, model, nfreqs, direction):
    raw = rod() if model == "rod" else S.grid_sphere(n=9, nside=1, nquads=5, nlev=3)
    f0, dd = raw.linedata[0].frequency[1], 8.0e3 / 2.99792458e8
    a = H.setup(raw, image_freqs=(f0 * (1 - dd), f0 * (1 + dd), nfreqs))
    d = np.array(direction)
    ref = O.Oracle(a).image_new(d, 17, 13)
    dev = _abi.DeviceModel(a)
    try:
        for precision in ("fp64", "split"):
            assert H.max_rel(dev.image_new(d, 17, 13, precision)["I"], ref["I"]) < 1e-5, precision
    finally:
        dev.close()
