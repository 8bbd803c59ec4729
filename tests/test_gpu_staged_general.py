"""The staged solve against the general kernel on the same ray pairs: a model of several lines with
its frequencies in reverse order takes the general kernel.

Bar: 1e-9 of each element of u.  The two take the same single-precision physics, and their rows
differ by their roundings, 2^-45 and 2^-46 a row over some hundred rows, with room for rows that
amplify a hundredfold; one single-precision rounding that differs is 6e-8."""
import ctypes as C
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


def with_velocity(a, velocity):
    """The model of arrays `a` given other velocities after its creation."""
    torch = pytest.importorskip("torch")
    dev = _abi.DeviceModel(a)
    v = torch.tensor(np.ascontiguousarray(velocity), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    _abi._check(_abi.load().mgr_model_set_velocity_device(dev.h, C.c_void_p(v.data_ptr())))
    dev.sync()
    return dev


def close_lines(nside=1, nquads=11, seed=0, npoints=1200):
    """Arrays of a model whose two lines lie 30 km/s apart, at rest nearly (0.3 km/s) and with 50
    times the velocities: at rest no pair reaches both lines, with the velocities many do, and a
    model created with them is the general kernel's."""
    raw = S.batch_model(npoints=npoints, nside=nside, nlev=3, nquads=nquads, seed=seed, sigma_v=0.3e3)
    ld = raw.linedata[0]
    f = np.array(ld.frequency, np.float64)
    f[1] = f[0] * (1.0 + 1.0e-4)
    raw = replace(raw, linedata=[replace(ld, frequency_given=f)])
    return H.setup(raw), H.setup(replace(raw, velocity=50.0 * raw.velocity))


def taken(dev):
    return dev.staged_statistics()[0]


def assert_same_u(a, bar=1e-9, precisions=("split",)):
    dev, general = _abi.DeviceModel(a), _abi.DeviceModel(in_reverse(a))
    try:
        for precision in precisions:
            u = dev.formal_solve_fo2(precision, want_u=True)["u"]
            assert taken(dev) == dev.P * dev.R
            g = general.formal_solve_fo2(precision, want_u=True)["u"][:, :, ::-1]
            assert taken(general) == 0
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


@pytest.mark.parametrize("seed", range(4))
def test_edge_of_an_elements_reach(gpu_lib, seed):
    """The same for the pairs of the trapezoid rule, whose elements decide by themselves: two of
    these four models have a line at the edge's rounding that shows."""
    raw = S.batch_model(npoints=6000, nside=2, nlev=5, nquads=31, seed=seed)
    assert_same_u(H.setup(raw, max_distance_opacity_contribution=1.5))


@pytest.mark.parametrize("nquads,approx", [(1, "None"), (5, "None"), (16, "OneLine"), (31, "CloseLines"),
                                           (32, "CloseLines"), (33, "CloseLines"), (50, "OneLine")])
def test_one_line(gpu_lib, nquads, approx):
    """The reverse order of one line's frequencies is its own, so the general kernel here is the
    (u, v) solve's, which is never staged.  Its origin row takes FP64 quotients where the other's
    has single-precision coefficients (three roundings of 2^-24 and one of 2^-22): 1e-6 in split
    precision.  FP64: the two positions' errors of 2^-53 line / width = 2e-10 on differences of
    0.35 and more, 1e-9 a pair, ten pairs alike: 1e-8."""
    raw = S.batch_model(npoints=1000, nside=1, nlev=2, nquads=nquads)
    dev = _abi.DeviceModel(H.setup(raw, approx=approx))
    try:
        for precision, bar in (("split", 1e-6), ("fp64", 1e-8)):
            u = dev.formal_solve_fo2(precision, want_u=True)["u"]
            assert taken(dev) == dev.P * dev.R
            v = dev.formal_solve_fo2_uv(precision)["u"]
            assert taken(dev) == 0
            assert H.max_rel(u, v) < bar, precision
    finally:
        dev.close()


@pytest.mark.parametrize("nside,nquads", [(1, 11), (1, 31), (2, 7)])
def test_pairs_left_to_the_general_kernel(gpu_lib, nside, nquads):
    """Ray pairs that reach both lines are listed, the others are not, and both are right: single,
    batched and as pixels."""
    at_rest, moving = close_lines(nside, nquads)
    dev, general = with_velocity(at_rest, moving["velocity"]), _abi.DeviceModel(moving)
    batch = _abi.Batch([dev])
    try:
        for precision, bar in (("split", 1e-9), ("fp64", 1e-8)):
            ref = general.formal_solve_fo2(precision, want_u=True)
            assert taken(general) == 0
            out = dev.formal_solve_fo2(precision, want_u=True)
            n, listed = dev.staged_statistics()
            assert n == dev.P * dev.R and 0 < listed < n, (n, listed)
            assert H.max_rel(out["u"], ref["u"]) < bar, precision
            assert H.max_rel(batch.formal_solve_fo2(precision)[0]["J"], ref["J"]) < bar, precision
            n, in_batch = dev.staged_statistics()
            assert n == dev.P * dev.R and in_batch == listed
    finally:
        batch.close()
        dev.close()
        general.close()


def test_pixels_left_to_the_general_kernel(gpu_lib):
    raw = S.grid_sphere(n=11, nside=1, nquads=5, nlev=3)
    ld = raw.linedata[0]
    f = np.array(ld.frequency, np.float64)
    f[1] = f[0] * (1.0 + 1.0e-4)
    slow = replace(raw, linedata=[replace(ld, frequency_given=f)], velocity=0.02 * raw.velocity)
    fast = replace(slow, velocity=raw.velocity)
    nu = (f[0] * (1.0 - 5.0e-5), f[0] * (1.0 + 1.5e-4), 41)
    d = np.array((0.48, 0.36, 0.8))
    fast = H.setup(fast, image_freqs=nu)
    dev, general = with_velocity(H.setup(slow, image_freqs=nu), fast["velocity"]), _abi.DeviceModel(fast)
    try:
        for precision, bar in (("split", 1e-9), ("fp64", 1e-8)):
            ref = general.image_new(d, 19, 14, precision)["I"]
            assert taken(general) == 0
            I = dev.image_new(d, 19, 14, precision)["I"]
            n, listed = dev.staged_statistics()
            assert n == 19 * 14 and 0 < listed, (n, listed)
            assert H.max_rel(I, ref, floor=1e-6 * ref.max()) < bar, precision
    finally:
        dev.close()
        general.close()


@pytest.mark.parametrize("npoints,nside,nquads,nlev,staged", [(9000, 2, 31, 3, True), (600, 2, 60, 42, False)])
def test_fixed_area(gpu_lib, npoints, nside, nquads, nlev, staged):
    """The 64 MiB of mgr_formal_solve_fo2_device_noalloc: several passes, each with its list, or
    the general kernel where the area's rays would not fill the GPU."""
    torch = pytest.importorskip("torch")
    if staged:
        at_rest, moving = close_lines(nside, nquads, npoints=npoints)
        dev, general = with_velocity(at_rest, moving["velocity"]), _abi.DeviceModel(moving)
    else:
        moving = H.setup(S.batch_model(npoints=npoints, nside=nside, nlev=nlev, nquads=nquads))
        dev, general = _abi.DeviceModel(moving), _abi.DeviceModel(in_reverse(moving))
    try:
        J = torch.empty((dev.P, dev.F), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        _abi._check(_abi.load().mgr_formal_solve_fo2_device_noalloc(dev.h, _abi.PRECISION["split"],
                                                                    C.c_void_p(J.data_ptr()), None, None))
        dev.sync()
        n, listed = dev.staged_statistics()
        assert n == (dev.P * dev.R if staged else 0) and (listed > 0) == staged
        ref = general.formal_solve_fo2("split")["J"]
        assert H.max_rel(J.cpu().numpy(), ref if staged else ref[:, ::-1]) < 1e-9
    finally:
        dev.close()
        general.close()


def hardly_any_listed(raw, share, bar=1e-9):
    """The staged solve takes all but `share` of the model's ray pairs by itself, and its u is the
    general kernel's."""
    a = H.setup(raw)
    dev, general = _abi.DeviceModel(a), _abi.DeviceModel(in_reverse(a))
    try:
        u = dev.formal_solve_fo2("split", want_u=True)["u"]
        n, listed = dev.staged_statistics()
        assert n == dev.P * dev.R and listed <= share * n, (n, listed)
        g = general.formal_solve_fo2("split", want_u=True)["u"][:, :, ::-1]
        assert H.max_rel(u, g) < bar
    finally:
        dev.close()
        general.close()


@pytest.mark.parametrize("step,boundary,share", [(1.0e12, S.BC_CMB, 0.0), (1.0e12, S.BC_ZERO, 0.01),
                                                 (1.0e7, S.BC_CMB, 0.0), (1.0e7, S.BC_ZERO, 0.01)])
def test_faint_rays(gpu_lib, step, boundary, share):
    """Pairs out of their line's reach have the minimum opacity's depth, 1e-26 per metre: 1e-14 with
    a step of 1e12 m, where a dark boundary leaves the sweep's source below 1e-28, and 1e-19 with
    one of 1e7 m; between points of a grid that lie at the same distance along the ray but for
    roundings it is 1e-30 and below.  The density keeps the depth of a pair in reach the same."""
    raw = S.batch_model(npoints=1500, nside=1, nlev=4, nquads=21, box=14 * step, n_h2=1.0e24 / step, sigma_v=2.0e3)
    hardly_any_listed(replace(raw, boundary_condition=np.full(len(raw.boundary2point), boundary, np.int32)), share)


def test_many_levels(gpu_lib):
    """30 levels at 10 to 100 K: sources over thirty powers of ten.  The general kernel takes its
    sources in true units and as zero below 1.2e-38; u is a mean of sources and boundary
    intensities, so that is off by 1.2e-38 at most."""
    a = H.setup(S.nlte_sphere(npoints=2000, nside=1, nlev=30, nquads=11))
    dev, general = _abi.DeviceModel(a), _abi.DeviceModel(in_reverse(a))
    try:
        u = dev.formal_solve_fo2("split", want_u=True)["u"]
        assert dev.staged_statistics() == (dev.P * dev.R, 0)
        g = general.formal_solve_fo2("split", want_u=True)["u"][:, :, ::-1]
        assert np.all(np.abs(u - g) < 1e-9 * np.abs(g) + 1.2e-38)
    finally:
        dev.close()
        general.close()


@pytest.mark.parametrize("precision", ["fp64", "split"])
def test_no_minimum_opacity(gpu_lib, precision):
    """Without a minimum opacity a pair out of its line's reach has no depth: a non-finite intensity,
    which every solve and the imager report."""
    raw = S.batch_model(npoints=300, nside=1, nlev=3, nquads=11, sigma_v=5.0e3)
    f0, dd = raw.linedata[0].frequency[0], 8.0e3 / S.CC
    d = np.array((0.48, 0.36, 0.8))
    dev, image = (_abi.DeviceModel(H.setup(raw, min_opacity=0.0, image_freqs=q))
                  for q in (None, (f0 * (1 - dd), f0 * (1 + dd), 11)))
    try:
        for call in (lambda: dev.formal_solve_fo2_uv(precision), lambda: dev.formal_solve_fo2(precision),
                     lambda: image.image_new(d, 9, 9, precision)):
            with pytest.raises(_abi.MgrError, match="non-finite"):
                call()
    finally:
        dev.close()
        image.close()


def test_negative_opacities(gpu_lib):
    """Every other point inverted, with an opacity of the minimum's size: the clamp at the minimum
    decides the sources beside thick pairs.  (FP64: as in test_one_line.)"""
    a = H.setup(S.batch_model(npoints=600, nside=1, nlev=3, nquads=11, sigma_v=2.0e3))
    op = a["opacity"].copy()
    op[::2] = -3.0e-22 * (1.0 + np.arange(len(op[::2]))[:, None] % 7)
    a = dict(a, opacity=op, interp_criterion=np.ones_like(op))
    assert_same_u(a, 1e-8, ("fp64",))
    assert_same_u(a)
