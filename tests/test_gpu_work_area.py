"""The memory a formal solve takes beside its results: half rays only where the solve walks them into
memory, less where the device has no room, and no allocation that a solve can do without inside a
stream capture."""
import ctypes as C

import numpy as np
import pytest

import helpers as H
from magritte_gb300 import _abi
from magritte_gb300 import synthetic as S

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MiB = 1 << 20


@pytest.fixture(scope="module")
def long_rays():
    """8k points, 24 ray pairs, one line x 5 frequencies: 8 MB of u, and 200 MB of half rays and more."""
    return H.setup(S.batch_model(npoints=8000, nside=2, nlev=2, nquads=5))


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


class Little:
    """Leaves `room` bytes of device memory to others."""

    def __init__(self, room):
        self.room = room

    def __enter__(self):
        torch.cuda.empty_cache()
        self.held = torch.empty(max(free_bytes() - self.room, 0), dtype=torch.uint8, device="cuda")

    def __exit__(self, *a):
        del self.held
        torch.cuda.empty_cache()


def test_banded_solve_holds_no_rays(gpu_lib, long_rays):
    dev = _abi.DeviceModel(long_rays)
    try:
        dev.set_n_off_diag(1)
        before = free_bytes()
        dev.formal_solve_fo2_alo()
        assert before - free_bytes() < 100 * MiB
    finally:
        dev.close()


@pytest.mark.parametrize("precision", ["split", "fp64"])
def test_solve_with_little_memory(gpu_lib, long_rays, precision):
    """Room for u and the ALO diagonal but not for the half rays: the general kernel's solve, as
    before there were any, and the first call of a solve that had its memory keeps it."""
    dev, ref = _abi.DeviceModel(long_rays), _abi.DeviceModel(long_rays)
    try:
        out = ref.formal_solve_fo2(precision)
        assert ref.staged_statistics()[0] == ref.P * ref.R
        with Little(100 * MiB):
            got = dev.formal_solve_fo2(precision)
            dev.staged_statistics()
            again = dev.formal_solve_fo2(precision)
            assert dev.staged_statistics()[0] in (0, dev.P * dev.R)
            assert np.array_equal(got["J"], again["J"])
        # FP64: the two kernels' depths differ by 1e-9 a pair (rounded positions)
        assert H.max_rel(got["J"], out["J"]) < (1e-9 if precision == "split" else 1e-8)
    finally:
        dev.close()
        ref.close()


def test_capture_of_a_first_solve(gpu_lib, long_rays):
    """A solve into the caller's u without the ALO diagonal needs no memory of its own: its first
    call may stand inside a stream capture."""
    warm, dev = _abi.DeviceModel(long_rays), _abi.DeviceModel(long_rays)
    try:
        ref = warm.formal_solve_fo2("split", want_u=True, want_lambda=False)  # loads the kernels
        warm.formal_solve_fo2_uv("split")
        J = torch.zeros((dev.P, dev.F), dtype=torch.float64, device="cuda")
        u = torch.zeros((dev.R, dev.P, dev.F), dtype=torch.float64, device="cuda")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(dev.stream())):
            dev.formal_solve_fo2_device("split", J.data_ptr(), u.data_ptr())
        graph.replay()
        torch.cuda.synchronize()
        assert H.max_rel(u.cpu().numpy(), ref["u"]) < 1e-9
        assert H.max_rel(J.cpu().numpy(), ref["J"]) < 1e-9
    finally:
        dev.close()
        warm.close()


@pytest.mark.parametrize("share,staged", [(1.2, True), (0.75, True), (0.3, False)])
def test_batch_with_little_memory(gpu_lib, long_rays, share, staged):
    """A share of the memory that a batch of two models takes, nearly all of it their half rays:
    both in a wave, one, or the general kernel."""
    devs = [_abi.DeviceModel(long_rays) for _ in range(2)]
    try:
        ref = devs[0].formal_solve_fo2("split")
        devs[0].staged_statistics()
        before = free_bytes()
        batch = _abi.Batch(devs)
        taken = before - free_bytes()
        batch.close()
        with Little(int(share * taken)):
            batch = _abi.Batch(devs)
        try:
            for out in batch.formal_solve_fo2("split"):
                assert H.max_rel(out["J"], ref["J"]) < 1e-9
        finally:
            batch.close()
        for d in devs:
            assert d.staged_statistics()[0] == (d.P * d.R if staged else 0)
    finally:
        for d in devs:
            d.close()


def smooth(dev, J):
    _abi._check(_abi.load().mgr_formal_solve_fo2_smooth_device(dev.h, None, 0, C.c_void_p(J.data_ptr())))
    return J.cpu().numpy()


def test_captured_solve_outlives_images_and_smooth_solves(gpu_lib):
    """A caller's graph of a formal solve holds the address of the work area: images and smooth
    solves, however large, leave that where it is."""
    a = H.setup(S.batch_model(npoints=1000, nside=1, nlev=3, nquads=11))
    dev = _abi.DeviceModel(a)
    try:
        ref = dev.formal_solve_fo2("split", want_lambda=False)["J"]
        J = torch.zeros((dev.P, dev.F), dtype=torch.float64, device="cuda")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(dev.stream())):
            dev.formal_solve_fo2_device("split", J.data_ptr())
        dev.image_new(np.array((0.48, 0.36, 0.8)), 301, 299, "split")
        smooth(dev, torch.zeros_like(J))
        keep = [torch.full((1 << 24,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(8)]
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(J.cpu().numpy(), ref)
        del keep
    finally:
        dev.close()


def test_smooth_solve_with_little_memory(gpu_lib):
    """48 MB of u for every origin at once; with 20 MiB left, several passes and the same J."""
    a = H.setup(S.batch_model(npoints=2000, nside=2, nlev=5, nquads=31))
    dev, ref = _abi.DeviceModel(a), _abi.DeviceModel(a)
    try:
        J = torch.zeros((dev.P, dev.F), dtype=torch.float64, device="cuda")
        want = smooth(ref, J).copy()
        with Little(20 * MiB):
            got = smooth(dev, J.zero_())
        assert np.array_equal(got, want)
    finally:
        dev.close()
        ref.close()


def test_captured_solve_outlives_larger_areas(gpu_lib):
    """Solves that need a larger area leave the one a caller's graph holds."""
    a = H.setup(S.batch_model(npoints=1000, nside=1, nlev=3, nquads=11))
    dev = _abi.DeviceModel(a)
    try:
        ref = dev.formal_solve_fo2("split", want_lambda=False)["J"]
        J = torch.zeros((dev.P, dev.F), dtype=torch.float64, device="cuda")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(dev.stream())):
            dev.formal_solve_fo2_device("split", J.data_ptr())
        dev.formal_solve_fo2("fp64")
        dev.formal_solve_sc0("split")
        keep = [torch.full((1 << 24,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(8)]
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(J.cpu().numpy(), ref)
        del keep
    finally:
        dev.close()
