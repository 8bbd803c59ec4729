"""The formal solve's frequency gradient is summed over the ray pairs in order: the same bits on
every call."""
import ctypes as C

import numpy as np
import pytest

import helpers as H
from magritte_gb300 import _abi
from magritte_gb300 import synthetic as S

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def gradients(dev, gJ, origins=None):
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device="cuda")
    g = [z(dev.P, dev.L) for _ in range(4)] + [z(dev.P, 3), z(dev.P, dev.F)]
    p = lambda t: C.c_void_p(t.data_ptr())
    torch.cuda.synchronize()
    _abi._check(_abi.load().mgr_formal_solve_fo2_adjoint_device(
        dev.h, None if origins is None else p(origins), 0 if origins is None else origins.numel(), p(gJ),
        *(p(t) for t in g)))
    return [t.cpu().numpy() for t in g]


def test_frequency_gradient_is_the_same_on_every_call(gpu_lib):
    """Some 40,000 sums of 24 terms: an order that varies shows in every call."""
    dev = _abi.DeviceModel(H.setup(S.batch_model(npoints=2000, nside=2, nlev=4, nquads=11)))
    try:
        gJ = torch.randn((dev.P, dev.F), dtype=torch.float64, device="cuda",
                         generator=torch.Generator(device="cuda").manual_seed(1))
        gJ[::3] = 0.0
        gJ[:, ::4] = 0.0
        first = gradients(dev, gJ)
        for _ in range(3):
            again = gradients(dev, gJ)
            assert np.array_equal(again[5], first[5])
            # the others are added with atomics; their largest sums have some thousand terms
            for a, b in zip(again[:5], first[:5]):
                assert np.max(np.abs(a - b)) < 1e-11 * np.max(np.abs(b))
        assert np.all(first[5][::3] == 0.0) and np.all(first[5][:, ::4] == 0.0) and np.any(first[5] != 0.0)
        # a list: those rows alone; an origin listed twice counts twice
        some = torch.tensor([4, 100, 7, 7], dtype=torch.int32, device="cuda")
        listed = gradients(dev, gJ, some)[5]
        want = np.zeros_like(listed)
        want[[4, 100]] = first[5][[4, 100]]
        want[7] = 2.0 * first[5][7]
        assert np.array_equal(listed, want)
    finally:
        dev.close()


def test_adjoint_with_little_memory(gpu_lib):
    """42 MB of frequency derivatives and some hundred MB of elimination scratch; with 90 MiB left,
    several passes of fewer warps and the same sums."""
    a = H.setup(S.batch_model(npoints=2000, nside=2, nlev=5, nquads=31))
    dev, ref = _abi.DeviceModel(a), _abi.DeviceModel(a)
    try:
        gJ = torch.ones((dev.P, dev.F), dtype=torch.float64, device="cuda")
        before = torch.cuda.mem_get_info()[0]
        want = gradients(ref, gJ)
        torch.cuda.empty_cache()
        took = before - torch.cuda.mem_get_info()[0]
        assert took > 120 << 20
        held = torch.empty(torch.cuda.mem_get_info()[0] - (90 << 20), dtype=torch.uint8, device="cuda")
        got = gradients(dev, gJ)
        del held
        assert np.array_equal(got[5], want[5])
        for a, b in zip(got[:5], want[:5]):
            assert np.max(np.abs(a - b)) < 1e-11 * np.max(np.abs(b))
    finally:
        torch.cuda.empty_cache()
        dev.close()
        ref.close()
