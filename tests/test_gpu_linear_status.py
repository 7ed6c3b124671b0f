"""The linear transform of the layers and its weight gradient when a bounded wait runs out (a test hook keeps one tile from
being handed over, the limit is a fraction of a millisecond): the kernels return, the record is readable through
check_device_status and gone afterwards, and the next call is right."""
import ctypes

import pytest
import torch

from helpers import randn, rel_err

pytestmark = pytest.mark.gpu
STALL = 2  # CXG_LINEAR_TEST_STALL


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


@pytest.fixture
def short_waits(cuda):
    import cxgnncomp_backend as be
    be.check_device_status("linear")
    be.set_wait_limit_cycles(200_000)  # ~0.1 ms
    yield be
    be.set_wait_limit_cycles(0)


@pytest.mark.parametrize("m", [1, 300, 40000])
def test_linear(short_waits, m):
    be = short_waits
    x, w = randn((m, 64), 1).cuda(), randn((48, 64), 2).cuda()
    y = torch.zeros(m, 48, device="cuda")
    rc = be._lib.cxg_linear_f32_ex(_p(x), _p(w), None, None, _p(y), ctypes.c_int64(m), 64, 48, ctypes.c_uint32(STALL), _stream())
    assert rc == 0
    with pytest.raises(RuntimeError, match="wait ran out"):
        be.check_device_status("linear")
    be.check_device_status("linear")  # told once
    be.set_wait_limit_cycles(0)
    with torch.no_grad():
        assert rel_err(be.linear(x, w).cpu(), x.cpu().double() @ w.cpu().double().t()) < 2e-6
    be.check_device_status("linear")


def test_weight_gradient(short_waits):
    be = short_waits
    x, g = randn((5000, 64), 3).cuda(), randn((5000, 36), 4).cuda()
    dw = torch.zeros(64, 36, device="cuda")
    need = ctypes.c_size_t(0)
    sizes = (ctypes.c_int64(5000), 64, 36)
    assert be._lib.cxg_dense_wgrad_f32_workspace_size(*sizes, ctypes.byref(need)) == 0
    ws = torch.zeros(need.value, dtype=torch.uint8, device="cuda")

    def run(flags):
        return be._lib.cxg_dense_wgrad_f32_ex(_p(x), _p(g), *sizes, ctypes.c_uint32(flags), _p(dw), _p(ws),
                                              ctypes.c_size_t(need.value), _stream())
    assert run(1) == 0
    with pytest.raises(RuntimeError, match="wait ran out"):
        be.check_device_status("linear")
    be.set_wait_limit_cycles(0)
    assert run(0) == 0
    be.check_device_status("linear")
    assert rel_err(dw.cpu(), x.cpu().double().t() @ g.cpu().double()) < 4e-6
