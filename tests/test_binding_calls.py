"""The Python binding's calls: what they accept and refuse, and what they allocate."""
import ctypes as C
import os
import re

import numpy as np
import pytest

from kraken_b200 import capi


@pytest.mark.gpu
def test_silu_mul_keeps_the_layout_of_its_inputs(cuda):
    import torch
    for shape, order in (((64, 32), (1, 0)), ((4, 6, 10), (2, 0, 1))):
        gate, up = (torch.randn(shape, device="cuda").permute(order) for _ in range(2))
        y = cuda.silu_mul(gate, up)
        assert y.stride() == gate.stride() and not y.requires_grad
        want = torch.nn.functional.silu(gate.double()) * up.double()
        assert (y - want).abs().max().item() < 1e-5


@pytest.mark.gpu
def test_backend_takes_every_form_of_pointer(cuda):
    """Integers, None where no pointer is needed, and what ctypes takes for a void pointer."""
    import torch
    be = cuda.Backend(0)
    w = torch.zeros(64 * 34, dtype=torch.uint8, device="cuda")
    w[0::34], w[1::34] = 0, 0x3C                      # Q8_0 blocks of scale 1.0
    w.view(64, 34)[:, 2:] = 1
    src = np.full(32, 2.0, np.float32)
    x, y = torch.zeros(32, device="cuda"), torch.zeros((2, 64), device="cuda")
    be.upload(C.c_void_p(x.data_ptr()), src.ctypes.data_as(C.POINTER(C.c_float)), src.nbytes)
    outs, ws = [y[0].data_ptr(), y[1].data_ptr()], [C.c_void_p(w.data_ptr()), w.data_ptr()]
    ran, fused = be.gemm_group(outs, None, ws, cuda.Q8_0, [64, 64], 32, xs=[x.data_ptr()] * 2)
    assert ran and not fused
    be.sync()
    assert (y == 64.0).all()
    be.upload(x.data_ptr(), src.tobytes(), src.nbytes)
    be.gemm(C.c_void_p(y.data_ptr()), x.data_ptr(), w.data_ptr(), cuda.Q8_0, 64, 32, 1)
    got = (C.c_float * 128)()
    be.download(got, y.data_ptr(), 512)
    assert list(got) == [64.0] * 128
    be.close()
    with pytest.raises(TypeError):
        be.upload(x.data_ptr(), src.ctypes.data, src.nbytes)


def test_addresses_are_checked_before_the_call():
    with pytest.raises((TypeError, C.ArgumentError)):
        capi._fc.backend_upload(1, 2.5, 0, 0, 0)


def test_every_launching_call_releases_the_interpreter_lock():
    """A launch can wait for room in the device's queue, and what empties it may be a host callback that needs the lock."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    text = open(os.path.join(root, "kraken_b200", "csrc", "py", "krk_fastcall.cpp")).read()
    calls = [m for m in re.finditer(r"\bkrk_cuda_\w+\(", text) if "workspace_bytes" not in m.group()]
    assert len(calls) >= 13
    for m in calls:
        line = text[text.rfind("\n", 0, m.start()) + 1:m.start()]
        assert "Py_BEGIN_ALLOW_THREADS" in line, m.group()


@pytest.mark.parametrize("longer", range(5))
def test_group_lists_of_unequal_length_are_refused(longer):
    import torch
    t = torch.zeros(64)
    lists = [[t, t], [t, t], [capi.Q8_0] * 2, [1, 1], [t, t]]   # xs, ws, wts, n_outs, outs
    if longer != 1:
        lists[longer] = lists[longer] + lists[longer][:1]
    else:
        lists = [l if i == 1 else l + l[:1] for i, l in enumerate(lists)]
    xs, ws, wts, n_outs, outs = lists
    with pytest.raises(ValueError):
        capi._fc.gemv_group(xs, ws, wts, n_outs, 32, outs, False, NoStream)
    addresses = lambda l: [0x1000] * len(l)   # noqa: E731
    with pytest.raises(ValueError):
        capi._fc.backend_gemm_group(0, addresses(outs), 0, addresses(ws), capi.Q8_0, n_outs, 32, 1, False, wts, addresses(xs))


class NoStream:
    cuda_stream = 0
