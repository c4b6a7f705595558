"""Two host threads that call one kernel with different sizes: neither call may fail because of the other."""
import ctypes
import threading

import pytest
import torch

from matterformer_b200 import _lib

pytestmark = pytest.mark.gpu


def _forward_call(N, D, dtype, bias, backend):
    """A prepared mf_simplicial_fwd call on its own stream and buffers, of an empty molecule: the host is what takes time."""
    g = torch.Generator(device="cuda").manual_seed(N)
    rows = [torch.randn(1, 1, N, D, generator=g, device="cuda").to(dtype) for _ in range(5)]
    coef = [torch.randn(1, 1, N, N, generator=g, device="cuda") for _ in range(3)] + [torch.randn(1, 1, N, generator=g, device="cuda")]
    mask = torch.zeros(1, N, dtype=torch.uint8, device="cuda")
    out, lse = torch.empty(1, 1, N, D, device="cuda"), torch.empty(1, 1, N, device="cuda")
    ws = torch.empty(1 << 16, dtype=torch.uint8, device="cuda")
    a = _lib.MfSimplicialFwdArgs(batch=1, heads=1, tokens=N, head_dim=D, dtype=_lib.MF_DTYPE_F32 if dtype == torch.float32 else _lib.MF_DTYPE_BF16,
                                 precision=_lib.MF_PRECISION["ieee_fp32" if dtype == torch.float32 else "bf16_tc"], backend=_lib.MF_BACKEND[backend])  # fmt: skip
    a.q, a.k1, a.v1, a.k2, a.v2 = (t.data_ptr() for t in rows)
    a.query_valid = a.pair_key_valid = mask.data_ptr()
    a.out, a.lse, a.workspace, a.workspace_bytes = out.data_ptr(), lse.data_ptr(), ws.data_ptr(), ws.numel()
    if bias:
        a.u, a.v_bias, a.w, a.gate = (t.data_ptr() for t in coef)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    entry, ref = _lib.lib().mf_simplicial_fwd, ctypes.byref(a)
    keep = (rows, coef, mask, out, lse, ws, stream, a)
    return (lambda: entry(ref, ctypes.c_void_p(stream.cuda_stream))), keep


@pytest.mark.parametrize("sizes,D,dtype,bias,backend",
                         [((33, 192), 64, torch.bfloat16, True, "tcgen05_tiles"), ((33, 192), 64, torch.bfloat16, False, "auto"),
                          ((9, 400), 128, torch.float32, False, "generic")], ids=["trilinear", "warp", "generic"])  # fmt: skip
def test_calls_of_different_sizes_at_once(sizes, D, dtype, bias, backend):
    failed = []

    def work(N, call):
        torch.cuda.set_device(0)
        for _ in range(2000):
            if call() != _lib.MF_OK:
                failed.append((N, _lib.last_error()))
                return

    calls = [_forward_call(N, D, dtype, bias, backend) for N in sizes]
    threads = [threading.Thread(target=work, args=(N, call)) for N, (call, _) in zip(sizes, calls)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed, failed
