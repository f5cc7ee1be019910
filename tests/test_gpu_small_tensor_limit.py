"""The scale of a small tensor while another thread changes the SM limit: which kernel takes the maximum is decided once per call."""
import ctypes as C
import shutil
import subprocess
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu
FLIP = "void flip(int (*set)(int), volatile int* stop) { while (!*stop) { set(1); set(0); } }"


def test_scale_while_the_sm_limit_changes(tmp_path):
    from arcquant_b200 import _lib, ops

    if shutil.which("gcc") is None:
        pytest.skip("needs a C compiler: a Python thread changes the limit too seldom")
    (tmp_path / "flip.c").write_text(FLIP)
    subprocess.check_call(["gcc", "-O1", "-shared", "-fPIC", "-o", str(tmp_path / "flip.so"), str(tmp_path / "flip.c")])
    flip = C.CDLL(str(tmp_path / "flip.so")).flip
    rows, k, ke, calls, lib = 8, 4096, 64, 5000, _lib.load()      # one launch on all SMs, two under a limit of one
    x = torch.randn(rows, k, device="cuda").bfloat16()
    idx = torch.randperm(k).to(torch.int16).cuda()
    q = torch.empty(rows, (k + ke) // 2, dtype=torch.uint8, device="cuda")
    sf = torch.empty(ops.sf_bytes(rows, k + ke), dtype=torch.uint8, device="cuda")
    scratch = torch.full((calls, _lib.SCALE_SCRATCH), 1e6, device="cuda")
    scales = torch.full((calls,), -1.0, device="cuda")
    stop, stream = C.c_int(0), ops._stream()
    before = lib.arcq_set_sm_limit(0)
    other = threading.Thread(target=flip, args=(C.cast(lib.arcq_set_sm_limit, C.c_void_p), C.byref(stop)))
    other.start()
    try:
        for i in range(calls):
            assert lib.arcq_quantize_tensor_scale(x.data_ptr(), None, 0, idx.data_ptr(), rows, k, ke, 16, q.data_ptr(), sf.data_ptr(),
                                                  scales[i].data_ptr(), scratch[i].data_ptr(), stream) == 0
    finally:
        stop.value = 1
        other.join()
        lib.arcq_set_sm_limit(before)
    want = x.abs().max().float() * (1.0 / 2688.0)
    assert int((scales != want).sum()) == 0
