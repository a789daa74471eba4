"""GPU tier, collected last: the entry point for callers that cannot allocate device memory.

``svtad_conv_wgrad_static`` is ``svtad_conv_wgrad`` with the workspace taken from an array built
into the library, for hosts that must not call cudaMalloc once they are running (device memory owned
by the host's own arena, allocation forbidden after start-up).  The test calls it through the C ABI several times in a row - the array is shared and keeps the previous call's contents - and checks every result
against the regular entry point and against the CPU oracle.
"""
import numpy as np
import pytest
import torch

from oracle import conv as oconv
from tests.helpers import f32np, make_conv_inputs, make_table

pytestmark = pytest.mark.gpu


def test_static_workspace_wgrad_matches_regular_entry_point_twice():
    from eccv26_tad_b200 import _lib, ops
    lib = _lib.load()
    assert lib.svtad_static_workspace_bytes() == 32 << 20
    cases = [(2, 40, 0.30, 192, torch.bfloat16, 301), (2, 40, 0.55, 192, torch.bfloat16, 302),
             (1, 8, 0.50, 64, torch.float32, 303)]
    for B, T, keep, C, dtype, seed in cases:
        _, _, table = make_table(B, T, 14, 14, keep, 3, seed)
        n = table.shape[0]
        x, w, b, gy = make_conv_inputs(n, C, C, 3, dtype, seed)
        tc, xc, gc = table.cuda(), x.cuda(), gy.cuda()
        ref_gw, ref_gb = ops.conv_wgrad(gc, xc, tc, 9)
        gw = torch.full((9, C, C), float("nan"), dtype=dtype, device="cuda")
        gb = torch.full((C,), float("nan"), dtype=dtype, device="cuda")
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        free_before = None
        for call in range(3):                    # calls in a row share the built-in array
            gw.fill_(float("nan")); gb.fill_(float("nan"))
            torch.cuda.synchronize()
            if call >= 1:
                # From the second call on (the first may make the driver load the kernels' code), the device's free
                # memory as the driver reports it must not move: that also sees a cudaMalloc made inside the
                # library, which torch's own counters cannot.
                free_before = torch.cuda.mem_get_info()[0]
            ops.conv_wgrad_static(gc, xc, tc, gw, gb)
            torch.cuda.synchronize()
            if free_before is not None:
                assert torch.cuda.mem_get_info()[0] == free_before, "device memory was allocated during the call"
            assert torch.cuda.memory_allocated() == before          # torch allocated nothing either
            assert torch.equal(gw, ref_gw) and torch.equal(gb, ref_gb)
        tol = 1e-5 if dtype == torch.float32 else 2e-2
        egw, egb = oconv.wgrad(f32np(gy), f32np(x), table.numpy(), 9)
        assert oconv.rel_err(f32np(gw), egw) < tol and oconv.rel_err(f32np(gb), egb) < tol
    assert ops.device_error() == 0


def test_static_workspace_rejects_oversized_problems():
    from eccv26_tad_b200 import _lib
    lib = _lib.load()
    n, C = 18880, 1024
    assert lib.svtad_workspace_bytes(_lib.OP_WGRAD, n, C, C, 9, _lib.BF16) > lib.svtad_static_workspace_bytes()
    dummy = torch.zeros(16, device="cuda")
    rc = lib.svtad_conv_wgrad_static(dummy.data_ptr(), dummy.data_ptr(), dummy.data_ptr(), dummy.data_ptr(), None,
                                     n, C, C, 9, 0, _lib.BF16, None)
    assert rc == _lib.ERR_WORKSPACE and "built-in" in _lib.last_error()


@pytest.mark.parametrize("T,keep,cin,cout,dtype,same", [
    (80, 0.30, 256, 256, torch.bfloat16, True),      # what the header promises
    (16, 0.30, 512, 512, torch.float16, True),
    (160, 0.30, 512, 1024, torch.bfloat16, False),   # the usual two token splits would take 36 MB
    (40, 0.30, 1024, 768, torch.bfloat16, None),
])
def test_static_workspace_takes_what_one_copy_of_the_gradient_fits(T, keep, cin, cout, dtype, same):
    from eccv26_tad_b200 import _lib, ops
    lib = _lib.load()
    table = make_table(1, T, 14, 14, keep, 3, 304)[2]
    n = table.shape[0]
    code = _lib.BF16 if dtype == torch.bfloat16 else _lib.F16
    assert same is None or (lib.svtad_workspace_bytes(_lib.OP_WGRAD, n, cin, cout, 9, code) <= lib.svtad_static_workspace_bytes()) == same
    x, w, b, gy = make_conv_inputs(n, cin, cout, 3, dtype, 304)
    tc, xc, gc = table.cuda(), x.cuda(), gy.cuda()
    ref_gw, ref_gb = ops.conv_wgrad(gc, xc, tc, 9)
    gw, gb = torch.full_like(ref_gw, float("nan")), torch.full_like(ref_gb, float("nan"))
    ops.conv_wgrad_static(gc, xc, tc, gw, gb)
    if same:
        assert torch.equal(gw, ref_gw) and torch.equal(gb, ref_gb)
    # the same fp32 sums in another order, rounded once: less than one 16-bit step apart
    assert oconv.rel_err(f32np(gw), f32np(ref_gw)) < 8e-3 and oconv.rel_err(f32np(gb), f32np(ref_gb)) < 8e-3
    assert ops.device_error() == 0
