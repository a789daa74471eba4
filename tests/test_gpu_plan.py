"""GPU tier: a table's work plan (row order, tile masks, pair lists) and the kernels that run by it."""
import numpy as np
import pytest
import torch

from oracle import conv as oconv
from tests.helpers import f32np, make_conv_inputs, make_table

pytestmark = pytest.mark.gpu
TILE = 128


def _build(table, tpb=0):
    from eccv26_tad_b200 import _lib
    lib = _lib.load()
    n, kk = table.shape
    nbytes = lib.svtad_plan_bytes(n, kk)
    plan = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    _lib.check(lib.svtad_plan_build(table.data_ptr(), n, kk, tpb, plan.data_ptr(), None))
    torch.cuda.synchronize()
    return plan


def _view(plan, n, kk):
    """Host view of the plan's parts, each on a 256-byte boundary."""
    raw, at, tiles = plan.cpu().numpy(), 0, -(-n // TILE)
    out = []
    for count, dtype in ((tiles * TILE, np.int32), (tiles, np.uint64), (tiles, np.int32), (kk, np.int32), (kk * n, np.int32), (kk * n, np.int32)):
        size = count * np.dtype(dtype).itemsize
        out.append(raw[at:at + size].view(dtype))
        at += -(-size // 256) * 256
    order, mask, seq, cnt, pi, pj = out
    return order, mask, seq, cnt, pi.reshape(kk, n), pj.reshape(kk, n)


@pytest.mark.parametrize("B,T,h,w,keep,ks", [(1, 1, 1, 1, 1.0, 3), (1, 3, 14, 14, 0.3, 3), (2, 40, 14, 14, 0.3, 5), (2, 80, 14, 14, 0.6, 3),
                                             (1, 20, 9, 7, 1.0, 7), (3, 100, 16, 16, 0.2, 3)])
def test_plan_of_a_table(B, T, h, w, keep, ks):
    table = make_table(B, T, h, w, keep, ks, 5)[2]
    n, kk = table.shape
    t = table.numpy()
    order, mask, seq, cnt, pi, pj = _view(_build(table.cuda()), n, kk)
    tiles = len(mask)
    assert sorted(order[:n]) == list(range(n)) and (order[n:] == -1).all()
    valid = t >= 0
    bits = np.array([[(int(m) >> k) & 1 for k in range(kk)] for m in mask], dtype=bool)
    for i in range(tiles):
        need = valid[order[i * TILE:min(n, (i + 1) * TILE)]].any(0)
        assert (bits[i] | ~need).all()
        if ks == 3:
            assert (bits[i] == need).all()            # the ring is the whole stencil
    assert sorted(seq) == list(range(tiles))
    assert (np.diff(bits.sum(1)[seq]) <= 0).all()
    for k in range(kk):
        rows = np.nonzero(valid[:, k])[0]
        assert cnt[k] == len(rows)
        assert (pi[k, :len(rows)] == rows).all() and (pj[k, :len(rows)] == t[rows, k]).all()


def test_plan_of_a_table_with_local_indices_and_bad_entries():
    tab = make_table(1, 4, 8, 8, 0.5, 3, 7)[2]
    tpb, B = tab.shape[0], 5
    local = tab.repeat(B, 1)
    local[3, 2] = 10 ** 6                              # out of range: no pair
    n = local.shape[0]
    _, _, _, cnt, pi, pj = _view(_build(local.cuda(), tpb), n, 9)
    t = local.numpy().astype(np.int64)
    for k in range(9):
        j = t[:, k] + np.arange(n) // tpb * tpb
        rows = np.nonzero((t[:, k] >= 0) & (j < n))[0]
        assert cnt[k] == len(rows) and (pi[k, :len(rows)] == rows).all() and (pj[k, :len(rows)] == j[rows]).all()


def _planned(table, x, w, b, gy, tpb=0, grad_fp32=False):
    from eccv26_tad_b200 import _lib
    lib = _lib.load()
    kk, cin, cout = w.shape
    n = x.shape[0]
    code = {torch.float32: _lib.F32, torch.bfloat16: _lib.BF16, torch.float16: _lib.F16}[x.dtype]
    plan = _build(table, tpb)
    y, gx = torch.empty(n, cout, dtype=x.dtype, device="cuda"), torch.empty(n, cin, dtype=x.dtype, device="cuda")
    gdt = torch.float32 if grad_fp32 else x.dtype
    gw, gb = torch.empty(kk, cin, cout, dtype=gdt, device="cuda"), torch.empty(cout, dtype=gdt, device="cuda")
    nbytes = lib.svtad_workspace_bytes(_lib.OP_BWD, n, cin, cout, kk, code)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(lib.svtad_conv_fwd_planned(x.data_ptr(), table.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), n, cin,
                                          cout, kk, tpb, code, plan.data_ptr(), st))
    _lib.check(lib.svtad_conv_bwd_typed(gy.data_ptr(), x.data_ptr(), table.data_ptr(), w.data_ptr(), gx.data_ptr(),
                                        gw.data_ptr(), gb.data_ptr(), n, cin, cout, kk, tpb, code,
                                        _lib.F32 if grad_fp32 else code, plan.data_ptr(), 3, None, ws.data_ptr(), nbytes, st))
    torch.cuda.synchronize()
    return y, gx, gw, gb


@pytest.mark.parametrize("B,T,keep,ks,cin,cout,dtype", [
    (1, 2, 0.3, 3, 256, 256, torch.bfloat16),          # fewer tiles than SMs
    (2, 80, 0.3, 3, 128, 192, torch.bfloat16),         # ragged last tile
    (4, 80, 0.3, 3, 192, 64, torch.float16),           # several tiles per CTA, short and long
    (1, 60, 0.5, 5, 160, 320, torch.bfloat16),         # partial chunks and column blocks, taps outside the sorted ring
    (4, 80, 0.6, 3, 64, 512, torch.bfloat16),          # one chunk per tap, two column blocks
    (1, 40, 1.0, 3, 96, 96, torch.bfloat16),           # the full grid
    (4, 18, 0.3, 3, 768, 768, torch.bfloat16),         # few tiles: the forward takes narrower column blocks than the input gradient
    (4, 40, 0.3, 3, 480, 96, torch.float16),           # weight gradient by blocks of 256 input channels, the last one partial
    (1, 20, 0.3, 3, 512, 288, torch.bfloat16),         # ... whole units and cut ones, a partial column block
])
def test_planned_kernels_give_the_unplanned_results(B, T, keep, ks, cin, cout, dtype):
    from eccv26_tad_b200 import ops
    table = make_table(B, T, 14, 14, keep, ks, 9)[2].cuda()
    x, w, b, gy = (t.cuda() for t in make_conv_inputs(table.shape[0], cin, cout, ks, dtype, 9, bias="random"))
    y, gx, gw, gb = _planned(table, x, w, b, gy)
    ey, egx = ops.conv_fwd(x, table, w, b), ops.conv_dgrad(gy, table, w, assume_symmetric=True)
    if T >= 80:                                        # few rows without a plan split the sums over a cluster
        assert torch.equal(y, ey) and torch.equal(gx, egx)
    assert oconv.rel_err(f32np(y), f32np(ey)) < 8e-3 and oconv.rel_err(f32np(gx), f32np(egx)) < 8e-3
    egw, egb = ops.conv_wgrad(gy, x, table, ks * ks)
    assert oconv.rel_err(f32np(gw), f32np(egw)) < 8e-3 and oconv.rel_err(f32np(gb), f32np(egb)) < 8e-3
    again = _planned(table, x, w, b, gy, grad_fp32=True)
    assert torch.equal(again[2], gw.float()) and torch.equal(again[3], gb.float()) and torch.equal(again[0], y)
    assert ops.device_error() == 0


@pytest.mark.parametrize("keep,table_kind", [(0.3, "built"), (0.5, "given"), (1.0, "given"), (1.0, "built")])
def test_module_with_a_layer_that_wants_a_plan(keep, table_kind):
    """C = 512 at 18 880 / 31 360 / 62 720 rows: the module's plan (first pass: the density is not known yet; later ones go
    by it), results as without one."""
    import eccv26_tad_b200 as sv
    from eccv26_tad_b200 import ops
    B = 4
    if keep == 1.0:
        table = sv.get_initial_neighbor_indices(14, 14, 80, "cuda", B)
    else:
        table = sv.build_neighbor_table(torch.randn(B * 80, 196, device="cuda"), keep, 14, 14)[1]
    table = table if table_kind == "built" else table.clone()
    n = table.numel() // 9
    C = 512
    m = sv.SparseConv2d(C, C).cuda().bfloat16()
    x = torch.randn(n, C, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    gy = torch.randn(n, C, device="cuda", dtype=torch.bfloat16)
    flat = table.reshape(-1, 9)
    ey = ops.conv_fwd(x.detach(), flat, m.weight.detach(), m.bias.detach())
    egx = ops.conv_dgrad(gy, flat, m.weight.detach(), assume_symmetric=True)
    egw, egb = ops.conv_wgrad(gy, x.detach(), flat, 9)
    for _ in range(3):
        y = m(x, table)
        gx, gw, gb = torch.autograd.grad(y, (x, m.weight, m.bias), gy)
        torch.cuda.synchronize()
        assert torch.equal(y, ey) and torch.equal(gx, egx)
        assert oconv.rel_err(f32np(gw), f32np(egw)) < 8e-3 and oconv.rel_err(f32np(gb), f32np(egb)) < 8e-3
    assert ops.device_error() == 0
