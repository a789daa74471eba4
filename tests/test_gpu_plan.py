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


@pytest.mark.parametrize("cin,cout", [(640, 640), (384, 800), (512, 928), (256, 960)])
def test_weight_gradient_in_narrower_column_blocks(cin, cout):
    """Five and seven (the last partial) blocks of 128 columns, five of 192 (the last partial or not) instead of 256."""
    from eccv26_tad_b200 import ops
    table = make_table(1, 24, 14, 14, 0.3, 3, 9)[2].cuda()
    x, w, b, gy = (t.cuda() for t in make_conv_inputs(table.shape[0], cin, cout, 3, torch.bfloat16, 9, bias="random"))
    gw, gb = _planned(table, x, w, b, gy)[2:]
    egw, egb = ops.conv_wgrad(gy, x, table, 9)
    assert oconv.rel_err(f32np(gw), f32np(egw)) < 8e-3 and oconv.rel_err(f32np(gb), f32np(egb)) < 8e-3
    assert ops.device_error() == 0


@pytest.mark.parametrize("keep,table_kind", [(0.3, "built"), (0.5, "given"), (1.0, "given"), (1.0, "built")])
def test_module_with_a_layer_that_wants_a_plan(keep, table_kind):
    """C = 512 at 18 880 / 31 360 / 62 720 rows: with the module's plan (a table built here that is sparse enough) and without
    one (the full grid; a caller's table whose density the call does not ask for), results as without one."""
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


# ---------------------------------------------------------------------------------------------------------------------
# The module's plans: made from what the table holds when the kernels run, by a rule that nothing asynchronous enters.
# C = 512 at 18 880 rows, keep 0.3: a layer whose forward, input gradient and weight gradient go by a plan.
# ---------------------------------------------------------------------------------------------------------------------
def _scores(T, seed):
    return torch.randn(T, 196, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))


def _layer(C, ks, n, seed, Co=None):
    import eccv26_tad_b200 as sv
    g = torch.Generator("cuda").manual_seed(seed)
    m = sv.SparseConv2d(C, Co or C, kernel_size=ks).cuda().bfloat16()
    x = torch.randn(n, C, device="cuda", generator=g).bfloat16().requires_grad_(True)
    gy = torch.randn(n, Co or C, device="cuda", generator=g).bfloat16()
    return m, x, gy


def _pass(m, x, table, gy):
    y = m(x, table)
    return (y.detach().reshape(gy.shape),) + torch.autograd.grad(y, (x, m.weight, m.bias), gy.reshape(y.shape))


def _unplanned(m, x, table, gy):
    from eccv26_tad_b200 import ops
    w, flat = m.weight.detach(), table.reshape(-1, m.weight.shape[0])
    xf = x.detach().reshape(-1, x.shape[-1])
    gw, gb = ops.conv_wgrad(gy, xf, flat, w.shape[0])
    return ops.conv_fwd(xf, flat, w, m.bias.detach()), ops.conv_dgrad(gy, flat, w, assume_symmetric=True), gw, gb


def _close(got, want):
    for a, b in zip(got, want):
        # both round the same fp32 sums, made in another order, once: less than one bf16 step apart
        assert oconv.rel_err(f32np(a).reshape(b.shape), f32np(b)) < 8e-3


def _wanted(n, C, kk, density):
    from eccv26_tad_b200 import _lib
    return _lib.load().svtad_plan_wanted(n, C, C, kk, _lib.BF16, density)


def test_a_table_rewritten_behind_the_version_counter():
    """The C ABI (or a replayed graph that holds the selection) writes another table into the same memory."""
    import eccv26_tad_b200 as sv
    from eccv26_tad_b200 import _lib
    T = 320
    kept, table = sv.build_neighbor_table(_scores(T, 1), 0.3, 14, 14)
    n = table.shape[0]
    assert _wanted(n, 512, 9, 0.35) == 3
    m, x, gy = _layer(512, 3, n, 1)
    for _ in range(2):
        _close(_pass(m, x, table, gy), _unplanned(m, x, table, gy))
        torch.cuda.synchronize()
    other, version = _scores(T, 2), table._version
    _lib.check(_lib.load().svtad_table_build(other.data_ptr(), T, 196, n // T, 14, 14, 3, kept.data_ptr(), table.data_ptr(),
                                             torch.cuda.current_stream().cuda_stream))
    assert table._version == version
    _close(_pass(m, x, table, gy), _unplanned(m, x, table, gy))


def test_graph_captured_behind_a_warm_up_on_the_same_stream():
    """Warm-up and capture on one stream; between replays the table is refreshed in place, and memory that the warm-up
    gave back is used by others."""
    import eccv26_tad_b200 as sv
    T = 320
    tables = [sv.build_neighbor_table(_scores(T, s), 0.3, 14, 14)[1] for s in (3, 4, 5)]
    table = tables[0]
    m, x, gy = _layer(512, 3, table.shape[0], 2)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        for _ in range(2):
            _pass(m, x, table, gy)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            out = _pass(m, x, table, gy)
    torch.cuda.current_stream().wait_stream(s)
    for new in tables[1:]:
        table.copy_(new)
        junk = [torch.full((1 << 20,), -7, dtype=torch.int32, device="cuda") for _ in range(4)]
        g.replay()
        torch.cuda.synchronize()
        _close(out, _unplanned(m, x, new, gy))
        del junk


def test_one_table_serves_layers_of_different_stencils():
    """225 * m entries are m * 25 rows of 9 taps as well as m * 9 rows of 25: each layer reads the table its own way."""
    import eccv26_tad_b200 as sv
    flat = sv.get_initial_neighbor_indices(15, 15, 40, "cuda", 1, 5).reshape(-1)          # 9 000 rows of 25
    flat = torch.where(torch.rand(flat.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(6)) < 0.3, flat, -1)
    for C, ks in ((512, 3), (512, 5), (512, 3)):
        kk = ks * ks
        n = flat.numel() // kk
        m, x, gy = _layer(C, ks, n, 3)
        x3 = x.detach().view(1, n, C).requires_grad_(True)                                 # [B, N, C]: the density is asked for
        y, gx, gw, gb = _pass(m, x3, flat, gy)
        ey, _, egw, egb = _unplanned(m, x3, flat, gy)
        _close((y, gw, gb), (ey, egw, egb))
        # not a symmetric table: the input gradient is the scatter form's
        w, egx = m.weight.detach(), torch.zeros(n, C, device="cuda")
        t = flat.view(n, kk).long()
        for k in range(kk):
            i = ((t[:, k] >= 0) & (t[:, k] < n)).nonzero().view(-1)
            egx.index_add_(0, t[i, k], gy[i].float() @ w[k].float().t())
        _close((gx.view(n, C),), (egx,))


@pytest.mark.parametrize("C,ks,T,keep,given", [(512, 3, 320, 0.3, True), (512, 3, 160, 0.5, True), (512, 3, 160, 0.6, True),
                                               (512, 3, 80, 1.0, True), (512, 5, 25, 0.38, False), (768, 3, 80, 0.3, False), (768, 3, 160, 0.3, True),
                                               (1024, 3, 30, 0.3, True), (256, 3, 1280, 0.3, False), (320, 3, 320, 0.2, False)])
def test_passes_repeat_bit_for_bit(C, ks, T, keep, given):
    """Neither the first pass on a table nor one that follows a synchronisation takes other kernels than the rest."""
    import eccv26_tad_b200 as sv
    if keep == 1.0:
        table = sv.get_initial_neighbor_indices(14, 14, T, "cuda", 1, ks)[0]
    else:
        table = sv.build_neighbor_table(_scores(T, 7), keep, 14, 14, ks)[1]
    n = table.shape[0]
    table = table.view(1, n, ks * ks)
    m, x, gy = _layer(C, ks, n, 4)
    x = x.detach().view(1, n, C).requires_grad_(True)
    first = None
    for i in range(6):
        t = table.clone() if given and i in (0, 3) else (table if first is None or not given else t)
        got = _pass(m, x, t, gy)
        if i % 2:
            torch.cuda.synchronize()
        first = first or got
        assert all(torch.equal(a, b) for a, b in zip(got, first))
    with torch.no_grad():
        assert torch.equal(m(x, t).view(n, C), first[0])
    _close(first, _unplanned(m, x, table, gy))


def test_two_streams_share_a_table():
    import eccv26_tad_b200 as sv
    table = sv.build_neighbor_table(_scores(320, 8), 0.3, 14, 14)[1]
    layers = [_layer(512, 3, table.shape[0], s) for s in (5, 6)]
    want = [_unplanned(m, x, table, gy) for m, x, gy in layers]
    streams = [torch.cuda.Stream() for _ in layers]
    torch.cuda.synchronize()
    outs = []
    for _ in range(3):
        for s, (m, x, gy) in zip(streams, layers):
            with torch.cuda.stream(s):
                outs.append(_pass(m, x, table, gy))
    torch.cuda.synchronize()
    for i, got in enumerate(outs):
        _close(got, want[i % 2])


def test_tables_made_in_inference_mode():
    import eccv26_tad_b200 as sv
    m, x, _ = _layer(512, 3, 62720, 9)
    with torch.inference_mode():
        full = sv.get_initial_neighbor_indices(14, 14, 320, "cuda", 1)
        sparse = sv.build_neighbor_table(_scores(320, 9), 0.3, 14, 14)[1]
        for table in (full, sparse):
            n = table.numel() // 9
            for _ in range(2):
                y = m(x[:n], table)
            assert torch.equal(y, m(x[:n], table.clone()))
