"""GPU tier: the reference-facing Python surface (module, autograd Function, pybind-module shim)."""
import numpy as np
import pytest
import torch

from oracle import conv as oconv
from tests.helpers import f32np, make_conv_inputs, make_table

pytestmark = pytest.mark.gpu


def _oracle_grads(table, x, w, b, gy, tpb=0):
    tn = table.numpy()
    xf, wf, bf, gf = (f32np(t) for t in (x, w, b, gy))
    y = oconv.fwd(xf, tn, wf, bf, tpb)
    gx = oconv.dgrad(gf, tn, wf, tpb)
    gw, gb = oconv.wgrad(gf, xf, tn, w.shape[0], tpb)
    return y, gx, gw, gb


def test_module_fp32_autograd_matches_oracle():
    from eccv26_tad_b200 import SparseConv2d
    _, _, table = make_table(1, 4, 14, 14, 0.5, 3, 31)
    n = table.shape[0]
    x, w, b, gy = make_conv_inputs(n, 64, 96, 3, torch.float32, 31, bias="random")
    m = SparseConv2d(64, 96).cuda()
    with torch.no_grad():
        m.weight.copy_(w); m.bias.copy_(b)
    xc = x.cuda().requires_grad_(True)
    y = m(xc, table.cuda())
    y.backward(gy.cuda())
    ey, egx, egw, egb = _oracle_grads(table, x, w, b, gy)
    assert oconv.rel_err(f32np(y), ey) < 1e-5
    assert oconv.rel_err(f32np(xc.grad), egx) < 1e-5
    assert oconv.rel_err(f32np(m.weight.grad), egw) < 1e-5
    assert oconv.rel_err(f32np(m.bias.grad), egb) < 1e-5


def test_module_autocast_bf16_batched_local_and_global_indices():
    """3-D input under bf16 autocast, fp32 master parameters (the reference's training setting)."""
    from eccv26_tad_b200 import SparseConv2d
    _, _, tab1 = make_table(1, 4, 14, 14, 0.3, 3, 32)
    N = tab1.shape[0]
    B = 3
    x, w, b, gy = make_conv_inputs(B * N, 192, 192, 3, torch.float32, 32, bias="random")
    m = SparseConv2d(192, 192).cuda()
    with torch.no_grad():
        m.weight.copy_(w); m.bias.copy_(b)
    local = tab1.unsqueeze(0).repeat(B, 1, 1).cuda()
    glob = torch.stack([torch.where(tab1 >= 0, tab1 + i * N, tab1) for i in range(B)]).cuda()
    # the oracle sees the bf16-rounded operands the autocast path produces
    xb, wb, bb, gb_ = (t.bfloat16() for t in (x, w, b, gy))
    ey, egx, egw, egb = _oracle_grads(glob.reshape(-1, 9).cpu(), xb, wb, bb, gb_)
    for table in (local, glob.long()):           # int64 tables are accepted like in the reference
        m.zero_grad()
        xc = x.view(B, N, 192).cuda().requires_grad_(True)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = m(xc, table)
        assert y.shape == (B, N, 192) and y.dtype == torch.bfloat16
        y.backward(gy.view(B, N, 192).cuda().bfloat16())
        assert xc.grad.shape == xc.shape and xc.grad.dtype == torch.float32
        assert m.weight.grad.dtype == torch.float32
        assert oconv.rel_err(f32np(y).reshape(-1, 192), ey) < 2e-2
        assert oconv.rel_err(f32np(xc.grad).reshape(-1, 192), egx) < 2e-2
        assert oconv.rel_err(f32np(m.weight.grad), egw) < 2e-2
        assert oconv.rel_err(f32np(m.bias.grad), egb) < 2e-2


def test_autocast_parameter_copies_are_cached_until_the_parameters_change():
    """The bf16 copies of fp32 parameters are made once per parameter version (two forwards of activation
    checkpointing share them) and refreshed after an in-place update; gradients come back in fp32."""
    from eccv26_tad_b200 import SparseConv2d, SparseConv2dFunction
    _, _, table = make_table(1, 4, 14, 14, 0.3, 3, 41)
    n = table.shape[0]
    x, w, b, gy = make_conv_inputs(n, 64, 64, 3, torch.float32, 41, bias="random")
    m = SparseConv2d(64, 64).cuda()
    with torch.no_grad():
        m.weight.copy_(w); m.bias.copy_(b)
    tc, xc, gc = table.cuda(), x.cuda(), gy.cuda().bfloat16()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y1 = m(xc, tc)
        w1 = m._cast_cache[1]
        y2 = m(xc, tc)
        assert m._cast_cache[1] is w1 and w1.dtype == torch.bfloat16
        assert torch.equal(y1, y2)
        # gradients equal those of the explicit-cast route through the reference-shaped Function
        xa = xc.clone().requires_grad_(True)
        m.zero_grad()
        m(xa, tc).backward(gc)
        xb = xc.clone().requires_grad_(True)
        wr = m.weight.detach().clone().requires_grad_(True)
        br = m.bias.detach().clone().requires_grad_(True)
        SparseConv2dFunction.apply(xb.bfloat16(), tc, wr.bfloat16(), br.bfloat16(), 0, 0).backward(gc)
        assert m.weight.grad.dtype == torch.float32 and torch.equal(m.weight.grad, wr.grad)
        assert torch.equal(m.bias.grad, br.grad) and torch.equal(xa.grad, xb.grad)
        with torch.no_grad():
            m.weight.mul_(0.5)
        y3 = m(xc, tc)
        assert m._cast_cache[1] is not w1
        assert not torch.equal(y3, y1)


def test_function_apply_signature_and_partial_grads():
    from eccv26_tad_b200 import SparseConv2dFunction
    _, _, table = make_table(1, 2, 14, 14, 0.5, 3, 33)
    n = table.shape[0]
    x, w, b, gy = make_conv_inputs(n, 64, 64, 3, torch.bfloat16, 33, bias="random")
    xc = x.cuda()                                   # no grad for x
    wc = w.cuda().requires_grad_(True)
    y = SparseConv2dFunction.apply(xc, table.cuda(), wc, None, 0, 4096)
    y.backward(gy.cuda())
    assert wc.grad is not None and wc.grad.shape == wc.shape
    ey, _, egw, _ = _oracle_grads(table, x, w, torch.zeros(64), gy)
    assert oconv.rel_err(f32np(y), ey) < 2e-2
    assert oconv.rel_err(f32np(wc.grad), egw) < 2e-2
    with pytest.raises(ValueError, match="divisible by 4"):
        SparseConv2dFunction.apply(torch.randn(4, 6).cuda(), torch.zeros(4, 9, dtype=torch.int32).cuda(),
                                   torch.randn(9, 6, 8).cuda())


def test_pybind_module_shim_signatures():
    from eccv26_tad_b200 import opentad_sparse_ops as lib
    _, _, table = make_table(1, 3, 14, 14, 0.5, 3, 34)
    n = table.shape[0]
    x, w, b, gy = make_conv_inputs(n, 128, 128, 3, torch.bfloat16, 34, bias="random")
    tc, xc, wc, bc, gc = (t.cuda() for t in (table, x, w, b, gy))
    ey, egx, egw, _ = _oracle_grads(table, x, w, b, gy)
    y0, _, _, _ = _oracle_grads(table, x, w, torch.zeros(128), gy)
    assert oconv.rel_err(f32np(lib.fwd(xc, tc, wc, 128, 0)), y0) < 2e-2
    assert oconv.rel_err(f32np(lib.implicit_gemm_fwd_v2(xc, tc, wc, bc, 0)), ey) < 2e-2
    assert oconv.rel_err(f32np(lib.implicit_gemm_fwd_v2(xc, tc, wc, torch.Tensor(), 0)), y0) < 2e-2
    assert oconv.rel_err(f32np(lib.implicit_gemm_fwd_v2_chunked(xc, tc, wc, bc, 0, 4096)), ey) < 2e-2
    assert oconv.rel_err(f32np(lib.bwd_in(gc, tc, wc, n, 128, 0)), egx) < 2e-2
    assert oconv.rel_err(f32np(lib.bwd_w(gc, xc, tc, 128, 0)), egw) < 2e-2
    import sys
    lib.install()
    assert sys.modules["opentad_sparse_ops"].fwd is lib.fwd
    del sys.modules["opentad_sparse_ops"]


def test_kernel_size_5_module():
    from eccv26_tad_b200 import SparseConv2d
    _, _, table = make_table(1, 3, 14, 14, 0.4, 5, 35)
    n = table.shape[0]
    x, w, b, gy = make_conv_inputs(n, 64, 64, 5, torch.bfloat16, 35, bias="random")
    m = SparseConv2d(64, 64, kernel_size=5).cuda().bfloat16()
    with torch.no_grad():
        m.weight.copy_(w); m.bias.copy_(b)
    xc = x.cuda().requires_grad_(True)
    y = m(xc, table.cuda())
    y.backward(gy.cuda())
    ey, egx, egw, egb = _oracle_grads(table, x, w, b, gy)
    assert oconv.rel_err(f32np(y), ey) < 2e-2
    assert oconv.rel_err(f32np(xc.grad), egx) < 2e-2
    assert oconv.rel_err(f32np(m.weight.grad), egw) < 2e-2


def test_reference_wrapper_runs_unchanged_on_top_of_the_shim():
    """The reference's own ``sparse_conv_layer.py`` (byte-compiled by ``oracle/build_ref.py`` into ``oracle/_ref``;
    its ``import opentad_sparse_ops`` answered by this package's module) - ITS SparseConv2d / SparseConv2dFunction,
    forward and backward under bf16 autocast with fp32 master parameters, 2-D and batched 3-D input, and in plain
    fp32 - against the oracle."""
    from oracle import build_ref
    from eccv26_tad_b200 import opentad_sparse_ops as shim
    ref = build_ref.load_wrapper(shim)
    if ref is None:
        pytest.skip("oracle/_ref/ref_sparse_conv_layer.bytecode has not been built")
    assert ref.sparse_lib_opt is shim                     # no JIT fallback to the reference's CUDA sources
    _, _, tab1 = make_table(1, 6, 14, 14, 0.3, 3, 71)
    N = tab1.shape[0]
    B = 2
    glob = torch.cat([torch.where(tab1 >= 0, tab1 + i * N, tab1) for i in range(B)])
    x, w, b, gy = make_conv_inputs(B * N, 192, 192, 3, torch.float32, 71, bias="random")
    m = ref.SparseConv2d(192, 192).cuda()
    assert tuple(m.weight.shape) == (9, 192, 192)
    with torch.no_grad():
        m.weight.copy_(w); m.bias.copy_(b)
    xb, wb, bb, gb_ = (t.bfloat16() for t in (x, w, b, gy))
    ey, egx, egw, egb = _oracle_grads(glob, xb, wb, bb, gb_)
    cases = [(x.cuda(), glob.cuda(), gy.cuda().bfloat16()),                                     # [N, C], global indices
             (x.view(B, N, 192).cuda(), tab1.unsqueeze(0).repeat(B, 1, 1).cuda().long(),        # [B, N, C], local, int64
              gy.view(B, N, 192).cuda().bfloat16())]
    for xin, table, g in cases:
        m.zero_grad()
        xc = xin.clone().requires_grad_(True)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = m(xc, table)
        assert y.dtype == torch.bfloat16 and y.shape[:-1] == xin.shape[:-1]
        y.backward(g)
        assert oconv.rel_err(f32np(y).reshape(-1, 192), ey) < 2e-2
        assert oconv.rel_err(f32np(xc.grad).reshape(-1, 192), egx) < 2e-2
        assert oconv.rel_err(f32np(m.weight.grad), egw) < 2e-2
        assert oconv.rel_err(f32np(m.bias.grad), egb) < 2e-2
    # fp32, small-channel branch of the reference wrapper (fwd + bias added by the wrapper, :86-87)
    x, w, b, gy = make_conv_inputs(N, 64, 64, 3, torch.float32, 72, bias="random")
    m = ref.SparseConv2d(64, 64).cuda()
    with torch.no_grad():
        m.weight.copy_(w); m.bias.copy_(b)
    xc = x.cuda().requires_grad_(True)
    y = m(xc, tab1.cuda())
    y.backward(gy.cuda())
    ey, egx, egw, egb = _oracle_grads(tab1, x, w, b, gy)
    assert oconv.rel_err(f32np(y), ey) < 1e-5 and oconv.rel_err(f32np(xc.grad), egx) < 1e-5
    assert oconv.rel_err(f32np(m.weight.grad), egw) < 1e-5 and oconv.rel_err(f32np(m.bias.grad), egb) < 1e-5
    from eccv26_tad_b200 import ops
    assert ops.device_error() == 0


@pytest.mark.parametrize("kind", ["built", "given", "given_late", "asymmetric", "local"])
@pytest.mark.parametrize("amp", [False, True])
def test_extension_path_by_what_is_known_about_the_table(kind, amp):
    """The module's one extension call against the oracle: a table this package built (no validation), a caller's
    table before and after its validation has come back to the host, an asymmetric one (scatter form) and one with
    indices local to each batch row (whose heuristic asks the device)."""
    from eccv26_tad_b200 import SparseConv2d, build_neighbor_table
    B, C = 3, 64
    scores, _, tab = make_table(B * 2, 1, 14, 14, 0.3, 3, 61)
    N = tab.shape[0] // B
    x, w, b, gy = make_conv_inputs(B * N, C, 128, 3, torch.bfloat16, 61, bias="random")
    glob = tab.clone()
    if kind == "built":
        table = build_neighbor_table(scores.cuda(), 0.3, 14, 14)[1]
    elif kind == "local":
        one = tab[:N]
        glob = torch.cat([torch.where(one >= 0, one + i * N, one) for i in range(B)])
        table = one.unsqueeze(0).repeat(B, 1, 1).cuda()
    else:
        if kind == "asymmetric":
            glob[5] = -1
        table = glob.view(B, N, 9).cuda()
    m = SparseConv2d(C, 128).cuda()
    with torch.no_grad():
        m.weight.copy_(w); m.bias.copy_(b)
    m = m if amp else m.bfloat16()
    ey, egx, egw, egb = _oracle_grads(glob, x, w, b, gy)
    for again in range(2):
        m.zero_grad()
        xc = x.view(B, N, C).cuda().requires_grad_(True)
        with torch.autocast("cuda", dtype=torch.bfloat16, enabled=amp):
            y = m(xc, table)
        if kind == "given_late":
            torch.cuda.synchronize()
        y.backward(gy.view(B, N, 128).cuda())
        assert m.weight.grad.dtype == m.weight.dtype and m.bias.grad.dtype == m.bias.dtype
        for got, ref in ((y, ey), (xc.grad, egx), (m.weight.grad, egw), (m.bias.grad, egb)):
            assert oconv.rel_err(f32np(got).reshape(ref.shape), ref) < 2e-2


def _small_layer(table, C=64, seed=81):
    """A bf16 layer with inputs for `table` (on the CPU), and what it has to give."""
    from eccv26_tad_b200 import SparseConv2d
    n, kk = table.shape
    ks = int(kk ** 0.5)
    x, w, b, gy = make_conv_inputs(n, C, C, ks, torch.bfloat16, seed, bias="random")
    m = SparseConv2d(C, C, kernel_size=ks).cuda().bfloat16()
    with torch.no_grad():
        m.weight.copy_(w); m.bias.copy_(b)
    return m, x.cuda().requires_grad_(True), gy.cuda(), _oracle_grads(table, x, w, b, gy)


def _run(m, x, table, gy):
    y = m(x, table)
    return (y.detach(),) + torch.autograd.grad(y, (x, m.weight, m.bias), gy)


def _check(got, want):
    for a, b in zip(got, want):
        assert oconv.rel_err(f32np(a), b) < 2e-2


@pytest.mark.parametrize("dtype", [torch.int64, torch.int32])
def test_what_one_stream_found_out_about_a_table_is_not_read_by_another_before_it_is_there(dtype):
    """The int32 form of an int64 table and the status word of an asymmetric one, asked for on a second stream while
    the first has not got to them yet."""
    _, _, table = make_table(1, 8, 14, 14, 0.4, 3, 81)
    table[7] = -1                                                       # asymmetric: the input gradient is the scatter form's
    m, x, gy, want = _small_layer(table)
    _check(_run(m, x, table.cuda(), gy), want)                          # kernels loaded
    t = table.to(dtype).cuda()
    busy, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(40_000_000)                                   # some 20 ms in front of the conversion and the check
        first = _run(m, x, t, gy)
    with torch.cuda.stream(other):
        second = _run(m, x, t, gy)
    torch.cuda.synchronize()
    _check(second, want)
    _check(first, want)


@pytest.mark.parametrize("dtype", [torch.int64, torch.int32])
@pytest.mark.parametrize("symmetric", [True, False])
def test_a_table_first_met_under_graph_capture(dtype, symmetric):
    """What a captured call finds out is in the graph's memory and there only when the graph has run: an eager call before
    the first replay asks anew, and the graph follows its table."""
    _, _, table = make_table(1, 8, 14, 14, 0.4, 3, 82)
    if not symmetric:
        table[9] = -1
    m, x, gy, want = _small_layer(table)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        for warm in (table.cuda(), table.to(dtype).cuda()):
            _run(m, x, warm, gy)
        s.synchronize()
        t = table.to(dtype).cuda()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            out = _run(m, x, t, gy)
        _check(_run(m, x, t, gy), want)
        torch.cuda.synchronize()
        for seed in (82, 83):
            _, _, new = make_table(1, 8, 14, 14, 0.4, 3, seed)
            if seed == 83:
                new[20] = -1                                            # symmetric no more
            else:
                new = table
            t.copy_(new.to(dtype))
            junk = torch.full((1 << 20,), -5, dtype=torch.int32, device="cuda")
            g.replay()
            torch.cuda.synchronize()
            _check(out, _oracle_grads(new, *(v.detach().cpu() for v in (x, m.weight, m.bias, gy))))
            del junk


def test_a_symmetric_table_read_with_another_stencil():
    """Rows of 9 taps that this package built are rows of 25 taps of no symmetry."""
    from eccv26_tad_b200 import build_neighbor_table
    scores, _, table = make_table(25, 1, 10, 10, 0.4, 3, 84)            # 1 000 rows of 9 = 360 of 25
    built = build_neighbor_table(scores.cuda(), 0.4, 10, 10)[1]
    assert torch.equal(built.cpu(), table)
    by25 = table.reshape(-1, 25)
    m, x, gy, want = _small_layer(torch.where(by25 < by25.shape[0], by25, -1))      # entries out of range read as zero
    _check(_run(m, x, built.reshape(-1, 25), gy), want)
    m, x, gy, want = _small_layer(table)
    _check(_run(m, x, built, gy), want)


def test_forward_mode_differentiation_is_refused():
    """There is no formula for it: a dual tensor must not come out without its tangent."""
    import torch.autograd.forward_ad as fwad
    _, _, table = make_table(1, 2, 14, 14, 0.4, 3, 85)
    m, x, _, want = _small_layer(table)
    t, params = table.cuda(), {"weight": m.weight.detach(), "bias": m.bias.detach()}
    with fwad.dual_level():
        for name in ("x", "weight", "bias"):
            v = x.detach() if name == "x" else params[name]
            dual = fwad.make_dual(v, torch.ones_like(v))
            with pytest.raises(NotImplementedError, match="forward mode"):
                torch.func.functional_call(m, {**params, name: dual} if name != "x" else params, (dual if name == "x" else x, t))
            with pytest.raises(NotImplementedError, match="forward mode"), torch.no_grad():
                torch.func.functional_call(m, {**params, name: dual} if name != "x" else params, (dual if name == "x" else x, t))
        assert oconv.rel_err(f32np(m(x, t)), want[0]) < 2e-2
    for transform in (lambda: torch.func.jvp(lambda v: m(v, t), (x.detach(),), (torch.ones_like(x),)),
                      lambda: torch.func.vmap(lambda v: m(v, t))(torch.stack([x.detach()] * 2)),
                      lambda: torch.func.grad(lambda v: m(v, t).sum())(x.detach())):
        with pytest.raises(RuntimeError):
            transform()


@pytest.mark.parametrize("kind", ["plain", "batched", "local", "amp"])
@pytest.mark.parametrize("grad", [True, False])
def test_a_traced_module_follows_its_inputs(kind, grad):
    """torch.jit.trace records the layer, not the features it was traced with."""
    from eccv26_tad_b200 import SparseConv2d
    _, _, table = make_table(2, 2, 14, 14, 0.4, 3, 86)
    n, C = table.shape[0], 64
    x, w, b, gy = (t.cuda() for t in make_conv_inputs(n, C, C, 3, torch.float32, 86, bias="random"))
    t, m = table.cuda(), SparseConv2d(C, C).cuda()
    with torch.no_grad():
        m.weight.copy_(w); m.bias.copy_(b)
    if kind != "plain":
        x, t = x.view(2, n // 2, C), t.view(2, n // 2, 9)
    if kind == "local":
        t = t[:1].repeat(2, 1, 1)
    other = torch.randn_like(x)
    with torch.set_grad_enabled(grad), torch.autocast("cuda", dtype=torch.bfloat16, enabled=kind == "amp"):
        traced = torch.jit.trace(m, (x, t), check_trace=False)
        for v in (x, other):
            v.requires_grad_(grad)
            got, want = traced(v, t), m(v, t)
            assert got.shape == want.shape and got.dtype == want.dtype and torch.equal(got, want)
            assert got.requires_grad == grad
            if grad:
                g = [torch.autograd.grad(y, (v, m.weight, m.bias), gy.view(y.shape).to(y.dtype)) for y in (got, want)]
                for a, e in zip(*g):
                    # under autocast the module rounds each gradient of a parameter once, as the cast in the trace does
                    assert a.dtype == e.dtype and oconv.rel_err(f32np(a), f32np(e)) < 1e-5


@pytest.mark.parametrize("known", [True, False])
def test_a_backward_without_a_plan_takes_no_workspace_for_one(known):
    """C = 256 at some 500 rows: a few MB of partial sums, not the 74 MB of the pair lists' pieces."""
    from eccv26_tad_b200 import ops
    _, _, table = make_table(1, 8, 14, 14, 0.3, 3, 87)
    m, x, gy, want = _small_layer(table, C=256)
    t = table.cuda()
    if known:
        ops.mark_symmetric(t)
    for run in (lambda: _run(m, x, t, gy)[1:], lambda: ops.conv_bwd(gy, x.detach(), t, m.weight.detach(), assume_symmetric=known)):
        _check(run(), want[1:])
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        run()
        torch.cuda.synchronize()
        assert torch.cuda.max_memory_allocated() - before < 24 << 20
