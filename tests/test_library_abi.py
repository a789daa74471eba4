"""CPU tier: the C-ABI library loads, exports every symbol the header declares, and rejects
bad arguments on the host (no kernel is launched by anything in this file)."""
import ctypes
import os
import re

import pytest

from eccv26_tad_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_symbols():
    text = open(os.path.join(ROOT, "include", "svtad.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(svtad_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_are_exported_and_bound():
    names = _declared_symbols()
    assert len(names) >= 12
    lib = ctypes.CDLL(_lib.LIB_PATH)
    for n in names:
        assert hasattr(lib, n), f"{n} declared in include/svtad.h but not exported"
        assert n in _lib.SIGNATURES, f"{n} has no ctypes signature"
    assert sorted(_lib.SIGNATURES) == names


def test_version_and_error_string():
    lib = _lib.load()
    assert lib.svtad_version() >= 100
    assert isinstance(_lib.last_error(), str)


def test_host_side_validation_returns_codes():
    lib = _lib.load()
    # C_in % 4 != 0 -> same complaint as the reference wrapper (sparse_conv_layer.py:39-42)
    rc = lib.svtad_conv_fwd(None, None, None, None, None, 10, 6, 8, 9, 0, _lib.F32, None, 0, None)
    assert rc == _lib.ERR_UNSUPPORTED and "divisible by 4" in _lib.last_error()
    rc = lib.svtad_conv_fwd(None, None, None, None, None, -1, 8, 8, 9, 0, _lib.F32, None, 0, None)
    assert rc == _lib.ERR_ARG
    rc = lib.svtad_conv_fwd(None, None, None, None, None, 4, 8, 8, 9, 0, 7, None, 0, None)
    assert rc == _lib.ERR_ARG and "dtype" in _lib.last_error()
    rc = lib.svtad_conv_fwd(None, None, None, None, None, 4, 8, 8, 9, 0, _lib.F32, None, 0, None)
    assert rc == _lib.ERR_ARG and "null" in _lib.last_error()
    rc = lib.svtad_conv_wgrad(None, None, None, None, None, 4, 8, 8, 9, 0, _lib.F32, None, 0, None)
    assert rc == _lib.ERR_ARG
    # a bias-gradient pointer at an odd offset is refused before any launch (the kernels store 8 bytes at a time)
    rc = lib.svtad_conv_wgrad(256, 256, 256, 256, 256 + 6, 4, 8, 8, 9, 0, _lib.BF16, 256, 1 << 20, None)
    assert rc == _lib.ERR_ARG and "gb" in _lib.last_error()
    rc = lib.svtad_table_build(None, 4, 196, 300, 14, 14, 3, None, None, None)
    assert rc == _lib.ERR_ARG and "k_keep" in _lib.last_error()
    rc = lib.svtad_table_build(None, 4, 200, 20, 14, 14, 3, None, None, None)
    assert rc == _lib.ERR_ARG
    rc = lib.svtad_table_init(1, 1, 14, 14, 4, None, None)
    assert rc == _lib.ERR_ARG and "odd" in _lib.last_error()
    with pytest.raises(ValueError):
        _lib.check(rc)
    # the one-call backward: something must be asked for, a bias gradient needs the weight gradient
    rc = lib.svtad_conv_bwd(None, None, None, None, None, None, None, 4, 8, 8, 9, 0, _lib.F32, None, None, 0, None)
    assert rc == _lib.ERR_ARG and "neither" in _lib.last_error()
    rc = lib.svtad_conv_bwd(None, None, None, None, 1, None, 1, 4, 8, 8, 9, 0, _lib.F32, None, None, 0, None)
    assert rc == _lib.ERR_ARG and "gb needs gw" in _lib.last_error()
    # fused selection + remap of a later round
    rc = lib.svtad_table_select_remap(None, None, 2, 100, 101, 9, None, None, None, None)
    assert rc == _lib.ERR_ARG and "k_keep" in _lib.last_error()
    rc = lib.svtad_table_select_remap(None, None, 2, 100, 50, 9, None, None, None, None)
    assert rc == _lib.ERR_ARG and "null" in _lib.last_error()
    rc = lib.svtad_table_select_remap(1, 1, 2, 60000, 50, 9, 1, None, 1, None)
    assert rc == _lib.ERR_UNSUPPORTED and "limit" in _lib.last_error()
    assert lib.svtad_table_select_remap(None, None, 0, 100, 50, 9, None, None, None, None) == 0
    assert lib.svtad_workspace_bytes(_lib.OP_BWD, 9440, 192, 192, 9, _lib.BF16) >= \
        lib.svtad_workspace_bytes(_lib.OP_WGRAD, 9440, 192, 192, 9, _lib.BF16) + 9440 * 192 * 4
    # empty problems are fine and touch nothing
    assert lib.svtad_conv_fwd(None, None, None, None, None, 0, 8, 8, 9, 0, _lib.F32, None, 0, None) == 0
    assert lib.svtad_table_init(0, 8, 14, 14, 3, None, None) == 0


def test_workspace_and_path_queries():
    lib = _lib.load()
    assert lib.svtad_workspace_bytes(_lib.OP_FWD, 9440, 192, 192, 9, _lib.BF16) == 0
    w = lib.svtad_workspace_bytes(_lib.OP_WGRAD, 9440, 192, 192, 9, _lib.BF16)
    assert w >= 9 * 192 * 192 * 4
    assert lib.svtad_workspace_bytes(_lib.OP_DGRAD, 100, 192, 192, 9, _lib.BF16) >= 100 * 192 * 4
    assert lib.svtad_path_for(_lib.OP_FWD, 9440, 192, 192, 9, _lib.BF16) == 1
    assert lib.svtad_path_for(_lib.OP_FWD, 784, 192, 192, 9, _lib.F32) == 0
    assert lib.svtad_path_for(_lib.OP_FWD, 784, 48, 48, 9, _lib.BF16) == 0


def test_module_surface_matches_reference():
    import inspect
    import torch
    from eccv26_tad_b200 import SparseConv2d, SparseConv2dFunction
    m = SparseConv2d(8, 12)
    assert tuple(m.weight.shape) == (9, 8, 12) and tuple(m.bias.shape) == (12,)
    assert m.chunk_size == 4096
    assert list(m.state_dict()) == ["weight", "bias"]
    assert SparseConv2d(8, 12, bias=False).bias is None
    assert tuple(SparseConv2d(8, 4, kernel_size=5).weight.shape) == (25, 8, 4)
    sig = inspect.signature(SparseConv2dFunction.forward)
    assert list(sig.parameters) == ["ctx", "x", "neighbor_indices", "weight", "bias", "tokens_per_batch", "chunk_size"]
    with pytest.raises(ValueError):   # no CPU path, loudly
        m(torch.zeros(4, 8), torch.zeros(4, 9, dtype=torch.int32))
    from eccv26_tad_b200 import opentad_sparse_ops as shim
    for name in ("fwd", "bwd_in", "bwd_w", "implicit_gemm_fwd_v2", "implicit_gemm_fwd_v2_chunked"):
        assert callable(getattr(shim, name))


def test_shape_mismatches_raise_before_any_launch():
    import torch
    from eccv26_tad_b200 import ops
    nbr = torch.zeros(5, 9, dtype=torch.int32)
    with pytest.raises(ValueError):
        ops._check_shapes("conv_fwd", 4, 9, nbr)
    with pytest.raises(ValueError):
        ops._check_shapes("conv_wgrad", 5, 9, nbr, grad_output=(torch.zeros(4, 8), 8))
    ops._check_shapes("conv_wgrad", 5, 9, nbr, grad_output=(torch.zeros(5, 8), 8))


def test_static_wgrad_wrapper_checks_shapes_before_the_library_sees_them():
    """conv_wgrad_static cannot copy or allocate, so every mismatch must be refused on the host."""
    import torch
    from eccv26_tad_b200 import ops

    class FakeCuda(torch.Tensor):          # CPU storage that claims to live on the device: nothing is launched
        is_cuda = True

    def t(*shape, dtype=torch.bfloat16):
        return torch.zeros(*shape, dtype=dtype).as_subclass(FakeCuda)

    n, c = 64, 8
    gw, gb = t(9, c, c), t(c)
    nbr = t(n, 9, dtype=torch.int32)
    with pytest.raises(ValueError, match="grad_output"):
        ops.conv_wgrad_static(t(n - 1, c), t(n, c), nbr, gw, gb)
    with pytest.raises(ValueError, match="neighbor table"):
        ops.conv_wgrad_static(t(n, c), t(n, c), t(n - 2, 9, dtype=torch.int32), gw, gb)
    with pytest.raises(ValueError, match="gb must hold"):
        ops.conv_wgrad_static(t(n, c), t(n, c), nbr, gw, t(c + 1))
    with pytest.raises(ValueError, match="gb must hold"):
        ops.conv_wgrad_static(t(n, c), t(n, c), nbr, gw, t(c, dtype=torch.float32))
    with pytest.raises(ValueError, match="16-byte aligned"):
        ops.conv_wgrad_static(t(n, c), t(n, c), nbr, gw, t(c + 3)[3:])


def test_tables_built_by_the_package_are_tagged_symmetric():
    import torch
    from eccv26_tad_b200 import ops
    a = torch.zeros(4, 9, dtype=torch.int32)
    assert not ops.is_known_symmetric(a)
    ops.mark_symmetric(a)
    assert ops.is_known_symmetric(a) and ops.is_known_symmetric(a.view(2, 2, 9))
    a[0, 0] = 1                                       # written to: the tag no longer holds
    assert not ops.is_known_symmetric(a)


def test_legacy_checkpoint_layout_is_remapped_on_load():
    """Weights stored as (C_in, 9, C_out) load into the (9, C_in, C_out) parameter, as with the reference's
    remap_legacy_sparse_conv_weights (opentad/utils/checkpoint.py:44-57)."""
    import torch
    from eccv26_tad_b200 import SparseConv2d, remap_legacy_sparse_conv_weights

    class Adapter(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.sparse_conv = SparseConv2d(8, 12)

    src = Adapter()
    legacy = {k: v.clone() for k, v in src.state_dict().items()}
    legacy["sparse_conv.weight"] = legacy["sparse_conv.weight"].permute(1, 0, 2).contiguous()   # (C_in, 9, C_out)
    assert legacy["sparse_conv.weight"].shape == (8, 9, 12)
    dst = Adapter()
    dst.load_state_dict({k: v.clone() for k, v in legacy.items()})
    assert torch.equal(dst.sparse_conv.weight, src.sparse_conv.weight)
    out = remap_legacy_sparse_conv_weights({k: v.clone() for k, v in legacy.items()}, Adapter().state_dict())
    assert torch.equal(out["sparse_conv.weight"], src.sparse_conv.weight)
    # current-layout checkpoints are left alone
    dst2 = Adapter()
    dst2.load_state_dict(src.state_dict())
    assert torch.equal(dst2.sparse_conv.weight, src.sparse_conv.weight)


def test_reference_wrapper_binds_to_the_shim_when_built():
    """Where ``oracle/_ref`` holds the byte-compiled reference wrapper, executing it with this package's
    ``opentad_sparse_ops`` in place picks the shim up (no JIT build of the reference's CUDA sources) and exposes
    the reference's class with the reference's constructor signature."""
    import inspect
    from oracle import build_ref
    from eccv26_tad_b200 import SparseConv2d, opentad_sparse_ops as shim
    ref = build_ref.load_wrapper(shim)
    if ref is None:
        pytest.skip("oracle/_ref/ref_sparse_conv_layer.bytecode has not been built")
    assert ref.sparse_lib_opt is shim
    theirs = list(inspect.signature(ref.SparseConv2d.__init__).parameters)
    ours = list(inspect.signature(SparseConv2d.__init__).parameters)
    assert ours[:len(theirs)] == theirs
    assert list(ref.SparseConv2d(8, 12).state_dict()) == list(SparseConv2d(8, 12).state_dict())


def test_top_level_opentad_sparse_ops_module():
    """``import opentad_sparse_ops`` (the module the reference wrapper looks for, built by the reference's setup.py as
    a CUDA extension) resolves to this package's callables without any install() call; setup.py ships it as a
    top-level module beside the package."""
    import importlib
    import sys
    sys.modules.pop("opentad_sparse_ops", None)
    mod = importlib.import_module("opentad_sparse_ops")
    from eccv26_tad_b200 import opentad_sparse_ops as shim
    for name in ("fwd", "bwd_in", "bwd_w", "implicit_gemm_fwd_v2", "implicit_gemm_fwd_v2_chunked"):
        assert getattr(mod, name) is getattr(shim, name)
    text = open(os.path.join(ROOT, "setup.py")).read()
    assert 'py_modules=["opentad_sparse_ops"]' in text and "libsvtad.so" in text


def test_concurrency_hint_round_trip_and_clamping():
    """The hint is host state of the library: settable and readable without a GPU, clamped to [1, 16]."""
    lib = _lib.load()
    start = lib.svtad_get_concurrency()
    try:
        assert lib.svtad_set_concurrency(3) == start and lib.svtad_get_concurrency() == 3
        assert lib.svtad_set_concurrency(0) == 3 and lib.svtad_get_concurrency() == 1
        assert lib.svtad_set_concurrency(99) == 1 and lib.svtad_get_concurrency() == 16
    finally:
        lib.svtad_set_concurrency(start)


def test_workspace_sizes_do_not_depend_on_the_concurrency_hint():
    """A workspace sized once must stay valid when the hint changes (svtad_conv_bwd plans its weight gradient for half
    the GPU whatever the caller's hint): svtad_workspace_bytes covers the plan under every hint."""
    lib = _lib.load()
    shapes = [(n, c, kk) for n in (4, 944, 3200, 9440, 17280, 18880, 40000, 226560) for c in (64, 192, 256, 768, 1024)
              for kk in (9, 25)]
    start = lib.svtad_get_concurrency()
    try:
        lib.svtad_set_concurrency(1)
        base = {s: [lib.svtad_workspace_bytes(op, s[0], s[1], s[1], s[2], _lib.BF16) for op in (_lib.OP_WGRAD, _lib.OP_BWD)]
                for s in shapes}
        for hint in (2, 3, 4, 7, 16):
            lib.svtad_set_concurrency(hint)
            for s in shapes:
                got = [lib.svtad_workspace_bytes(op, s[0], s[1], s[1], s[2], _lib.BF16) for op in (_lib.OP_WGRAD, _lib.OP_BWD)]
                assert got == base[s], (hint, s)
    finally:
        lib.svtad_set_concurrency(start)


def test_a_plan_is_wanted_where_one_layer_pays_for_it():
    """svtad_plan_wanted: what a plan saves one layer in one pass has to exceed what making it takes."""
    lib = _lib.load()

    def wanted(n, c, kk, density, dtype=_lib.BF16):
        return lib.svtad_plan_wanted(n, c, c, kk, dtype, density)
    assert wanted(18880, 1024, 9, 0.35) == 3 and wanted(18880, 512, 9, 0.35) == 3 and wanted(18880, 384, 9, 0.35, _lib.F16) == 3
    assert wanted(4720, 768, 9, 0.35) == 3 and wanted(3920, 1024, 9, 0.51) == 0 and wanted(75520, 256, 9, 0.59) == 0
    assert wanted(19600, 192, 9, 0.51) == 0 and wanted(43200, 128, 9, 0.55) == 0            # 17 to 25 us for 5 to 15
    assert wanted(18880, 256, 9, 0.35) == 0 and wanted(1770, 1024, 9, 0.35) == 0
    assert wanted(62720, 512, 9, 0.91) == 0 and wanted(50240, 384, 9, 0.75) == 0            # hardly a neighbor missing
    assert wanted(18880, 256, 25, 0.28) == 2 and wanted(2360, 512, 25, 0.52) == 0           # 5x5: the lists alone
    assert wanted(12800, 320, 9, 0.27) == 3 and wanted(113280, 192, 9, 0.35) == 1           # lists of 256 channels for 192: rows alone
    for n, c, density, alone in ((18880, 512, 0.35, 1), (113280, 384, 0.35, 1), (75520, 256, 0.35, 0), (50240, 512, 0.75, 0),
                                 (4720, 768, 0.35, 0), (9440, 768, 0.35, 1), (7840, 768, 0.51, 1), (18880, 256, 0.35, 0)):
        fwd = lib.svtad_plan_wanted_fwd(n, c, c, 9, _lib.BF16, density)
        assert fwd == alone and fwd <= (wanted(n, c, 9, density) & 1)
    assert wanted(18880, 1024, 9, 0.35, _lib.F32) == 0 and wanted(140000, 1024, 9, 0.35) == 0 and wanted(18880, 1024, 1, 0.35) == 0


@pytest.mark.parametrize("n,cin,cout,density,wanted", [
    (8736, 384, 384, 0.20, 0), (9700, 384, 384, 0.20, 1),        # one wave of tile pairs, two
    (37760, 320, 320, 0.35, 1), (34496, 768, 192, 0.45, 1), (75520, 256, 256, 0.35, 0),
    (5120, 1024, 1024, 0.20, 0), (5121, 1024, 1024, 0.20, 1),
])
def test_a_forward_s_row_order_is_wanted_by_the_waves_it_saves(n, cin, cout, density, wanted):
    lib = _lib.load()
    assert lib.svtad_plan_wanted_fwd(n, cin, cout, 9, _lib.BF16, density) == wanted
    assert lib.svtad_plan_wanted_fwd(n, cin, cout, 9, _lib.F32, density) == 0


@pytest.mark.parametrize("n,cin,cout,density,wanted", [
    (18940, 512, 192, 0.188, 0), (8960, 640, 256, 0.188, 0), (7644, 512, 384, 0.266, 0),      # the longest tile takes what the order saves
    (8960, 640, 768, 0.188, 1), (10192, 1024, 1024, 0.509, 1), (56252, 384, 384, 0.508, 1),
])
def test_no_row_order_for_a_forward_whose_longest_tile_decides(n, cin, cout, density, wanted):
    assert _lib.load().svtad_plan_wanted_fwd(n, cin, cout, 9, _lib.BF16, density) == wanted


@pytest.mark.parametrize("cin,cout,halves,bn", [(640, 640, 1, 128), (896, 896, 1, 128), (512, 960, 2, 192), (640, 1024, 1, 256),
                                                (512, 640, 2, 256), (320, 320, 1, 192), (1024, 1024, 2, 256)])
def test_column_block_of_a_weight_gradient_by_pairs(cin, cout, halves, bn):
    """By what its own steps take, which shows in the pieces its workspace holds: two of 128 * halves rows and a block's columns, and
    a record, for each of 148 CTAs."""
    lib = _lib.load()
    each = 2 * 128 * halves * bn * 4 + 16
    assert lib.svtad_bwd_workspace_bytes(18880, cin, cout, 9, _lib.BF16, 2, 0) == (148 * each + 255) // 256 * 256


def test_workspace_sizes_count_the_pair_lists_only_where_a_plan_is_used():
    """The weight gradient by pair lists parks pieces of its sums (74 MB at C = 256); a call without a plan does not."""
    lib = _lib.load()
    mb = 1 << 20
    for dtype in (_lib.BF16, _lib.F16):
        for n, most in ((100, 5), (4720, 16), (18880, 19)):
            assert lib.svtad_workspace_bytes(_lib.OP_WGRAD, n, 256, 256, 9, dtype) < most * mb
            plain, listed = (lib.svtad_bwd_workspace_bytes(n, 256, 256, 9, dtype, use, 0) for use in (0, 2))
            assert plain < most * mb < listed
            assert lib.svtad_bwd_workspace_bytes(n, 256, 256, 9, dtype, 1, 0) == plain             # the row order takes none
            scatter = lib.svtad_workspace_bytes(_lib.OP_DGRAD, n, 256, 256, 9, dtype)
            assert lib.svtad_bwd_workspace_bytes(n, 256, 256, 9, dtype, 0, 1) == plain + scatter
            assert lib.svtad_workspace_bytes(_lib.OP_BWD, n, 256, 256, 9, dtype) == listed + scatter
        assert lib.svtad_workspace_bytes(_lib.OP_WGRAD, 18880, 192, 192, 9, dtype) <= lib.svtad_static_workspace_bytes()
    # fp32: several ranges' partials fit the built-in workspace, one range's where they can
    for c in (64, 192, 256, 320, 384, 512, 704, 768):
        assert lib.svtad_workspace_bytes(_lib.OP_WGRAD, 18880, c, c, 9, _lib.F32) <= lib.svtad_static_workspace_bytes()
    assert lib.svtad_bwd_workspace_bytes(0, 256, 256, 9, _lib.BF16, 3, 1) == 0


def test_entering_a_table_costs_the_same_however_many_tables_are_alive():
    import time
    import torch
    from eccv26_tad_b200 import ops

    def per_table(count):
        tables = [torch.zeros(1, 9, dtype=torch.int32) for _ in range(count)]
        t0 = time.perf_counter()
        for t in tables:
            ops.mark_symmetric(t)
        return (time.perf_counter() - t0) / count, tables
    per_table(200)
    few, _ = per_table(200)
    _, alive = per_table(30000)
    many, more = per_table(2000)
    assert many < 20 * few + 20e-6          # a look at each of 30 000 would take hundreds of microseconds
    assert all(ops.is_known_symmetric(t) for t in alive + more)


def test_a_symmetric_table_is_symmetric_in_rows_of_its_own_length():
    import torch
    from eccv26_tad_b200 import ops
    t = ops.mark_symmetric(torch.zeros(100, 9, dtype=torch.int32))
    assert ops.is_known_symmetric(t) and ops.is_known_symmetric(t.view(4, 25, 9)) and ops.is_known_symmetric(t[:50])
    assert not ops.is_known_symmetric(t.view(36, 25)) and not ops.is_known_symmetric(t.view(1, 36, 25))
    assert ops.is_known_symmetric(t.view(-1))           # no row length to go by
