"""GPU tier: the fp32 kernels that split their operands into bf16 planes for the tensor cores (csrc/conv_f32_tc.cu), at the
edges of their tiles and at values that the planes cannot hold, against sums over the existing pairs in 64 bits."""
import numpy as np
import pytest
import torch

from tests.helpers import make_conv_inputs, make_table

pytestmark = pytest.mark.gpu

# Relative error (2-norm).  A step of 64 products takes four instructions into one accumulator, each of which cuts off less than
# one unit (2^-23) of it: 4.8e-7 if all cut alike; the steps' sums are then rounded to nearest, half a unit each, at random.
BOUND = 5e-7


def _ops():
    from eccv26_tad_b200 import ops
    return ops


def _chain(n, kk, density, seed):
    """A symmetric table of any number of rows: tap kk - 1 - k undoes tap k."""
    rng = np.random.default_rng(seed)
    t = np.full((n, kk), -1, np.int32)
    t[:, kk // 2] = np.arange(n)
    for k in range(kk // 2):
        d = kk // 2 - k
        i = np.nonzero(rng.random(max(0, n - d)) < density)[0]
        t[i, k] = i + d
        t[i + d, kk - 1 - k] = i
    return torch.from_numpy(t)


def _pairs(table, k, tpb):
    i = torch.nonzero(table[:, k] >= 0).flatten()
    j = table[i, k].long() + (torch.div(i, tpb, rounding_mode="floor") * tpb if tpb else 0)
    return i, j


def _truth(table, x, w, b, gy, tpb=0):
    x, w, b, gy = x.double(), w.double(), b.double(), gy.double()
    y, gx, gw = torch.zeros(len(x), w.shape[2]).double(), torch.zeros_like(x), torch.zeros_like(w)
    for k in range(table.shape[1]):
        i, j = _pairs(table, k, tpb)
        y.index_add_(0, i, x[j] @ w[k])
        gx.index_add_(0, j, gy[i] @ w[k].T)
        gw[k] = x[j].T @ gy[i]
    return y + b, gx, gw, gy.sum(0)


def _run(table, x, w, b, gy, tpb=0):
    ops = _ops()
    t, x, w, b, gy = (v.cuda() for v in (table, x, w, b, gy))
    y = ops.conv_fwd(x, t, w, b, tpb)
    gx = ops.conv_dgrad(gy, t, w, tpb, assume_symmetric=True)
    gw, gb = ops.conv_wgrad(gy, x, t, w.shape[0], tpb)
    torch.cuda.synchronize()
    assert ops.device_error() == 0
    return [v.cpu() for v in (y, gx, gw, gb)]


def _close(got, truth):
    for name, a, e in zip(("y", "gx", "gw", "gb"), got, truth):
        err = (a.double() - e).norm() / e.norm().clamp_min(1e-300)
        assert err < BOUND, f"{name}: {err:.2e}"


@pytest.mark.parametrize("n,cin,cout,kk", [
    (1, 4, 4, 1),                # one row, one tap
    (127, 64, 64, 9), (128, 64, 128, 9), (129, 128, 64, 9),      # edges of a row tile
    (300, 60, 68, 9),            # a partial chunk, a partial column block behind a whole one
    (640, 132, 4, 25), (639, 132, 4, 25),      # the weight gradient's rule on both sides; a second block of 4 channels
    (700, 32, 36, 49),           # 49 taps
    (2000, 192, 192, 9),         # a half block of channels; K steps not shared
    (200, 1024, 64, 9),          # K steps shared by eight
    (30011, 8, 12, 9),           # several lists per range of tokens
])
def test_edges_of_tiles_chunks_and_lists(n, cin, cout, kk):
    table = _chain(n, kk, 0.35, n)
    x, w, b, gy = make_conv_inputs(n, cin, cout, int(kk ** 0.5), torch.float32, n, bias="random")
    _close(_run(table, x, w, b, gy), _truth(table, x, w, b, gy))


@pytest.mark.parametrize("n,kk,density", [(n, kk, d) for n in (3, 4, 8, 64, 65) for kk, d in ((9, 0.0), (49, 0.03), (49, 1.0))])
def test_taps_without_a_neighbor_are_left_out_of_few_rows(n, kk, density):
    table = _chain(n, kk, density, n)
    x, w, b, gy = make_conv_inputs(n, 192, 68, int(kk ** 0.5), torch.float32, n, bias="random")
    _close(_run(table, x, w, b, gy), _truth(table, x, w, b, gy))
    if n == 64:                 # nothing at all: the bias, and zeros
        table[:] = -1
        y, gx, gw, gb = _run(table, x, w, b, gy)
        assert torch.equal(y, b.expand(n, -1)) and not gx.any() and not gw.any()


@pytest.mark.parametrize("n,cin,cout,kk", [(1898, 64, 64, 9), (1899, 64, 64, 9), (2599, 16, 20, 9), (2600, 16, 20, 9),
                                           (899, 64, 1024, 49), (900, 64, 1024, 49)])
def test_both_sides_of_the_weight_gradient_s_rule(n, cin, cout, kk):
    table = _chain(n, kk, 0.2, n)
    x, w, b, gy = make_conv_inputs(n, cin, cout, int(kk ** 0.5), torch.float32, n, bias="random")
    _close(_run(table, x, w, b, gy), _truth(table, x, w, b, gy))


def test_rows_that_are_16_but_not_32_byte_aligned_and_batch_local_indices():
    n, c = 900, 64
    table = _chain(n // 3, 9, 0.5, 3).repeat(3, 1)
    x, w, b, gy = make_conv_inputs(n, c, c, 3, torch.float32, 11, bias="random")
    shifted = [torch.empty(v.numel() + 4, device="cuda")[4:].copy_(v.flatten().cuda()).view(v.shape) for v in (x, w, gy)]
    assert all(v.data_ptr() % 32 == 16 for v in shifted)
    tpb = n // 3
    truth = _truth(table, x, w, b, gy, tpb)
    aligned = _run(table, x, w, b, gy, tpb)
    _close(aligned, truth)
    got = _run(table, shifted[0], shifted[1], b, shifted[2], tpb)
    assert all(torch.equal(a, e) for a, e in zip(got, aligned))


@pytest.mark.parametrize("sx,sw", [(2.0 ** 100, 2.0 ** -90), (2.0 ** -60, 2.0 ** -30), (2.0 ** -100, 1.0)])
def test_precision_does_not_hang_on_the_scale(sx, sw):
    _, _, table = make_table(1, 14, 14, 14, 0.3, 3, 5)
    x, w, b, gy = make_conv_inputs(table.shape[0], 64, 64, 3, torch.float32, 5)
    x, w = x * sx, w * sw
    gy = gy * sx if 2.0 ** -80 < sx < 1 else gy      # the weight gradient's products stay in range
    _close(_run(table, x, w, b, gy), _truth(table, x, w, b, gy))


@pytest.mark.parametrize("small", ["x", "w", "gy"])
@pytest.mark.parametrize("scale", [2.0 ** -112, 2.0 ** -120, 2.0 ** -127])
def test_the_planes_hold_values_down_to_the_last_bit_of_fp32(small, scale):
    """Down to subnormal values, the other operands large enough for results in the normal range."""
    _, _, table = make_table(1, 8, 14, 14, 0.5, 3, 6)
    x, w, b, gy = make_conv_inputs(table.shape[0], 64, 64, 3, torch.float32, 6)
    t = {"x": x, "w": w, "gy": gy}
    t = {name: v * (scale if name == small else 2.0 ** 36) for name, v in t.items()}
    got, truth = _run(table, t["x"], t["w"], b, t["gy"]), _truth(table, t["x"], t["w"], b, t["gy"])
    _close(got[:3], truth[:3])


@pytest.mark.parametrize("where", ["x", "w", "gy"])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.4e38])
@pytest.mark.parametrize("n", [700, 200])
def test_values_beyond_the_planes(where, value, n):
    """Infinities, NaN and values that round up beyond bf16's range: the same infinities and NaN as in the sums over the pairs
    themselves, and nothing in the rows, columns and taps that they have no part in."""
    table = _chain(n, 9, 0.3, 9)
    x, w, b, gy = make_conv_inputs(n, 64, 96, 3, torch.float32, 9, bias="random")
    t = {"x": x, "w": w, "gy": gy}[where]
    t.view(-1)[t.numel() // 2 + 5] = value
    if where == "w":
        t.view(-1)[7] = 0.25 * value
    got = _run(table, x, w, b, gy)
    want = []
    for e in _truth(table, x, w, b, gy):
        want.append(e.float())
    for name, a, e in zip(("y", "gx", "gw", "gb"), got, want):
        assert torch.equal(a.isnan(), e.isnan()), name
        assert torch.equal(a.isinf(), e.isinf()) and torch.equal(a[a.isinf()], e[e.isinf()]), name
        ok = e.isfinite()
        # finite sums: as above, but for the size of the largest product of their own that a fp32 sum is rounded at
        err = (a[ok].double() - e[ok].double()).abs() / e[ok].double().abs().clamp_min(1.0)
        assert err.max() < 1e-4, (name, err.max())


def test_sums_beyond_the_scaled_range_are_those_of_the_fp32_values():
    """2^16 times each value: sums above 2^96 leave fp32's range before they are brought back, and are made again."""
    n = 9000                                # several lists per range of tokens
    table = _chain(n, 9, 0.3, 2)
    x, w, b, gy = make_conv_inputs(n, 8, 12, 3, torch.float32, 2)
    x, w, gy = x * 2.0 ** 62, w * 2.0 ** 45, gy * 2.0 ** 50
    x[n // 2] *= 2.0 ** -62                 # rows of one tile on both sides of the line
    got, truth = _run(table, x, w, b, gy), _truth(table, x, w, b, gy)
    _close(got[:3], truth[:3])


def test_infinities_cost_a_small_multiple_of_an_ordinary_call():
    """One value, a row, all of them: 5 to 7 times an ordinary call's time were measured, 20 to 450 with a thread per element."""
    ops = _ops()
    n, c = 4720, 192
    table = _chain(n, 9, 0.2, 1).cuda()
    plain = [t.cuda() for t in make_conv_inputs(n, c, c, 3, torch.float32, 1)]

    def times(x, w, gy):
        out = []
        for f in (lambda: ops.conv_fwd(x, table, w), lambda: ops.conv_dgrad(gy, table, w, assume_symmetric=True),
                  lambda: ops.conv_wgrad(gy, x, table, 9)):
            best = 1e9
            for _ in range(5):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                for _ in range(8):
                    f()
                b.record()
                b.synchronize()
                best = min(best, a.elapsed_time(b))
            out.append(best)
        return out

    ordinary = times(plain[0], plain[1], plain[3])
    for where in ("one", "row", "all"):
        x, w, gy = plain[0].clone(), plain[1].clone(), plain[3].clone()
        for t in (x, gy):
            t.view(-1)[{"one": slice(5000, 5001), "row": slice(5 * c, 6 * c), "all": slice(None)}[where]] = float("inf")
        if where == "one":
            w.view(-1)[5000] = float("inf")
        for ours, usual in zip(times(x, w, gy), ordinary):
            assert ours < 14 * usual, (where, ours, usual)


@pytest.mark.parametrize("what,n,cin,cout,kk,density", [("fwd", 8, 512, 512, 49, 0.0), ("dgrad", 32, 512, 512, 49, 0.0),
                                                        ("wgrad", 800, 64, 1024, 49, 0.05), ("wgrad", 1100, 64, 64, 9, 1.0)])
def test_the_tensor_cores_do_not_take_what_the_cuda_cores_do_faster(what, n, cin, cout, kk, density, monkeypatch):
    """Few rows without neighbors (2.3 to 2.9 times the time with every tap worked through), weight gradients of many CTAs with
    few pairs each (1.5 times) or of little work on a full table (1.3 times)."""
    ops = _ops()
    table = _chain(n, kk, density, n).cuda()
    x, w, _, gy = (t.cuda() for t in make_conv_inputs(n, cin, cout, int(kk ** 0.5), torch.float32, n))
    f = {"fwd": lambda: ops.conv_fwd(x, table, w), "dgrad": lambda: ops.conv_dgrad(gy, table, w, assume_symmetric=True),
         "wgrad": lambda: ops.conv_wgrad(gy, x, table, kk)}[what]

    def time(path):
        monkeypatch.setenv("SVTAD_FORCE_PATH", path)
        f()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(20):
                f()
        best = 1e9
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    assert time("") < 1.2 * time("simt")
