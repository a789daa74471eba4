"""GPU tier: the fp32 kernels on the CUDA cores (csrc/conv_f32.cu), which the tensor-core ones leave very wide layers, very few
rows and, under SVTAD_FORCE_PATH=simt, everything, against sums over the existing pairs in 64 bits."""
import pytest
import torch

from tests.helpers import make_conv_inputs
from tests.test_gpu_f32_tc import _chain, _ops, _run, _truth

pytestmark = pytest.mark.gpu

# Relative error (2-norm): a chain of m fp32 additions rounds half a unit (2^-24) of a partial sum each time, at random: sqrt(m) 2^-24;
# the longest here has 16 000 (4 100 channels, four taps).
BOUND = 128 * 2.0 ** -24


def _close(got, truth):
    for name, a, e in zip(("y", "gx", "gw", "gb"), got, truth):
        err = (a.double() - e).norm() / e.norm().clamp_min(1e-300)
        assert err < BOUND, f"{name}: {err:.2e}"


@pytest.mark.parametrize("n,cin,cout,kk", [
    (1, 4, 4, 1), (63, 64, 64, 9), (65, 60, 68, 9), (129, 192, 192, 9),      # tiles of 64 rows, steps shared by a cluster
    (200, 512, 64, 25), (700, 36, 32, 49),
    (4000, 32, 320, 9),          # tiles of 128 rows, shared
    (8000, 16, 320, 9),          # ... and not shared; several ranges of the weight gradient
])
def test_forced_to_the_cuda_cores(n, cin, cout, kk, monkeypatch):
    monkeypatch.setenv("SVTAD_FORCE_PATH", "simt")
    table = _chain(n, kk, 0.35, n)
    x, w, b, gy = make_conv_inputs(n, cin, cout, int(kk ** 0.5), torch.float32, n, bias="random")
    _close(_run(table, x, w, b, gy), _truth(table, x, w, b, gy))


def test_batch_local_indices_and_an_asymmetric_table(monkeypatch):
    monkeypatch.setenv("SVTAD_FORCE_PATH", "simt")
    n, tpb = 900, 300
    local = _chain(tpb, 9, 0.5, 3).repeat(3, 1)
    x, w, b, gy = make_conv_inputs(n, 64, 96, 3, torch.float32, 11, bias="random")
    _close(_run(local, x, w, b, gy, tpb), _truth(local, x, w, b, gy, tpb))
    table = _chain(n, 9, 0.5, 4)
    table[5, 0] = 700                       # a neighbor that does not have row 5 for its own
    t = [v.cuda() for v in (table, x, w, gy)]
    gx, gw, gb = _ops().conv_bwd(t[3], t[1], t[0], t[2])
    _close([gx.cpu(), gw.cpu(), gb.cpu()], _truth(table, x, w, b, gy)[1:])


@pytest.mark.parametrize("n,cin,cout", [(40, 4096, 8), (40, 4100, 8), (40, 8, 4100), (3, 64, 64), (4, 64, 64)])
def test_where_the_two_kinds_meet(n, cin, cout):
    table = _chain(n, 9, 0.35, n)
    x, w, b, gy = make_conv_inputs(n, cin, cout, 3, torch.float32, n, bias="random")
    _close(_run(table, x, w, b, gy), _truth(table, x, w, b, gy))
