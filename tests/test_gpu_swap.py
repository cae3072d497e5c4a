"""GPU: edges of the operand-swapped tensor-core kernel: row counts around its tile sizes, one scale group, column tiles
that are half empty, more tiles than SMs, groups of projections.

Bound per value: half an fp16 ulp of the result (2^-11 |y|), one more where the kernel and the oracle round to different
neighbours, and fp32 sums of exact products over k, k 2^-24 sum |x||w| each.  Up to 16 rows the kernel multiplies by the
unrounded (code - 8) * scale, the oracle by its fp16 rounding: 2^-11 sum |x||w| more."""
import numpy as np
import pytest
import torch

from helpers import make_acts, quantized_layer
from oracle import uniql_oracle as orc

pytestmark = pytest.mark.gpu


def _dev(layer):
    b = torch.from_numpy(layer["bias"]).cuda() if layer["bias"] is not None else None
    return torch.from_numpy(layer["packed"]).cuda(), torch.from_numpy(layer["scales"]).cuda(), b, layer["n"]


def _check(y, x, layer):
    ref = orc.linear_ref(x.numpy(), None, None, layer["bias"], layer["n"], w_deq=layer["w_deq"]).astype(np.float64)
    mass = np.abs(x.numpy().astype(np.float64)) @ np.abs(layer["w_deq"][:, :layer["n"]].astype(np.float64))
    bound = 2.0 ** -10 * np.abs(ref) + (2 * layer["k"] * 2.0 ** -24 + (2.0 ** -11 if x.shape[0] <= 16 else 0)) * mass + 1e-7
    assert (np.abs(y.cpu().numpy().astype(np.float64) - ref) <= bound).all()


@pytest.mark.parametrize("n,k", [(128, 128), (192, 640), (320, 256), (1024, 3968), (19200, 256)])
@pytest.mark.parametrize("m", [5, 16, 17, 32, 33, 65, 97, 113, 128])
def test_rows_and_widths(m, n, k):
    from uniql_b200 import ops
    layer = quantized_layer(n + k, n, k, bias=(n == 320))
    x = make_acts(m, m, k)
    w, s, b, _ = _dev(layer)
    for _ in range(3):          # the rings' timing differs between cold and cached weights
        _check(ops.w4a16_linear(x.cuda(), w, s, b, n), x, layer)


@pytest.mark.parametrize("n,k", [(128, 128), (192, 640), (4096, 1024), (9600, 256)])
@pytest.mark.parametrize("m", [129, 209, 225, 256, 257, 301, 600])
def test_more_than_128_rows(m, n, k):
    """Row tiles of 144 to 256 rows (four, three and two stages), several row tiles, split over k, and the 256 x 256 tiles
    of the prefill kernel where they are chosen."""
    from uniql_b200 import ops
    layer = quantized_layer(n + k, n, k, bias=(n == 192))
    x = make_acts(m, m, k)
    w, s, b, _ = _dev(layer)
    for _ in range(2):
        _check(ops.w4a16_linear(x.cuda(), w, s, b, n), x, layer)


@pytest.mark.parametrize("m", [7, 16, 18, 64, 128])
@pytest.mark.parametrize("widths,k", [((192, 128, 448), 384), ((9600, 9664), 256)])
def test_groups(m, widths, k):
    from uniql_b200 import ops
    layers = [quantized_layer(7 * i + n + k, n, k, bias=(i == 1)) for i, n in enumerate(widths)]
    x = make_acts(m, m, k)
    for y, layer in zip(ops.w4a16_linear_group(x.cuda(), [_dev(la) for la in layers]), layers):
        _check(y, x, layer)


@pytest.mark.parametrize("m", [5, 16])
@pytest.mark.parametrize("n,k", [(192, 128), (200, 640), (9600, 256)])
def test_swiglu_pair_and_residual(m, n, k):
    """Half-empty tiles, one scale group, more pair tiles than SMs; the epilogue against separate launches of the plain
    kernel (identical sums, so only the elementwise roundings are compared: they are the same)."""
    from uniql_b200 import ops
    g, u = (_dev(quantized_layer(i + n + k, n, k, bias=(n == 200))) for i in (1, 2))
    x = make_acts(m, m, k).cuda()
    res = make_acts(m + 1, m, n, outliers=False).cuda()
    a, b = ops.w4a16_linear_group(x, [g])[0], ops.w4a16_linear_group(x, [u])[0]
    want = torch.nn.functional.silu(a) * b
    (got,) = ops.w4a16_linear_group(x, [g, u], epilogue="swiglu")
    assert torch.equal(got, want)
    (got,) = ops.w4a16_linear_group(x, [g], residual=res)
    assert torch.equal(got, a + res)


@pytest.mark.parametrize("m", [5, 16, 17, 64, 256])
def test_packed_ring_refilled_many_times(m):
    """Every CTA streams more scale groups than the packed ring has slots (40 and 80 against at most 16), so each slot is
    handed back and refilled by TMA while other warps still read: a slot released before all lanes of a warp have read it
    gives wrong weights.  The sums are deterministic, so cold and cached weights must give the same bits."""
    from uniql_b200 import ops
    n, k = 148 * 128 + 64, 5120
    layer = quantized_layer(n + k, n, k)
    x = make_acts(m, m, k)
    w, s, b, _ = _dev(layer)
    first = ops.w4a16_linear(x.cuda(), w, s, b, n)
    _check(first, x, layer)
    for _ in range(20):
        assert torch.equal(ops.w4a16_linear(x.cuda(), w, s, b, n), first)


@pytest.mark.parametrize("m", [1, 5, 16, 17, 128])
def test_prefetch_hint(m):
    """The ranges are asked for by every grouped launch, whole 128-byte lines inside them only, and change no result.
    (Lines are dealt out over CTAs and lanes: no line, one, fewer than lanes, many.)"""
    from uniql_b200 import ops
    n, k = 1024, 1024
    layer = quantized_layer(n + k, n, k)
    x = make_acts(m, m, k).cuda()
    hints = [(torch.zeros(nb, dtype=torch.uint8, device="cuda"), nb) for nb in (100, 128, 3000, 1 << 22)]
    (want,) = ops.w4a16_linear_group(x, [_dev(layer)])
    (got,) = ops.w4a16_linear_group(x, [_dev(layer)], prefetch=hints)
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    _check(got, x.cpu(), layer)
    assert ops.read_and_clear_status("cuda") == 0


@pytest.mark.parametrize("m", [5, 8, 16])
@pytest.mark.parametrize("n,k", [(64, 1024), (200, 2304), (2048, 2048), (1024, 4096)])
def test_swiglu_pair_and_residual_shared_by_a_cluster(m, n, k):
    """1 to 32 pair tiles, so that a cluster shares each over k and the epilogue works on sums fetched from its CTAs' shared
    memory.  Bounds: gate and up as in _check (ends in fp16 roundings of their own: included); |silu'| < 1.1; then the fp16
    roundings of silu, product and sum, half an ulp = 2^-11 each, 2^-25 where the result is subnormal."""
    from uniql_b200 import ops
    gl, ul = (quantized_layer(i + n + k, n, k, bias=(n == 200)) for i in (1, 2))
    x = make_acts(m, m, k)
    res = make_acts(m + 1, m, n, outliers=False)

    def parts(layer):
        ref = orc.linear_ref(x.numpy(), None, None, layer["bias"], n, w_deq=layer["w_deq"]).astype(np.float64)
        mass = np.abs(x.numpy().astype(np.float64)) @ np.abs(layer["w_deq"][:, :n].astype(np.float64))
        return ref, 2.0 ** -10 * np.abs(ref) + (2 * layer["k"] * 2.0 ** -24 + 2.0 ** -11) * mass + 1e-7

    (g, eg), (u, eu) = parts(gl), parts(ul)
    act = g / (1.0 + np.exp(-g))
    want = act * u
    bound = 1.1 * eg * (np.abs(u) + eu) + np.abs(act) * eu
    bound = bound + 2.0 ** -11 * (np.abs(act) + 1.1 * eg) * (np.abs(u) + eu) + 2.0 ** -25 * (np.abs(u) + eu)
    bound = bound + 2.0 ** -11 * (np.abs(want) + bound) + 2.0 ** -24
    for _ in range(3):
        (got,) = ops.w4a16_linear_group(x.cuda(), [_dev(gl), _dev(ul)], epilogue="swiglu")
        assert (np.abs(got.cpu().numpy().astype(np.float64) - want) <= bound).all()
        (got,) = ops.w4a16_linear_group(x.cuda(), [_dev(gl)], residual=res.cuda())
        summed = g + res.numpy().astype(np.float64)
        assert (np.abs(got.cpu().numpy().astype(np.float64) - summed) <= eg + 2.0 ** -11 * (np.abs(summed) + eg) + 1e-7).all()
    assert ops.read_and_clear_status("cuda") == 0
