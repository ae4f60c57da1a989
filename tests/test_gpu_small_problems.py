"""The kernels that small problems take (conv_small.cu, dw3x3_few_kernel) at the sizes where they can go wrong - remainders of
the 16 x 32 tiles, K of less than a step and not a multiple of one, splits of K over 1 .. 8 warps, windows that leave the frame -
and the kernels of the large ones at the same sizes (TB200_NO_SMALL=1). All bit-exact against the oracle."""
import numpy as np
import pytest

from torq_b200.oplist import Graph
from torq_b200.quant import quantize_multipliers
from torq_b200.runtime import Executable
from oracle_exec import run_graph
from gpu_exec import run_graph_gpu

pytestmark = pytest.mark.gpu


def _ms(rng, n, k):
    return quantize_multipliers(rng.uniform(0.5, 1.5, n) * 40.0 / (np.sqrt(k) * 74 * 74))


def _both(device, g, xs, monkeypatch):
    want = run_graph(g, xs)
    for off in ("0", "1"):
        monkeypatch.setenv("TB200_NO_SMALL", off)
        got = run_graph_gpu(device, g, xs)
        assert all((a == b).all() for a, b in zip(got, want)), off


# N, H, W, IC, OC, k, stride, pad: K of 16 .. 2304 bytes, splits of every size, odd frames, OC around the 32-column tile
CONVS = [
    (1, 5, 7, 16, 33, 1, 1, 0), (1, 16, 1, 16, 32, 1, 1, 0), (3, 7, 7, 160, 24, 1, 1, 0), (1, 4, 4, 24, 10, 1, 1, 0), (1, 3, 5, 960, 31, 1, 1, 0),
    (1, 9, 11, 32, 16, 3, 1, 1), (2, 8, 8, 48, 40, 3, 2, 1), (1, 6, 6, 256, 64, 3, 1, 1), (1, 13, 10, 64, 72, 5, 1, 2), (1, 56, 56, 64, 64, 3, 1, 1),
    (1, 15, 17, 3, 16, 3, 2, 1), (2, 9, 6, 3, 40, 3, 1, 1), (1, 3, 3, 3, 8, 3, 1, 0),
]


@pytest.mark.parametrize("case", CONVS)
@pytest.mark.parametrize("clamp,table", [((-128, 127), False), ((4, 120), True)])
def test_small_convolution(device, case, clamp, table, monkeypatch):
    N, H, W, IC, OC, k, st, pad = case
    rng = np.random.default_rng(1234 + H + IC + OC)
    g = Graph()
    m, s = _ms(rng, OC, k * k * IC)
    y = g.conv2d(g.input((N, H, W, IC)), rng.integers(-127, 128, (OC, k, k, IC), dtype=np.int8),
                 np.round(rng.normal(0, 900, OC)).astype(np.int32), m, s, stride=(st, st), pad=(pad,) * 4, input_zp=-9, out_zp=4, clamp=clamp)
    g.output(g.table(y, rng.permutation(np.arange(-128, 128)).astype(np.int8)) if table else y)
    _both(device, g, [rng.integers(-128, 128, (N, H, W, IC), dtype=np.int8)], monkeypatch)


@pytest.mark.parametrize("IC,kh,kw", [(6048, 3, 3), (7216, 3, 3), (8512, 2, 2), (7008, 2, 3)])
def test_channels_beyond_a_short_reciprocal(device, IC, kh, kw, monkeypatch):
    """Chunks of the K axis whose tap a 20-bit reciprocal got wrong, with every tap at a border of the frame somewhere."""
    rng = np.random.default_rng(IC)
    g = Graph()
    m, s = _ms(rng, 32, kh * kw * IC)
    g.output(g.conv2d(g.input((1, 4, 4, IC)), rng.integers(-127, 128, (32, kh, kw, IC), dtype=np.int8), np.full(32, 50, np.int32), m, s,
                      pad=(kh // 2, kh // 2, kw // 2, kw // 2), input_zp=-9, out_zp=4))
    _both(device, g, [rng.integers(-128, 128, (1, 4, 4, IC), dtype=np.int8)], monkeypatch)


def test_stem_of_few_pixels_on_a_frame_beyond_two_gigabytes(device):
    """A wide stride leaves few output pixels, but the offsets into the frame need 64 bits."""
    from oracle import oracle_np as onp
    rng = np.random.default_rng(5)
    S, st, OC = 26760, 110, 16
    x = np.frombuffer(rng.bytes(S * S * 3), np.int8).reshape(1, S, S, 3)
    w = rng.integers(-127, 128, (OC, 3, 3, 3), dtype=np.int8)
    m, s = _ms(rng, OC, 27)
    g = Graph()
    g.output(g.conv2d(g.input(x.shape), w, np.full(OC, 50, np.int32), m, s, stride=(st, st), input_zp=-9, out_zp=4))
    got = run_graph_gpu(device, g, [x])[0][0]
    n = (S - 3) // st + 1
    taps = [x[0, kh:kh + st * n:st, kw:kw + st * n:st][:n, :n].astype(np.int64) + 9 for kh in range(3) for kw in range(3)]
    acc = sum(np.einsum("hwi,oi->hwo", t, w.reshape(OC, 9, 3)[:, k].astype(np.int64)) for k, t in enumerate(taps)) + 50
    want = onp.requant(onp.wrap32(acc.reshape(-1, OC)), m, s, 4, -128, 127)
    assert (got.reshape(-1, OC) == want).all()


@pytest.mark.parametrize("C,H,W,st,clamp", [(4, 1, 1, 1, (-128, 127)), (20, 5, 7, 1, (-128, 127)), (36, 9, 8, 2, (4, 127)), (128, 6, 33, 1, (-20, 90)),
                                            (16, 12, 3, 2, (-128, 127))])
def test_few_depthwise_outputs(device, C, H, W, st, clamp, monkeypatch):
    rng = np.random.default_rng(C + W)
    g = Graph()
    m, s = _ms(rng, C, 9)
    g.output(g.depthwise_conv2d(g.input((2, H, W, C)), rng.integers(-127, 128, (3, 3, C, 1), dtype=np.int8),
                                np.round(rng.normal(0, 500, C)).astype(np.int32), m, s, stride=(st, st), pad=(1, 1, 1, 1), input_zp=5, out_zp=4,
                                clamp=clamp))
    _both(device, g, [rng.integers(-128, 128, (2, H, W, C), dtype=np.int8)], monkeypatch)


@pytest.mark.parametrize("S,K,OC,conv_first", [(7, 32, 40, True), (5, 96, 24, False), (4, 576, 33, True)])
def test_add_between_intermediates_rides_in_the_convolution(device, S, K, OC, conv_first, monkeypatch):
    from torq_b200.runtime import Executable
    rng = np.random.default_rng(S + K)
    g = Graph()
    x = g.input((1, S, S, K))
    m, s = _ms(rng, OC, K)
    conv = lambda: g.conv2d(x, rng.integers(-127, 128, (OC, 1, 1, K), dtype=np.int8), np.full(OC, 77, np.int32), m, s, input_zp=-5, out_zp=4)
    r, h = conv(), conv()
    g.output(g.add(*((h, r) if conv_first else (r, h)), a_zp=4, a_ms=(1 << 30, 11), b_zp=4, b_ms=(1395864371, 12), out_ms=(1093202297, 49),
                   out_zp=-3, clamp=(-110, 120)))
    monkeypatch.setenv("TB200_NO_SMALL", "0")
    ex = Executable(device, g.serialize())
    assert ex.launch_count == 2, ex.op_kernels()
    ex.destroy()
    _both(device, g, [rng.integers(-128, 128, (1, S, S, K), dtype=np.int8)], monkeypatch)


@pytest.mark.parametrize("M,K,N", [(5, 4096, 256), (64, 4096, 4096), (65, 2064, 1024), (128, 1040, 2500), (100, 1001, 2077), (17, 8192, 8192), (321, 2048, 2600)])
@pytest.mark.parametrize("table", [False, True])
def test_few_dozen_rows(device, M, K, N, table, monkeypatch):
    rng = np.random.default_rng(M + K + N)
    g = Graph()
    m, s = _ms(rng, N, K)
    y = g.fully_connected(g.input((M, K)), rng.integers(-127, 128, (N, K), dtype=np.int8), np.round(rng.normal(0, 900, N)).astype(np.int32), m, s,
                          input_zp=-7, out_zp=3)
    g.output(g.table(y, rng.permutation(np.arange(-128, 128)).astype(np.int8)) if table else y)
    _both(device, g, [rng.integers(-128, 128, (M, K), dtype=np.int8)], monkeypatch)


@pytest.mark.parametrize("shape,OC,stride,pad", [((1, 211, 90, 3), 16, 2, (0, 1, 0, 1)), ((3, 70, 75, 3), 32, 1, (1, 1, 1, 1)), ((2, 65, 43, 3), 48, 2, (1, 1, 1, 1)),
                                                 ((37, 5, 7, 3), 64, 1, (2, 0, 2, 0)), ((40, 31, 17, 3), 16, 1, (1, 1, 1, 1)),
                                                 ((3, 67, 132, 3), 16, 2, (0, 1, 0, 1)), ((2, 30, 140, 3), 32, 2, (1, 1, 1, 1)), ((5, 9, 64, 3), 96, 2, (1, 0, 2, 3)),
                                                 ((2, 90, 4, 3), 16, 2, (1, 1, 1, 1)), ((37, 101, 77, 3), 16, 1, (1, 1, 1, 1)), ((5, 230, 299, 3), 48, 1, (0, 1, 1, 0))])
@pytest.mark.parametrize("table", [False, True])
@pytest.mark.parametrize("double_round,clamp", [(True, (-128, 127)), (False, (3, 100))])
def test_stem_of_large_frames(device, shape, OC, stride, pad, table, double_round, clamp, monkeypatch):
    """The stem kernel of the frames the small-problem kernels leave: pixel counts that end inside a warp, rows shorter than a warp, windows
    over every edge, one and several passes over the channels, one pixel a thread and (from 1536 an SM on) several."""
    monkeypatch.setenv("TB200_NO_SMALL", "1")
    rng = np.random.default_rng(OC + shape[1])
    g = Graph()
    m, s = quantize_multipliers(rng.uniform(0.002, 0.004, OC))
    y = g.conv2d(g.input(shape), rng.integers(-127, 128, (OC, 3, 3, 3), dtype=np.int8), rng.integers(-3000, 3000, OC).astype(np.int32), m, s,
                 stride=(stride, stride), pad=pad, input_zp=-7, out_zp=3, double_round=double_round, clamp=clamp)
    g.output(g.table(y, rng.integers(-128, 128, 256).astype(np.int8)) if table else y)
    ex = Executable(device, g.serialize())
    assert ex.op_kernels()[0] == "conv2d_stem333_mma", ex.op_kernels()
    ex.destroy()
    x = rng.integers(-128, 128, shape, dtype=np.int8)
    assert (run_graph_gpu(device, g, [x])[0] == run_graph(g, [x])[0]).all()
