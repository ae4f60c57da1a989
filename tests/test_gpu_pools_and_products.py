"""The strip pooling kernels, the one-step rescaled add and the tiled products at the sizes where they can go wrong: odd
frames and channel counts, windows that hang over every edge, tile remainders, folded transposes, scalars and casts."""
import numpy as np
import pytest
from gpu_exec import run_graph_gpu
from oracle_exec import run_graph
from torq_b200.bf16 import from_bf16, to_bf16
from torq_b200.oplist import Graph
from torq_b200.quant import add_rescale_params
from torq_b200.runtime import Executable

pytestmark = pytest.mark.gpu


def _check(device, g, inputs):
    for want, got in zip(run_graph(g, inputs), run_graph_gpu(device, g, inputs)):
        assert want.shape == got.shape and (want == got).all(), int((want != got).sum())


@pytest.mark.parametrize("k,s", [(2, 2), (3, 1), (3, 2), (5, 1)])
@pytest.mark.parametrize("shape", [(1, 5, 7, 3), (2, 9, 6, 20), (1, 13, 11, 32), (3, 40, 33, 64)])
@pytest.mark.parametrize("table", [False, True])
def test_strip_pools(device, k, s, shape, table):
    rng = np.random.default_rng(k * 100 + s)
    x = rng.integers(-128, 128, shape, dtype=np.int8)
    t = rng.integers(-128, 128, 256).astype(np.int8)
    pad = ((k - 1) // 2, k // 2) * 2
    for kind in ("max", "avg"):
        g = Graph()
        xi = g.input(shape)
        y = g.maxpool2d(xi, (k, k), (s, s), pad, pad_value=-77) if kind == "max" else \
            g.avg_pool2d(xi, (k, k), (s, s), pad, input_zp=-9, output_zp=5)
        g.output(g.table(y, t) if table else y)
        if table:
            ex = Executable(device, g.serialize())
            assert ex.launch_count == 1, ex.op_kernels()
            ex.destroy()
        _check(device, g, [x])


@pytest.mark.parametrize("kind", ["max", "avg"])
@pytest.mark.parametrize("shape", [(65535, 2, 2, 4), (65536, 2, 2, 4), (1, 131070, 2, 3), (1, 131074, 2, 3)])
def test_table_behind_a_pool_at_the_strips_grid_limits(device, kind, shape):
    """More images or rows than a strip's grid takes: the pool and its table run as two launches."""
    rng = np.random.default_rng(shape[1])
    x = rng.integers(-128, 128, shape, dtype=np.int8)
    g = Graph()
    xi = g.input(shape)
    y = g.maxpool2d(xi, (2, 2), (2, 2)) if kind == "max" else g.avg_pool2d(xi, (2, 2), (2, 2), input_zp=-9, output_zp=5)
    g.output(g.table(y, rng.integers(-128, 128, 256).astype(np.int8)))
    ex = Executable(device, g.serialize())
    assert ex.launch_count == (1 if max(shape[0], shape[1] // 2) <= 65535 else 2), ex.op_kernels()
    ex.destroy()
    _check(device, g, [x])


@pytest.mark.parametrize("n", [1, 15, 16, 4099])
@pytest.mark.parametrize("scales", [(0.02, 0.1, 0.05), (0.07, 0.03, 0.09), (0.05, 0.05, 0.02), (0.05, 0.05, 0.0008)])  # the last too steep for the linear form
def test_rescaled_add_covers_every_operand_pair(device, n, scales):
    rng = np.random.default_rng(n)
    m0, m1, mo = add_rescale_params(*scales)
    a, b = (rng.integers(-128, 128, (1, n), dtype=np.int8) for _ in range(2))
    if n == 4099:  # all 65536 pairs
        p = np.arange(65536)
        a, b = (p >> 8).astype(np.uint8).view(np.int8).reshape(1, -1), (p & 255).astype(np.uint8).view(np.int8).reshape(1, -1)
    for fn, clamp in (("add", (-128, 127)), ("sub", (-100, 90))):
        g = Graph()
        g.output(getattr(g, fn)(g.input(a.shape), g.input(b.shape), a_zp=7, a_ms=m0, b_zp=-10, b_ms=m1, out_ms=mo, out_zp=3, clamp=clamp))
        _check(device, g, [a, b])


# the second row: stages' edges of the 16 x 16, 32 x 32 and 64 x 32 tiles, aligned rows and odd ones (which take 64 x 64 where there are
# enough); the third: 64 x 64 tiles of aligned rows, over the edges of tiles and stages
@pytest.mark.parametrize("M,K,N", [(1, 1, 1), (16, 128, 17), (33, 130, 31), (160, 65, 190), (300, 36, 900), (520, 129, 512),
                                   (40, 256, 16), (17, 515, 24), (31, 769, 33), (300, 64, 304), (310, 191, 297), (1300, 63, 520), (1291, 128, 512),
                                   (2500, 64, 1008), (2441, 80, 1008)])
@pytest.mark.parametrize("dtype", ["bf16", "f32", "i16", "i8"])
@pytest.mark.parametrize("transposed", [False, True])
def test_tiled_products(device, M, K, N, dtype, transposed):
    rng = np.random.default_rng(M + K + N)
    shape_b = (N, K) if transposed else (K, N)
    if dtype[0] == "i":
        lim = 128 if dtype == "i8" else 32768
        a, b = (rng.integers(-lim, lim, s).astype(np.int8 if dtype == "i8" else np.int16) for s in ((M, K), shape_b))
    else:
        a, b = (rng.normal(0, 1, s).astype(np.float32) for s in ((M, K), shape_b))
        if dtype == "bf16":
            a, b = to_bf16(a), to_bf16(b)
    g = Graph()
    ai, bi = g.input((M, K), dtype), g.input(shape_b, dtype)
    bt = g.transpose(bi, (1, 0)) if transposed else bi
    g.output(g.matmul_i32(ai, bt, a_zp=3, b_zp=-2) if dtype[0] == "i" else g.matmul_f(ai, bt, "f32"))
    ex = Executable(device, g.serialize())
    assert ex.launch_count == 1, ex.op_kernels()
    ex.destroy()
    _check(device, g, [a, b])


@pytest.mark.parametrize("M,K,N", [(65536 * 64 + 5, 3, 2), (2, 3, 65536 * 64 + 5)])
@pytest.mark.parametrize("dtype", ["bf16", "i8"])
def test_products_of_more_tiles_than_a_second_grid_dimension_takes(device, M, K, N, dtype):
    rng = np.random.default_rng(K)
    a, b = (rng.integers(-128, 128, s, dtype=np.int8) for s in ((M, K), (K, N)))
    if dtype == "bf16":
        a, b = to_bf16(a.astype(np.float32)), to_bf16(b.astype(np.float32))
    g = Graph()
    ai, bi = g.input((M, K), dtype), g.input((K, N), dtype)
    g.output(g.matmul_i32(ai, bi, a_zp=3, b_zp=-2) if dtype == "i8" else g.matmul_f(ai, bi, "f32"))
    _check(device, g, [a, b])


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 255), (5, 256), (7, 500), (2, 1024), (4, 1100)])
def test_softmax_with_its_scalar_and_cast(device, rows, cols):
    x = np.random.default_rng(cols).normal(0, 3, (rows, cols)).astype(np.float32)
    g = Graph()
    p = g.softmax(g.ew("mul", g.input(x.shape, "f32"), g.const(np.full((1, 1), 0.37, np.float32))))
    g.output(g.ew("cast", p, out_dtype="bf16"))
    if x.size > 1:
        ex = Executable(device, g.serialize())
        assert ex.launch_count == 1, ex.op_kernels()
        ex.destroy()
    got = from_bf16(run_graph_gpu(device, g, [x])[0])
    e = np.exp((x * np.float32(0.37)).astype(np.float64) - (x * np.float32(0.37)).max(-1, keepdims=True))
    assert np.allclose(got, e / e.sum(-1, keepdims=True), rtol=2 ** -7, atol=1e-30)


@pytest.mark.parametrize("cols", [200, 500, 1000, 1025, 3000])
def test_folded_scalar_rounds_as_the_multiplication_does(device, cols):
    """softmax(x * s) in one launch against the same two ops apart (the product is an output too): the same bits."""
    x = np.random.default_rng(cols).normal(0, 20, (64, cols)).astype(np.float32)
    got = []
    for apart in (False, True):
        g = Graph()
        y = g.ew("mul", g.input(x.shape, "f32"), g.const(np.full((1, 1), 0.37, np.float32)))
        g.output(g.softmax(y))
        if apart:
            g.output(y)
        ex = Executable(device, g.serialize())
        assert ex.launch_count == 1 + apart, ex.op_kernels()
        ex.destroy()
        got.append(run_graph_gpu(device, g, [x])[0])
    assert (got[0].view(np.uint32) == got[1].view(np.uint32)).all(), int((got[0] != got[1]).sum())


def _pools_and_add(shape, k, s, table, max_first, fn="add", pad_value=-128):
    """fn of the max pool (a table behind it) and the average pool of one tensor."""
    rng = np.random.default_rng(shape[1])
    m0, m1, mo = add_rescale_params(0.02, 0.03, 0.04)
    pad = ((k - 1) // 2, k // 2) * 2
    g = Graph()
    x = g.input(shape)
    mx = g.maxpool2d(x, (k, k), (s, s), pad, pad_value=pad_value)
    if table:
        mx = g.table(mx, rng.integers(-128, 128, 256).astype(np.int8))
    av = g.avg_pool2d(x, (k, k), (s, s), pad, input_zp=-9, output_zp=100)  # saturates
    a, b = (mx, av) if max_first else (av, mx)
    g.output(getattr(g, fn)(a, b, a_zp=-7, a_ms=m0, b_zp=10, b_ms=m1, out_ms=mo, out_zp=2, clamp=(-120, 127) if table else (-128, 127)))
    return g


@pytest.mark.parametrize("k,s", [(2, 2), (3, 1), (3, 2), (5, 1)])
@pytest.mark.parametrize("shape", [(1, 5, 7, 3), (2, 9, 6, 20), (1, 13, 11, 32), (3, 40, 33, 64), (9, 112, 107, 32), (20, 61, 64, 64), (5, 90, 91, 100)])
@pytest.mark.parametrize("table,max_first,fn", [(True, True, "add"), (False, False, "add"), (True, False, "sub")])
def test_two_pools_and_their_sum_in_one_launch(device, k, s, shape, table, max_first, fn):
    g = _pools_and_add(shape, k, s, table, max_first, fn)
    ex = Executable(device, g.serialize())
    assert ex.launch_count == 1 and ex.op_kernels()[-1] == "pool_add", ex.op_kernels()
    ex.destroy()
    _check(device, g, [np.random.default_rng(k).integers(-128, 128, shape, dtype=np.int8)])


def test_two_pools_and_their_sum_one_by_one(device):
    """Another pad value, or a result that lies over the pooled tensor: the three ops as they are."""
    shape = (2, 24, 24, 16)
    x = np.random.default_rng(0).integers(-128, 128, shape, dtype=np.int8)
    g = _pools_and_add(shape, 3, 2, True, True, pad_value=-77)
    ex = Executable(device, g.serialize())
    assert ex.launch_count == 3, ex.op_kernels()
    ex.destroy()
    _check(device, g, [x])
    g = _pools_and_add(shape, 3, 1, True, True)
    ex = Executable(device, g.serialize())
    buf = device.alloc(x.nbytes)
    buf.upload(x)
    ex.dispatch([buf], [buf])
    got = buf.download(shape, np.int8)
    buf.free(), ex.destroy()
    assert (got == run_graph(g, [x])[0]).all()
