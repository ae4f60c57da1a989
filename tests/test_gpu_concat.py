"""Concatenations of intermediates in one launch: two to eight operands, copied and rescaled, results of odd widths, operands that
other ops read too, rows that do not fill a block. Bit-exact against the oracle."""
import numpy as np
import pytest

from gpu_exec import run_graph_gpu
from oracle_exec import run_graph
from torq_b200.oplist import Graph
from torq_b200.quant import quantize_multiplier
from torq_b200.runtime import Executable

pytestmark = pytest.mark.gpu
IDENT = ((1 << 30), 30)


@pytest.mark.parametrize("shape,channels,rescaled", [((1, 1, 1), (16, 16), ()), ((2, 9, 7), (16, 48, 32), (1,)), ((1, 20, 21), (128, 16, 16, 64), (0, 3)),
                                                     ((3, 64, 64), (32, 32), (0, 1)), ((1, 5, 3), (16,) * 8, (2, 7)), ((1, 6, 5), (16, 24), (1,)),
                                                     ((40, 64, 64), (16, 48, 16), (1, 2)), ((37, 65, 67), (32, 64), ()), ((41, 64, 64), (96, 32, 32), (0, 2))])
@pytest.mark.parametrize("factor", [lambda k: 0.6 + 0.2 * k, lambda k: 0.31 + 0.02 * k], ids=["one multiply-add", "tables"])
def test_concat_of_intermediates(device, shape, channels, rescaled, factor):
    """Rescales that one multiply-add gives for every byte, and ones below a half, whose double rounding none does."""
    rng = np.random.default_rng(sum(channels))
    g = Graph()
    xs = [rng.integers(-128, 128, shape + (c,), dtype=np.int8) for c in channels]
    parts = [g.table(g.input(x.shape), rng.permutation(np.arange(-128, 128)).astype(np.int8)) for x in xs]
    ms = [quantize_multiplier(factor(k)) if k in rescaled else IDENT for k in range(len(parts))]
    zp = [4 if k not in rescaled else k - 3 for k in range(len(parts))]
    acc = g.concat(parts[0], parts[1], a_zp=zp[0], a_ms=ms[0], b_zp=zp[1], b_ms=ms[1], out_zp=4)
    for k in range(2, len(parts)):
        acc = g.concat(acc, parts[k], a_zp=4, a_ms=IDENT, b_zp=zp[k], b_ms=ms[k], out_zp=4)
    g.output(g.table(acc, np.arange(-128, 128, dtype=np.int8)[::-1].copy()))
    g.output(g.table(parts[1], np.arange(-128, 128, dtype=np.int8)))  # another reader of an operand
    if all(c % 16 == 0 for c in channels):
        ex = Executable(device, g.serialize())
        assert ex.launch_count == len(parts) + 1 + 2, ex.op_kernels()
        ex.destroy()
    for a, b in zip(run_graph_gpu(device, g, xs), run_graph(g, xs)):
        assert (a == b).all()
