"""What the planner folds into a neighbour is what the folded op would have taken by itself: graphs that its own checks refuse stay
refused."""
import numpy as np
import pytest

from torq_b200.oplist import Graph
from torq_b200.runtime import Executable, TorqB200Error

pytestmark = pytest.mark.gpu


def _softmax_graph(mul_from=(4, 8), cast_to=(4, 8)):
    g = Graph()
    y = g.ew("mul", g.input(mul_from, "f32"), g.const(np.full((1, 1), 0.5, np.float32)))
    y.shape = (4, 8)
    z = g.output(g.ew("cast", g.softmax(y), out_dtype="bf16"))
    z.shape = cast_to
    return g


def _concat_graph(inner_channels):
    g = Graph()
    parts = [g.table(g.input((1, 2, 2, 16)), np.arange(-128, 128).astype(np.int8)) for _ in range(3)]
    kw = dict(a_zp=0, a_ms=(1 << 30, 30), b_zp=0, b_ms=(1 << 30, 30), out_zp=0)
    inner = g.concat(parts[0], parts[1], **kw)
    inner.shape = (1, 2, 2, inner_channels)
    mid = g.concat(inner, parts[2], **kw)
    mid.shape = (1, 2, 2, 48)
    g.output(g.table(g.concat(mid, g.table(g.input((1, 2, 2, 16)), np.arange(-128, 128).astype(np.int8)), **kw), np.arange(-128, 128).astype(np.int8)))
    return g


@pytest.mark.parametrize("good,bad", [
    (_softmax_graph(), [_softmax_graph(mul_from=(8, 4)), _softmax_graph(cast_to=(8, 4))]),
    (_concat_graph(32), [_concat_graph(16), _concat_graph(48)]),
])
def test_refused_shapes_stay_refused(device, good, bad):
    Executable(device, good.serialize()).destroy()
    for g in bad:
        with pytest.raises(TorqB200Error):
            Executable(device, g.serialize())
