"""What the planner folds into a neighbour is what the folded op would have taken by itself: graphs that its own checks refuse stay
refused, and a state tensor is written where its op stands, not earlier."""
import numpy as np
import pytest

from torq_b200.oplist import Graph
from torq_b200.quant import quantize_multipliers
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


@pytest.mark.parametrize("producer", ["conv", "pool"])
def test_table_into_a_state_is_written_in_its_place(device, producer):
    """The state is read between the producer and the table that writes it: the reader sees the step before."""
    rng = np.random.default_rng(3)
    C, ident = 16, np.arange(-128, 128).astype(np.int8)
    x = rng.integers(-128, 128, (1, 4, 4, C), dtype=np.int8)
    g = Graph()
    xi = g.input(x.shape)
    if producer == "conv":
        m, s = quantize_multipliers(np.full(C, 0.01))
        h = g.conv2d(xi, rng.integers(-127, 128, (C, 1, 1, C), dtype=np.int8), np.zeros(C, np.int32), m, s)
    else:
        h = g.maxpool2d(xi, (2, 2), (2, 2))
    state = g.state(h.shape, "i8")
    g.output(g.table(state, ident))
    t = g.table(h, ident[::-1].copy())
    g.ops[-1].outputs = [state]
    g.tensors.remove(t)  # the last tensor made: ids stay dense
    for k, tt in enumerate(g.tensors):
        tt.id = k
    ex = Executable(device, g.serialize())
    d_in, d_out = device.alloc(x.nbytes), device.alloc(int(np.prod(h.shape)))
    got = []
    for step in range(2):
        d_in.upload(x)
        ex.dispatch([d_in], [d_out])
        got.append(d_out.download(h.shape, np.int8))
    d_in.free(), d_out.free(), ex.destroy()
    assert (got[0] == 0).all() and len(np.unique(got[1])) > 2
