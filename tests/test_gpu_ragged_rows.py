"""Layers whose rows are no multiple of 16 bytes: read by the small-problem kernel as they are, or padded and trimmed around the
tensor-core kernels - odd channels in and out, last words of a tensor, few rows, strides, tables. Bit-exact against the oracle."""
import numpy as np
import pytest

from gpu_exec import run_graph_gpu
from oracle_exec import run_graph
from torq_b200.oplist import Graph
from torq_b200.quant import quantize_multipliers

pytestmark = pytest.mark.gpu


def _check(device, g, xs, monkeypatch):
    want = run_graph(g, xs)
    for off in ("0", "1"):  # the small-problem kernel where it applies, then the padded copies
        monkeypatch.setenv("TB200_NO_SMALL", off)
        for a, b in zip(run_graph_gpu(device, g, xs), want):
            assert (a == b).all(), (off, int((a != b).sum()))


@pytest.mark.parametrize("M,K,N", [(1, 515, 33), (3, 1001, 517), (5, 37, 9), (129, 63, 65), (300, 1023, 1001), (1100, 100, 251), (513, 513, 513)])
@pytest.mark.parametrize("table", [False, True])
def test_fully_connected(device, M, K, N, table, monkeypatch):
    rng = np.random.default_rng(M + K + N)
    m, s = quantize_multipliers(rng.uniform(0.5, 1.5, N) * 40.0 / (np.sqrt(K) * 74 * 74))
    g = Graph()
    y = g.fully_connected(g.input((M, K)), rng.integers(-127, 128, (N, K), dtype=np.int8), np.round(rng.normal(0, 900, N)).astype(np.int32), m, s,
                          input_zp=-7, out_zp=3)
    g.output(g.table(y, rng.permutation(np.arange(-128, 128)).astype(np.int8)) if table else y)
    _check(device, g, [rng.integers(-128, 128, (M, K), dtype=np.int8)], monkeypatch)


@pytest.mark.parametrize("N,H,W,IC,OC,k,st", [(1, 7, 5, 5, 7, 3, 1), (1, 12, 9, 24, 30, 3, 1), (2, 28, 28, 100, 77, 3, 1), (3, 30, 29, 9, 33, 3, 2),
                                              (2, 16, 16, 40, 17, 5, 1), (4, 33, 31, 33, 65, 1, 1), (1, 64, 64, 17, 16, 3, 2), (2, 40, 40, 16, 50, 3, 1)])
def test_convolution(device, N, H, W, IC, OC, k, st, monkeypatch):
    rng = np.random.default_rng(H + IC + OC)
    m, s = quantize_multipliers(rng.uniform(0.5, 1.5, OC) * 40.0 / (np.sqrt(k * k * IC) * 74 * 74))
    p = k // 2
    g = Graph()
    g.output(g.conv2d(g.input((N, H, W, IC)), rng.integers(-127, 128, (OC, k, k, IC), dtype=np.int8),
                      np.round(rng.normal(0, 900, OC)).astype(np.int32), m, s, stride=(st, st), pad=(p,) * 4, input_zp=-9, out_zp=4))
    _check(device, g, [rng.integers(-128, 128, (N, H, W, IC), dtype=np.int8)], monkeypatch)
