"""The op-by-op decode kernels (decode_linear.cu) where they can go wrong: tile and token remainders, one and many K groups, K slices
that meet in a cluster, products that walk their tiles with the arg max riding along, caches shorter and longer than a round of
keys, one to four query heads. Against fp32 torch."""
import numpy as np
import pytest
import torch

from gpu_exec import run_graph_gpu
from torq_b200.bf16 import from_bf16, to_bf16
from torq_b200.oplist import Graph
from torq_b200.runtime import Executable

pytestmark = pytest.mark.gpu


def _bf(t):
    return t.to(torch.bfloat16).to(torch.float32)


def _product(rng, B, K, N):
    x = to_bf16(rng.normal(0, 1, (B, K)).astype(np.float32))
    w = rng.integers(-128, 128, (N, K), dtype=np.int8)
    s = to_bf16(rng.uniform(0.5, 1.5, N).astype(np.float32) / (73.0 * np.sqrt(K)))
    want = (torch.from_numpy(from_bf16(x)) @ torch.from_numpy(w.astype(np.float32)).T) * torch.from_numpy(from_bf16(s))
    return x, w, s, want


@pytest.mark.parametrize("B,K,N", [(1, 64, 1), (3, 64, 33), (8, 192, 32), (9, 8192, 31), (16, 6912, 100), (32, 6912, 1152), (25, 4096, 70),
                                   (2, 128, 60001), (32, 1152, 30001), (8, 6912, 28500), (8, 3072, 38000), (7, 3072, 28500)])
def test_products(device, B, K, N):
    rng = np.random.default_rng(B + K + N)
    x, w, s, want = _product(rng, B, K, N)
    g = Graph()
    y = g.gemv_w8(g.input((B, K), "bf16"), w, s, out_dtype="f32")
    g.output(y), g.output(g.argmax(y))
    got, ids = run_graph_gpu(device, g, [x])
    assert np.abs(got - want.numpy()).max() <= 1e-5 * np.abs(want.numpy()).max()
    assert (ids == got.argmax(-1)).all()


@pytest.mark.parametrize("B,K,N", [(1, 1152, 40), (2, 6912, 33), (7, 64, 32), (8, 1152, 30001)])
@pytest.mark.parametrize("spread", [0, 8, 40, 120])
def test_products_of_few_tokens_over_magnitudes(device, B, K, N, spread):
    """The two sizes whose K no warps share take the activations as fixed-point numbers, the others as they are: magnitudes 2^-spread .. 1
    side by side, subnormals at the far end.
    Against 64 bits; the bound is that of an fp32 sum of K terms: K 2^-24 of the sum of magnitudes."""
    rng = np.random.default_rng(B + K + spread)
    x = to_bf16((rng.normal(0, 1, (B, K)) * np.exp2(rng.uniform(-spread, 0, (B, K)) - (100 if spread == 40 else 0))).astype(np.float32))
    x[0, : K // 2] = 0
    w = rng.integers(-128, 128, (N, K), dtype=np.int8)
    s = to_bf16(np.ones(N, np.float32))
    g = Graph()
    g.output(g.gemv_w8(g.input((B, K), "bf16"), w, s, out_dtype="f32"))
    got = run_graph_gpu(device, g, [x])[0].astype(np.float64)
    xd, wd = from_bf16(x).astype(np.float64), w.astype(np.float64)
    bound = K * 2.0 ** -24 * (np.abs(xd) @ np.abs(wd).T) + 1e-44
    assert (np.abs(got - xd @ wd.T) <= bound).all(), np.max(np.abs(got - xd @ wd.T) / bound)


@pytest.mark.parametrize("B,K,N", [(1, 1152, 30001), (2, 4096, 28500), (5, 1152, 28500), (8, 1600, 30001)])
@pytest.mark.parametrize("gap", [16, 22, 30])
def test_rows_with_an_outlier_keep_what_lies_below_it(device, B, K, N, gap):
    """One activation of a row 2^gap above the rest, meeting weights of zero: what is left is the sum of the others, to the bound of an fp32
    sum of K terms. Rows without an outlier beside it give the same bits as without such neighbours, and the arg max ranges over both."""
    rng = np.random.default_rng(B + K + gap)
    x = rng.normal(0, 1, (B, K)).astype(np.float32)
    x = np.where(np.abs(x) < 2.0 ** -9, 2.0 ** -9, x)
    plain = to_bf16(x)
    at = [b * K // B for b in range(B)]
    outliers = [b for b in range(B) if b % 2 == 0]
    for b in outliers:
        x[b, at[b]] = 2.0 ** gap
    w = rng.integers(-128, 128, (N, K), dtype=np.int8)
    w[:, at] = 0
    g = Graph()
    y = g.gemv_w8(g.input((B, K), "bf16"), w, to_bf16(np.ones(N, np.float32)), out_dtype="f32")
    g.output(y), g.output(g.argmax(y))
    bits = to_bf16(x)
    got, ids = run_graph_gpu(device, g, [bits])
    xd = torch.from_numpy(from_bf16(bits)).double()
    wd = torch.from_numpy(w).double()
    xd[outliers, [at[b] for b in outliers]] = 0.0  # meets zeros only
    want, bound = (xd @ wd.T).numpy(), K * 2.0 ** -24 * (xd.abs() @ wd.abs().T).numpy()
    assert (np.abs(got - want) <= bound).all(), np.max(np.abs(got - want) / bound)
    assert (ids == got.argmax(-1)).all()
    rest = [b for b in range(B) if b not in outliers]
    beside = run_graph_gpu(device, g, [plain])[0]
    assert (got[rest].view(np.uint32) == beside[rest].view(np.uint32)).all()


@pytest.mark.parametrize("B,K,N", [(1, 64, 40), (3, 1152, 33), (8, 1152, 30001)])
def test_products_of_few_tokens_with_infinities_and_nans(device, B, K, N):
    rng = np.random.default_rng(K)
    x, w, s, _ = _product(rng, B, K, N)
    x[0, 5], x[B - 1, K - 1] = 0x7f80, (0x7fc0 if B > 1 else 0x7f80)
    g = Graph()
    g.output(g.gemv_w8(g.input((B, K), "bf16"), w, s, out_dtype="f32"))
    got = run_graph_gpu(device, g, [x])[0]
    with np.errstate(invalid="ignore"):
        want = (from_bf16(x)[:, None, :] * w.astype(np.float32)[None]).sum(-1) * from_bf16(s)[None]
    assert (np.isnan(got) == np.isnan(want)).all() and (np.isposinf(got) == np.isposinf(want)).all() and (np.isneginf(got) == np.isneginf(want)).all()
    ok = np.isfinite(want)
    assert not ok.any() or np.abs(got[ok] - want[ok]).max() <= 1e-5 * np.abs(want[ok]).max()


@pytest.mark.parametrize("B,K,I", [(1, 64, 1), (5, 1152, 17), (32, 1152, 6912), (17, 4096, 100)])
def test_geglu_behind_the_product(device, B, K, I):
    rng = np.random.default_rng(B + K + I)
    x, w, s, want = _product(rng, B, K, 2 * I)
    g = Graph()
    g.output(g.geglu(g.gemv_w8(g.input((B, K), "bf16"), w, s)))
    ex = Executable(device, g.serialize())
    assert ex.launch_count == 1, ex.op_kernels()
    ex.destroy()
    got = from_bf16(run_graph_gpu(device, g, [x])[0])
    want = _bf(want)
    want = (_bf(torch.nn.functional.gelu(want[:, :I], approximate="tanh")) * want[:, I:]).numpy()
    assert (np.abs(got - want) <= 2.0 ** -6 * np.maximum(np.abs(want), 0.05)).all()


@pytest.mark.parametrize("B,K,I", [(1, 64, 20), (8, 1152, 14400), (3, 1536, 15000)])
def test_geglu_behind_a_product_of_one_group_changes_no_bit(device, B, K, I, monkeypatch):
    """Products whose K no warps share, as wide gate / up ones: the same bits with GeGLU in the launch and behind it."""
    rng = np.random.default_rng(B + K)
    x, w, s, _ = _product(rng, B, K, 2 * I)
    g = Graph()
    g.output(g.geglu(g.gemv_w8(g.input((B, K), "bf16"), w, s)))
    got = run_graph_gpu(device, g, [x])[0]
    monkeypatch.setenv("TB200_NO_DECODER_FUSION", "1")
    ex = Executable(device, g.serialize())
    assert ex.op_kernels() == ["linear_w8", "geglu"], ex.op_kernels()
    ex.destroy()
    alone = run_graph_gpu(device, g, [x])[0]
    assert (got == alone).all(), int((got != alone).sum())


@pytest.mark.parametrize("n_q,B,window", [(1, 1, 0), (2, 3, 20), (4, 9, 130)])
def test_attention_over_short_and_long_caches(device, n_q, B, window):
    rng = np.random.default_rng(n_q)
    D, T = 256, 700
    g = Graph()
    qkv, pos_in = g.input((B, (n_q + 2) * D), "bf16"), g.input((1,), "i32")
    kc, vc = g.state((B, T, D), "bf16"), g.state((B, T, D), "bf16")
    one = to_bf16(np.zeros(D, np.float32))
    q = g.rope_kv(qkv, pos_in, one, one, kc, vc, n_q=n_q, n_kv=1, head_dim=D, theta=10000.0, eps=1e-6)
    g.output(q), g.output(g.attn_decode(q, pos_in, kc, vc, n_q=n_q, n_kv=1, head_dim=D, window=window, scale=D ** -0.5))
    ex = Executable(device, g.serialize())
    d_in, d_pos = device.alloc(B * (n_q + 2) * D * 2), device.alloc(4)
    outs = [device.alloc(B * n_q * D * 2) for _ in range(2)]
    half = D // 2
    inv = torch.pow(torch.tensor(10000.0), -torch.arange(half, dtype=torch.float32) / half)
    K, V = torch.zeros(B, T, D), torch.zeros(B, T, D)
    for pos in range(600):
        t = torch.from_numpy(rng.normal(0, 1, (B, (n_q + 2) * D)).astype(np.float32))
        bits = to_bf16(t.numpy())
        d_in.upload(bits), d_pos.upload(np.array([pos], np.int32))
        ex.dispatch([d_in, d_pos], outs)
        t = torch.from_numpy(from_bf16(bits))
        k = t[:, n_q * D:(n_q + 1) * D]
        k = _bf(k * torch.rsqrt((k * k).mean(-1, keepdim=True) + 1e-6))
        cs, sn = torch.cos(pos * inv), torch.sin(pos * inv)
        K[:, pos] = _bf(torch.cat([k[:, :half] * cs - k[:, half:] * sn, k[:, half:] * cs + k[:, :half] * sn], -1))
        V[:, pos] = t[:, (n_q + 1) * D:]
        if pos in (0, 1, 15, 16, 127, 128, 129, 512, 599):
            qg, got = (from_bf16(o.download((B, n_q * D), np.uint16)) for o in outs)
            lo = max(0, pos - window + 1) if window else 0
            p = torch.softmax(torch.einsum("bhd,btd->bht", torch.from_numpy(qg).reshape(B, n_q, D) * D ** -0.5, K[:, lo:pos + 1]), -1)
            want = torch.einsum("bht,btd->bhd", p, V[:, lo:pos + 1]).reshape(B, -1).numpy()
            assert np.abs(got - want).max() <= 2.0 ** -6 * np.abs(want).max(), pos
    for b in [d_in, d_pos] + outs:
        b.free()
    ex.destroy()


@pytest.mark.parametrize("behind", ["geglu", "rope_kv"])
@pytest.mark.parametrize("B", [1, 2])
def test_norms_in_front_of_a_product_over_the_callers_own_rows(device, B, behind):
    """A residual updated in place, and a result bound over rows that the norm reads: the product's blocks read these rows while others
    store, so the norm has to run before it. The same bits as with buffers of their own, which the norm in the product's launch takes."""
    H, I, n_q, D, T = 1152, 6912, 4, 256, 8
    rng = np.random.default_rng(B)
    x, r = (to_bf16(rng.normal(0, 1, (B, H)).astype(np.float32)) for _ in range(2))
    w1, w2, wd = (to_bf16(rng.normal(0, 0.1, n).astype(np.float32)) for n in (H, H, D))
    N = 2 * I if behind == "geglu" else (n_q + 2) * D
    _, w, s, _ = _product(rng, B, H, N)
    g = Graph()
    xi, ri = g.input((B, H), "bf16"), g.input((B, H), "bf16")
    y1 = g.rmsnorm(xi, w1, 1e-6, residual=ri)
    y = g.gemv_w8(g.rmsnorm(y1, w2, 1e-6), w, s)
    if behind == "geglu":
        y, width = g.geglu(y), I
    else:
        pos = g.input((1,), "i32")
        kc, vc = g.state((B, T, D), "bf16"), g.state((B, T, D), "bf16")
        y, width = g.rope_kv(y, pos, wd, wd, kc, vc, n_q=n_q, n_kv=1, head_dim=D, theta=10000.0, eps=1e-6), n_q * D
    g.output(y1), g.output(y)
    ex = Executable(device, g.serialize())
    assert any(k.startswith("norm_linear_w8") for k in ex.op_kernels()), ex.op_kernels()
    bx, br, b1, by = (device.alloc(2 * B * max(H, width)) for _ in range(4))
    bp = device.alloc(4)
    bp.upload(np.array([3], np.int32))
    want = None
    for o1, oy in ((b1, by), (br, by), (bx, by), (b1, bx), (b1, br), (br, bx)):
        for _ in range(1 if want is None else 20):
            bx.upload(x), br.upload(r)
            ex.dispatch([bx, br] + ([bp] if behind == "rope_kv" else []), [o1, oy])
            got = [o1.download((B, H), np.uint16), oy.download((B, width), np.uint16)]
            want = want or got
            assert all((a == b).all() for a, b in zip(got, want)), (o1 is b1, oy is by)
    for b in (bx, br, b1, by, bp):
        b.free()
    ex.destroy()
