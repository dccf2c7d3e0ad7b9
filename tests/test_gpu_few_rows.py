"""Linear layers of at most 16 rows (csrc/skinny_cluster.cu) and the fused decode attention (csrc/attention_decode.cu) at the edges of
their tiles: one row, odd feature counts, K below and across a step, K ranges over a cluster, folded LayerNorm, exact bfloat16
weights; cache positions around a group of keys and head sizes 32, 64 and 128."""
import numpy as np
import pytest

from mimir_framework_b200 import abi, configs
from mimir_framework_b200.abi import make_desc
from oracle import port

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt():
    from mimir_framework_b200 import runtime

    runtime.init(0)
    return runtime


@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("m,n,k", [(1, 1, 4), (3, 33, 128), (4, 31, 132), (5, 100, 768), (8, 4737, 300), (9, 768, 3072), (16, 2304, 768), (16, 65, 4096), (2, 40, 1028)])
def test_few_rows_against_float64(rt, norm, m, n, k):
    r = np.random.default_rng(m * 31 + n)
    x = r.standard_normal((m, k)).astype(np.float32)
    w, b = (r.standard_normal((n, k)) / np.sqrt(k)).astype(np.float32), r.standard_normal(n).astype(np.float32)
    g, be = (1 + 0.1 * r.standard_normal(k)).astype(np.float32), r.standard_normal(k).astype(np.float32)
    lin = make_desc("l", "Linear", inputs=["h" if norm else "x"], output="y", in_features=k, out_features=n, seq_len=m, use_bias=1, params_count=n * k + n)
    descs = ([make_desc("n", "LayerNorm", inputs=["x"], output="h", in_features=k, affine=1, use_bias=1, eps=1e-5, params_count=2 * k)] if norm else []) + [
        lin, make_desc("s", "SiLU", inputs=["y"], output="x")]
    weights = ([np.concatenate([g, be])] if norm else []) + [np.concatenate([w.ravel(), b]), None]
    mod = rt.GraphModel(descs)
    for i, t in enumerate(weights):
        mod.upload_weights(i, t)
    mod.plan({"x": (m * k, False)}, 1)
    got = mod.forward({"x": (x.ravel(), False)}, 1, m * n).reshape(m, n)
    mod.close()
    h = x.astype(np.float64)
    if norm:
        h = (h - h.mean(1, keepdims=True)) / np.sqrt(h.var(1, keepdims=True) + 1e-5) * g + be
    y = h @ w.astype(np.float64).T + b
    want = y / (1 + np.exp(-y))
    assert np.linalg.norm(got - want) <= 2e-6 * np.linalg.norm(want) + 1e-7


@pytest.mark.parametrize("shift", [0, 1, 2])
@pytest.mark.parametrize("m,n,k,micro", [(1, 1, 4, 1), (5, 100, 768, 1), (16, 65, 4096, 1), (2, 40, 1028, 1), (3, 33, 12, 3)])
def test_folded_layernorm_of_a_device_input_at_any_address(rt, m, n, k, micro, shift):
    """The norm of a graph input (here behind an alias) is folded at plan time; the caller's buffer, and each micro-batch in it, may
    start anywhere."""
    import torch

    r = np.random.default_rng(m + n)
    x = r.standard_normal((micro, m, k)).astype(np.float32)
    w, b = (r.standard_normal((n, k)) / np.sqrt(k)).astype(np.float32), r.standard_normal(n).astype(np.float32)
    g, be = (1 + 0.1 * r.standard_normal(k)).astype(np.float32), r.standard_normal(k).astype(np.float32)
    descs = [make_desc("i", "Identity", inputs=["x"], output="a"),
             make_desc("n", "LayerNorm", inputs=["a"], output="h", in_features=k, affine=1, use_bias=1, eps=1e-5, params_count=2 * k),
             make_desc("l", "Linear", inputs=["h"], output="x", in_features=k, out_features=n, seq_len=m, use_bias=1, params_count=n * k + n)]
    mod = rt.GraphModel(descs, pipeline=micro)
    mod.upload_weights(1, np.concatenate([g, be]))
    mod.upload_weights(2, np.concatenate([w.ravel(), b]))
    mod.plan({"x": (m * k, False)}, micro)
    buf = torch.zeros(micro * m * k + 4, device="cuda")
    buf[shift:shift + x.size] = torch.from_numpy(x.ravel())
    out = torch.empty(micro * m * n, device="cuda")
    h = x.astype(np.float64)
    want = (((h - h.mean(-1, keepdims=True)) / np.sqrt(h.var(-1, keepdims=True) + 1e-5) * g + be) @ w.astype(np.float64).T + b).ravel()
    for _ in range(3):  # layer by layer, captured, replayed
        out.zero_()
        mod.forward_device({"x": (buf[shift:].data_ptr(), m * k, False)}, micro, out.data_ptr(), out.numel(), torch.cuda.current_stream().cuda_stream)
        got = out.cpu().numpy()
        assert np.linalg.norm(got - want) <= 2e-6 * np.linalg.norm(want) + 1e-7
    mod.close()


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("batch,heads,hd,prefix", [(1, 3, 64, 15), (2, 4, 32, 31), (3, 2, 128, 7), (16, 4, 64, 16), (1, 1, 64, 1)])
def test_decode_steps_against_the_full_forward(rt, bf16, batch, heads, hd, prefix):
    """Two steps behind a prefix; each row must be the last row of the full causal forward."""
    E, V, steps = heads * hd, 77, 2
    ids = np.random.default_rng(5).integers(0, V, (batch, prefix + steps)).astype(np.float32)
    cfg = dict(layers=2, d_model=E, heads=heads, ffn=4 * E, vocab=V, norm="layer")
    weights = configs.seeded_weights(configs.gpt_decoder(seq=prefix, **cfg), seed=2, std=0.05, bf16=bf16)
    m = rt.GraphModel(configs.gpt_decoder(seq=prefix, **cfg), abi.PREC_BF16W if bf16 else abi.PREC_BF16X2)
    for i, w in enumerate(weights):
        m.upload_weights(i, w)
    m.plan({"x": (prefix, False)}, batch)
    m.decode_begin({"x": (1, False)}, batch, prefix + steps)
    m.forward({"x": (ids[:, :prefix].copy().ravel(), False)}, batch, prefix * V)
    for t in range(prefix, prefix + steps):
        got = m.decode_step({"x": (ids[:, t].copy(), False)}, batch, t, V).reshape(batch, V)
        descs = configs.gpt_decoder(seq=t + 1, **cfg)
        for b in range(batch):
            want = port.run_graph(descs, weights, {"x": ids[b, : t + 1]}).reshape(t + 1, V)[-1]
            assert np.linalg.norm(got[b] - want) <= 2e-5 * np.linalg.norm(want)
    m.close()


@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("m,n,k", [(1, 1, 8), (3, 33, 128), (8, 17, 40), (9, 31, 1032), (16, 768, 3072), (16, 65, 4096), (5, 4737, 768), (16, 4752, 1024), (7, 100, 264)])
def test_exact_bfloat16_weights_against_float64(rt, norm, m, n, k):
    """A step of a token-wise layer whose weights are bfloat16 values (csrc/skinny_mma.cu): one tile and a walk over many, K below a unit, over
    all warps and over a cluster; every warp's accumulators are exact products summed in fp32, as in the fp32 kernel above."""
    r = np.random.default_rng(m * 31 + n)
    x = (r.standard_normal((m, k)) + 1).astype(np.float32)
    w = (r.standard_normal((n, k)) / np.sqrt(k)).astype(np.float32)
    w, b = (w.view(np.uint32) & 0xffff0000).view(np.float32), r.standard_normal(n).astype(np.float32)
    g, be = (1 + 0.1 * r.standard_normal(k)).astype(np.float32), r.standard_normal(k).astype(np.float32)
    lin = make_desc("l", "Linear", inputs=["h" if norm else "x"], output="y", in_features=k, out_features=n, seq_len=1, use_bias=1, params_count=n * k + n)
    descs = ([make_desc("n", "LayerNorm", inputs=["x"], output="h", in_features=k, affine=1, use_bias=1, eps=1e-5, params_count=2 * k)] if norm else []) + [
        lin, make_desc("s", "SiLU", inputs=["y"], output="x")]
    mod = rt.GraphModel(descs, abi.PREC_BF16W)
    for i, t in enumerate(([np.concatenate([g, be])] if norm else []) + [np.concatenate([w.ravel(), b]), None]):
        mod.upload_weights(i, t)
    mod.plan({"x": (k, False)}, m)
    mod.decode_begin({"x": (k, False)}, m, 2)
    h = x.astype(np.float64)
    if norm:
        h = (h - h.mean(1, keepdims=True)) / np.sqrt(h.var(1, keepdims=True) + 1e-5) * g + be
    y = h @ w.astype(np.float64).T + b
    want = y / (1 + np.exp(-y))
    got = mod.decode_step({"x": (x, False)}, m, 0, n).reshape(m, n)
    assert np.linalg.norm(got - want) <= 2e-6 * np.linalg.norm(want) + 1e-7
    x[0, 0] = np.inf  # stays what it is: infinite where the weight is not zero, and the other rows keep their bits
    again = mod.decode_step({"x": (x, False)}, m, 0, n).reshape(m, n)
    mod.close()
    assert np.array_equal(again[1:], got[1:])
    if not norm:
        with np.errstate(invalid="ignore", over="ignore"):
            y = x[:1] @ w.T + b
            want = y / (1 + np.exp(-y))
        assert np.array_equal(np.isnan(again[0]), np.isnan(want[0])) and np.array_equal(np.isposinf(again[0]), np.isposinf(want[0]))


@pytest.mark.parametrize("precision", [abi.PREC_BF16W, abi.PREC_BF16X2])
@pytest.mark.parametrize("what", ["beta", "-gamma", "overflow"])
@pytest.mark.parametrize("m,n,k", [(3, 33, 128), (9, 31, 1032), (16, 65, 4096), (5, 4737, 768), (16, 4752, 1024), (7, 100, 264)])
def test_infinities_that_a_layernorm_makes(rt, precision, what, m, n, k):
    """An infinite beta or gamma, and a gamma that takes a finite row past fp32: the Linear behind that LayerNorm has infinities where the
    weight is not zero and NaN where it is, with exact bfloat16 weights as with fp32 ones."""
    r = np.random.default_rng(m * 31 + n)
    x = (r.standard_normal((m, k)) + 1).astype(np.float32)
    w = (r.standard_normal((n, k)) / np.sqrt(k)).astype(np.float32)
    b = r.standard_normal(n).astype(np.float32)
    if precision == abi.PREC_BF16W:
        w = (w.view(np.uint32) & 0xffff0000).view(np.float32)
    at = k - 5
    w[1::3, at] = 0.0
    g, be = (1 + 0.1 * r.standard_normal(k)).astype(np.float32), r.standard_normal(k).astype(np.float32)
    if what == "beta":
        be[at] = np.inf
    elif what == "-gamma":
        g[at] = -np.inf
    else:
        g[at] = 3e38
        x[:, at] = 1 + 4 * (-1.0) ** np.arange(m)  # about four deviations off either way
    descs = [make_desc("n", "LayerNorm", inputs=["x"], output="h", in_features=k, affine=1, use_bias=1, eps=1e-5, params_count=2 * k),
             make_desc("l", "Linear", inputs=["h"], output="x", in_features=k, out_features=n, seq_len=1, use_bias=1, params_count=n * k + n)]
    mod = rt.GraphModel(descs, precision)
    mod.upload_weights(0, np.concatenate([g, be]))
    mod.upload_weights(1, np.concatenate([w.ravel(), b]))
    mod.plan({"x": (k, False)}, m)
    mod.decode_begin({"x": (k, False)}, m, 2)
    got = mod.decode_step({"x": (x, False)}, m, 0, n).reshape(m, n)
    mod.close()
    with np.errstate(invalid="ignore", over="ignore"):
        h = x.astype(np.float64)
        h = ((h - h.mean(1, keepdims=True)) / np.sqrt(h.var(1, keepdims=True) + 1e-5) * g + be).astype(np.float32)
        want = h[:, at:at + 1] * w[:, at]
    assert np.all(np.isinf(h[:, at])) and np.isnan(want).any() and np.isinf(want).any()
    assert np.array_equal(got, want, equal_nan=True)


def test_a_linear_on_host_arrays_whose_budget_ends_at_its_planes(rt):
    """Room for the arrays and the operand planes to the byte, and none for the word of the weights' largest magnitude."""
    rows, k, n = 256, 256, 256
    r = np.random.default_rng(7)
    x, w = (r.standard_normal(s).astype(np.float32) for s in ((rows, k), (n, k)))
    want = rt.linear_forward(x, w, None, rows, k, n).copy()
    need = 4 * (rows * k + n * k + rows * n) + 4 * rows * k + 4 * n * k  # two planes of two bytes
    stats = rt.guard_stats()
    rt.check(rt.lib().mimir_b200_guard_set_limit(stats["current"] + need))
    try:
        got = rt.linear_forward(x, w, None, rows, k, n)
        rt.check(rt.lib().mimir_b200_guard_set_limit(stats["current"] + need - 1))
        with pytest.raises(rt.MimirB200Error):
            rt.linear_forward(x, w, None, rows, k, n)
    finally:
        rt.check(rt.lib().mimir_b200_guard_set_limit(stats["limit"]))
    assert np.array_equal(got, want)
