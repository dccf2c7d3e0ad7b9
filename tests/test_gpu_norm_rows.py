"""Norms and softmax of rows in registers (csrc/norm_rows.cu) at the edges of their forms: a warp, one CTA, clusters; lengths that are no
multiple of four (rows start between 16-byte boundaries); channels that end inside a vector; tensors that are not 16-byte aligned; and the
one-pass RMSNorm of longer rows (csrc/norms.cu)."""
import numpy as np
import pytest

from mimir_framework_b200 import abi
from mimir_framework_b200.abi import make_desc
from oracle import port

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt():
    from mimir_framework_b200 import runtime

    runtime.init(0)
    return runtime


def close(got, want):
    assert np.all(np.isfinite(got)) and np.linalg.norm(got.ravel() - want.ravel()) <= 3e-6 * np.linalg.norm(want)


@pytest.mark.parametrize("rows,n", [(1, 1), (3, 5), (200, 31), (7, 1024), (301, 1025), (5, 1027), (2000, 2050), (150, 16381), (149, 16383), (2, 16385), (3, 40001), (1, 131069), (160, 17001)])
def test_layernorm_rmsnorm_softmax(rt, rows, n):
    r = np.random.default_rng(n)
    x = (r.standard_normal((rows, n)) * 2 + 0.5).astype(np.float32)
    g, b = (1 + 0.1 * r.standard_normal(n)).astype(np.float32), r.standard_normal(n).astype(np.float32)
    d = x.astype(np.float64)
    if n > 1:
        close(rt.layernorm(x, g, b, rows, n), (d - d.mean(1, keepdims=True)) / np.sqrt(d.var(1, keepdims=True) + 1e-5) * g + b)
    e = np.exp(d - d.max(1, keepdims=True))
    close(rt.softmax(x, rows, n), e / e.sum(1, keepdims=True))
    if n <= 16384:
        ng = n - n // 3  # gamma applies to a prefix
        want = d / np.sqrt((d * d).mean(1, keepdims=True) + 1e-5)
        want[:, :ng] *= g[:ng]
        close(rt.rmsnorm(x, g[:ng], rows, n), want)


@pytest.mark.parametrize("batch,ch,h,w,groups", [(2, 32, 1, 1, 32), (3, 64, 3, 1, 16), (1, 96, 7, 9, 32), (2, 64, 16, 12, 8), (9, 64, 53, 53, 32), (1, 64, 101, 101, 4), (2, 32, 2, 1, 4)])
@pytest.mark.parametrize("act", [-1, abi.ELT_SILU])
def test_groupnorm(rt, batch, ch, h, w, groups, act):
    r = np.random.default_rng(ch + h)
    x = r.standard_normal((batch, groups, ch // groups * h * w)).astype(np.float32)
    g, b = (1 + 0.1 * r.standard_normal(ch)).astype(np.float32), r.standard_normal(ch).astype(np.float32)
    d = x.astype(np.float64)
    d = ((d - d.mean(2, keepdims=True)) / np.sqrt(d.var(2, keepdims=True) + 1e-5)).reshape(batch, ch, h * w) * g[None, :, None] + b[None, :, None]
    close(rt.groupnorm(x, g, b, batch, ch, h, w, groups, 1e-5, act), d / (1 + np.exp(-d)) if act >= 0 else d)


@pytest.mark.parametrize("rows,n", [(3, 5), (7, 768), (5, 1027), (9, 4096), (3, 16381), (2, 40001), (160, 20004)])
@pytest.mark.parametrize("scale", [1e15, 3e19, 3e28])
def test_variances_at_and_beyond_the_largest_float(rt, rows, n, scale):
    """The reference's variance overflows to infinity there and its rows become beta; so do rows in registers and swept rows."""
    r = np.random.default_rng(n)
    x = (r.standard_normal((rows, n)) * scale).astype(np.float32)
    b = r.standard_normal(n).astype(np.float32)
    got = np.asarray(rt.layernorm(x, np.ones(n, np.float32), b, rows, n)).reshape(rows, n)
    if scale < 1e18:
        d = x.astype(np.float64)
        close(got, (d - d.mean(1, keepdims=True)) / d.std(1, keepdims=True) + b)
    else:
        assert np.abs(got - b).max() <= 1e-6 * np.abs(b).max()


@pytest.mark.parametrize("hw", [(2, 2), (3, 1)])
def test_silu_over_its_whole_range(rt, hw):
    """gamma = 0 and beta = v make every value of a channel silu(v): dense around zero, both ends of the exponential's range, the
    largest floats and the infinities.  Two special-function instructions of 2^-22 each and a few roundings: 2^-21 relative; where
    the reciprocal is flushed the true value is below 1.2e-36."""
    v = np.concatenate([np.linspace(-100, 100, 7993), [0.0, -0.0, 1e-30, -1e-30, 1e-40, -87.3, -87.4, -88.0, -88.8, -1e4, -1e35, -3.4e38, 88.8, 1e35, 2.4e38, 3.4e38,
                        np.inf, 64.0, 64.1]]).astype(np.float32)
    v = np.append(v, np.zeros(-len(v) % 32, np.float32))
    x = np.random.default_rng(0).standard_normal((1, v.size, *hw)).astype(np.float32)
    got = np.asarray(rt.groupnorm(x, np.zeros(v.size, np.float32), v, 1, v.size, *hw, 32, 1e-5, abi.ELT_SILU)).reshape(v.size, -1)
    d = v.astype(np.float64)[:, None]
    with np.errstate(over="ignore"):
        want = np.broadcast_to(d / (1 + np.exp(-d)), got.shape)
    far = np.isinf(want)
    assert np.array_equal(got[far], want[far])
    assert (np.abs(got[~far] - want[~far]) <= 2.0**-21 * np.abs(want[~far]) + 1.2e-36).all()
    v[:] = -np.inf
    assert np.isnan(rt.groupnorm(x, np.zeros(v.size, np.float32), v, 1, v.size, *hw, 32, 1e-5, abi.ELT_SILU)).all()


def test_unaligned_device_tensors(rt):
    import torch

    x, rows, n = torch.randn(4 * 301 + 1, device="cuda"), 4, 301
    y = torch.empty(4 * 301 + 1, device="cuda")
    rt.check(rt.lib().mimir_b200_dev_softmax(x[1:].data_ptr(), y[1:].data_ptr(), rows, n, 0, None))
    torch.cuda.synchronize()
    assert torch.allclose(y[1:].view(rows, n), torch.softmax(x[1:].view(rows, n), 1), atol=1e-6, rtol=1e-5)


@pytest.mark.parametrize("rows,n,ng", [(1, 16388, 16388), (1, 24576, 24576), (2, 16386, 16386), (3, 24580, 24576), (1, 24577, 24577), (148, 24576, 24576), (149, 24576, 24576), (5, 32768, 7)])
def test_one_pass_rmsnorm_gamma(rt, rows, n, ng):
    """Gamma through shared memory (up to three chunks per SM) and from L2, whole and ragged last chunks, gamma shorter than the row."""
    r = np.random.default_rng(rows + n)
    x, g = r.standard_normal((rows, n)).astype(np.float32), r.standard_normal(ng).astype(np.float32)
    got = np.asarray(rt.rmsnorm(x.ravel(), g, rows, n)).reshape(rows, n)
    for i in sorted({0, rows // 2, rows - 1}):
        want = port.rmsnorm(x[i], g, 1e-5)
        assert np.abs(got[i] - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("batch,seq", [(1, 256), (1, 300), (3, 257), (40, 300)])
def test_one_pass_rmsnorm_into_planes(rt, batch, seq):
    """The next Linear's operand planes written by the norm: whole chunks, a ragged last one, few and many CTAs."""
    E, out = 128, 8
    r = np.random.default_rng(seq)
    x = r.standard_normal((batch, seq * E)).astype(np.float32)
    g, w = r.standard_normal(seq * E).astype(np.float32), (r.standard_normal(out * E) / np.sqrt(E)).astype(np.float32)
    descs = [make_desc("n", "RMSNorm", inputs=["x"], output="t", params_count=g.size),
             make_desc("l", "Linear", inputs=["t"], output="x", in_features=E, out_features=out, seq_len=seq, use_bias=False, params_count=w.size)]
    m = rt.GraphModel(descs, abi.PREC_BF16X2)
    m.upload_weights(0, g)
    m.upload_weights(1, w)
    m.plan({"x": (seq * E, False)}, batch)
    got = m.forward({"x": (x, False)}, batch, seq * out)
    m.close()
    for i in sorted({0, batch // 2, batch - 1}):
        want = port.rmsnorm(x[i], g, float(descs[0].eps)).reshape(seq, E).astype(np.float64) @ w.reshape(out, E).T.astype(np.float64)
        assert np.linalg.norm(got[i] - want.ravel()) <= 1e-5 * np.linalg.norm(want)


@pytest.mark.parametrize("rows,n,tickets,flag", [(1, 24576, 0, 1), (3, 24577, 12, 1), (3, 24577, 12, 0), (3, 24577, 5, 1), (40, 40960, 2**31 - 1, 1), (40, 40960, 2**31 - 1, 0)])
def test_rmsnorms_behind_one_that_gave_up_write_nothing(rt, rows, n, tickets, flag):
    """After a bounded wait of the one-pass RMSNorm ran out its ticket counter stands where the launch left it.  The norms queued behind
    it have no row to work on: they leave their output alone and report the timeout, and the first norm after the report is right."""
    import torch

    lib = rt.lib()
    rt.check(lib.mimir_b200_check_device(None))
    x = torch.randn(rows, n, device="cuda")
    y = torch.full((rows, n), 7.0, device="cuda")
    torch.cuda.synchronize()
    run = lambda: rt.check(lib.mimir_b200_dev_rmsnorm(x.data_ptr(), None, 0, y.data_ptr(), rows, n, 1e-5, None))
    rt.check(lib.mimir_b200_selftest_norm_gave_up(tickets, flag, None))
    run()
    run()
    assert lib.mimir_b200_check_device(None) == abi.E_TIMEOUT
    assert bool((y == 7.0).all())
    assert lib.mimir_b200_check_device(None) == abi.OK
    run()
    rt.check(lib.mimir_b200_check_device(None))
    want = x.double() / torch.sqrt((x.double() ** 2).mean(1, keepdim=True) + 1e-5)
    # (the reference's sequential fp32 sum, which the kernel follows, is off by up to n roundings of 2^-24 of the sum of squares)
    assert float((y - want).abs().max()) <= (1e-6 + n * 2.0**-25) * float(want.abs().max())


def contraction_bound(k):
    """fp32 inputs and their split to 2e-6; three MMAs per 16 of K, each of which loses 1.5e-8 to 3.6e-8 of the sum by truncation, of which
    the epilogue puts 1.5e-8 back."""
    return 2e-6 + 3 * (k + 15) // 16 * 2.1e-8


@pytest.mark.parametrize("tokens,d,whole", [(17, 64, False), (200, 128, False), (33, 1088, False), (40, 100, False), (128, 4096, False),
                                            (20, 64, True), (160, 192, True), (128, 256, True), (333, 1024, True), (20, 100, True)])
def test_layernorm_into_operand_planes(rt, tokens, d, whole):
    """A LayerNorm that only a contraction reads writes its operand planes: a row for a warp, a CTA and a cluster, one row of all
    tokens, one too long for registers, and (100 elements, whose planes are padded) the form that stays apart."""
    r = np.random.default_rng(tokens + d)
    n, batch, f = tokens * d, 3, 40
    x = (r.standard_normal((batch, n)) + 0.5).astype(np.float32)
    ln = n if whole else d
    g, be = (1 + 0.1 * r.standard_normal(ln)).astype(np.float32), r.standard_normal(ln).astype(np.float32)
    w, b = (r.standard_normal((f, d)) / np.sqrt(d)).astype(np.float32), r.standard_normal(f).astype(np.float32)
    descs = [abi.make_desc("a", "ReLU", inputs=["x"], output="a"),
             abi.make_desc("n", "LayerNorm", inputs=["a"], output="h", in_features=0 if whole else d, affine=1, use_bias=1, eps=1e-5, params_count=2 * ln),
             abi.make_desc("l", "Linear", inputs=["h"], output="x", in_features=d, out_features=f, seq_len=tokens, use_bias=1, params_count=f * d + f)]
    mod = rt.GraphModel(descs)
    mod.upload_weights(1, np.concatenate([g, be]))
    mod.upload_weights(2, np.concatenate([w.ravel(), b]))
    mod.plan({"x": (n, False)}, batch)
    h = np.maximum(x, 0).astype(np.float64).reshape(batch, -1, ln)
    h = (h - h.mean(-1, keepdims=True)) / np.sqrt(h.var(-1, keepdims=True) + 1e-5) * g + be
    want = h.reshape(batch, tokens, d) @ w.astype(np.float64).T + b
    for _ in range(3):  # layer by layer, captured, replayed
        got = mod.forward({"x": (x.ravel(), False)}, batch, tokens * f).reshape(want.shape)
        assert np.linalg.norm(got - want) <= contraction_bound(d) * np.linalg.norm(want)
    mod.close()


@pytest.mark.parametrize("rows,k,n", [(17, 64, 64), (40, 130, 1000), (300, 96, 70), (1000, 256, 768), (20000, 64, 300)])
def test_linear_with_a_residual_into_operand_planes(rt, rows, k, n):
    """x = act(a) + lin(act(a)), read by one Linear only: the sum leaves the first Linear as the second one's planes."""
    r = np.random.default_rng(rows)
    x = r.standard_normal((rows, k)).astype(np.float32)
    w0, w1, w2 = ((r.standard_normal(s) / np.sqrt(s[1])).astype(np.float32) for s in ((n, k), (n, n), (64, n)))
    lin = lambda name, i, o, w: abi.make_desc(name, "Linear", inputs=[i], output=o, in_features=w.shape[1], out_features=w.shape[0], seq_len=rows, use_bias=0,
                                              params_count=w.size)
    descs = [lin("l0", "x", "a", w0), lin("l1", "a", "b", w1), abi.make_desc("s", "Add", inputs=["a", "b"], output="c"), lin("l2", "c", "x", w2)]
    mod = rt.GraphModel(descs)
    for i, w in ((0, w0), (1, w1), (3, w2)):
        mod.upload_weights(i, w.ravel())
    mod.plan({"x": (rows * k, False)}, 1)
    a = x.astype(np.float64) @ w0.astype(np.float64).T
    want = (a + a @ w1.astype(np.float64).T) @ w2.astype(np.float64).T
    got = mod.forward({"x": (x.ravel(), False)}, 1, rows * 64).reshape(want.shape)
    mod.close()
    assert np.linalg.norm(got - want) <= (contraction_bound(k) + 2 * contraction_bound(n)) * np.linalg.norm(want)


@pytest.mark.parametrize("tokens,d", [(40, 64), (200, 128), (33, 1088), (128, 4096)])
def test_layernorm_into_a_single_operand_plane(rt, tokens, d):
    """PREC_BF16, one plane: the bits of the LayerNorm and the Linear one after the other."""
    r = np.random.default_rng(tokens * d)
    n, batch, f = tokens * d, 2, 72
    x = (r.standard_normal((batch, n)) + 0.5).astype(np.float32)
    g, be = (1 + 0.1 * r.standard_normal(d)).astype(np.float32), r.standard_normal(d).astype(np.float32)
    w, b = (r.standard_normal((f, d)) / np.sqrt(d)).astype(np.float32), r.standard_normal(f).astype(np.float32)
    lin = lambda i: abi.make_desc("l", "Linear", inputs=[i], output="x", in_features=d, out_features=f, seq_len=tokens, use_bias=1, params_count=f * d + f)  # noqa: E731
    norm = lambda o: abi.make_desc("n", "LayerNorm", inputs=["a"], output=o, in_features=d, affine=1, use_bias=1, eps=1e-5, params_count=2 * d)  # noqa: E731
    act = abi.make_desc("a", "ReLU", inputs=["x"], output="a")

    def run(descs, values, per_in, per_out):
        mod = rt.GraphModel(descs, abi.PREC_BF16)
        for i, desc in enumerate(descs):
            if desc.params_count:
                mod.upload_weights(i, np.concatenate([g, be]) if desc.type == b"LayerNorm" else np.concatenate([w.ravel(), b]))
        mod.plan({"x": (per_in, False)}, batch)
        got = mod.forward({"x": (values, False)}, batch, per_out).copy()
        mod.close()
        return got

    got = run([act, norm("h"), lin("h")], x.ravel(), n, tokens * f)
    h = run([act, norm("x")], x.ravel(), n, n)
    assert np.array_equal(got, run([lin("x")], h.ravel(), n, tokens * f))
    # what one plane of 8 or 11 bits per operand leaves
    want = h.reshape(batch, tokens, d).astype(np.float64) @ w.astype(np.float64).T + b
    assert np.linalg.norm(got.reshape(want.shape) - want) <= 2.0**-7 * np.linalg.norm(want)
