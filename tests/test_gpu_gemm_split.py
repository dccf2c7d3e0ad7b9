"""The split-K contraction kernel (csrc/gemm_split.cu) at the sizes where it can go wrong: one row, tile edges in every direction,
K shorter than a block per split, every width and split count, row-major and channel-major outputs."""
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


@pytest.mark.parametrize("precision", [abi.PREC_BF16X2, abi.PREC_BF16W, abi.PREC_BF16])
@pytest.mark.parametrize("form,m,n,k", [("16,1", 17, 1, 64), ("16,8", 17, 129, 520), ("32,4", 33, 127, 300), ("48,2", 97, 256, 128), ("64,8", 65, 70, 1000),
                                        ("96,1", 200, 300, 65), ("48,10", 50, 131, 700), ("32,12", 33, 70, 1000), ("64,5", 100, 129, 520), ("128,1", 129, 128, 1), ("128,8", 257, 385, 2048), ("", 40, 1000, 4100), ("", 333, 1000, 1000)])
def test_linear_against_float64(rt, monkeypatch, precision, form, m, n, k):
    if form:
        monkeypatch.setenv("MIMIR_B200_GEMM_SPLIT", form)
    r = np.random.default_rng(m * 7 + n)
    x = r.standard_normal((m, k)).astype(np.float32)
    w = (r.standard_normal((n, k)) / np.sqrt(k)).astype(np.float32)
    if precision != abi.PREC_BF16X2:
        w = (w.view(np.uint32) & 0xffff0000).view(np.float32)  # exact in one plane
    b, res = r.standard_normal(n).astype(np.float32), r.standard_normal((m, n)).astype(np.float32)
    descs = [make_desc("l", "Linear", inputs=["x"], output="h", in_features=k, out_features=n, seq_len=m, use_bias=1, params_count=n * k + n),
             make_desc("g", "GELU", inputs=["h"], output="a"), make_desc("s", "Add", inputs=["r", "a"], output="x")]
    mod = rt.GraphModel(descs, precision)
    mod.upload_weights(0, np.concatenate([w.ravel(), b]))
    mod.plan({"x": (m * k, False), "r": (m * n, False)}, 1)
    got = mod.forward({"x": (x.ravel(), False), "r": (res.ravel(), False)}, 1, m * n).reshape(m, n)
    mod.close()
    h = x.astype(np.float64) @ w.astype(np.float64).T + b
    want = h * 0.5 * (1 + np.tanh(0.7978845608 * (h + 0.044715 * h ** 3))) + res
    tol = 2e-3 if precision == abi.PREC_BF16 else 1e-5
    assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)


@pytest.mark.parametrize("precision", [abi.PREC_BF16X2, abi.PREC_BF16W])
@pytest.mark.parametrize("m,n,k", [(257, 6000, 2100), (1025, 4100, 2100), (1409, 2700, 2500), (1537, 2304, 1100), (100, 38000, 520)])
def test_around_one_wave_of_big_tiles(rt, precision, m, n, k):
    """72, 153, 132, 117 and 149 tiles of 128 x 256, where narrow tiles give way to big ones (cut in two in the last wave, in pairs and alone)."""
    r = np.random.default_rng(m + n)
    x = r.standard_normal((m, k)).astype(np.float32)
    w = (r.standard_normal((n, k)) / np.sqrt(k)).astype(np.float32)
    if precision != abi.PREC_BF16X2:
        w = (w.view(np.uint32) & 0xffff0000).view(np.float32)
    b = r.standard_normal(n).astype(np.float32)
    mod = rt.GraphModel([make_desc("l", "Linear", in_features=k, out_features=n, seq_len=m, use_bias=1, params_count=n * k + n)], precision)
    mod.upload_weights(0, np.concatenate([w.ravel(), b]))
    mod.plan({"x": (m * k, False)}, 1)
    got = mod.forward({"x": (x.ravel(), False)}, 1, m * n).reshape(m, n)
    mod.close()
    rows = np.unique(np.concatenate([np.arange(0, m, 37), np.arange(m - 5, m)]))
    want = x[rows].astype(np.float64) @ w.astype(np.float64).T + b
    assert np.all(np.isfinite(got)) and np.linalg.norm(got[rows] - want) <= 1e-5 * np.linalg.norm(want)
    cols = np.unique(np.concatenate([np.arange(0, n, 61), np.arange(n - 5, n)]))
    want = x.astype(np.float64) @ w[cols].astype(np.float64).T + b[cols]
    assert np.linalg.norm(got[:, cols] - want) <= 1e-5 * np.linalg.norm(want)


@pytest.mark.parametrize("form", ["16,1", "48,2", "48,5", "128,8", ""])
@pytest.mark.parametrize("batch,ic,oc,h,w,k,stride,pad", [(1, 64, 130, 9, 7, 3, 1, 1), (3, 32, 40, 5, 11, 1, 1, 0), (2, 96, 16, 8, 8, 5, 1, 2), (2, 3, 70, 17, 19, 7, 2, 3)])
def test_convolution_against_the_port(rt, monkeypatch, form, batch, ic, oc, h, w, k, stride, pad):
    if form:
        monkeypatch.setenv("MIMIR_B200_GEMM_SPLIT", form)
    r = np.random.default_rng(batch * ic + oc)
    x = r.standard_normal((batch, ic * h * w)).astype(np.float32)
    wt = (r.standard_normal(oc * ic * k * k) / np.sqrt(ic * k * k)).astype(np.float32)
    got = rt.conv2d(x, wt, batch, ic, oc, h, w, k, stride, pad).reshape(batch, -1)
    want = np.stack([port.conv2d(x[i], wt, ic, oc, h, w, k, stride, pad, False).ravel() for i in range(batch)])
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)


@pytest.mark.parametrize("form", ["16,1", "16,5", "48,3", "48,10", "96,6", "128,2", ""])
@pytest.mark.parametrize("m,k,n", [(1, 40, 33), (50, 70, 131), (97, 200, 255), (130, 129, 64)])
def test_chain_through_operand_planes(rt, monkeypatch, form, m, k, n):
    """Linear -> GELU -> Linear: the first layer writes the second one's operand planes (zero up to a multiple of 64 columns), odd row
    lengths go element by element, cluster sizes that are no power of two included."""
    if form:
        monkeypatch.setenv("MIMIR_B200_GEMM_SPLIT", form)
    r = np.random.default_rng(m + n)
    x = r.standard_normal((m, k)).astype(np.float32)
    w = [(r.standard_normal((o, i)) / np.sqrt(i)).astype(np.float32) for i, o in ((k, n), (n, n))]
    b = [r.standard_normal(n).astype(np.float32) for _ in range(2)]
    descs = [make_desc("l", "Linear", inputs=["x"], output="h", in_features=k, out_features=n, seq_len=m, use_bias=1, params_count=n * k + n),
             make_desc("g", "GELU", inputs=["h"], output="a"),
             make_desc("m", "Linear", inputs=["a"], output="x", in_features=n, out_features=n, seq_len=m, use_bias=1, params_count=n * n + n)]
    mod = rt.GraphModel(descs)
    for layer, i in ((0, 0), (2, 1)):
        mod.upload_weights(layer, np.concatenate([w[i].ravel(), b[i]]))
    mod.plan({"x": (m * k, False)}, 1)
    got = mod.forward({"x": (x.ravel(), False)}, 1, m * n).reshape(m, n)
    mod.close()
    h = x.astype(np.float64) @ w[0].astype(np.float64).T + b[0]
    a = h * 0.5 * (1 + np.tanh(0.7978845608 * (h + 0.044715 * h ** 3)))
    want = a @ w[1].astype(np.float64).T + b[1]
    # two contractions of at most 255 products, a few 1e-6 each (operand planes and accumulation)
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)


@pytest.mark.parametrize("precision", [abi.PREC_BF16X2, abi.PREC_BF16W])
@pytest.mark.parametrize("form", ["64,1", "128,1", "32,3"])
@pytest.mark.parametrize("ic,stride", [(512, 1), (512, 2), (1024, 1), (1024, 0)])
def test_mean_loss_of_the_sums_is_put_back_once(rt, monkeypatch, precision, form, ic, stride):
    """The tensor core's truncating adds make every sum a little too small, by a share that K fixes; the kernel puts the mean of it back, in
    channel-major results (3 x 3 convolutions, stride 2 over im2col rows) and row-major ones (stride 0 here: a Linear) alike."""
    monkeypatch.setenv("MIMIR_B200_GEMM_SPLIT", form)
    r = np.random.default_rng(ic + stride)
    oc, k = 130, 9 * ic
    w = (r.standard_normal((oc, k)) / np.sqrt(k)).astype(np.float32)
    if precision != abi.PREC_BF16X2:
        w = (w.view(np.uint32) & 0xffff0000).view(np.float32)
    if stride:
        h = 9 if stride == 1 else 18
        x = r.standard_normal((2, ic, h, h)).astype(np.float32)
        desc = make_desc("c", "Conv2d", in_channels=ic, out_channels=oc, input_height=h, input_width=h, kernel=3, stride=stride, padding=1, params_count=w.size)
        taps = np.lib.stride_tricks.sliding_window_view(np.pad(x, ((0, 0), (0, 0), (1, 1), (1, 1))), (3, 3), (2, 3))[:, :, ::stride, ::stride]
        rows = taps.transpose(0, 2, 3, 1, 4, 5).reshape(2, -1, k)
        want = (rows.astype(np.float64) @ w.T.astype(np.float64)).transpose(0, 2, 1)
        batch = 2
    else:
        x = r.standard_normal((162, k)).astype(np.float32)
        desc = make_desc("l", "Linear", in_features=k, out_features=oc, seq_len=162, use_bias=0, params_count=w.size)
        want = (x.astype(np.float64) @ w.T.astype(np.float64))[None]
        batch = 1
    mod = rt.GraphModel([desc], precision)
    mod.upload_weights(0, w.ravel())
    mod.plan({"x": (x.size // batch, False)}, batch)
    got = mod.forward({"x": (x.reshape(batch, -1), False)}, batch, want[0].size).reshape(want.shape)
    mod.close()
    # Normal operands lose 1.5e-8 of the sum per instruction, measured to within 1e-9 at every K; a correction that is missing, or there
    # twice, is 1.5e-8 x one or two of the products per 16 of K.
    products = 3 if precision == abi.PREC_BF16X2 else 2
    assert abs(np.vdot(got - want, want) / np.vdot(want, want)) <= 2e-9 * products * k / 16
