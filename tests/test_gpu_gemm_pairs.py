"""The CTA-pair form of the GEMM kernel (tcgen05 cta_group::2) is taken by default only for launches of a full wave of
tiles; MIMIR_B200_GEMM_PAIR=1 (read once per process, hence the child process) forces it wherever the form allows, so that
ragged shapes reach it: an odd number of row tiles (the last pair's second CTA has no rows), row and column counts that
are not multiples of the tile, K-block counts of 1 and more, every precision mode, bias / GELU / residual epilogues, the
operand-plane hand-off between two layers, and a convolution in the shifted-GEMM form."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import sys, os
import numpy as np
sys.path.insert(0, os.path.join(ROOT, "tests")); sys.path.insert(0, ROOT)
from conftest import assert_close
from mimir_framework_b200 import abi, configs, runtime as rt
from oracle import port
rt.init(0, 0)
r = np.random.default_rng(3)
def run(descs, weights, x, out_n, prec):
    m = rt.GraphModel(descs, prec)
    for i, w in enumerate(weights): m.upload_weights(i, w)
    m.plan({"x": (x.size, False)}, 1)
    y = m.forward({"x": (x, False)}, 1, out_n); m.close(); return y.ravel()
n = 0
for rows, k, nout in [(300, 64, 70), (129, 512, 256), (640, 96, 520), (1000, 768, 300), (257, 32, 33)]:
    for prec in (abi.PREC_BF16X2, abi.PREC_BF16W):
        w = (r.standard_normal(k * nout + nout) * 0.05).astype(np.float32)
        if prec == abi.PREC_BF16W: w = configs.round_to_bf16(w)
        x = r.standard_normal(rows * k).astype(np.float32)
        d = [abi.make_desc("l", "Linear", in_features=k, out_features=nout, seq_len=rows, params_count=w.size)]
        assert_close(run(d, [w], x, rows * nout, prec), port.run_graph(d, [w], {"x": x}), f"linear {rows}x{k}x{nout} prec {prec}")
        n += 1
# Linear + GELU -> Linear + residual: planes handed from one pair launch to the next
rows, k = 700, 128
w1 = (r.standard_normal(k * 320 + 320) * 0.05).astype(np.float32); w2 = (r.standard_normal(320 * k + k) * 0.05).astype(np.float32)
d = [abi.make_desc("f1", "Linear", output="h", in_features=k, out_features=320, seq_len=rows, params_count=w1.size),
     abi.make_desc("g", "GELU", inputs=["h"], output="g"),
     abi.make_desc("f2", "Linear", inputs=["g"], output="o", in_features=320, out_features=k, seq_len=rows, params_count=w2.size),
     abi.make_desc("a", "Add", inputs=["o", "__input__"], output="x")]
x = r.standard_normal(rows * k).astype(np.float32)
assert_close(run(d, [w1, None, w2, None], x, rows * k, abi.PREC_BF16X2), port.run_graph(d, [w1, None, w2, None], {"x": x}), "ffn with residual"); n += 1
# convolution, 256 output channels (the unswapped channel-major form), 3 x 3 and 1 x 1
for ks in (3, 1):
    ic, oc, hw = 64, 256, 20
    cw = (r.standard_normal(oc * ic * ks * ks) * np.sqrt(2 / (ic * ks * ks))).astype(np.float32)
    d = [abi.make_desc("c", "Conv2d", in_channels=ic, out_channels=oc, input_height=hw, input_width=hw, kernel=ks, stride=1, padding=ks // 2, params_count=cw.size)]
    x = r.standard_normal(ic * hw * hw).astype(np.float32)
    assert_close(run(d, [cw], x, oc * hw * hw, abi.PREC_BF16X2), port.run_graph(d, [cw], {"x": x}), f"conv {ks}x{ks}"); n += 1
rt.check(rt.lib().mimir_b200_check_device(None))
print("PAIR_CASES_OK", n)
"""


def test_forced_cta_pairs_on_ragged_shapes():
    env = dict(os.environ, MIMIR_B200_GEMM_PAIR="1")
    out = subprocess.run([sys.executable, "-c", "ROOT = %r\n" % ROOT + CHILD], env=env, capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout[-2000:] + out.stderr[-4000:]
    assert "PAIR_CASES_OK 13" in out.stdout, out.stdout[-2000:]


@pytest.mark.parametrize("precision", ["x2", "w"])
@pytest.mark.parametrize("whole,cut,n,k", [(9472, 9600, 1024, 256), (12800, 8192, 256, 616), (9472, 9500, 1000, 1032)])
def test_tiles_cut_in_two_keep_their_bits(precision, whole, cut, n, k):
    """The last wave's tiles run as two of 128 columns where it would leave half of the CTAs idle (`cut` rows: 4 of 74 pair tiles, and 64 of
    148 single ones) and whole elsewhere (`whole` rows): the rows the two launches share have the same bits."""
    import numpy as np
    from mimir_framework_b200 import abi, configs, runtime as rt

    rt.init(0)
    r = np.random.default_rng(n)
    w = (r.standard_normal(n * k + n) * 0.05).astype(np.float32)
    if precision == "w":
        w = configs.round_to_bf16(w)
    x = r.standard_normal((max(whole, cut), k)).astype(np.float32)
    got = []
    for rows in (whole, cut):
        m = rt.GraphModel([abi.make_desc("l", "Linear", in_features=k, out_features=n, seq_len=rows, use_bias=1, params_count=w.size),
                           abi.make_desc("g", "GELU", inputs=["x"], output="x")], abi.PREC_BF16X2 if precision == "x2" else abi.PREC_BF16W)
        m.upload_weights(0, w)
        m.plan({"x": (rows * k, False)}, 1)
        got.append(m.forward({"x": (x[:rows].ravel(), False)}, 1, rows * n).reshape(rows, n))
        m.close()
    both = min(whole, cut)
    assert np.array_equal(got[0][:both], got[1][:both])
    want = x[-40:].astype(np.float64) @ w[: n * k].reshape(n, k).T.astype(np.float64) + w[n * k:]
    want = want * 0.5 * (1 + np.tanh(0.7978845608 * (want + 0.044715 * want ** 3)))
    big = got[0] if whole > cut else got[1]
    assert np.linalg.norm(big[-40:] - want) <= 1e-5 * np.linalg.norm(want)


@pytest.mark.parametrize("precision", ["x2", "w"])
@pytest.mark.parametrize("what", ["residual", "planes"])
@pytest.mark.parametrize("whole,cut,n,k", [(9472, 9600, 1024, 256), (12800, 8192, 256, 616), (9472, 9500, 1000, 1032)])
def test_cut_tiles_of_every_epilogue_keep_their_bits(precision, what, whole, cut, n, k):
    """As above, for tiles that add a residual and tiles that write the next layer's operand planes (whose own tiles are cut as well)."""
    import numpy as np
    from mimir_framework_b200 import abi, configs, runtime as rt

    rt.init(0)
    r = np.random.default_rng(n + k)
    weights = [(r.standard_normal(o * i + o) * 0.05).astype(np.float32) for i, o in ((k, n), (n, n))]
    if precision == "w":
        weights = [configs.round_to_bf16(w) for w in weights]
    x, res = (r.standard_normal((max(whole, cut), c)).astype(np.float32) for c in (k, n))
    got = []
    for rows in (whole, cut):
        descs = [abi.make_desc("l", "Linear", inputs=["x"], output="h", in_features=k, out_features=n, seq_len=rows, use_bias=1, params_count=weights[0].size)]
        if what == "residual":
            descs.append(abi.make_desc("s", "Add", inputs=["h", "r"], output="x"))
        else:
            descs.append(abi.make_desc("m", "Linear", inputs=["h"], output="x", in_features=n, out_features=n, seq_len=rows, use_bias=1, params_count=weights[1].size))
        m = rt.GraphModel(descs, abi.PREC_BF16X2 if precision == "x2" else abi.PREC_BF16W)
        m.upload_weights(0, weights[0])
        inputs = {"x": (x[:rows].ravel(), False)}
        if what == "residual":
            inputs["r"] = (res[:rows].ravel(), False)
        else:
            m.upload_weights(1, weights[1])
        m.plan({name: (v.size, bc) for name, (v, bc) in inputs.items()}, 1)
        got.append(m.forward(inputs, 1, rows * n).reshape(rows, n))
        m.close()
    both = min(whole, cut)
    assert np.array_equal(got[0][:both], got[1][:both])
    want = x[-40:].astype(np.float64) @ weights[0][: n * k].reshape(n, k).T.astype(np.float64) + weights[0][n * k:]
    if what == "residual":
        want = want + res[-40:]
    else:
        want = want @ weights[1][: n * n].reshape(n, n).T.astype(np.float64) + weights[1][n * n:]
    big = got[0] if whole > cut else got[1]
    # 1e-5 for each contraction
    assert np.linalg.norm(big[-40:] - want) <= (1e-5 if what == "residual" else 2e-5) * np.linalg.norm(want)
