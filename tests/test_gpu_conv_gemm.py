"""The spatial-tile convolution kernel (csrc/conv_gemm.cu), forced on images at the edges of its 16 x 16 tiles: one tile, one pixel more
and less, several output-channel tiles, 32 and more input channels, kernels of 3, 5 and 7, every precision, residual and ReLU."""
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
@pytest.mark.parametrize("batch,ic,oc,h,w,k", [(1, 32, 16, 16, 16, 3), (2, 64, 130, 17, 33, 3), (3, 96, 40, 31, 15, 5), (1, 32, 260, 5, 48, 7), (2, 256, 128, 32, 32, 3),
                                               (5, 32, 33, 1, 1, 3), (2, 64, 128, 20, 40, 1), (2, 32, 64, 9, 64, 5)])
def test_forced_spatial_tiles_against_the_port(rt, monkeypatch, precision, batch, ic, oc, h, w, k):
    monkeypatch.setenv("MIMIR_B200_CONV_SPATIAL", "1")
    r = np.random.default_rng(batch * ic + oc + k)
    x = r.standard_normal((batch, ic * h * w)).astype(np.float32)
    res = r.standard_normal((batch, oc * h * w)).astype(np.float32)
    wt = (r.standard_normal(oc * ic * k * k) / np.sqrt(ic * k * k)).astype(np.float32)
    if precision != abi.PREC_BF16X2:
        wt = (wt.view(np.uint32) & 0xffff0000).view(np.float32)  # exact in one plane
    descs = [make_desc("c", "Conv2d", inputs=["x"], output="y", in_channels=ic, out_channels=oc, input_height=h, input_width=w, kernel=k, stride=1,
                       padding=k // 2, params_count=wt.size), make_desc("a", "Add", inputs=["y", "r"], output="x")]
    m = rt.GraphModel(descs, precision)
    m.upload_weights(0, wt)
    m.plan({"x": (ic * h * w, False), "r": (oc * h * w, False)}, batch)
    got = m.forward({"x": (x, False), "r": (res, False)}, batch, oc * h * w)
    m.close()
    want = np.stack([port.conv2d(x[i], wt, ic, oc, h, w, k, 1, k // 2, False).ravel() for i in range(batch)]) + res
    tol = 2e-3 if precision == abi.PREC_BF16 else 1e-5
    assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)


@pytest.mark.parametrize("batch,ic,oc,h,k,stride,pad", [(2, 3, 64, 37, 7, 2, 3), (1, 40, 130, 20, 3, 2, 1), (3, 4, 70, 18, 3, 1, 1)])
def test_im2col_rows_as_pixels(rt, monkeypatch, batch, ic, oc, h, k, stride, pad):
    monkeypatch.setenv("MIMIR_B200_CONV_SPATIAL", "1")
    r = np.random.default_rng(ic)
    x = r.standard_normal((batch, ic * h * h)).astype(np.float32)
    wt = (r.standard_normal(oc * ic * k * k) / np.sqrt(ic * k * k)).astype(np.float32)
    got = rt.conv2d(x, wt, batch, ic, oc, h, h, k, stride, pad).reshape(batch, -1)
    want = np.stack([port.conv2d(x[i], wt, ic, oc, h, h, k, stride, pad, False).ravel() for i in range(batch)])
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)


def test_relu_and_many_tiles(rt):
    """The default dispatch: more tiles than SMs, ReLU in the epilogue."""
    batch, ic, oc, h = 20, 32, 24, 48
    r = np.random.default_rng(1)
    x = r.standard_normal((batch, ic * h * h)).astype(np.float32)
    wt = (r.standard_normal(oc * ic * 9) / np.sqrt(ic * 9)).astype(np.float32)
    got = rt.conv2d(x, wt, batch, ic, oc, h, h, 3, 1, 1, relu=True).reshape(batch, -1)
    want = np.stack([port.conv2d(x[i], wt, ic, oc, h, h, 3, 1, 1, True).ravel() for i in range(batch)])
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)
