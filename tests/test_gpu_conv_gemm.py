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


@pytest.mark.parametrize("skip_conv", [False, True])
@pytest.mark.parametrize("batch,ic,oc,h,w", [(40, 32, 130, 12, 10), (10, 64, 64, 34, 18), (150, 32, 32, 1, 1), (2, 32, 32, 8, 8)])
def test_residual_block_behind_an_upsample(rt, batch, ic, oc, h, w, skip_conv):
    """Up -> conv -> conv, plus the upsampled image itself or a 1 x 1 convolution of it, which stands after the other two."""
    oc = oc if skip_conv else ic
    r = np.random.default_rng(batch + oc)
    x = r.standard_normal((batch, ic * h * w)).astype(np.float32)
    shapes = [(oc, ic, 3), (oc, oc, 3), (oc, ic, 1)]
    ws = [(r.standard_normal(o * i * k * k) / np.sqrt(i * k * k)).astype(np.float32) for o, i, k in shapes]
    conv = lambda name, a, b, j: make_desc(name, "Conv2d", inputs=[a], output=b, in_channels=shapes[j][1], out_channels=oc, input_height=2 * h,  # noqa: E731
                                           input_width=2 * w, kernel=shapes[j][2], stride=1, padding=shapes[j][2] // 2, params_count=ws[j].size)
    descs = [make_desc("u", "UpsampleNearest", inputs=["x"], output="u", in_channels=ic, out_h=h, out_w=w, scale_h=2, scale_w=2),
             conv("c1", "u", "t", 0), conv("c2", "t", "y", 1)]
    if skip_conv:
        descs.append(conv("c3", "u", "s", 2))
    descs.append(make_desc("a", "Add", inputs=["y", "s" if skip_conv else "u"], output="x"))
    m = rt.GraphModel(descs, abi.PREC_BF16X2)
    for j in range(3 if skip_conv else 2):
        m.upload_weights(1 + j, ws[j])
    m.plan({"x": (ic * h * w, False)}, batch)
    got = m.forward({"x": (x, False)}, batch, oc * 4 * h * w)
    m.close()
    for i in range(0, batch, 3):
        u = x[i].reshape(ic, h, w).repeat(2, 1).repeat(2, 2).ravel()
        t = port.conv2d(u, ws[0], ic, oc, 2 * h, 2 * w, 3, 1, 1, False).ravel()
        want = port.conv2d(t, ws[1], oc, oc, 2 * h, 2 * w, 3, 1, 1, False).ravel()
        want = want + (port.conv2d(u, ws[2], ic, oc, 2 * h, 2 * w, 1, 1, 0, False).ravel() if skip_conv else u)
        assert np.linalg.norm(got[i] - want) <= 2e-5 * np.linalg.norm(want)


@pytest.mark.parametrize("precision", [abi.PREC_BF16X2, abi.PREC_BF16W])
@pytest.mark.parametrize("batch,ic,oc,h,w,k,up", [(1, 32, 16, 16, 16, 3, 0), (2, 64, 130, 17, 33, 3, 0), (3, 96, 40, 31, 15, 5, 0), (1, 32, 260, 9, 48, 7, 0), (5, 32, 33, 1, 1, 3, 0),
                                                  (2, 64, 128, 20, 40, 1, 0), (3, 64, 70, 3, 43, 1, 0), (40, 32, 32, 12, 10, 3, 1)])
def test_tiles_of_128_pixels_keep_the_bits_of_256(rt, monkeypatch, precision, batch, ic, oc, h, w, k, up):
    """Half of a tile's pixels, the same sums in the same order: 8 rows of 16, or 128 of a line; with a residual, plain or read at half size."""
    monkeypatch.setenv("MIMIR_B200_CONV_SPATIAL", "1")
    r = np.random.default_rng(batch * ic + oc + k)
    wt = (r.standard_normal(oc * ic * k * k) / np.sqrt(ic * k * k)).astype(np.float32)
    if precision != abi.PREC_BF16X2:
        wt = (wt.view(np.uint32) & 0xffff0000).view(np.float32)
    s = 2 if up else 1
    conv = lambda name, a, b: make_desc(name, "Conv2d", inputs=[a], output=b, in_channels=ic, out_channels=oc, input_height=s * h, input_width=s * w,  # noqa: E731
                                        kernel=k, stride=1, padding=k // 2, params_count=wt.size)
    if up:
        descs = [make_desc("u", "UpsampleNearest", inputs=["x"], output="u", in_channels=ic, out_h=h, out_w=w, scale_h=2, scale_w=2), conv("c", "u", "t"), conv("d", "t", "y"),
                 make_desc("a", "Add", inputs=["y", "u"], output="x")]
    else:
        descs = [conv("c", "x", "y"), make_desc("a", "Add", inputs=["y", "r"], output="x")]
    ins = {"x": (r.standard_normal((batch, ic * h * w)).astype(np.float32), False)}
    if not up:
        ins["r"] = (r.standard_normal((batch, oc * h * w)).astype(np.float32), False)
    got = []
    for px in ("256", "128"):
        monkeypatch.setenv("MIMIR_B200_CONV_PX", px)
        m = rt.GraphModel(descs, precision)
        for j, d in enumerate(descs):
            if d.type == b"Conv2d":
                m.upload_weights(j, wt)
        m.plan({n: (a.shape[1], bc) for n, (a, bc) in ins.items()}, batch)
        got.append(m.forward(ins, batch, oc * s * s * h * w))
        m.close()
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("form", ["skip", "chain", "plain"])
@pytest.mark.parametrize("batch,ic,oc,h,w,groups", [(20, 64, 128, 58, 58, 32), (33, 32, 64, 63, 65, 16), (3, 32, 256, 120, 99, 8), (45, 32, 160, 37, 33, 5), (80, 32, 64, 48, 48, 32),
                                                  (2, 32, 64, 40, 34, 8), (1, 64, 40, 32, 32, 8)])
def test_groupnorm_statistics_of_a_large_result(rt, form, batch, ic, oc, h, w, groups):
    """Conv -> GroupNorm -> SiLU on 32 MB and more: the moments come from the convolution's epilogue where a GroupNorm of four channels and more
    to a group is folded behind few rows or a long sum, else from a sweep.  Then a 1 x 1 convolution that the normalised tensor is
    added to, a convolution that reads it, or nothing.  Tiles cut at the right and the lower edge; values with a mean of several deviations."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(batch + oc)
    randn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    x = randn(batch, ic, h, w) + 2.0
    w1 = (randn(oc, ic, 3, 3) + 0.3) / (9 * ic) ** 0.5
    g, b = 1 + 0.2 * randn(oc), 0.1 * randn(oc)
    k2 = 1 if form == "skip" else 3
    w2 = randn(oc, ic if form == "skip" else oc, k2, k2) / (k2 * k2 * oc) ** 0.5
    conv = lambda name, i, o, c, k: make_desc(name, "Conv2d", inputs=[i], output=o, in_channels=c, out_channels=oc, input_height=h, input_width=w,  # noqa: E731
                                              kernel=k, stride=1, padding=k // 2, params_count=oc * c * k * k)
    descs = [conv("c1", "x", "a", ic, 3),
             make_desc("g", "GroupNorm", inputs=["a"], output="b", in_channels=oc, input_height=h, input_width=w, num_groups=groups, affine=1, use_bias=1, eps=1e-5,
                       params_count=2 * oc), make_desc("s", "SiLU", inputs=["b"], output="x" if form == "plain" else "c")]
    if form == "skip":
        descs += [conv("c2", "x", "d", ic, 1), make_desc("add", "Add", inputs=["c", "d"], output="x")]
    elif form == "chain":
        descs += [conv("c2", "c", "x", oc, 3)]
    m = rt.GraphModel(descs)
    m.upload_weights(0, w1.cpu().numpy().ravel())
    m.upload_weights(1, torch.cat([g, b]).cpu().numpy())
    if form != "plain":
        m.upload_weights(3, w2.cpu().numpy().ravel())
    m.plan({"x": (ic * h * w, False)}, batch)
    got = torch.empty(batch, oc, h, w, device="cuda")
    d = lambda t: t.double()  # noqa: E731
    c = torch.nn.functional.silu(torch.nn.functional.group_norm(torch.nn.functional.conv2d(d(x), d(w1), padding=1), groups, d(g), d(b), 1e-5))
    want = c + torch.nn.functional.conv2d(d(x), d(w2)) if form == "skip" else torch.nn.functional.conv2d(c, d(w2), padding=1) if form == "chain" else c
    torch.cuda.synchronize()
    for _ in range(3):  # layer by layer, captured, replayed
        got.zero_()
        m.forward_device({"x": (x.data_ptr(), ic * h * w, False)}, batch, got.data_ptr(), got.numel())
        torch.cuda.synchronize()
        # two contractions (4e-6 each, of values that the norm then takes a mean of up to five deviations from)
        assert (got - want).norm() <= 3e-5 * want.norm()
    m.close()


def test_planes_are_not_kept_where_the_budget_has_no_room(rt):
    """Conv -> conv -> Add with a 1 x 1 convolution of the input, which reads the first one's planes; planned again with a budget that
    these would exceed, it lays out its own, and gives the same."""
    batch, c, h = 4, 64, 64
    r = np.random.default_rng(3)
    x = r.standard_normal((batch, c * h * h)).astype(np.float32)
    ws = [(r.standard_normal(c * c * k * k) / np.sqrt(c * k * k)).astype(np.float32) for k in (3, 3, 1)]
    conv = lambda name, i, o, k: make_desc(name, "Conv2d", inputs=[i], output=o, in_channels=c, out_channels=c, input_height=h, input_width=h, kernel=k,  # noqa: E731
                                           stride=1, padding=k // 2, params_count=c * c * k * k)
    descs = [conv("c1", "x", "a", 3), conv("c2", "a", "b", 3), conv("c3", "x", "d", 1), make_desc("add", "Add", inputs=["b", "d"], output="x")]

    def run():
        m = rt.GraphModel(descs)
        for i, w in enumerate(ws):
            m.upload_weights(i, w)
        m.plan({"x": (c * h * h, False)}, batch)
        used, arena = rt.guard_stats()["current"], rt.stats()["arena_peak_bytes"]
        got = m.forward({"x": (x, False)}, batch, c * h * h).copy()
        m.close()
        return got, used, arena

    before = rt.guard_stats()["limit"]
    want, used, arena = run()
    rt.check(rt.lib().mimir_b200_guard_set_limit(used - (1 << 20)))
    try:
        got, _, less = run()
    finally:
        rt.check(rt.lib().mimir_b200_guard_set_limit(before))
    assert less < arena
    assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)


@pytest.mark.parametrize("silu", [True, False])
@pytest.mark.parametrize("batch,ic,oc,h,w,k,groups", [(9, 64, 3, 120, 124, 3, 32), (3, 96, 1, 171, 172, 5, 8), (35, 32, 8, 65, 128, 1, 32), (2, 160, 4, 203, 132, 7, 40)])
def test_direct_convolution_normalises_its_input(rt, silu, batch, ic, oc, h, w, k, groups):
    """GroupNorm (+ SiLU) read by a convolution to a handful of channels only, on more than 32 MB: tiles cut at every edge, whose ring stays zero (in
    one launch where that is faster, test_direct_convolution_normalises_where_that_is_faster)."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(ic + oc)
    randn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    x = randn(batch, ic, h, w) + 1.0
    g, b, wt = 1 + 0.2 * randn(ic), 0.5 * randn(ic), randn(oc, ic, k, k) / (ic * k * k) ** 0.5
    descs = [make_desc("r", "LeakyReLU", inputs=["x"], output="a"),
             make_desc("g", "GroupNorm", inputs=["a"], output="b", in_channels=ic, input_height=h, input_width=w, num_groups=groups, affine=1, use_bias=1, eps=1e-5,
                       params_count=2 * ic)]
    if silu:
        descs.append(make_desc("s", "SiLU", inputs=["b"], output="c"))
    descs.append(make_desc("c", "Conv2d", inputs=["c" if silu else "b"], output="x", in_channels=ic, out_channels=oc, input_height=h, input_width=w, kernel=k, stride=1,
                           padding=k // 2, params_count=wt.numel()))
    m = rt.GraphModel(descs)
    m.upload_weights(1, torch.cat([g, b]).cpu().numpy())
    m.upload_weights(len(descs) - 1, wt.cpu().numpy().ravel())
    m.plan({"x": (ic * h * w, False)}, batch)
    got = torch.empty(batch, oc, h, w, device="cuda")
    n = torch.nn.functional.group_norm(torch.nn.functional.leaky_relu(x.double(), 0.01), groups, g.double(), b.double(), 1e-5)
    want = torch.nn.functional.conv2d(torch.nn.functional.silu(n) if silu else n, wt.double(), padding=k // 2)
    torch.cuda.synchronize()
    for _ in range(3):  # layer by layer, captured, replayed
        got.zero_()
        m.forward_device({"x": (x.data_ptr(), ic * h * w, False)}, batch, got.data_ptr(), got.numel())
        torch.cuda.synchronize()
        assert (got - want).norm() <= 3e-6 * want.norm()  # fp32 throughout: 2^-21 for SiLU, a few 2^-24 for the norm and the sums
    m.close()


def skip_block(c, oc, h):
    """conv -> conv -> Add with a 1 x 1 convolution of the input: operand planes that the first one laid out are read again."""
    conv = lambda name, i, o, ic, k: make_desc(name, "Conv2d", inputs=[i], output=o, in_channels=ic, out_channels=oc, input_height=h, input_width=h, kernel=k,  # noqa: E731
                                               stride=1, padding=k // 2, params_count=oc * ic * k * k)
    descs = [conv("c1", "x", "a", c, 3), conv("c2", "a", "b", oc, 3), conv("c3", "x", "d", c, 1), make_desc("add", "Add", inputs=["b", "d"], output="x")]
    r = np.random.default_rng(c + oc)
    return descs, [(r.standard_normal(d.params_count) / np.sqrt(d.in_channels * d.kernel**2)).astype(np.float32) if d.params_count else None for d in descs]


def plan_and_run(rt, descs, ws, x, batch, out):
    """The result, the arena's size and the memory that uploading and planning took."""
    before = rt.guard_stats()["current"]
    m = rt.GraphModel(descs)
    try:
        for i, w in enumerate(ws):
            if w is not None:
                m.upload_weights(i, w)
        uploaded = rt.guard_stats()["current"]
        m.plan({"x": (x.shape[1], False)}, batch)
        used, arena = rt.guard_stats()["current"] - before, rt.stats()["arena_peak_bytes"]
        got = m.forward({"x": (x, False)}, batch, out).copy()
    finally:
        m.close()
    return got, used, arena, uploaded - before


@pytest.mark.parametrize("missing", ["arena", "weights"])
def test_a_plan_goes_without_kept_planes_where_the_weight_planes_would_not_fit(rt, monkeypatch, missing):
    """A budget with room for the plan that keeps no planes, to the byte: the larger arena does not fit (16 images of 128^2), or does,
    and the weight planes behind it do not (two of 56^2, 512 channels)."""
    batch, c, oc, h = (16, 64, 64, 128) if missing == "arena" else (2, 512, 512, 56)
    descs, ws = skip_block(c, oc, h)
    x = np.random.default_rng(5).standard_normal((batch, c * h * h)).astype(np.float32)
    want, used, arena, _ = plan_and_run(rt, descs, ws, x, batch, oc * h * h)
    monkeypatch.setenv("MIMIR_B200_FUSE_GN_CONV", "0")
    plain, least, least_arena, uploaded = plan_and_run(rt, descs, ws, x, batch, oc * h * h)
    monkeypatch.delenv("MIMIR_B200_FUSE_GN_CONV")
    assert least < used, "the kept planes cost memory here, or this test shows nothing"
    # the weight planes are what does not fit: the larger arena alone does
    assert (uploaded + arena > least) == (missing == "arena")
    before, base = rt.guard_stats()["limit"], rt.guard_stats()["current"]
    rt.check(rt.lib().mimir_b200_guard_set_limit(base + least))
    try:
        got, now, got_arena, _ = plan_and_run(rt, descs, ws, x, batch, oc * h * h)
    finally:
        rt.check(rt.lib().mimir_b200_guard_set_limit(before))
    assert (now, got_arena) == (least, least_arena)
    assert np.array_equal(got, plain)
    assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)


def head_graph(ic, oc, h, w, k, groups, silu=True):
    """LeakyReLU -> GroupNorm (-> SiLU) -> convolution to a handful of channels."""
    d = [make_desc("r", "LeakyReLU", inputs=["x"], output="a"),
         make_desc("g", "GroupNorm", inputs=["a"], output="b", in_channels=ic, input_height=h, input_width=w, num_groups=groups, affine=1, use_bias=1, eps=1e-5,
                   params_count=2 * ic)]
    if silu:
        d.append(make_desc("s", "SiLU", inputs=["b"], output="c"))
    return d + [make_desc("c", "Conv2d", inputs=["c" if silu else "b"], output="x", in_channels=ic, out_channels=oc, input_height=h, input_width=w, kernel=k, stride=1,
                          padding=k // 2, params_count=oc * ic * k * k)]


def run_on_device(rt, descs, weights, x, out_shape, passes=1):
    import torch

    m = rt.GraphModel(descs)
    for i, wt in weights.items():
        m.upload_weights(i, wt.cpu().numpy().ravel())
    per = x[0].numel()
    m.plan({"x": (per, False)}, x.shape[0])
    got = torch.empty(out_shape, device="cuda")
    torch.cuda.synchronize()
    for _ in range(passes):  # layer by layer, captured, replayed
        got.zero_()
        m.forward_device({"x": (x.data_ptr(), per, False)}, x.shape[0], got.data_ptr(), got.numel())
        torch.cuda.synchronize()
    m.close()
    return got


@pytest.mark.parametrize("batch,ic,oc,h,w,k,groups,folded", [(2, 64, 3, 300, 300, 3, 32, False),     # few rows, not long enough: the GroupNorm stays apart
                                                            (9, 64, 3, 120, 124, 3, 32, False),     # a tensor of L2's size
                                                            (100, 64, 3, 128, 128, 3, 32, False),   # short rows
                                                            (12, 128, 5, 260, 256, 5, 32, False),   # a large kernel
                                                            (12, 128, 3, 260, 256, 3, 32, True), (3, 64, 8, 420, 424, 5, 16, True), (25, 64, 1, 260, 260, 5, 8, True), (1, 64, 3, 400, 400, 3, 2, True), (2, 96, 7, 368, 368, 3, 24, True)])
def test_direct_convolution_normalises_where_that_is_faster(rt, monkeypatch, batch, ic, oc, h, w, k, groups, folded):
    """Which form ran shows in the bits: a GroupNorm that stays apart gives those of a plan without the fold."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(ic + oc)
    randn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    x = randn(batch, ic, h, w) + 1.0
    g, b, wt = 1 + 0.2 * randn(ic), 0.5 * randn(ic), randn(oc, ic, k, k) / (ic * k * k) ** 0.5
    descs, weights = head_graph(ic, oc, h, w, k, groups), {1: torch.cat([g, b]), 3: wt}
    got = run_on_device(rt, descs, weights, x, (batch, oc, h, w), 3)
    monkeypatch.setenv("MIMIR_B200_FUSE_GN_CONV", "0")
    apart = run_on_device(rt, descs, weights, x, (batch, oc, h, w))
    assert torch.equal(got, apart) != folded
    for i in range(0, batch, 4):
        n = torch.nn.functional.group_norm(torch.nn.functional.leaky_relu(x[i:i + 4].double(), 0.01), groups, g.double(), b.double(), 1e-5)
        want = torch.nn.functional.conv2d(torch.nn.functional.silu(n), wt.double(), padding=k // 2)
        assert (got[i:i + 4] - want).norm() <= 3e-6 * want.norm()  # fp32 throughout: 2^-21 for SiLU, a few 2^-24 for the norm and the sums


def residual_graph(ic, oc, h, w, k1, k2, groups, silu=True, act=None):
    """conv -> GroupNorm (-> SiLU) added to another convolution of the input."""
    conv = lambda name, o, k: make_desc(name, "Conv2d", inputs=["x"], output=o, in_channels=ic, out_channels=oc, input_height=h, input_width=w, kernel=k,  # noqa: E731
                                        stride=1, padding=k // 2, params_count=oc * ic * k * k)
    d = [conv("c1", "a", k1), make_desc("g", "GroupNorm", inputs=["a"], output="b", in_channels=oc, input_height=h, input_width=w, num_groups=groups, affine=1, use_bias=1,
                                        eps=1e-5, params_count=2 * oc)]
    if silu:
        d.append(make_desc("s", "SiLU", inputs=["b"], output="c"))
    return d + [conv("c2", "d", k2), make_desc("add", "Add", inputs=["c" if silu else "b", "d"], output="x")]


def residual_case(ic, oc, k1, k2, batch, h, w, seed):
    import torch

    gen = torch.Generator(device="cuda").manual_seed(seed)
    randn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    half = lambda t: (t.view(torch.int32) & -65536).view(torch.float32)  # noqa: E731  (weights that are bfloat16 values, for every precision)
    w1, w2 = (half(randn(oc, ic, k, k) / (k * k * ic) ** 0.5) for k in (k1, k2))
    return randn(batch, ic, h, w) + 0.5, w1, 1 + 0.2 * randn(oc), 0.1 * randn(oc), w2


def residual_want(x, w1, g, b, w2, groups, silu=True):
    import torch

    f = torch.nn.functional
    n = f.group_norm(f.conv2d(x.double(), w1.double(), padding=w1.shape[2] // 2), groups, g.double(), b.double(), 1e-5)
    return (f.silu(n) if silu else n) + f.conv2d(x.double(), w2.double(), padding=w2.shape[2] // 2)


@pytest.mark.parametrize("precision", [abi.PREC_BF16X2, abi.PREC_BF16W])
@pytest.mark.parametrize("batch,ic,oc,h,w,k2,groups,silu", [(9, 64, 128, 97, 95, 3, 16, True), (5, 128, 160, 113, 112, 3, 5, True), (10, 32, 96, 96, 96, 5, 32, False)])
def test_a_normed_residual_leaves_a_3_x_3_convolution_its_weight_slots(rt, monkeypatch, precision, batch, ic, oc, h, w, k2, groups, silu):
    """The coefficients' 4 KB do not fit beside two activation tiles and three weight planes in blocks of 64 channels (two activation planes, 3 x 3,
    tiles of 256 pixels): blocks of 32 then, whose sums are in another order, so that the bits show which ran (the first convolution, 5 x 5, takes
    blocks of 32 in any case).  No planes are kept here: the form that normalises and reads planes of its own."""
    import torch

    monkeypatch.setenv("MIMIR_B200_CONV_PX", "256")
    x, w1, g, b, w2 = residual_case(ic, oc, 5, k2, batch, h, w, oc + k2)
    descs = residual_graph(ic, oc, h, w, 5, k2, groups, silu)
    weights = {0: w1, 1: torch.cat([g, b]), len(descs) - 2: w2}
    got = run_residual(rt, descs, weights, x, oc, precision, 3)
    want = residual_want(x, w1, g, b, w2, groups, silu)
    assert (got - want).norm() <= 3e-5 * want.norm()  # two contractions (4e-6 each), one of them normalised
    monkeypatch.setenv("MIMIR_B200_CONV_BK", "32")
    assert torch.equal(run_residual(rt, descs, weights, x, oc, precision), got)
    monkeypatch.setenv("MIMIR_B200_FUSE_GN_CONV", "0")
    assert not torch.equal(run_residual(rt, descs, weights, x, oc, precision), got), "the residual was not normalised by the convolution"


def run_residual(rt, descs, weights, x, oc, precision=abi.PREC_BF16X2, passes=1):
    import torch

    m = rt.GraphModel(descs, precision)
    for i, wt in weights.items():
        m.upload_weights(i, wt.cpu().numpy().ravel())
    per = x[0].numel()
    m.plan({"x": (per, False)}, x.shape[0])
    got = torch.empty(x.shape[0], oc, *x.shape[2:], device="cuda")
    torch.cuda.synchronize()
    for _ in range(passes):
        got.zero_()
        m.forward_device({"x": (x.data_ptr(), per, False)}, x.shape[0], got.data_ptr(), got.numel())
        torch.cuda.synchronize()
    m.close()
    return got


@pytest.mark.parametrize("batch,ic,oc,h,groups,folded", [(20, 32, 64, 88, 16, False), (40, 64, 32, 90, 8, False), (20, 32, 64, 87, 16, True), (14, 32, 96, 87, 24, True), (3, 64, 256, 111, 2, True),
                                                             (2, 32, 64, 300, 4, True), (1, 64, 32, 520, 2, True), (1, 32, 64, 376, 64, True)])
def test_a_residual_of_few_channels_is_normalised_apart(rt, monkeypatch, batch, ic, oc, h, groups, folded):
    """Fewer than 96 channels: the GroupNorm of its own, whose bits a plan without the fold has, unless it has few long rows or channels of an odd size."""
    import torch

    x, w1, g, b, w2 = residual_case(ic, oc, 3, 3, batch, h, h, oc)
    descs, weights = residual_graph(ic, oc, h, h, 3, 3, groups), {0: w1, 1: torch.cat([g, b]), 3: w2}
    got = run_residual(rt, descs, weights, x, oc)
    want = residual_want(x, w1, g, b, w2, groups)
    assert (got - want).norm() <= 3e-5 * want.norm()
    monkeypatch.setenv("MIMIR_B200_FUSE_GN_CONV", "0")
    assert torch.equal(run_residual(rt, descs, weights, x, oc), got) != folded


@pytest.mark.parametrize("batch,c,oc,h,w,k,kept", [(4, 128, 128, 96, 96, 3, False), (4, 64, 256, 64, 64, 3, False), (8, 64, 64, 32, 32, 3, False), (2, 64, 64, 96, 96, 7, False), (2, 64, 64, 128, 128, 7, True),
                                                  (3, 64, 100, 61, 67, 3, True), (40, 64, 160, 33, 33, 3, True), (8, 64, 64, 33, 33, 5, False), (5, 128, 72, 131, 103, 5, True), (1, 32, 64, 64, 200, 3, True)])
def test_planes_are_kept_where_their_ring_costs_less_than_laying_them_out(rt, monkeypatch, batch, c, oc, h, w, k, kept):
    """A second wave of tiles, twice as many outputs as inputs and more, a wide ring: planes of its own.  Whether planes are kept shows in the
    arena.  The kept ones: ragged lines and channels, rings of one and two pixels, a residual added."""
    conv = lambda name, i, o, ic, ks: make_desc(name, "Conv2d", inputs=[i], output=o, in_channels=ic, out_channels=oc, input_height=h, input_width=w,  # noqa: E731
                                                kernel=ks, stride=1, padding=ks // 2, params_count=oc * ic * ks * ks)
    descs = [conv("c1", "x", "a", c, k), conv("c3", "x", "d", c, 1), make_desc("add", "Add", inputs=["a", "d"], output="x")]
    r = np.random.default_rng(h + oc)
    ws = [(r.standard_normal(d.params_count) / np.sqrt(d.in_channels * d.kernel**2)).astype(np.float32) if d.params_count else None for d in descs]
    x = r.standard_normal((batch, c * h * w)).astype(np.float32)
    got, _, arena, _ = plan_and_run(rt, descs, ws, x, batch, oc * h * w)
    monkeypatch.setenv("MIMIR_B200_FUSE_GN_CONV", "0")
    apart, _, least, _ = plan_and_run(rt, descs, ws, x, batch, oc * h * w)
    assert (arena > least) == kept
    assert np.array_equal(got, apart)  # the same sums in the same order


def silu_arguments(n):
    """fp32 values over the range where SiLU is no subnormal, and their SiLU in 64 bits."""
    import torch

    beta = torch.linspace(-87.0, 70.0, n, device="cuda") + torch.rand(n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
    return beta, torch.nn.functional.silu(beta.double())


# two special-function instructions of 2^-22 each; rounding of the product and, where a sum follows, of the sum
SILU_BOUND = 2.0**-21 + 2.0**-23


def test_silu_of_a_normed_residual_over_the_whole_range(rt):
    """gamma = 0: the residual is SiLU(beta) of each channel, and the convolution that it is added to adds zeros."""
    import torch

    batch, ic, oc, h = 5, 32, 160, 120
    x, w1, _, _, w2 = residual_case(ic, oc, 3, 3, batch, h, h, 1)
    beta, want = silu_arguments(oc)
    got = run_residual(rt, residual_graph(ic, oc, h, h, 3, 3, 32), {0: w1, 1: torch.cat([torch.zeros_like(beta), beta]), 3: torch.zeros_like(w2)}, x, oc)
    want = want.view(1, oc, 1, 1)
    assert bool(((got - want).abs() <= SILU_BOUND * want.abs()).all())


@pytest.mark.parametrize("oc,groups", [(8, 4), (3, 2)])
def test_silu_of_a_direct_convolution_over_the_whole_range(rt, oc, groups):
    """gamma = 0, and an output channel takes one input channel with weight one."""
    import torch

    batch, ic, h, w = 1, 64, 1024, 512  # 128 MB in a few rows: the convolution normalises
    beta, want = silu_arguments(ic)
    x = torch.randn(batch, ic, h, w, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    for first in range(0, ic, oc):
        pick = [min(first + o, ic - 1) for o in range(oc)]
        wt = torch.zeros(oc, ic, 1, 1, device="cuda")
        wt[range(oc), pick] = 1.0
        got = run_on_device(rt, head_graph(ic, oc, h, w, 1, groups), {1: torch.cat([torch.zeros_like(beta), beta]), 3: wt}, x, (batch, oc, h, w))
        exact = want[pick].view(1, oc, 1, 1)
        assert bool(((got - exact).abs() <= SILU_BOUND * exact.abs()).all())


@pytest.mark.parametrize("form", ["apart", "residual"])
def test_moments_of_infinities_overflows_and_far_means(rt, form):
    """conv + r -> GroupNorm -> SiLU on more than 96 MB, of which r gives one group of a sample an infinity or a NaN (the group becomes NaN, and no
    other changes a bit), values whose squares overflow (beta is left), or a mean of 700 deviations."""
    import torch

    batch, ic, oc, h, groups = 42, 32, 96, 80, 24
    gen = torch.Generator(device="cuda").manual_seed(9)
    randn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    x, w1, w2 = randn(batch, ic, h, h), randn(oc, ic, 3, 3) / (9 * ic) ** 0.5, randn(oc, ic, 3, 3) / (9 * ic) ** 0.5
    g, b = 1 + 0.2 * randn(oc), 0.5 * randn(oc)
    conv = lambda name, i, o: make_desc(name, "Conv2d", inputs=[i], output=o, in_channels=ic, out_channels=oc, input_height=h, input_width=h, kernel=3, stride=1,  # noqa: E731
                                        padding=1, params_count=w1.numel())
    sums = [conv("c1", "x", "a"), make_desc("add", "Add", inputs=["a", "r"], output="s")]
    norm = [make_desc("g", "GroupNorm", inputs=["s"], output="n", in_channels=oc, input_height=h, input_width=h, num_groups=groups, affine=1, use_bias=1, eps=1e-5,
                      params_count=2 * oc), make_desc("silu", "SiLU", inputs=["n"], output="x" if form == "apart" else "t")]
    rest = [] if form == "apart" else [conv("c2", "x", "d"), make_desc("add2", "Add", inputs=["t", "d"], output="x")]

    def run(descs, r, launches=None):
        m = rt.GraphModel(descs)
        m.upload_weights(0, w1.cpu().numpy().ravel())
        if len(descs) > 2:
            m.upload_weights(2, torch.cat([g, b]).cpu().numpy())
        if len(descs) > 4:
            m.upload_weights(4, w2.cpu().numpy().ravel())
        m.plan({"x": (ic * h * h, False), "r": (oc * h * h, False)}, batch)
        got = torch.empty(batch, oc, h, h, device="cuda")
        torch.cuda.synchronize()
        before = rt.stats()["kernels_launched"]
        m.forward_device({"x": (x.data_ptr(), ic * h * h, False), "r": (r.data_ptr(), oc * h * h, False)}, batch, got.data_ptr(), got.numel())
        torch.cuda.synchronize()
        if launches is not None:  # planes, convolution, moments merged, then the GroupNorm or (coefficients, planes, convolution)
            assert rt.stats()["kernels_launched"] - before == launches
        m.close()
        return got

    last = [make_desc("add", "Add", inputs=["a", "r"], output="x")]
    run_all = lambda r: run(sums + norm + rest, r, 4 if form == "apart" else 6)  # noqa: E731
    r0 = randn(batch, oc, h, h)
    clean = run_all(r0)
    for value in (float("inf"), float("-inf"), float("nan")):
        r = r0.clone()
        r[1, 5, h - 1, 17] = value
        got = run_all(r)
        assert bool(got[1, 4:8].isnan().all())
        got[1, 4:8] = clean[1, 4:8]
        assert torch.equal(got, clean)
    r = r0.clone()
    r[2, 8:12] *= 1e22
    r[3, 12:16] += 700.0
    got, plain = run_all(r), run([sums[0]] + last, r)
    other = torch.nn.functional.conv2d(x.double(), w2.double(), padding=1) if rest else torch.zeros_like(got)
    want = torch.nn.functional.silu(b.double())[8:12].view(4, 1, 1) + other[2, 8:12]
    assert bool(((got[2, 8:12] - want).abs() <= 2e-6 * (1 + want.abs()) + (4e-5 if rest else 0.0)).all())  # (the second convolution's own error: 4e-6 of its norm)
    n = torch.nn.functional.group_norm(plain[3:4].double(), groups, g.double(), b.double(), 1e-5)
    want = torch.nn.functional.silu(n)[0, 12:16] + other[3, 12:16]
    # the mean, its product with 1 / std and the sum are rounded at 700 deviations each
    assert bool(((got[3, 12:16] - want).abs() <= 4 * 700 * 2.0**-24 * 1.1 * g[12:16].abs().max() + (4e-5 if rest else 0.0)).all())
    got[2, 8:12], got[3, 12:16] = clean[2, 8:12], clean[3, 12:16]
    assert torch.equal(got, clean)


@pytest.mark.parametrize("batch,ic,oc,h,k,groups,emits", [(16, 32, 128, 96, 3, 32, False), (16, 64, 64, 168, 1, 16, False), (16, 64, 64, 112, 3, 16, False), (22, 64, 96, 112, 1, 24, True), (35, 32, 64, 108, 3, 8, True),
                                                            (16, 64, 128, 96, 3, 32, True), (14, 128, 128, 93, 3, 32, False)])
def test_moments_are_taken_where_a_sweep_costs_more(rt, batch, ic, oc, h, k, groups, emits):
    """A convolution and a GroupNorm of its own, by launches: planes, convolution, GroupNorm, and one that merges the moments."""
    import torch

    x, w1, g, b, _ = residual_case(ic, oc, k, 1, batch, h, h, oc + h)
    descs = residual_graph(ic, oc, h, h, k, 1, groups)[:3]
    descs[2] = make_desc("s", "SiLU", inputs=["b"], output="x")
    m = rt.GraphModel(descs)
    m.upload_weights(0, w1.cpu().numpy().ravel())
    m.upload_weights(1, torch.cat([g, b]).cpu().numpy())
    m.plan({"x": (ic * h * h, False)}, batch)
    got = torch.empty(batch, oc, h, h, device="cuda")
    torch.cuda.synchronize()
    before = rt.stats()["kernels_launched"]
    m.forward_device({"x": (x.data_ptr(), ic * h * h, False)}, batch, got.data_ptr(), got.numel())
    torch.cuda.synchronize()
    assert rt.stats()["kernels_launched"] - before == (4 if emits else 3)
    m.close()
    f = torch.nn.functional
    for i in range(0, batch, 8):
        want = f.silu(f.group_norm(f.conv2d(x[i:i + 8].double(), w1.double(), padding=k // 2), groups, g.double(), b.double(), 1e-5))
        assert (got[i:i + 8] - want).norm() <= 3e-5 * want.norm()


@pytest.mark.parametrize("precision", [abi.PREC_BF16X2, abi.PREC_BF16W, abi.PREC_BF16])
@pytest.mark.parametrize("form,launches", [("apart", 4), ("kept planes", 5), ("own planes", 6)])
@pytest.mark.parametrize("silu", [True, False])
def test_moments_and_normed_residuals_of_ragged_images(rt, precision, form, launches, silu):
    """63 x 76 pixels, cut by every tile, and a mean of half a deviation, by launches: planes, convolution, moments merged, then the GroupNorm, or
    coefficients and the convolution that normalises its residual, on the planes of the first one or on its own."""
    import torch

    batch, ic, oc, h, w, groups = 43, 64, 128, 63, 76, 16
    k2 = 3 if form == "own planes" else 1
    x, w1, g, b, w2 = residual_case(ic, oc, 3, k2, batch, h, w, 63)
    descs = residual_graph(ic, oc, h, w, 3, k2, groups, silu)
    weights = {0: w1, 1: torch.cat([g, b]), len(descs) - 2: w2}
    if form == "apart":
        descs = descs[:2 + silu]
        descs[-1] = make_desc("s", "SiLU", inputs=["b"], output="x") if silu else make_desc(
            "g", "GroupNorm", inputs=["a"], output="x", in_channels=oc, input_height=h, input_width=w, num_groups=groups, affine=1, use_bias=1, eps=1e-5, params_count=2 * oc)
        weights = {0: w1, 1: torch.cat([g, b])}
    m = rt.GraphModel(descs, precision)
    for i, wt in weights.items():
        m.upload_weights(i, wt.cpu().numpy().ravel())
    m.plan({"x": (ic * h * w, False)}, batch)
    got = torch.empty(batch, oc, h, w, device="cuda")
    torch.cuda.synchronize()
    before = rt.stats()["kernels_launched"]
    m.forward_device({"x": (x.data_ptr(), ic * h * w, False)}, batch, got.data_ptr(), got.numel())
    torch.cuda.synchronize()
    assert rt.stats()["kernels_launched"] - before == launches
    m.close()
    for i in range(0, batch, 12):
        want = residual_want(x[i:i + 12], w1, g, b, w2, groups, silu)
        if form == "apart":
            want = want - torch.nn.functional.conv2d(x[i:i + 12].double(), w2.double(), padding=k2 // 2)
        # two contractions of 4e-6, or of one plane of 11 bits per operand (the weights are bfloat16 values)
        assert (got[i:i + 12] - want).norm() <= (2.0**-9 if precision == abi.PREC_BF16 else 3e-5) * want.norm()


@pytest.mark.parametrize("batch,ic,oc,h", [(6, 64, 128, 112), (9, 64, 256, 64)])
def test_planes_are_kept_for_a_convolution_that_normalises_its_residual(rt, batch, ic, oc, h):
    """A fifth wave of half tiles to four, four times as many outputs as inputs: by launches, planes, convolution, moments merged, coefficients,
    convolution."""
    import torch

    x, w1, g, b, w2 = residual_case(ic, oc, 3, 1, batch, h, h, oc)
    descs = residual_graph(ic, oc, h, h, 3, 1, 16)
    m = rt.GraphModel(descs)
    for i, wt in ((0, w1), (1, torch.cat([g, b])), (3, w2)):
        m.upload_weights(i, wt.cpu().numpy().ravel())
    m.plan({"x": (ic * h * h, False)}, batch)
    got = torch.empty(batch, oc, h, h, device="cuda")
    torch.cuda.synchronize()
    before = rt.stats()["kernels_launched"]
    m.forward_device({"x": (x.data_ptr(), ic * h * h, False)}, batch, got.data_ptr(), got.numel())
    torch.cuda.synchronize()
    assert rt.stats()["kernels_launched"] - before == 5
    m.close()
    want = residual_want(x, w1, g, b, w2, 16)
    assert (got - want).norm() <= 3e-5 * want.norm()
