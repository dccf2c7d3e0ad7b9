"""Workloads of the forward path, as a program that uses the framework runs them.

Each case names a family and its sizes:

  encoder   the registry's transformer encoder (whole-vector LayerNorm, MLP over the flattened sequence), fp32
  linear    the stand-alone Linear + bias + GELU stack, fp32
  decoder   the GPT-style causal decoder over a whole prompt (prefill), bf16-exact or fp32 weights
  step      one token of that decoder (token-wise LayerNorm) against the key / value cache
  conv      the vision stack: stem 7 x 7 s2, then Conv 3 x 3 -> GroupNorm -> SiLU -> residual blocks, fp32
  unet      the UNet mid + up path: ResBlocks, one wide attention head, nearest upsampling, bf16-exact weights
  norm      one normalisation or softmax on data that already is on the GPU (the device-pointer calls)
  hook      one Linear on host arrays, weights included (the call that replaces the per-layer accelerator hook)

Graph cases run on device pointers, or on host arrays where `host` is set.  Weights and inputs are seeded synthetic data with
the distributions of the benchmark configurations (mimir_framework_b200/configs.py).
"""
from __future__ import annotations

import numpy as np
import torch

from mimir_framework_b200 import abi, configs
from mimir_framework_b200 import runtime as rt

PRECISION = {"x2": abi.PREC_BF16X2, "w": abi.PREC_BF16W, "one": abi.PREC_BF16}


def listed():
    cfg = configs.TRANSFORMER_CFG
    enc = dict(family="encoder", seq=cfg["seq_len"], heads=cfg["num_heads"], head_dim=cfg["d_model"] // cfg["num_heads"], mlp=cfg["mlp_hidden"],
               layers=cfg["num_layers"], out=cfg["output_dim"], vocab=cfg["vocab_size"])
    d = configs.DECODER_CFG
    dec = dict(layers=d["layers"], heads=d["heads"], head_dim=d["d_model"] // d["heads"], ffn=d["ffn"], vocab=d["vocab"])
    return [
        # one request at a time, host arrays in and out: what a script that calls the model per sample waits for
        dict(enc, name="encoder_b1_host", batch=1, host=True),
        # configuration 1 as it is stated: eight samples
        dict(enc, name="encoder_b8", batch=8, host=False),
        # a server that gathers requests: more rows than a handful, far fewer than a GEMM tile's worth per SM
        dict(enc, name="encoder_b40", batch=40, host=False),
        # configuration 2 at its smallest row count
        dict(family="linear", name="linear_4096", rows=4096, width=4096, layers=3),
        # the same stack on a ragged batch and a width that is no multiple of a tile
        dict(family="linear", name="linear_333x1000", rows=333, width=1000, layers=3),
        # configuration 3 as it is stated: prefill of 32 prompts
        dict(dec, family="decoder", name="decoder_b32", batch=32, seq=1024, precision="w"),
        # one prompt of a length that is no multiple of a tile
        dict(dec, family="decoder", name="decoder_b1_s1000", batch=1, seq=1000, precision="w"),
        # token-by-token generation behind a prefix of about a thousand tokens
        dict(dec, family="step", name="step_b16", batch=16, pos=991, precision="w"),
        # configuration 4 as it is stated
        dict(family="conv", name="conv_b64", batch=64, image=224, width=64),
        # configuration 5 as it is stated
        dict(family="unet", name="unet_b16", batch=16, latent=64, base=512),
        # token-wise LayerNorm of a batch of sequences (a layer that a host program runs on its own device buffers)
        dict(family="norm", name="layernorm_32768x768", op="layernorm", rows=32768, n=768),
        # a feed-forward layer called on host arrays
        dict(family="hook", name="hook_512x768x3072", rows=512, k=768, n=3072),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    family = rng.choice(["encoder", "linear", "decoder", "step", "conv", "unet", "norm", "hook"])
    if family == "encoder":
        return dict(family=family, batch=_log(rng, 1, 64), host=rng.random() < 0.5, seq=rng.randint(16, 160), heads=rng.choice([2, 3, 4, 6]),
                    head_dim=rng.choice([32, 48, 64]), mlp=_log(rng, 200, 1500), layers=rng.randint(1, 3), out=rng.randint(64, 512), vocab=8192)
    if family == "linear":
        return dict(family=family, rows=_log(rng, 8, 32768), width=_log(rng, 250, 4096), layers=rng.randint(1, 3))
    if family == "decoder":
        return dict(family=family, batch=_log(rng, 1, 16), seq=_log(rng, 32, 1024), layers=rng.randint(2, 12), heads=rng.randint(4, 12), head_dim=64,
                    ffn=256 * rng.randint(4, 12), vocab=_log(rng, 1000, 32000), precision=rng.choice(["w", "w", "x2", "one"]))
    if family == "step":
        return dict(family=family, batch=_log(rng, 1, 24), pos=_log(rng, 16, 1023), layers=rng.randint(2, 12), heads=rng.randint(4, 12), head_dim=64,
                    ffn=256 * rng.randint(4, 12), vocab=_log(rng, 1000, 32000), precision=rng.choice(["w", "x2"]))
    if family == "conv":
        return dict(family=family, batch=_log(rng, 1, 48), image=rng.randint(64, 224), width=rng.choice([32, 64]))
    if family == "unet":
        return dict(family=family, batch=rng.randint(1, 16), latent=4 * rng.randint(6, 16), base=rng.choice([256, 512]))
    if family == "hook":
        return dict(family=family, rows=_log(rng, 1, 2048), k=_log(rng, 100, 4096), n=_log(rng, 100, 4096))
    op = rng.choice(["layernorm", "rmsnorm", "groupnorm", "softmax"])
    if op == "layernorm":
        n = _log(rng, 64, 4096)
        return dict(family=family, op=op, rows=max(1, _log(rng, 1000, 100_000_000) // n), n=n)
    if op == "rmsnorm":
        n = _log(rng, 2000, 800_000)
        return dict(family=family, op=op, rows=max(1, _log(rng, 10_000, 100_000_000) // n), n=n)
    if op == "softmax":
        n = _log(rng, 100, 50_000)
        return dict(family=family, op=op, rows=max(1, _log(rng, 10_000, 100_000_000) // n), n=n)
    return dict(family=family, op=op, rows=_log(rng, 1, 48), channels=32 * rng.randint(2, 16), side=rng.randint(8, 112))


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _host(t):
    return t.cpu().numpy()


def _weights(descs, gen, bf16):
    """N(0, 0.02) with zero Linear biases and identity norms, like configs.seeded_weights (made on the GPU: these are large)."""
    out = []
    for d in descs:
        n, t = int(d.params_count), d.type.decode()
        if n == 0:
            out.append(None)
        elif t in ("LayerNorm", "GroupNorm", "RMSNorm"):
            w = np.ones(n, np.float32)
            if t != "RMSNorm" and d.use_bias:
                w[n // 2:] = 0.0
            out.append(w)
        else:
            w = torch.randn(n, device="cuda", generator=gen) * 0.02
            if t == "Linear" and d.use_bias:
                w[n - d.out_features:] = 0.0
            out.append(_host(w.bfloat16().float() if bf16 else w))
    return out


def _model(descs, weights, precision):
    m = rt.GraphModel(descs, precision)
    for i, w in enumerate(weights):
        m.upload_weights(i, w)
    return m


def _device_graph(descs, weights, precision, inputs, batch, out_per_sample):
    """inputs: name -> (device tensor, broadcast)."""
    m = _model(descs, weights, precision)
    per = {k: t.numel() if bc else t.numel() // batch for k, (t, bc) in inputs.items()}
    m.plan({k: (per[k], bc) for k, (_, bc) in inputs.items()}, batch)
    return dict(how="device", model=m, batch=batch, keep=inputs, spec={k: (t.data_ptr(), per[k], bc) for k, (t, bc) in inputs.items()},
                out=torch.empty(batch, out_per_sample, device="cuda"))


def _encoder(c):
    return dict(seq_len=c["seq"], d_model=c["heads"] * c["head_dim"], vocab_size=c["vocab"], num_layers=c["layers"], num_heads=c["heads"],
                mlp_hidden=c["mlp"], output_dim=c["out"])


def _decoder(c, seq, norm):
    return dict(layers=c["layers"], d_model=c["heads"] * c["head_dim"], heads=c["heads"], ffn=c["ffn"], vocab=c["vocab"], seq=seq, norm=norm)


def _conv_channels(c):
    return (c["width"], 2 * c["width"], 2 * c["width"], 4 * c["width"], 4 * c["width"])


def prepare(case, seed):
    rt.init(0)
    gen = _generator(seed)
    c, family = case, case["family"]

    def randn(*shape):
        return torch.randn(*shape, device="cuda", generator=gen)

    if family == "encoder":
        cfg = _encoder(c)
        descs = configs.transformer_encoder(**cfg)
        ids = torch.randint(0, c["vocab"], (c["batch"], c["seq"]), device="cuda", generator=gen).float()
        inputs = {"x": (ids, False), "mag": (randn(cfg["d_model"]) * 0.02, True), "mod": (randn(cfg["d_model"]) * 0.02, True)}
        weights = _weights(descs, gen, bf16=False)
        if not c["host"]:
            return _device_graph(descs, weights, abi.PREC_BF16X2, inputs, c["batch"], c["out"])
        m = _model(descs, weights, abi.PREC_BF16X2)
        m.plan({"x": (c["seq"], False), "mag": (cfg["d_model"], True), "mod": (cfg["d_model"], True)}, c["batch"])
        return dict(how="host", model=m, batch=c["batch"], inputs={k: (_host(t), bc) for k, (t, bc) in inputs.items()}, out_n=c["out"])
    if family == "linear":
        k = c["width"]
        descs = configs.linear_gelu_stack(c["rows"], k, c["layers"])
        bound, weights = k ** -0.5, []
        for _ in range(c["layers"]):
            w = torch.rand(k * k + k, device="cuda", generator=gen) * 2 - 1
            w[: k * k] *= bound
            w[k * k:] *= 0.1
            weights += [_host(w), None]
        return _device_graph(descs, weights, abi.PREC_BF16X2, {"x": (randn(c["rows"], k), False)}, 1, c["rows"] * k)
    if family == "decoder":
        descs = configs.gpt_decoder(**_decoder(c, c["seq"], "rms"))
        ids = torch.randint(0, c["vocab"], (c["batch"], c["seq"]), device="cuda", generator=gen).float()
        weights = _weights(descs, gen, bf16=c["precision"] != "x2")
        return _device_graph(descs, weights, PRECISION[c["precision"]], {"x": (ids, False)}, c["batch"], c["seq"] * c["vocab"])
    if family == "step":
        # a prefix of `pos` tokens goes through the ordinary forward, which fills the cache
        descs = configs.gpt_decoder(**_decoder(c, c["pos"], "layer"))
        ids = torch.randint(0, c["vocab"], (c["batch"], c["pos"] + 1), device="cuda", generator=gen).float()
        m = _model(descs, _weights(descs, gen, bf16=c["precision"] != "x2"), PRECISION[c["precision"]])
        m.plan({"x": (c["pos"], False)}, c["batch"])
        m.decode_begin({"x": (1, False)}, c["batch"], max(1024, c["pos"] + 1))
        prefix = ids[:, : c["pos"]].contiguous()
        logits = torch.empty(c["batch"] * c["pos"] * c["vocab"], device="cuda")
        m.forward_device({"x": (prefix.data_ptr(), c["pos"], False)}, c["batch"], logits.data_ptr(), logits.numel())
        torch.cuda.synchronize()
        return dict(how="step", model=m, batch=c["batch"], pos=c["pos"], inputs={"x": (_host(ids[:, c["pos"]].contiguous()), False)}, out_n=c["vocab"])
    if family == "conv":
        descs = configs.conv_stack(c["image"], _conv_channels(c))
        weights = []
        for d in descs:
            n, t = int(d.params_count), d.type.decode()
            if t == "Conv2d":
                weights.append(_host(randn(n) * (2.0 / (d.in_channels * d.kernel * d.kernel)) ** 0.5))
            elif t == "GroupNorm":
                weights.append(np.concatenate([np.ones(n // 2, np.float32), np.zeros(n - n // 2, np.float32)]))
            else:
                weights.append(None)
        x = torch.rand(c["batch"], 3 * c["image"] * c["image"], device="cuda", generator=gen)
        hw = (c["image"] - 1) // 2 + 1
        return _device_graph(descs, weights, abi.PREC_BF16X2, {"x": (x, False)}, c["batch"], 4 * c["width"] * hw * hw)
    if family == "unet":
        descs = configs.unet_mid_up(c["latent"], c["base"])
        weights = _weights(descs, gen, bf16=True)
        x = randn(c["batch"], 4 * c["latent"] * c["latent"])
        return _device_graph(descs, weights, abi.PREC_BF16W, {"x": (x, False)}, c["batch"], 3 * (4 * c["latent"]) ** 2)
    if family == "hook":
        k, n = c["k"], c["n"]
        return dict(how="hook", x=_host(randn(c["rows"] * k)), w=_host(randn(n * k) * 0.02), b=_host(randn(n) * 0.02), rows=c["rows"], k=k, n=n)
    if c["op"] == "groupnorm":
        x, params = randn(c["rows"], c["channels"] * c["side"] * c["side"]), c["channels"]
    else:
        x, params = randn(c["rows"], c["n"]), c["n"]
    return dict(how="norm", case=c, x=x, y=torch.empty_like(x), gamma=1 + 0.1 * randn(params), beta=0.1 * randn(params))


def run(s):
    how = s["how"]
    if how == "device":
        s["model"].forward_device(s["spec"], s["batch"], s["out"].data_ptr(), s["out"].numel())
        return s["out"]
    if how == "host":
        return s["model"].forward(s["inputs"], s["batch"], s["out_n"])
    if how == "step":
        return s["model"].decode_step(s["inputs"], s["batch"], s["pos"], s["out_n"])
    if how == "hook":
        return rt.linear_forward(s["x"], s["w"], s["b"], s["rows"], s["k"], s["n"])
    c, lib = s["case"], rt.lib()
    x, y, g, b = s["x"].data_ptr(), s["y"].data_ptr(), s["gamma"].data_ptr(), s["beta"].data_ptr()
    if c["op"] == "layernorm":
        rt.check(lib.mimir_b200_dev_layernorm(x, g, b, y, c["rows"], c["n"], 1e-5, None))
    elif c["op"] == "rmsnorm":
        rt.check(lib.mimir_b200_dev_rmsnorm(x, g, c["n"], y, c["rows"], c["n"], 1e-5, None))
    elif c["op"] == "softmax":
        rt.check(lib.mimir_b200_dev_softmax(x, y, c["rows"], c["n"], 0, None))
    else:
        rt.check(lib.mimir_b200_dev_groupnorm(x, g, b, y, c["rows"], c["channels"], c["side"], c["side"], 32, 1e-5, abi.ELT_SILU, None))
    return s["y"]


def _params(descs):
    """Weights that a pass reads whole: everything but the embedding table."""
    return sum(int(d.params_count) for d in descs if d.type.decode() != "Embedding")


def work(case):
    c, family = case, case["family"]
    if family == "encoder":
        B, S, E, H, L = c["batch"], c["seq"], c["heads"] * c["head_dim"], c["mlp"], c["layers"]
        per_layer = 8 * S * E * E + 4 * S * S * E + 4 * S * E * H
        values = _params(configs.transformer_encoder(**_encoder(c))) + B * (S + S * E + c["out"])
        return {"bytes": 4 * values, "flops": B * (L * per_layer + 2 * S * E * c["out"])}
    if family == "linear":
        k = c["width"]
        return {"bytes": 4 * (c["layers"] * (k * k + k) + 2 * c["rows"] * k), "flops": configs.linear_gelu_stack_flops(c["rows"], k, c["layers"])}
    if family == "decoder":
        cfg = _decoder(c, c["seq"], "rms")
        rows = c["batch"] * c["seq"]
        values = _params(configs.gpt_decoder(**cfg)) + rows * (1 + cfg["d_model"] + c["vocab"])
        cfg.pop("norm")
        return {"bytes": 4 * values, "flops": c["batch"] * configs.gpt_decoder_flops(**cfg)}
    if family == "step":
        E, L, B = c["heads"] * c["head_dim"], c["layers"], c["batch"]
        weights = L * (4 * E * E + 2 * E * c["ffn"] + c["ffn"] + 5 * E) + 2 * E + E * c["vocab"]
        values = weights + B * (1 + E + c["vocab"]) + 2 * L * B * (c["pos"] + 1) * E
        return {"bytes": 4 * values, "flops": 2 * B * (L * (4 * E * E + 2 * E * c["ffn"] + 2 * (c["pos"] + 1) * E) + E * c["vocab"])}
    if family in ("conv", "unet"):
        if family == "conv":
            descs, flops = configs.conv_stack(c["image"], _conv_channels(c)), 0
            hw = (c["image"] - 1) // 2 + 1
            per = 3 * c["image"] ** 2 + 4 * c["width"] * hw * hw
        else:
            descs = configs.unet_mid_up(c["latent"], c["base"])
            tokens, E = (c["latent"] // 4) ** 2, c["base"]
            per, flops = (4 + 3 * 16) * c["latent"] ** 2, 8 * tokens * E * E + 4 * tokens * tokens * E
        return {"bytes": 4 * (_params(descs) + c["batch"] * per), "flops": c["batch"] * (flops + configs.conv_flops(descs))}
    if family == "hook":
        return {"bytes": 4 * (c["rows"] * (c["k"] + c["n"]) + c["n"] * (c["k"] + 1)), "flops": 2 * c["rows"] * c["k"] * c["n"]}
    n, params = (c["channels"] * c["side"] ** 2, c["channels"]) if c["op"] == "groupnorm" else (c["n"], c["n"])
    return {"bytes": 4 * (2 * c["rows"] * n + (0 if c["op"] == "softmax" else 2 if c["op"] != "rmsnorm" else 1) * params), "flops": 10 * c["rows"] * n}


def tolerance(case):
    """fp32 results throughout.  Contractions carry fp32 operands as 16-bit plane pairs with fp32 accumulation in the tensor
    core: a few 1e-6 per layer, which add up over the depth of a graph.  `one` rounds each operand to one 16-bit plane."""
    family = case["family"]
    if family == "decoder" and case["precision"] == "one":
        return {"rel": 5e-3}
    if family in ("decoder", "step", "unet"):
        return {"rel": 1e-4}
    if family in ("encoder", "linear", "conv"):
        return {"rel": 5e-5}
    if family == "hook":
        return {"rel": 2e-5}
    return {"rel": 1e-5}
