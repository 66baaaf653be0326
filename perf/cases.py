"""Performance cases: the calls that a program built on this package makes, over the sizes that it makes them at.

Training is one step of the language model handle (forward, checkpointed backward, every parameter gradient), as one
CUDA graph replay for the larger models and through the host-buffer call for the small one, plus the optimizer step on
the flat parameter buffer.  A program that builds its own model calls single blocks (forward and backward) or residual
stacks; a server calls the block forward on prompts of any length (prefill) and the one-token step (decode); the scan is
also an operator of its own.  Sizes are those of the benchmark's and the tests' configurations, and generic ones between.

`listed()` are fixed points, `draw(rng)` another point of the same ranges.  `prepare` builds what such a program has in
hand before the call (weights on the GPU, inputs, a model handle or a captured step), `run` makes the call.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "photon-mamba2-llm_b200"))


# -------------------------------------------------------------------------------------------------
# the cases
# -------------------------------------------------------------------------------------------------

def listed():
    return [
        # the headline benchmark: ~100M parameters, fp32, one training step as a graph replay
        {"name": "train_flat_fp32_b4_t512", "kind": "lm", "dtype": "fp32", "layers": 24, "level1": 0, "heads": 24, "d_head": 64,
         "d_state": 64, "vocab": 50257, "batch": 4, "seq": 512, "chunk": 256, "host": False},
        # the two-level model at token rate and quarter rate, bf16 storage
        {"name": "train_two_level_bf16_b8_t1024", "kind": "lm", "dtype": "bf16", "layers": 12, "level1": 12, "heads": 24, "d_head": 64,
         "d_state": 64, "vocab": 50257, "batch": 8, "seq": 1024, "chunk": 256, "host": False},
        # long-context training, bf16 storage: the largest step
        {"name": "train_flat_bf16_b8_t2048", "kind": "lm", "dtype": "bf16", "layers": 24, "level1": 0, "heads": 24, "d_head": 64,
         "d_state": 64, "vocab": 50257, "batch": 8, "seq": 2048, "chunk": 256, "host": False},
        # a small model stepped from host token buffers (copies in, loss out): launch and host time dominate
        {"name": "train_small_host_fp32_b2_t128", "kind": "lm", "dtype": "fp32", "layers": 2, "level1": 0, "heads": 8, "d_head": 32,
         "d_state": 16, "vocab": 1000, "batch": 2, "seq": 128, "chunk": 64, "host": True},
        # one block, forward and backward, at the single-block configuration (the smallest dimensions in use)
        {"name": "block_small_fp32_b2_t128", "kind": "block", "dtype": "fp32", "heads": 8, "d_head": 32, "d_state": 16,
         "batch": 2, "seq": 128, "chunk": 64},
        # one block, forward and backward, bf16 storage, on sequences whose length no chunk divides
        {"name": "block_bf16_b2_t1000", "kind": "block", "dtype": "bf16", "heads": 24, "d_head": 64, "d_state": 64,
         "batch": 2, "seq": 1000, "chunk": 256},
        # a residual stack with block-input checkpoints, called eagerly, three half-chunks long
        {"name": "stack_fp32_l4_b2_t384", "kind": "stack", "dtype": "fp32", "layers": 4, "heads": 24, "d_head": 64, "d_state": 64,
         "batch": 2, "seq": 384, "chunk": 256},
        # prefill of one prompt of odd length through one block
        {"name": "prefill_fp32_b1_t1337", "kind": "prefill", "dtype": "fp32", "heads": 24, "d_head": 64, "d_state": 64,
         "batch": 1, "seq": 1337, "chunk": 256},
        # decode of a single stream: the smallest call
        {"name": "decode_fp32_b1_h24", "kind": "decode", "heads": 24, "d_head": 64, "d_state": 64, "expand": 2, "batch": 1},
        # decode of a large batch at the decode benchmark's dimensions (d_model equals the inner width there)
        {"name": "decode_fp32_b256_h32", "kind": "decode", "heads": 32, "d_head": 64, "d_state": 128, "expand": 1, "batch": 256},
        # the scan operator, forward and backward, bf16 inputs and fp32 state: the scan benchmark
        {"name": "scan_bf16_b16_t8192", "kind": "scan", "dtype": "bf16", "batch": 16, "seq": 8192, "heads": 32, "groups": 1,
         "d_head": 64, "d_state": 128, "chunk": 256},
        # gradient norm, clipping and AdamW over the flat buffer of the ~100M-parameter model
        {"name": "adamw_clip_100m", "kind": "adamw", "params": 126_000_000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lm", "lm", "block", "block", "stack", "prefill", "prefill", "decode", "decode", "scan", "scan", "adamw"])
    if kind == "lm":
        # training sequences are cut to a fixed length: multiples of 64 tokens, not all of them multiples of the chunk
        dtype = rng.choice(["fp32", "bf16"])
        heads = rng.choice([8, 16, 24])
        batch = rng.randint(1, 8)
        seq = 64 * _log_int(rng, 4, 16) if rng.random() < 0.5 else 256 * _log_int(rng, 2, 8)
        level1 = rng.randint(2, 6) if seq % 256 == 0 and rng.random() < 0.3 else 0
        if dtype == "fp32":
            batch = max(1, min(batch, 8192 // seq))
        return {"kind": "lm", "dtype": dtype, "layers": rng.randint(2, 12), "level1": level1, "heads": heads, "d_head": 64, "d_state": 64,
                "vocab": _log_int(rng, 1000, 50257), "batch": batch, "seq": seq, "chunk": rng.choice([128, 256]),
                "host": rng.random() < 0.3}
    if kind == "block":
        small = rng.random() < 0.3
        return {"kind": "block", "dtype": rng.choice(["fp32", "bf16"]), "heads": rng.choice([8, 16]) if small else rng.choice([8, 16, 24, 32]),
                "d_head": 32 if small else 64, "d_state": rng.choice([16, 32]) if small else rng.choice([64, 64, 128]),
                "batch": rng.randint(1, 4), "seq": _log_int(rng, 48, 1600), "chunk": 64 if small else rng.choice([128, 256])}
    if kind == "stack":
        return {"kind": "stack", "dtype": "fp32", "layers": rng.randint(2, 6), "heads": rng.choice([8, 16, 24]), "d_head": 64, "d_state": 64,
                "batch": rng.randint(1, 4), "seq": _log_int(rng, 64, 1024), "chunk": rng.choice([128, 256])}
    if kind == "prefill":
        seq = _log_int(rng, 17, 2500)
        return {"kind": "prefill", "dtype": rng.choice(["fp32", "bf16"]), "heads": rng.choice([8, 16, 24, 32]), "d_head": 64,
                "d_state": rng.choice([64, 64, 128]), "batch": max(1, min(_log_int(rng, 1, 8), 8192 // seq)), "seq": seq, "chunk": 256}
    if kind == "decode":
        return {"kind": "decode", "heads": rng.choice([8, 16, 24, 32]), "d_head": 64, "d_state": rng.choice([64, 128]),
                "expand": rng.choice([1, 2]), "batch": _log_int(rng, 1, 256)}
    if kind == "scan":
        # sequences of whole chunks, as the operator is called by a program that pads, and of any length
        dtype = rng.choice(["fp32", "bf16"])
        chunk = rng.choice([128, 256])
        whole = rng.random() < 0.6
        seq = chunk * _log_int(rng, 2, 8192 // chunk) if whole else _log_int(rng, 100, 1500)
        heads = rng.choice([8, 16, 32])
        most = 8192 if not whole else 131072 if dtype == "bf16" else 32768
        batch = max(1, min(_log_int(rng, 1, 16), most // seq))
        groups = heads if whole and seq <= 2048 and rng.random() < 0.3 else 1
        return {"kind": "scan", "dtype": dtype, "batch": batch, "seq": seq, "heads": heads, "groups": groups,
                "d_head": 64, "d_state": rng.choice([64, 128]), "chunk": chunk}
    return {"kind": "adamw", "params": _log_int(rng, 1_000_000, 126_000_000)}


# -------------------------------------------------------------------------------------------------
# inputs
# -------------------------------------------------------------------------------------------------

def _config(case):
    import pm_b200
    heads, d_head = case["heads"], case["d_head"]
    # expand 2 (inner width heads * d_head) unless the case says otherwise
    d_model = heads * d_head // case.get("expand", 2)
    return pm_b200.Mamba2Config(d_model=d_model, d_state=case["d_state"], d_head=d_head, n_heads=heads, n_groups=1, d_conv=4,
                                block_len=case.get("chunk", 256))


def _block_params(cfg, g):
    """The distributions of the package's own initialiser, drawn on the GPU: projections uniform in 1/sqrt(fan_in),
    A = -exp(U[log 1, log 16]), dt_bias = softplus^-1(U[1e-3, 1e-1]), D = 1, norm weight 1."""
    sh = cfg.param_shapes()

    def uni(name, fan_in):
        return (torch.rand(sh[name], device="cuda", generator=g) * 2 - 1) / math.sqrt(fan_in)

    dt = torch.rand(sh["dt_bias"], device="cuda", generator=g) * (1e-1 - 1e-3) + 1e-3
    return {"in_proj_weight": uni("in_proj_weight", cfg.d_model), "conv1d_weight": uni("conv1d_weight", cfg.d_conv),
            "conv1d_bias": torch.zeros(sh["conv1d_bias"], device="cuda"),
            "a_log": torch.rand(sh["a_log"], device="cuda", generator=g) * math.log(16.0), "d_skip": torch.ones(sh["d_skip"], device="cuda"),
            "dt_bias": dt + torch.log(-torch.expm1(-dt)), "norm_weight": torch.ones(sh["norm_weight"], device="cuda"),
            "out_proj_weight": uni("out_proj_weight", cfg.d_inner)}


def _owned(lm, view):
    """The handle owns the memory behind its views: a view that a program hands on keeps the handle with it."""
    t = view.view(-1)
    t.owner = lm
    return t


def prepare(case, seed):
    import pm_b200 as pm
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    kind = case["kind"]
    td = torch.bfloat16 if case.get("dtype") == "bf16" else torch.float32

    def randn(*shape):
        return torch.randn(*shape, device="cuda", generator=g)

    if kind == "adamw":
        n = case["params"]
        # gradients of a mean loss: small elements, with a norm above the clipping threshold
        return {"kind": kind, "opt": pm.AdamW(randn(n) * 0.02, lr=3e-4, weight_decay=0.1), "grads": randn(n) * 1e-2}
    if kind == "scan":
        B, T, H, G, P, N = (case[k] for k in ("batch", "seq", "heads", "groups", "d_head", "d_state"))
        dt = torch.nn.functional.softplus(randn(B, T, H) * 0.5 - 2.0)
        a = dt * -torch.exp(torch.rand(H, device="cuda", generator=g) * math.log(16.0))
        x = (randn(B, T, H, P) * dt.unsqueeze(-1)).to(td)            # the operator takes x dt
        b, c, dy = randn(B, T, G, N).to(td), randn(B, T, G, N).to(td), randn(B, T, H, P).to(td)
        cls = pm.SsdScanBf16 if td == torch.bfloat16 else pm.SsdScan
        return {"kind": kind, "scan": cls(x, a, b, c, case["chunk"]), "dy": dy}
    cfg = _config(case)
    if kind == "lm":
        lm = pm.FlatMamba(cfg, case["layers"], case["vocab"], case["batch"], case["seq"], compute_dtype=td,
                          level1_layers=case["level1"], group=4)
        n = case["layers"] + case["level1"]
        wproj = (torch.rand(cfg.d_model, cfg.d_model, device="cuda", generator=g) * 2 - 1) / math.sqrt(cfg.d_model) if case["level1"] else None
        lm.load(randn(case["vocab"], cfg.d_model) * 0.02, [_block_params(cfg, g) for _ in range(n)], wproj=wproj)
        ids = torch.randint(0, case["vocab"], (case["batch"], case["seq"]), device="cuda", generator=g)
        targets = torch.roll(ids, -1, dims=1).contiguous()
        state = {"kind": kind, "lm": lm, "loss": _owned(lm, lm.loss_dev), "grads": _owned(lm, lm.flat_grads)}
        if case["host"]:
            state.update(kind="lm_host", ids=ids.cpu().pin_memory(), targets=targets.cpu().pin_memory())
        else:
            state.update(ids=ids, targets=targets, step=lm.capture_step())
        return state
    B = case["batch"]
    if kind == "decode":
        blk = pm.Mamba2Block(cfg, _block_params(cfg, g))
        st = blk.zero_state(B)
        st["ssm_state"].copy_(randn(*st["ssm_state"].shape) * 0.1)
        st["conv_window"].copy_(randn(*st["conv_window"].shape) * 0.5)
        return {"kind": kind, "block": blk, "x": randn(B, 1, cfg.d_model), "state": st}
    T = case["seq"]
    x, dout = randn(B, T, cfg.d_model).to(td), randn(B, T, cfg.d_model).to(td)
    if kind == "stack":
        return {"kind": kind, "enc": pm.ContextEncoder(cfg, [_block_params(cfg, g) for _ in range(case["layers"])]), "x": x, "dout": dout}
    return {"kind": kind, "block": pm.Mamba2Block(cfg, _block_params(cfg, g), compute_dtype=td), "x": x, "dout": dout}


# -------------------------------------------------------------------------------------------------
# one pass
# -------------------------------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "lm":
        state["step"](state["ids"], state["targets"])
        return {"loss": state["loss"], "grads": state["grads"]}
    if kind == "lm_host":
        loss = state["lm"].step_host(state["ids"], state["targets"])
        return {"loss": loss, "grads": state["grads"]}
    if kind == "block":
        out = state["block"].forward(state["x"], residual=state["x"])
        dx, grads = state["block"].backward(state["x"], state["dout"], dx_accum=state["dout"])
        return {"out": out, "dx": dx, "grads": grads}
    if kind == "stack":
        out, saved = state["enc"].forward_checkpointed(state["x"])
        dx, grads = state["enc"].checkpoint_backward(saved, state["dout"])
        return {"out": out, "dx": dx, "grads": grads}
    if kind == "prefill":
        return state["block"].forward(state["x"], residual=state["x"])
    if kind == "decode":
        y, st = state["block"].step(state["x"], state["state"])
        return {"y": y, "ssm_state": st["ssm_state"], "conv_window": st["conv_window"]}
    if kind == "scan":
        y = state["scan"].forward()
        dx, da, db, dc = state["scan"].backward(state["dy"])
        return {"y": y, "dx": dx, "da": da, "db": db, "dc": dc}
    sumsq = state["opt"].step(state["grads"], max_norm=1.0)
    return {"params": state["opt"].p, "m": state["opt"].m, "v": state["opt"].v, "sumsq": sumsq}


# -------------------------------------------------------------------------------------------------
# the work of one pass, and how closely two implementations agree
# -------------------------------------------------------------------------------------------------

def _scan_flops_per_token(H, P, N, G, Q):
    """Chunked scan, causal half of the in-chunk products.  Forward: C B^T, masked product with x, states, C h.
    Backward: the transposed products, and dG with its two products."""
    fwd = Q * N * G + H * (Q * P + 4.0 * N * P)
    bwd = H * (2.0 * Q * P + 8.0 * N * P) + 3.0 * Q * N * G
    return fwd, bwd


def _block_counts(D, H, P, N, Q):
    """Matmul flops per token and direction, scan flops per token forward and backward, parameters."""
    inner = H * P
    J = 2 * inner + 2 * N + H
    fwd, bwd = _scan_flops_per_token(H, P, N, 1, Q)
    return 2.0 * (D * J + inner * D), fwd, bwd, D * J + inner * D + (inner + 2 * N) * 5 + inner + 3 * H


def work(case):
    kind = case["kind"]
    if kind == "adamw":
        n = case["params"]
        return {"bytes": 28.0 * n, "flops": 15.0 * n}                # p, g, m, v in; p, m, v out
    H, P, N = case["heads"], case["d_head"], case["d_state"]
    esz = 2 if case.get("dtype") == "bf16" else 4
    if kind == "scan":
        G, tok = case["groups"], float(case["batch"] * case["seq"])
        fwd, bwd = _scan_flops_per_token(H, P, N, G, min(case["chunk"], case["seq"]))
        # x, b, c, dy in; y, dx, db, dc out; a in, da out
        return {"bytes": tok * (esz * (4 * H * P + 4 * G * N) + 8 * H), "flops": tok * (fwd + bwd)}
    D = H * P // case.get("expand", 2)
    if kind == "decode":
        B = case["batch"]
        mm, _, _, params = _block_counts(D, H, P, N, 1)
        X = H * P + 2 * N
        return {"bytes": 4.0 * params + B * (8.0 * D + 8.0 * H * N * P + 24.0 * X), "flops": B * (mm + 6.0 * H * N * P)}
    tok = float(case["batch"] * case["seq"])
    mm, sf, sb, params = _block_counts(D, H, P, N, min(case["chunk"], case["seq"]))
    if kind == "prefill":
        return {"bytes": tok * D * 2 * esz + params * 4.0, "flops": tok * (mm + sf)}
    if kind == "block":
        return {"bytes": tok * D * 4 * esz + params * 8.0, "flops": tok * (3 * mm + sf + sb)}
    if kind == "stack":
        return {"bytes": tok * D * 4 * 4 + case["layers"] * params * 8.0, "flops": case["layers"] * tok * (3 * mm + sf + sb)}
    layers = case["layers"] + case["level1"] / 4.0                   # level 1 runs at a quarter of the token rate
    n_params = (case["layers"] + case["level1"]) * params + case["vocab"] * D
    return {"bytes": 8.0 * n_params + 16.0 * tok, "flops": tok * (layers * (3 * mm + sf + sb) + 6.0 * case["vocab"] * D)}


def tolerance(case):
    kind = case["kind"]
    if kind == "adamw":
        return {"rel": 1e-5}
    if case.get("dtype") == "bf16":
        return {"rel": 2e-2, "max": 0.8}          # bf16 operands and storage; the decay's gradient is a difference of large sums
    if kind == "lm":
        return {"rel": 3e-4}                      # fp32 products on bf16 pairs (16 mantissa bits), through up to 24 blocks and back
    if kind == "decode":
        return {"rel": 5e-5}
    return {"rel": 1e-4 if kind == "prefill" else 2e-4}
