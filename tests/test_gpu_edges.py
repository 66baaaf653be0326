"""GPU tests of the kernel variants at the sizes where their tiling or dispatch changes: edges of tiles, remainders,
the smallest and largest sizes of a rule.  Oracle or plain fp32 / fp64 torch as the reference."""
import pathlib
import subprocess
import sys
import threading

import pytest
import torch

from oracle import mamba2_oracle as orc
from util import FP32_TOL, assert_close, block_params, cuda_params, rand, randn, tol_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pm():
    import __graft_entry__ as ge
    ge.build()
    import pm_b200
    assert torch.cuda.is_available()
    return pm_b200


@pytest.mark.parametrize("offset", [0, 1])        # 1: buffers off the 16-byte grid take the scalar kernels
@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 4099, 1024 * 1024 + 2])
def test_adamw_sizes_and_alignment(pm, n, offset):
    p0, g = randn((n,), 1), randn((n,), 2)
    p_ref, m_ref, v_ref = [p0.clone()], [torch.zeros(n)], [torch.zeros(n)]
    buf = torch.zeros(n + 1, device="cuda")
    buf[offset:offset + n] = p0.cuda()
    opt = pm.AdamW(buf[offset:offset + n], lr=3e-3, weight_decay=0.1)
    sumsq = opt.step(g.cuda(), max_norm=0.5)
    g_ref = [g.clone()]
    norm = orc.clip_grad_norm(g_ref, 0.5)
    orc.adamw_step(p_ref, g_ref, m_ref, v_ref, 1, lr=3e-3, wd=0.1)
    assert abs(float(sumsq.item()) ** 0.5 - norm) < 1e-5 * norm
    assert_close(buf[offset:offset + n], p_ref[0], tol=1e-5, what="params")
    assert_close(opt.m, m_ref[0], what="m")
    assert_close(opt.v, v_ref[0], what="v")       # (1 - beta in fp32 on the device, in fp64 in the oracle)


def _block(pm, D, H, P, N, G, Q, dtype, seed=3):
    cfg = orc.Mamba2Config(d_model=D, d_state=N, d_head=P, n_heads=H, n_groups=G, d_conv=4, block_len=Q)
    p = orc.init_block_params(cfg, seed=seed)
    pc = pm.Mamba2Config(d_model=D, d_state=N, d_head=P, n_heads=H, n_groups=G, d_conv=4, block_len=Q)
    return cfg, p, pm.Mamba2Block(pc, {k: v.cuda() for k, v in p.items()}, compute_dtype=dtype)


# lengths around the 128-token step of the one-kernel scan, one and two 64-wide blocks of d_state, narrow heads and states
@pytest.mark.parametrize("B,T", [(1, 1), (2, 17), (1, 127), (2, 128), (3, 129), (1, 500)])
@pytest.mark.parametrize("P,N,G", [(64, 64, 1), (64, 128, 1), (32, 16, 1), (16, 8, 4), (64, 64, 4), (48, 96, 1)])
def test_block_forward_lengths(pm, B, T, P, N, G):
    D, H = 64, 4
    cfg, p, blk = _block(pm, D, H, P, N, G, 256, torch.float32)
    x = randn((B, T, D), 5)
    out = blk.forward(x.cuda())
    torch.cuda.synchronize()
    assert pm.device_status() == 0
    assert_close(out, orc.block_forward(p, cfg, x), what=f"B={B} T={T} P={P} N={N} G={G}")


# the same for the backward, with sequences long enough to be walked in segments (eight heads: in_proj's width is a multiple of 8 and
# the chain kernels serve the backward; four: the FMA contractions)
@pytest.mark.parametrize("B,T", [(1, 1), (2, 17), (1, 127), (2, 128), (3, 129), (1, 256), (1, 640), (2, 1024)])
@pytest.mark.parametrize("P,N,G,H", [(64, 64, 1, 4), (64, 64, 1, 8), (32, 16, 1, 4), (32, 16, 1, 8), (64, 64, 4, 4), (64, 64, 8, 8), (64, 24, 1, 4), (64, 24, 1, 8), (48, 40, 1, 8)])
def test_block_backward_lengths(pm, B, T, P, N, G, H):
    D, Q = 64, 128 if P == 64 else 64
    cfg, p, blk = _block(pm, D, H, P, N, G, Q, torch.float32)
    x, cot = randn((B, T, D), 5), randn((B, T, D), 6)
    dx, grads = blk.backward(x.cuda(), cot.cuda())
    torch.cuda.synchronize()
    assert pm.device_status() == 0
    leaves = {k: v.clone().requires_grad_(True) for k, v in p.items()}
    xr = x.clone().requires_grad_(True)
    orc.block_forward(leaves, cfg, xr).backward(cot)
    chunk = Q if T % Q == 0 else T
    chain = H == 8 and (chunk <= (256 if P == 64 else 64) or (P == N == 64 and chunk % 128 == 0))
    assert_close(dx, xr.grad, what="dx")
    for k, g in grads.items():
        if T > 1 or k != "a_log":      # (one token: d(a_log) is exactly zero)
            assert_close(g, leaves[k].grad, tol=FP32_TOL if chain else tol_for(k), what=k)


# inputs of the size that a model's embeddings have, where D x outweighs the scan's part of y a thousand times: d(a_log) and d(dt_bias) do not
# go through y - D x, on the FMA contractions (odd widths, ragged lengths, d_head beyond 64), 3xTF32 (d_state 128 on whole chunks), and the chains
@pytest.mark.parametrize("P,N,H,T,Q", [(64, 128, 8, 256, 128), (64, 128, 8, 300, 128), (64, 64, 8, 300, 128), (64, 64, 6, 256, 128), (32, 16, 4, 200, 64), (24, 40, 6, 128, 64),
                                       (128, 64, 4, 128, 64), (5, 7, 3, 60, 32)])
def test_block_gradients_of_small_inputs(pm, P, N, H, T, Q):
    D, B = 64, 2
    cfg, p, blk = _block(pm, D, H, P, N, 1, Q, torch.float32)
    x, cot = randn((B, T, D), 5, 0.02), randn((B, T, D), 6, 1e-3)
    dx, grads = blk.backward(x.cuda(), cot.cuda())
    assert pm.device_status() == 0
    leaves = {k: v.double().requires_grad_(True) for k, v in p.items()}
    xr = x.double().requires_grad_(True)
    orc.block_forward(leaves, cfg, xr).backward(cot.double())
    assert_close(dx, xr.grad, what="dx")
    for k, g in grads.items():
        assert_close(g, leaves[k].grad, tol=tol_for(k), what=k)


# the same in a model, whose token embeddings are of that size: every engine of the scan's backward, fp32 and bf16 storage (2e-2 as for any
# bf16 gradient)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("P,N,H,T,Q", [(64, 128, 8, 256, 128), (64, 128, 8, 300, 128), (32, 16, 8, 200, 64), (24, 40, 8, 128, 64), (32, 16, 4, 200, 64), (128, 64, 8, 128, 64)])
def test_model_decay_gradients(pm, dtype, P, N, H, T, Q):
    D, B, V, L = 128, 2, 200, 2
    if dtype == torch.bfloat16 and H % 8:
        pytest.skip("bf16 storage wants widths that are multiples of 8")
    cfg = orc.Mamba2Config(d_model=D, d_state=N, d_head=P, n_heads=H, n_groups=1, d_conv=4, block_len=Q)
    layers, embed = [block_params(cfg, seed=61 + l) for l in range(L)], randn((V, D), 13, 0.02)
    lm = pm.FlatMamba(pm.Mamba2Config(d_model=D, d_state=N, d_head=P, n_heads=H, n_groups=1, d_conv=4, block_len=Q), L, V, B, T, compute_dtype=dtype)
    lm.load(embed.cuda(), [cuda_params(p) for p in layers])
    ids, tg, _ = orc.lcg_batch(17, B, T, V)
    lm.step_device(ids.cuda(), tg.cuda())
    er, ls = embed.double().requires_grad_(True), [{k: v.double().requires_grad_(True) for k, v in p.items()} for p in layers]
    orc.lm_loss(er, ls, cfg, ids, tg, cdt=torch.float64).backward()
    assert pm.device_status() == 0
    _, gl = lm.grads()
    for l in range(L):
        for k in ("a_log", "dt_bias", "in_proj_weight", "d_skip"):
            assert_close(gl[l][k], ls[l][k].grad, tol=tol_for(k) if dtype == torch.float32 else 2e-2, what=f"layer {l} {k}")
    lm.close()


# token counts at which the weight gradients of the bf16-storage block split K or not, with and without whole tiles
@pytest.mark.parametrize("B,T", [(1, 40), (1, 1100), (3, 1024)])
def test_block_bf16_weight_gradient_splits(pm, B, T):
    D, H, P, N = 128, 8, 32, 16
    cfg, p, blk = _block(pm, D, H, P, N, 1, 64, torch.bfloat16)
    x, cot = randn((B, T, D), 5).bfloat16(), randn((B, T, D), 6).bfloat16()
    dx, grads = blk.backward(x.cuda(), cot.cuda())
    torch.cuda.synchronize()
    assert pm.device_status() == 0
    leaves = {k: v.clone().requires_grad_(True) for k, v in p.items()}
    xr = x.float().requires_grad_(True)
    orc.block_forward(leaves, cfg, xr).backward(cot.float())
    assert_close(dx.float(), xr.grad, tol=3e-2, what="dx")
    for k in ("in_proj_weight", "out_proj_weight"):
        assert_close(grads[k], leaves[k].grad, tol=2e-2, what=k)


# bf16 storage on whole chunks, on either side of the lines between the scan as chains and chunk by chunk: both as chains, the recompute chunk by
# chunk, both chunk by chunk; chunks of one and two steps.  Tolerances of the tests above.
@pytest.mark.parametrize("B,T", [(5, 512), (1, 512), (1, 1024)])
@pytest.mark.parametrize("Q", [128, 256])
def test_block_bf16_chains_or_chunks(pm, B, T, Q):
    cfg, p, blk = _block(pm, 64, 8, 64, 64, 1, Q, torch.bfloat16)
    x, cot = randn((B, T, 64), 5).bfloat16(), randn((B, T, 64), 6).bfloat16()
    out = blk.forward(x.cuda())
    dx, grads = blk.backward(x.cuda(), cot.cuda())
    torch.cuda.synchronize()
    assert pm.device_status() == 0
    leaves = {k: v.clone().requires_grad_(True) for k, v in p.items()}
    xr = x.float().requires_grad_(True)
    ref = orc.block_forward(leaves, cfg, xr)
    ref.backward(cot.float())
    assert_close(out.float(), ref, tol=2e-2, what="out")
    assert_close(dx.float(), xr.grad, tol=3e-2, what="dx")
    for k, v in leaves.items():
        assert_close(grads[k], v.grad, tol=2e-2, what=k)


# batch sizes around the switch from streamed FMA to tensor-core projections and its tile widths; widths with ragged column
# tiles; the last ones are served by the general kernels, or have an odd d_state per head under the vectorised state step
@pytest.mark.parametrize("B", [1, 2, 3, 5, 9, 16, 17, 33, 70, 130, 300])
@pytest.mark.parametrize("D,H,P,N,G", [(64, 4, 32, 16, 1), (72, 6, 24, 40, 6), (200, 8, 64, 128, 1), (36, 3, 5, 7, 1), (64, 2, 8, 7, 2), (64, 4, 8, 5, 4)])
def test_decode_batches(pm, B, D, H, P, N, G):
    cfg, p, blk = _block(pm, D, H, P, N, G, 64, torch.float32)
    st = blk.zero_state(B)
    ref = {"ssm_state": randn((B, H, N, P), 7, 0.3), "conv_window": randn((B, cfg.xbc_dim, 3), 8, 0.5)}
    st["ssm_state"].copy_(ref["ssm_state"]); st["conv_window"].copy_(ref["conv_window"])
    for step in range(2):
        x = randn((B, 1, D), 20 + step)
        y, st = blk.step(x.cuda(), st)
        y_ref, ref = orc.block_step(p, cfg, x, ref)
        assert_close(y, y_ref, what=f"y step {step}")
        assert_close(st["ssm_state"], ref["ssm_state"], what="state")
        assert_close(st["conv_window"], ref["conv_window"], what="window")
    assert pm.device_status() == 0


# as many sequences as tiles of 128 of them fit on the SMs at once (in_proj has nine column tiles), and one more, which is alone in a tile of
# 256; as many as leave out_proj two splits of its 24 k-tiles (seven column tiles), and one more
@pytest.mark.parametrize("B,D,H,P", [(2048, 200, 8, 64), (2049, 200, 8, 64), (1280, 800, 24, 64), (1281, 800, 24, 64)])
def test_decode_tiles_of_many_sequences(pm, B, D, H, P):
    N = 16
    cfg, p, blk = _block(pm, D, H, P, N, 1, 64, torch.float32)
    ref = {"ssm_state": randn((B, H, N, P), 7, 0.3), "conv_window": randn((B, cfg.xbc_dim, 3), 8, 0.5)}
    x = randn((B, 1, D), 20)
    y, st = blk.step(x.cuda(), {k: v.cuda() for k, v in ref.items()})
    y_ref, ref = orc.block_step(p, cfg, x, ref)
    assert_close(y, y_ref, what="y")
    assert_close(st["ssm_state"], ref["ssm_state"], what="state")
    assert_close(st["conv_window"], ref["conv_window"], what="window")
    assert pm.device_status() == 0


# weight rows that take a thread more than one pass of its groups, with a remainder, on both products; beyond 16 sequences the two widths
# that convert the token themselves, with a part of a tile at the end; offset 1: the token and the norm's weight off the 16-byte grid
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("B,D", [(1, 1028), (2, 1028), (4, 1028), (8, 1028), (16, 1028), (17, 1032), (32, 1032), (50, 1032), (64, 1032)])
def test_decode_long_rows(pm, B, D, offset):
    def off_grid(t):
        return torch.cat([t.new_zeros(offset), t.flatten()])[offset:].view(t.shape)

    H, P, N = 13, 128, 12
    cfg, p, blk = _block(pm, D, H, P, N, 1, 64, torch.float32)
    blk.params["norm_weight"] = off_grid(blk.params["norm_weight"])
    ref = {"ssm_state": randn((B, H, N, P), 7, 0.3), "conv_window": randn((B, cfg.xbc_dim, 3), 8, 0.5)}
    st = {k: v.cuda() for k, v in ref.items()}
    x = randn((B, 1, D), 20)
    y, st = blk.step(off_grid(x.cuda()), st)
    y_ref, ref = orc.block_step(p, cfg, x, ref)
    assert_close(y, y_ref, what="y")
    assert_close(st["ssm_state"], ref["ssm_state"], what="state")
    assert_close(st["conv_window"], ref["conv_window"], what="window")


# steps that follow one another without a pause read what the step before wrote, and weights that a product just wrote: the same bits as with
# the device idle in between; the projections on FMA, on the tensor cores and on the general kernels
@pytest.mark.parametrize("B,D", [(1, 128), (16, 128), (40, 128), (400, 128), (400, 132)])
def test_decode_steps_back_to_back(pm, B, D):
    cfg, p, blk = _block(pm, D, 4, 64, 64, 1, 64, torch.float32)
    x = [randn((B, 1, D), 20 + i).cuda() for i in range(12)]
    eye, w = torch.eye(D, device="cuda"), [randn(tuple(blk.params["in_proj_weight"].shape), 40 + i, 0.1).cuda() for i in range(3)]

    def run(pause):
        st, ys = blk.zero_state(B), []
        for i, xt in enumerate(x):
            if i % 4 == 3:
                pm.matmul(eye, w[i // 4], out=blk.params["in_proj_weight"])
                pause()
            y, st = blk.step(xt, st)
            pause()
            ys.append(y)
        torch.cuda.synchronize()
        return ys + [st["ssm_state"], st["conv_window"]]

    first = blk.params["in_proj_weight"].clone()
    want = run(torch.cuda.synchronize)
    blk.params["in_proj_weight"].copy_(first)
    for got, ref in zip(run(lambda: None), want):
        assert torch.equal(got, ref)


# more sequences than a grid has rows, on the general and on the tensor-core route of the projections
@pytest.mark.parametrize("D,H,P,N", [(16, 1, 8, 4), (16, 2, 4, 7)])
def test_decode_many_sequences(pm, D, H, P, N):
    B = 65537
    cfg, p, blk = _block(pm, D, H, P, N, 1, 64, torch.float32)
    st = blk.zero_state(B)
    ref = {"ssm_state": randn((B, H, N, P), 7, 0.3), "conv_window": randn((B, cfg.xbc_dim, 3), 8, 0.5)}
    st["ssm_state"].copy_(ref["ssm_state"]); st["conv_window"].copy_(ref["conv_window"])
    x = randn((B, 1, D), 20)
    y, st = blk.step(x.cuda(), st)
    y_ref, ref = orc.block_step(p, cfg, x, ref)
    assert_close(y, y_ref, what="y")
    assert_close(st["ssm_state"], ref["ssm_state"], what="state")
    assert_close(st["conv_window"], ref["conv_window"], what="window")
    assert pm.device_status() == 0


# a captured step is replayed after the block has stepped at more batch sizes than it keeps workspaces for, and after memory has been
# handed out again
def test_captured_decode_outlives_other_batches(pm):
    D, H, P, N, B = 64, 4, 32, 16, 3
    cfg, p, blk = _block(pm, D, H, P, N, 1, 64, torch.float32)
    start = {"ssm_state": randn((B, H, N, P), 7, 0.3).cuda(), "conv_window": randn((B, cfg.xbc_dim, 3), 8, 0.5).cuda()}
    x, st = randn((B, 1, D), 20).cuda(), {k: v.clone() for k, v in start.items()}
    want, _ = blk.step(x, {k: v.clone() for k, v in start.items()})
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        blk.step(x, {k: v.clone() for k, v in start.items()})              # warm-up on the stream that captures
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        y, _ = blk.step(x, st)
    for stream in (side, torch.cuda.current_stream()):
        with torch.cuda.stream(stream):
            for batch in range(1, 12):
                blk.step(randn((batch, 1, D), batch).cuda(), blk.zero_state(batch))
            guards = [torch.full((64 * k,), 7, dtype=torch.uint8, device="cuda") for k in range(1, 200)]
    torch.cuda.synchronize()
    for k in st:
        st[k].copy_(start[k])
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want) and pm.device_status() == 0
    assert all(bool((g == 7).all()) for g in guards)


# the bf16-input scan off the 128-token grid keeps everything but its outputs at fp32 precision: lengths around a step, segments,
# narrow heads and states, one and two halves of d_state, tensors that start off a 16-byte boundary
@pytest.mark.parametrize("B,T", [(1, 1), (2, 127), (1, 129), (3, 200), (1, 700)])
@pytest.mark.parametrize("P,N,G,off", [(64, 64, 1, 0), (64, 128, 1, 0), (64, 128, 4, 0), (32, 16, 1, 0), (64, 72, 1, 3)])
def test_scan_bf16_lengths(pm, B, T, P, N, G, off):
    H = 4

    def put(t):
        return torch.cat([torch.zeros(off, dtype=t.dtype), t.flatten()]).cuda()[off:].view(t.shape)
    x, b, c, dy = randn((B, T, H, P), 1).bfloat16(), randn((B, T, G, N), 2).bfloat16(), randn((B, T, G, N), 3).bfloat16(), randn((B, T, H, P), 4).bfloat16()
    a = -torch.nn.functional.softplus(randn((B, T, H), 5) - 2.0)
    init = randn((B, H, N, P), 6)
    scan = pm.SsdScanBf16(put(x), a.cuda(), put(b), put(c), 128)
    y, last = scan.forward(init_state=put(init), want_final_state=True)
    y0 = scan.forward()
    dx, da, db, dc = scan.backward(put(dy))
    torch.cuda.synchronize()
    assert pm.device_status() == 0
    leaves = [t.float().requires_grad_(True) for t in (x, a, b, c)]
    be, ce = (t.expand(B, T, H, N) for t in leaves[2:])
    ref, _ = orc.ssd_scan_chunked(leaves[0], leaves[1], be, ce, T, return_final_state=True)
    ref.backward(dy.float())
    with torch.no_grad():
        ref_i, last_i = orc.ssd_scan_chunked(leaves[0], leaves[1], be, ce, T, initial_state=init, return_final_state=True)
    for got, want, tol, what in ((y0.float(), ref, 5e-3, "y"), (y.float(), ref_i, 5e-3, "y from a state"), (last, last_i, 1e-4, "final state"),
                                 (dx.float(), leaves[0].grad, 5e-3, "dx"), (da, leaves[1].grad, 1e-4, "da"),
                                 (db.float(), leaves[2].grad, 5e-3, "db"), (dc.float(), leaves[3].grad, 5e-3, "dc")):
        if T > 1 or what != "da":      # (one token: da is exactly zero)
            assert_close(got, want, tol=tol, what=what)


# the state that the bf16-input scan hands on is formed in fp32 off the whole chunks (whole ones round what they form): fp32 sums of up to
# 700 decaying terms stay within 2e-6 of fp64, sums of bf16 pairs are 5e-6 off.
@pytest.mark.parametrize("B,T", [(1, 1), (2, 127), (1, 129), (3, 200), (1, 700)])
@pytest.mark.parametrize("P,N,G,off", [(64, 64, 1, 0), (64, 128, 4, 0), (32, 16, 1, 0), (8, 40, 1, 3)])
def test_scan_bf16_final_state_in_fp32(pm, B, T, P, N, G, off):
    H = 4
    x, b, c = randn((B, T, H, P), 1).bfloat16(), randn((B, T, G, N), 2).bfloat16(), randn((B, T, G, N), 3).bfloat16()
    a = -torch.nn.functional.softplus(randn((B, T, H), 5) - 2.0)
    init = torch.cat([torch.zeros(off), randn((B, H, N, P), 6).flatten()]).cuda()[off:].view(B, H, N, P)
    be, ce = (t.double().expand(B, T, H, N) for t in (b, c))
    for i0 in (None, init):
        _, want = orc.ssd_scan_chunked(x.double(), a.double(), be, ce, T, initial_state=None if i0 is None else i0.cpu().double(), return_final_state=True)
        _, last = pm.SsdScanBf16(x.cuda(), a.cuda(), b.cuda(), c.cuda(), 128).forward(init_state=i0, want_final_state=True)
        assert pm.device_status() == 0
        assert_close(last, want, tol=2e-6, what="final state")


# chunks of several steps: a state is rounded to bf16 between the steps only where that leaves da (fp32) about as far off as one rounding
# per chunk does; a single chunk, two chunks of two steps and chunks of more steps keep da and the state at fp32 precision
@pytest.mark.parametrize("T,Q", [(256, 256), (512, 256), (384, 384), (768, 384), (1024, 512), (1024, 1024)])
@pytest.mark.parametrize("N,G", [(64, 1), (128, 4)])
def test_scan_bf16_chunks_of_several_steps(pm, T, Q, N, G):
    B, H, P = 2, 4, 64
    x, b, c, dy = randn((B, T, H, P), 1).bfloat16(), randn((B, T, G, N), 2).bfloat16(), randn((B, T, G, N), 3).bfloat16(), randn((B, T, H, P), 4).bfloat16()
    a = -torch.nn.functional.softplus(randn((B, T, H), 5) - 2.0)
    scan = pm.SsdScanBf16(x.cuda(), a.cuda(), b.cuda(), c.cuda(), Q)
    y, last = scan.forward(want_final_state=True)
    dx, da, db, dc = scan.backward(dy.cuda())
    assert pm.device_status() == 0
    leaves = [t.double().requires_grad_(True) for t in (x, a, b, c)]
    ref, last_ref = orc.ssd_scan_chunked(leaves[0], leaves[1], *(t.expand(B, T, H, N) for t in leaves[2:]), Q, return_final_state=True)
    ref.backward(dy.double())
    for got, want, tol, what in ((y.float(), ref, 5e-3, "y"), (last, last_ref, 1e-4, "final state"), (dx.float(), leaves[0].grad, 5e-3, "dx"),
                                 (da, leaves[1].grad, 1e-4, "da"), (db.float(), leaves[2].grad, 5e-3, "db"), (dc.float(), leaves[3].grad, 5e-3, "dc")):
        assert_close(got, want, tol=tol, what=what)


# bf16 storage with a long vocabulary: the gradient of a row tile's hidden rows runs on a stream of its own under the next tile, and the
# tiles alternate between two buffers.  Four whole tiles and a remainder; the second buffer in the blocks' workspace, or (small blocks) of
# its own.  Everything on one stream, eagerly and as a graph replay, is the same sums in the same order.
@pytest.mark.parametrize("D,H,P,N,Q,own", [(64, 8, 8, 8, 32, True), (256, 8, 64, 64, 128, False)])
def test_lm_head_lane(pm, D, H, P, N, Q, own):
    B, T, V = 9, 512, 8200
    cfg = orc.Mamba2Config(d_model=D, d_state=N, d_head=P, n_heads=H, n_groups=1, d_conv=4, block_len=Q)
    p, embed = block_params(cfg, seed=61), randn((V, D), 13, 0.3)
    lm = pm.FlatMamba(pm.Mamba2Config(d_model=D, d_state=N, d_head=P, n_heads=H, n_groups=1, d_conv=4, block_len=Q), 1, V, B, T, compute_dtype=torch.bfloat16)
    lm.load(embed.cuda(), [cuda_params(p)])
    tile = 1024 * V * 4
    assert (lm.activation_detail["lm_head_transient"] >= 2 * tile) == own and (lm.activation_detail["block_workspace"] >= tile) == (not own)
    graph = lm.capture_step()
    n_embed = V * D
    for seed in range(3):
        ids, tg, _ = orc.lcg_batch(17 + seed, B, T, V)
        pm.set_concurrency(False)
        try:
            loss = lm.step_device(ids.cuda(), tg.cuda()).clone()
        finally:
            pm.set_concurrency(True)
        want = lm.flat_grads.clone()
        if seed == 0:
            er, leaves = embed.clone().requires_grad_(True), {k: v.clone().requires_grad_(True) for k, v in p.items()}
            ref = orc.lm_loss(er, [leaves], cfg, ids, tg)
            ref.backward()
            assert abs(float(loss) - float(ref)) < 2e-2 * float(ref)
            ge, gl = lm.grads()
            assert_close(ge, er.grad, tol=2e-2, what="embed")
            for k in ("in_proj_weight", "out_proj_weight", "norm_weight"):
                assert_close(gl[0][k], leaves[k].grad, tol=2e-2, what=k)
        for run in (lm.step_device, lm.step_device, graph, graph):
            lm.flat_grads.zero_()
            assert torch.equal(run(ids.cuda(), tg.cuda()).reshape(-1), loss.reshape(-1))
            assert torch.equal(lm.flat_grads[n_embed:], want[n_embed:])
            assert_close(lm.flat_grads[:n_embed], want[:n_embed], tol=1e-6, what="embed")      # (its token rows are added atomically)
    assert pm.device_status() == 0
    del graph
    lm.close()


# two threads with a block and a stream each share the library's internal streams, not the events that order them
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_blocks_on_two_threads(pm, dtype):
    work = []
    for k, (B, T) in enumerate([(2, 512), (1, 700)]):
        cfg, p, blk = _block(pm, 128, 8, 64, 64, 1, 128, dtype, seed=3 + k)
        x, cot = (randn((B, T, 128), s + k).cuda().to(dtype) for s in (5, 15))
        dx, grads = blk.backward(x, cot)
        work.append((blk, x, cot, dx, grads))
    torch.cuda.synchronize()
    off = [[], []]

    def run(k):
        blk, x, cot, dx, grads = work[k]
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(40):
                got, g = blk.backward(x, cot)
                off[k].append((got != dx).any() | torch.stack([(g[n] != grads[n]).any() for n in g]).any())
            torch.cuda.current_stream().synchronize()
    threads = [threading.Thread(target=run, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert [len(o) for o in off] == [40, 40] and not any(bool(o) for k in off for o in k)
    assert pm.device_status() == 0


FIRST_CALLS = """
import threading, torch, pm_b200 as pm
cfg = pm.Mamba2Config(d_model=64, d_state=64, d_head=64, n_heads=8, block_len=128)
g = torch.Generator().manual_seed(1)
params = {k: (0.1 * torch.randn(s, generator=g)).cuda() for k, s in cfg.param_shapes().items()}
x = torch.randn(2, 256, 64, generator=g).cuda()
torch.cuda.synchronize()
start, got = threading.Barrier(6), [None] * 6
def first(k):
    blk = pm.Mamba2Block(cfg, params)
    with torch.cuda.stream(torch.cuda.Stream()):
        start.wait()
        got[k] = (blk.forward(x), *blk.backward(x, x)[1].values())
        torch.cuda.current_stream().synchronize()
threads = [threading.Thread(target=first, args=(k,)) for k in range(6)]
[t.start() for t in threads]; [t.join() for t in threads]
assert all(g is not None and all(torch.equal(a, b) for a, b in zip(g, got[0])) for g in got), got
assert pm.device_status() == 0
print("same")
"""


# what the library sets up on first use (the driver's entry point, internal streams, kernel attributes, tensor maps), asked for by six
# threads at the same time in a process of its own
def test_first_calls_on_several_threads(pm):
    r = subprocess.run([sys.executable, "-c", FIRST_CALLS], cwd=pathlib.Path(pm.__file__).parent.parent, capture_output=True, text=True, timeout=200)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr[-2000:]


# an allocation that the driver refuses fails the call that asked for it, and no later one
def test_refused_call_does_not_fail_the_next(pm):
    assert pm.lib.pmb_gemm_reserve_scratch(1 << 60) != 0
    a, b = randn((64, 32), 1).cuda(), randn((32, 64), 2).cuda()
    assert_close(pm.matmul(a, b), a.double() @ b.double(), tol=3e-5, what="product")


# the CTA-pair GEMM's ways of storing a result: ragged edges (odd widths, rows past the last whole tile), fp32 and bf16, a residual
# loaded ahead, a result added onto C, and the two tile widths (few tiles with a long K take the narrow one on pairs)
@pytest.mark.parametrize("M,N,K", [(2048, 768, 1536), (1100, 1411, 200), (300, 4616, 72)])
@pytest.mark.parametrize("out16,res", [(0, 0), (1, 0), (1, 1), (0, 1), (0, 2)])
def test_gemm_pair_tiles_store(pm, M, N, K, out16, res):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, b = (torch.randn(*s, device="cuda", generator=g, dtype=torch.bfloat16) for s in ((M, K), (K, (N + 7) // 8 * 8)))
    ld = (N + 7) // 8 * 8
    dt = torch.bfloat16 if out16 else torch.float32
    c = torch.randn(M, ld, device="cuda", generator=g).to(dt)
    r = c if res == 2 else torch.randn(M, ld, device="cuda", generator=g).to(dt)
    want = a.float() @ b[:, :N].float() + (r[:, :N].float() if res else 0.0)
    past = c[:, N:].clone()
    st = pm.lib.pmb_gemm_bf16(pm._stream(), 0, 0, M, N, K, a.data_ptr(), K, b.data_ptr(), ld, c.data_ptr(), ld, r.data_ptr() if res else None, out16)
    assert st == 0 and pm.device_status() == 0
    assert_close(c[:, :N].float(), want, tol=5e-3 if out16 else 1e-5, what=f"{M}x{N}x{K}")
    assert torch.equal(c[:, N:], past)                  # nothing beyond the result's columns


@pytest.mark.parametrize("M,N,K", [(2048, 768, 1536), (1000, 1224, 136)])
def test_gemm_pair_tiles_on_pairs(pm, M, N, K):
    a, b = randn((M, K), 1).cuda(), randn((K, N), 2).cuda()
    out = pm.matmul(a, b)
    assert pm.device_status() == 0
    assert_close(out, a.double() @ b.double(), tol=3e-5, what=f"{M}x{N}x{K}")


# the conv's strips: 16 runs of 8, 16 or 32 steps to a CTA (130 and 240 sequences of 160 channels), four channels per
# thread, the next four rows in shared memory (the oracle's fp32 sums in another order: 1e-5 of the largest)
@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("B,T", [(1, 1), (2, 7), (1, 8), (1, 63), (2, 65), (3, 300), (40, 260), (130, 260), (240, 260)])
@pytest.mark.parametrize("H,P,N", [(4, 4, 4), (4, 16, 8), (8, 16, 16)])
def test_conv_strips(pm, B, T, K, H, P, N):
    cfg = pm.Mamba2Config(d_model=32, d_state=N, d_head=P, n_heads=H, n_groups=1, d_conv=K, block_len=T)
    I, X, J = cfg.d_inner, cfg.xbc_dim, cfg.in_proj_dim
    xzd, w, b, dact = randn((B, T, J), 1).requires_grad_(True), randn((X, 1, K), 2, 0.5).requires_grad_(True), randn((X,), 3, 0.1).requires_grad_(True), randn((B, T, X), 5)
    conv = torch.nn.functional.conv1d(xzd[..., I:I + X].transpose(1, 2), w, None, padding=K - 1, groups=X) + b.reshape(-1, 1)
    want = orc.silu(conv[..., :T].transpose(1, 2))
    act, _ = pm.conv_silu_dt_fwd(cfg, xzd.detach().cuda(), w.detach().cuda(), b.detach().cuda(), torch.zeros(H).cuda())
    assert_close(act, want, tol=1e-5, what="act")
    (want * dact).sum().backward()
    dxzd, dw, db = pm.conv_silu_bwd(cfg, xzd.detach().cuda(), w.detach().cuda(), b.detach().cuda(), dact.cuda())
    for got, want, what in ((dxzd[..., I:I + X], xzd.grad[..., I:I + X], "dx"), (dw, w.grad, "dw"), (db, b.grad, "db")):
        assert_close(got, want, tol=1e-5, what=what)


# decays that underflow inside a step of 128 tokens: the scan's masked tiles are formed by factors of 32-token blocks, each of which is a
# decay of its own.  bf16 inputs (rounded and kept as pairs), ragged and whole lengths, segments; as in the tests above.
@pytest.mark.parametrize("T,Q", [(128, 128), (200, 128), (512, 128), (1500, 256), (2048, 256)])
@pytest.mark.parametrize("N,strength", [(64, 3.0), (128, 30.0)])
def test_scan_bf16_strong_decay(pm, T, Q, N, strength):
    B, H, P = 1, 4, 64
    x, b, c, dy = randn((B, T, H, P), 1).bfloat16(), randn((B, T, 1, N), 2).bfloat16(), randn((B, T, 1, N), 3).bfloat16(), randn((B, T, H, P), 4).bfloat16()
    a = -strength * torch.nn.functional.softplus(randn((B, T, H), 5) - 1.0)
    scan = pm.SsdScanBf16(x.cuda(), a.cuda(), b.cuda(), c.cuda(), Q)
    y = scan.forward()
    dx, da, db, dc = scan.backward(dy.cuda())
    assert pm.device_status() == 0
    leaves = [t.double().requires_grad_(True) for t in (x, a, b, c)]
    orc.ssd_scan_chunked(leaves[0], leaves[1], *(t.expand(B, T, H, N) for t in leaves[2:]), Q if T % Q == 0 else T).backward(dy.double())
    ref = orc.ssd_scan_chunked(*(t.detach() for t in leaves[:2]), *(t.detach().expand(B, T, H, N) for t in leaves[2:]), Q if T % Q == 0 else T)
    for got, want, tol, what in ((y.float(), ref, 5e-3, "y"), (dx.float(), leaves[0].grad, 5e-3, "dx"), (da, leaves[1].grad, 1e-3, "da"),
                                 (db.float(), leaves[2].grad, 5e-3, "db"), (dc.float(), leaves[3].grad, 5e-3, "dc")):
        assert_close(got, want, tol=tol, what=what)


# a that is positive for a while: inside a step S rises (falls) by `rise` and comes back, so that the factors of a block beyond 88 are inf and 0
# where the rows outside have ordinary exponentials.  Rows inside the excursion overflow and are left out, as are dx of the rise and y of the
# fall, whose states do.  bf16 inputs (rounded and kept as pairs), ragged and whole lengths, segments; bf16 results as in the tests above.
@pytest.mark.parametrize("T,Q", [(128, 128), (200, 128), (512, 128), (1500, 256)])
@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("rise", [12.0, 30.0, 100.0])
def test_scan_bf16_positive_a(pm, T, Q, N, rise):
    B, H, P = 1, 4, 64
    x, b, c, dy = randn((B, T, H, P), 1).bfloat16(), randn((B, T, 1, N), 2).bfloat16(), randn((B, T, 1, N), 3).bfloat16(), randn((B, T, H, P), 4).bfloat16()
    for sign, first, end, what in ((1.0, 20, 40, "y"), (-1.0, 70, 100, "dx")):
        a = -torch.nn.functional.softplus(randn((B, T, H), 5) - 2.0)
        out = torch.ones(T, dtype=torch.bool)
        for t0 in range(0, T - end, 128):
            a[:, t0 + first] += sign * rise
            a[:, t0 + end] -= sign * rise
            out[t0 + first:t0 + end] = False
        scan = pm.SsdScanBf16(x.cuda(), a.cuda(), b.cuda(), c.cuda(), Q)
        got = scan.forward()
        xd = x.double().requires_grad_(True)
        want = orc.ssd_scan_chunked(xd, a.double(), *(t.double().expand(B, T, H, N) for t in (b, c)), Q if T % Q == 0 else T)
        if what == "dx":
            got = scan.backward(dy.cuda())[0]
            want, = torch.autograd.grad(want, xd, dy.double())
        assert pm.device_status() == 0
        assert_close(got.float()[:, out], want.detach()[:, out], tol=5e-3, what=what)


# products whose columns go to tiles of two widths: two rounds of tiles, a cut inside and one before the last tile, B in either order, a residual
@pytest.mark.parametrize("M,N,K", [(2048, 3224, 768), (1337, 3224, 136), (1000, 5000, 64), (14630, 296, 64)])
@pytest.mark.parametrize("tb,res", [(False, False), (True, True)])
def test_gemm_columns_cut(pm, M, N, K, tb, res):
    a, b, r = randn((M, K), 1).cuda(), randn((N, K) if tb else (K, N), 2).cuda(), randn((M, N), 3).cuda()
    out = pm.matmul(a, b, trans_b=tb, residual=r if res else None)
    assert pm.device_status() == 0
    want = a.double() @ (b.T if tb else b).double() + (r.double() if res else 0.0)
    assert_close(out, want, tol=3e-5, what=f"{M}x{N}x{K}")


# kernels that start while the one before them in the stream is still at work wait for it before they touch memory: calls one after the
# other on buffers that each of them overwrites give what they give one at a time (the sums have fixed orders: equal bits)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D,H,P,N,B,T,Q", [(128, 8, 32, 16, 2, 128, 64), (256, 8, 64, 64, 2, 300, 128), (768, 24, 64, 64, 1, 640, 256)])
def test_calls_one_after_the_other(pm, dtype, D, H, P, N, B, T, Q):
    _, _, blk = _block(pm, D, H, P, N, 1, Q, dtype)
    xs, cots = [randn((B, T, D), 5 + i).cuda().to(dtype) for i in range(4)], [randn((B, T, D), 15 + i).cuda().to(dtype) for i in range(4)]

    def call(i):
        return blk.forward(xs[i], residual=xs[i]), *blk.backward(xs[i], cots[i])
    want = []
    for i in range(4):
        want.append(call(i))
        torch.cuda.synchronize()
    for _ in range(5):
        for i, got in enumerate([call(i) for i in range(4)]):
            assert torch.equal(got[0], want[i][0]) and torch.equal(got[1], want[i][1])
            assert all(torch.equal(got[2][k], want[i][2][k]) for k in got[2])
    assert pm.device_status() == 0


# more chains than the machine has SMs: those of a last round that fills less than a third of it are walked in segments beside the others
# (one chain more than a round, a few, just under a third; just over and two full rounds, which stay whole)
@pytest.mark.parametrize("B,H", [(149, 1), (19, 8), (24, 8), (25, 8), (37, 8)])
@pytest.mark.parametrize("T", [770, 896])
def test_scan_last_round_in_segments(pm, B, H, T):
    P, N, G = 16, 24, 1
    x, b, c, dy = randn((B, T, H, P), 1).bfloat16(), randn((B, T, G, N), 2).bfloat16(), randn((B, T, G, N), 3).bfloat16(), randn((B, T, H, P), 4).bfloat16()
    a = -torch.nn.functional.softplus(randn((B, T, H), 5) - 2.0)
    init = randn((B, H, N, P), 6)
    scan = pm.SsdScanBf16(x.cuda(), a.cuda(), b.cuda(), c.cuda(), 128)
    y, last = scan.forward(init_state=init.cuda(), want_final_state=True)
    scan.forward()
    dx, da, db, dc = scan.backward(dy.cuda())
    torch.cuda.synchronize()
    assert pm.device_status() == 0
    leaves = [t.float().requires_grad_(True) for t in (x, a, b, c)]
    be, ce = (t.expand(B, T, H, N) for t in leaves[2:])
    orc.ssd_scan_chunked(leaves[0], leaves[1], be, ce, T // 7, return_final_state=True)[0].backward(dy.float())
    with torch.no_grad():
        ref, ref_last = orc.ssd_scan_chunked(leaves[0], leaves[1], be, ce, T // 7, initial_state=init, return_final_state=True)
    for got, want, tol, what in ((y.float(), ref, 5e-3, "y"), (last, ref_last, 5e-3, "final state"), (dx.float(), leaves[0].grad, 5e-3, "dx"), (da, leaves[1].grad, 5e-3, "da"),
                                 (db.float(), leaves[2].grad, 5e-3, "db"), (dc.float(), leaves[3].grad, 5e-3, "dc")):
        assert_close(got, want, tol=tol, what=what)


# the launches of such a call overlap one another and the next call's: the same bits as with the device idle in between, and in a graph
@pytest.mark.parametrize("B", [19, 24])
def test_scans_in_segments_back_to_back(pm, B):
    T, H, P, N = 896, 8, 16, 24
    scans = []
    for k in range(2):
        x, b, c, dy = (randn(sh, 10 * k + i).bfloat16().cuda() for i, sh in enumerate([(B, T, H, P), (B, T, 1, N), (B, T, 1, N), (B, T, H, P)]))
        a = -torch.nn.functional.softplus(randn((B, T, H), 10 * k + 5) - 2.0).cuda()
        scans.append((pm.SsdScanBf16(x, a, b, c, 128), dy))

    def run(pause):
        out = []
        for _ in range(3):
            for scan, dy in scans:
                out.append(scan.forward())
                pause()
                out.extend(scan.backward(dy))
                pause()
        torch.cuda.synchronize()
        return out

    want = run(torch.cuda.synchronize)
    for got, ref in zip(run(lambda: None), want):
        assert torch.equal(got, ref)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        for scan, dy in scans:
            scan.forward(); scan.backward(dy)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        out = [t for scan, dy in scans for t in (scan.forward(), *scan.backward(dy))]
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    for got, ref in zip(out, want):
        assert torch.equal(got, ref)
    assert pm.device_status() == 0


@pytest.mark.parametrize("B", [19, 24])
def test_block_last_round_in_segments(pm, B):
    D, H, P, N, T, Q = 64, 8, 16, 16, 770, 64
    cfg, p, blk = _block(pm, D, H, P, N, 1, Q, torch.float32)
    x, cot = randn((B, T, D), 5), randn((B, T, D), 6)
    out = blk.forward(x.cuda())
    dx, grads = blk.backward(x.cuda(), cot.cuda())
    torch.cuda.synchronize()
    assert pm.device_status() == 0
    leaves = {k: v.clone().requires_grad_(True) for k, v in p.items()}
    xr = x.clone().requires_grad_(True)
    ref = orc.block_forward(leaves, cfg, xr)
    ref.backward(cot)
    assert_close(out, ref.detach(), what="out")
    assert_close(dx, xr.grad, what="dx")
    for k, g in grads.items():
        # (the sums for a_log and dt_bias cancel over 15000 tokens: 1.9e-4 and 2.2e-4 from fp64 also with 144 chains, which stay whole)
        assert_close(g, leaves[k].grad, tol=5e-4 if k in ("a_log", "dt_bias") else FP32_TOL, what=k)


# rows of the pooling, the shifted repeat and their adjoints, and the token rows' gradient: a part of a warp, a warp and a bit, two blocks
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [8, 136, 1032])
def test_two_level_widths(pm, D, dtype):
    B, T, V, group = 2, 24, 50, 4
    cfg = orc.Mamba2Config(d_model=D, d_state=8, d_head=8, n_heads=8, block_len=24)
    layers = [block_params(cfg, seed=30 + i) for i in range(2)]
    embed, wproj = randn((V, D), 9, 0.5), randn((D, D), 10, D ** -0.5)
    ids, tg, _ = orc.lcg_batch(11, B, T, V)
    er, wr, ls = embed.clone().requires_grad_(True), wproj.clone().requires_grad_(True), [{k: v.clone().requires_grad_(True) for k, v in p.items()} for p in layers]
    ref = orc.hier_lm_loss(er, wr, ls[:1], ls[1:], cfg, ids, tg, group=group)
    ref.backward()
    lm = pm.FlatMamba(pm.Mamba2Config(d_model=D, d_state=8, d_head=8, n_heads=8, block_len=24), 1, V, B, T, compute_dtype=dtype, level1_layers=1, group=group)
    lm.load(embed.cuda(), [cuda_params(p) for p in layers], wproj=wproj.cuda())
    loss = lm.step_device(ids.cuda(), tg.cuda())
    tol = 1e-4 if dtype == torch.float32 else 5e-2       # (the reference's bound for gradients in bf16)
    assert abs(float(loss) - float(ref)) < tol * abs(float(ref))
    assert_close(lm.grads()[0], er.grad, tol=tol, what="d_embed")
    assert_close(lm.view(lm.flat_grads, -2), wr.grad, tol=tol, what="d_wproj")
    assert pm.device_status() == 0
    lm.close()


# the backward of whole chunks on plain operands (csrc/ssd_dx.cu): one and several row blocks to a chunk, one chunk, B and C per head, more
# CTAs than fit the machine at once, and a decay that underflows inside a block of columns.  bf16 operands and storage: 2e-2.
@pytest.mark.parametrize("B,T,Q", [(1, 128, 128), (2, 256, 256), (2, 768, 128), (3, 1024, 256), (2, 4096, 256)])
@pytest.mark.parametrize("G,decay", [(1, 0.0), (1, 3.0), (8, 0.0)])
def test_block_bf16_backward_of_chunks(pm, B, T, Q, G, decay):
    cfg, p, blk = _block(pm, 256, 8, 64, 64, G, Q, torch.bfloat16)
    p["a_log"] = p["a_log"] + decay
    blk = pm.Mamba2Block(blk.config, {k: v.cuda() for k, v in p.items()}, compute_dtype=torch.bfloat16)
    x, cot = randn((B, T, 256), 32).bfloat16(), randn((B, T, 256), 33).bfloat16()
    leaves = {k: v.clone().requires_grad_(True) for k, v in p.items()}
    xr = x.float().requires_grad_(True)
    orc.block_forward(leaves, cfg, xr).backward(cot.float())
    dx, grads = blk.backward(x.cuda(), cot.cuda())
    assert_close(dx.float(), xr.grad, tol=2e-2, what="dx")
    for k, v in leaves.items():
        assert_close(grads[k], v.grad, tol=2e-2, what=k)
    assert pm.device_status() == 0


# more chains than SMs: every SM takes an equal stretch of all chains' steps, and the state of a chain that two SMs share goes through memory.
# Bit by bit what the same sequences give one batch at a time, where each chain is walked whole; twice, and in a graph.  (db and dc are sums over
# heads in an order that depends on the number of batches, rounded to bf16: two of them lie one step apart, at most 2^-7 of the value.)
@pytest.mark.parametrize("B,H,T,P,N,Q", [(2, 80, 512, 64, 64, 128), (2, 80, 700, 64, 128, 128), (3, 100, 640, 64, 128, 128), (2, 75, 513, 8, 8, 64),
                                         (2, 140, 1024, 64, 64, 256), (7, 96, 512, 32, 64, 512), (4, 76, 1200, 64, 64, 256)])
def test_scan_of_more_chains_than_sms(pm, B, H, T, P, N, Q):
    x, b, c, dy = (randn(s, i).bfloat16().cuda() for i, s in enumerate([(B, T, H, P), (B, T, 1, N), (B, T, 1, N), (B, T, H, P)]))
    a = (-torch.nn.functional.softplus(randn((B, T, H), 5) - 1.0)).cuda()
    init = randn((B, H, N, P), 6).cuda()
    scan = pm.SsdScanBf16(x, a, b, c, Q)

    def call(s, dy, init):
        y, last = s.forward(init, True)
        return y, last, *s.backward(dy)

    want = [torch.cat(v) for v in zip(*(call(pm.SsdScanBf16(x[i:i + 1], a[i:i + 1], b[i:i + 1], c[i:i + 1], Q), dy[i:i + 1], init[i:i + 1]) for i in range(B)))]
    side, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    got = [call(scan, dy, init) for _ in range(2)]
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(g, stream=side):
        got.append(call(scan, dy, init))
    for _ in range(2):
        g.replay()
    torch.cuda.synchronize()
    assert pm.device_status() == 0
    for run in got:
        for u, v, what in zip(run, want, ("y", "last", "dx", "da", "db", "dc")):
            if what in ("db", "dc"):
                assert_close(u.float(), v.float(), tol=2.0 ** -7, what=what)
            else:
                assert torch.equal(u, v), what


# the same inside bf16-storage blocks, with what a backward reads (chunks of one and of two steps).  dx: the sums over heads and the recompute of
# half the batch take other orders there, bf16 storage's own tolerance.
@pytest.mark.parametrize("B,T,Q", [(8, 1024, 256), (7, 768, 256), (7, 1280, 128)])
def test_bf16_block_of_more_chains_than_sms(pm, B, T, Q):
    cfg = pm.Mamba2Config(d_model=256, d_state=64, d_head=64, n_heads=24, n_groups=1, d_conv=4, block_len=Q)
    p = {k: v.cuda() for k, v in orc.init_block_params(orc.Mamba2Config(256, 64, 64, 24, 1, 4, Q), seed=3).items()}
    blk = pm.Mamba2Block(cfg, p, compute_dtype=torch.bfloat16)
    x, dout = randn((B, T, 256), 1).bfloat16().cuda(), randn((B, T, 256), 2).bfloat16().cuda()
    out = blk.forward(x)
    dx, _ = blk.backward(x, dout)
    half = B // 2                              # 72 or 96 chains: each walked whole
    for lo, hi in ((0, half), (half, B)):
        assert torch.equal(out[lo:hi], blk.forward(x[lo:hi].contiguous()))
        assert_close(dx[lo:hi].float(), blk.backward(x[lo:hi].contiguous(), dout[lo:hi].contiguous())[0].float(), tol=2e-2, what="dx")
    assert pm.device_status() == 0


# the sums of in_proj's K splits with the conv step: four columns to a thread where the window and the conv weights lie on the 16-byte grid and
# the taps are four, a column to a thread elsewhere.  Against the oracle's step, as above.
@pytest.mark.parametrize("K,offset", [(4, 0), (4, 1), (3, 0), (2, 0)])
@pytest.mark.parametrize("B,N", [(17, 64), (33, 4), (200, 128)])
def test_decode_finish(pm, B, N, K, offset):
    cfg = orc.Mamba2Config(64, N, 32, 4, 1, K, 64)
    p = orc.init_block_params(cfg, seed=5)
    blk = pm.Mamba2Block(pm.Mamba2Config(d_model=64, d_state=N, d_head=32, n_heads=4, n_groups=1, d_conv=K, block_len=64), {k: v.cuda() for k, v in p.items()})
    st, st_o = blk.zero_state(B), orc.zero_state(cfg, B)
    win = torch.empty(st["conv_window"].numel() + offset, device="cuda")[offset:].view_as(st["conv_window"])
    win.copy_(randn(tuple(win.shape), 2).cuda())
    st["conv_window"] = win
    st_o["conv_window"] = win.cpu().clone()
    for t in range(2):
        x = randn((B, 1, 64), 10 + t)
        y, st = blk.step(x.cuda(), st)
        y_o, st_o = orc.block_step(p, cfg, x, st_o)
        assert_close(y, y_o, what="y")
        assert_close(st["conv_window"], st_o["conv_window"], what="window")


# the states that a backward reads leave in boxes of 32 rows: d_state at and around the boxes' edges, d_head below the box's width (a box that wrote
# past its state would change the next head's).  On bf16 (several chunks of 128) and as pairs (a ragged length); bounds as in the tests above.
@pytest.mark.parametrize("N,P", [(8, 8), (24, 64), (32, 40), (40, 64), (64, 56), (72, 64), (96, 24), (104, 8), (128, 64)])
@pytest.mark.parametrize("T", [384, 300])
def test_scan_bf16_kept_states(pm, T, N, P):
    B, H, G = 2, 6, 1
    x, b, c, dy = randn((B, T, H, P), 1).bfloat16(), randn((B, T, G, N), 2).bfloat16(), randn((B, T, G, N), 3).bfloat16(), randn((B, T, H, P), 4).bfloat16()
    a = -torch.nn.functional.softplus(randn((B, T, H), 5) - 2.0)
    scan = pm.SsdScanBf16(x.cuda(), a.cuda(), b.cuda(), c.cuda(), 128)
    scan.forward()
    dx, da, db, dc = scan.backward(dy.cuda())
    assert pm.device_status() == 0
    leaves = [t.double().requires_grad_(True) for t in (x, a, b, c)]
    orc.ssd_scan_chunked(leaves[0], leaves[1], *(t.expand(B, T, H, N) for t in leaves[2:]), 128 if T % 128 == 0 else T).backward(dy.double())
    for got, ref, tol, what in ((dx.float(), leaves[0].grad, 5e-3, "dx"), (da, leaves[1].grad, 5e-3, "da"), (db.float(), leaves[2].grad, 5e-3, "db"), (dc.float(), leaves[3].grad, 5e-3, "dc")):
        assert_close(got, ref, tol=tol, what=what)


# decays between e^-92 and e^-88, below the smallest normal number: every second x and every other dY are zero, so that rows of the results consist of such
# terms alone.  A masked element is kept in bf16 (pairs), whose steps there are 2^-133: 2^-134 |x| of a result's largest, 3e-37, and a bf16 result's 2^-9.
@pytest.mark.parametrize("dtype,T,N,Q", [(torch.float32, 256, 64, 128), (torch.float32, 512, 64, 256), (torch.bfloat16, 256, 64, 128), (torch.bfloat16, 512, 128, 256),
                                         (torch.bfloat16, 200, 64, 128)])
def test_scan_of_subnormal_decays(pm, dtype, T, N, Q):
    B, H, P = 2, 4, 64
    x, b, c, dy = (randn(s, i + 1).to(dtype) for i, s in enumerate([(B, T, H, P), (B, T, 1, N), (B, T, 1, N), (B, T, H, P)]))
    x[:, 1::2] = 0
    dy[:, 0::2] = 0
    a = -88.0 - 4.0 * rand((B, T, H), 5)
    scan = (pm.SsdScan if dtype == torch.float32 else pm.SsdScanBf16)(x.cuda(), a.cuda(), b.cuda(), c.cuda(), Q if T % Q == 0 else T)
    y = scan.forward()
    _, da, db, dc = scan.backward(dy.cuda())
    assert pm.device_status() == 0
    leaves = [t.double().requires_grad_(True) for t in (x, a, b, c)]
    ref = orc.ssd_scan_chunked(leaves[0], leaves[1], *(t.expand(B, T, H, N) for t in leaves[2:]), Q if T % Q == 0 else T)
    ref.backward(dy.double())
    for got, want, what in ((y[:, 1::2], ref[:, 1::2], "y"), (da, leaves[1].grad, "da"), (db, leaves[2].grad, "db"), (dc, leaves[3].grad, "dc")):
        assert_close(got.float(), want, tol=5e-3, what=what)


# the same in the backward of whole chunks on plain operands (csrc/ssd_dx.cu): d_a_log is a sum of such terms.  The reference takes the diagonal, which does
# not depend on the decays, by itself: its row and column sums would leave 1e-16 of it.
@pytest.mark.parametrize("T,Q", [(128, 128), (256, 256), (512, 256)])
def test_block_bf16_backward_of_subnormal_decays(pm, monkeypatch, T, Q):
    def scan(x, a, b, c, block_len):
        S = torch.cumsum(a, 1).transpose(1, 2)
        below = torch.ones(T, T, dtype=torch.bool).tril(-1)
        G = torch.einsum("bthn,bshn->bhts", c, b)
        M = G * torch.exp((S.unsqueeze(3) - S.unsqueeze(2)).masked_fill(~below, -float("inf"))) + G * torch.eye(T, dtype=G.dtype)
        return torch.einsum("bhts,bshp->bthp", M, x)

    cfg, p, blk = _block(pm, 256, 8, 64, 64, 1, Q, torch.bfloat16)
    p["in_proj_weight"][:, -cfg.n_heads:] = 0                       # dt = softplus(0.5413) = 1 everywhere
    p["dt_bias"].fill_(0.541324854612918)
    p["a_log"] = torch.log(88.5 + torch.arange(cfg.n_heads) * 0.25)
    blk = pm.Mamba2Block(blk.config, {k: v.cuda() for k, v in p.items()}, compute_dtype=torch.bfloat16)
    x, cot = randn((2, T, 256), 32).bfloat16(), (randn((2, T, 256), 33) * 1e4).bfloat16()
    _, grads = blk.backward(x.cuda(), cot.cuda())
    monkeypatch.setattr(orc, "ssd_scan_ops_default", scan)
    leaves = {k: v.double().requires_grad_(True) for k, v in p.items()}
    orc.block_forward(leaves, cfg, x.double()).backward(cot.double())
    assert float(leaves["a_log"].grad.abs().max()) < 1e-30
    assert_close(grads["a_log"], leaves["a_log"].grad, tol=2e-2, what="d_a_log")
    assert pm.device_status() == 0


# more chains than SMs where every head has its own B and C, while another stream's kernels hold SMs that the first blocks would be placed on: the same bits
# as whole walks of a batch at a time (no sums over heads here)
@pytest.mark.parametrize("B,H,T,P,N,Q", [(2, 80, 512, 64, 64, 128), (3, 64, 700, 64, 128, 128)])
def test_scan_of_more_chains_than_sms_beside_another_stream(pm, B, H, T, P, N, Q):
    x, b, c, dy = (randn(s, i).bfloat16().cuda() for i, s in enumerate([(B, T, H, P), (B, T, H, N), (B, T, H, N), (B, T, H, P)]))
    a = (-torch.nn.functional.softplus(randn((B, T, H), 5) - 1.0)).cuda()

    def call(i, j):
        s = pm.SsdScanBf16(x[i:j], a[i:j], b[i:j], c[i:j], Q)
        return s.forward(), *s.backward(dy[i:j])

    want = [torch.cat(v) for v in zip(*(call(i, i + 1) for i in range(B)))]
    other, m = torch.cuda.Stream(), torch.randn(4096, 4096, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(other):
        for _ in range(8):
            m = torch.tanh(m @ m)
    got = [call(0, B) for _ in range(4)]
    torch.cuda.synchronize()
    assert pm.device_status() == 0
    for run in got:
        for u, v, what in zip(run, want, ("y", "dx", "da", "db", "dc")):
            assert torch.equal(u, v), what
