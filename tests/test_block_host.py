"""What a block object keeps on the host between calls: the library is replaced by a recorder, no kernel is launched."""
import copy
import pickle
import threading

import pytest
import torch


class Recorder:
    """Stands in for the library: notes the workspace that each step was handed."""

    def __init__(self):
        self.steps = []
        self.inside = threading.Barrier(1)

    def pmb_mamba2_step_workspace_bytes(self, cfg, batch):
        return 256 * batch

    def pmb_mamba2_block_workspace_bytes(self, cfg, batch, seqlen):
        return 64 * batch * seqlen

    pmb_stack_workspace_bytes = pmb_mamba2_block_workspace_bytes

    def pmb_mamba2_block_fwd(self, stream, cfg, params, batch, seqlen, x, residual, out, ws, n):
        self.steps.append((threading.get_ident(), ws, n))
        self.inside.wait(10)
        return 0

    def pmb_stack_fwd_ckpt(self, stream, cfg, layers, params, batch, seqlen, saved, ws, n):
        return self.pmb_mamba2_block_fwd(stream, cfg, params, batch, seqlen, saved, None, None, ws, n)

    def pmb_stack_bwd(self, stream, cfg, layers, params, grads, batch, seqlen, saved, dh, ws, n, cb, user):
        return self.pmb_mamba2_block_fwd(stream, cfg, params, batch, seqlen, saved, None, None, ws, n)

    def pmb_mamba2_step(self, stream, cfg, params, batch, x, state, window, y, ws, n):
        self.config, self.params = cfg._obj, params._obj
        self.steps.append((threading.get_ident(), ws, n))
        self.inside.wait(10)
        return 0


@pytest.fixture
def pm(monkeypatch):
    import __graft_entry__ as ge
    ge.build()
    import pm_b200
    monkeypatch.setattr(pm_b200, "lib", Recorder())
    monkeypatch.setattr(pm_b200, "_dev", lambda t, name: t)
    monkeypatch.setattr(pm_b200.Mamba2Block, "_io", lambda self, t, name: t)
    pm_b200.on_stream = 7
    monkeypatch.setattr(pm_b200, "_stream", lambda: pm_b200.on_stream)
    pm_b200.capturing = False
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: pm_b200.capturing)
    yield pm_b200
    del pm_b200.capturing, pm_b200.on_stream


def make(pm):
    cfg = pm.Mamba2Config(d_model=16, d_state=8, d_head=8, n_heads=2)
    return pm.Mamba2Block(cfg, {k: torch.ones(s) for k, s in cfg.param_shapes().items()})


def step(blk, batch=2, device="cpu"):
    blk.step(torch.zeros(batch, 1, 16, device=device), blk.zero_state(batch, device))


def test_captured_step_owns_its_workspace(pm):
    blk = make(pm)
    step(blk)                        # warm-up on the stream that captures
    pm.capturing = True
    held = []
    empty = torch.empty
    pm_ws = []

    def keep(*a, **k):               # (what the capture's pool does: memory handed out inside it stays with the graph)
        t = empty(*a, **k)
        held.append(t)
        pm_ws.append(t.data_ptr())
        return t
    torch.empty = keep
    try:
        step(blk)
    finally:
        torch.empty = empty
        pm.capturing = False
    captured = pm.lib.steps[-1][1]
    assert captured in pm_ws
    for batch in (2, *range(3, 14)):  # more keys than the object keeps, and the captured one's again
        step(blk, batch)
    step(blk)
    assert captured not in [ws for _, ws, _ in pm.lib.steps[2:]] and pm.lib.steps[0][1] != captured
    assert all(n == 256 * b for (_, _, n), b in zip(pm.lib.steps, (2, 2, 2, *range(3, 14), 2)))


def test_kept_workspaces_are_reused_and_bounded(pm):
    blk = make(pm)
    for _ in range(2):
        step(blk)
    assert pm.lib.steps[0][1] == pm.lib.steps[1][1]
    for batch in range(1, 40):
        step(blk, batch)
    assert len(blk._step_ws.__dict__) <= 8


def test_threads_do_not_share_a_workspace(pm):
    blk = make(pm)
    pm.lib.inside = threading.Barrier(2)             # both calls are inside the library at the same time
    threads = [threading.Thread(target=step, args=(blk,)) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    (a, wa, _), (b, wb, _) = pm.lib.steps
    assert a != b and wa != wb


def test_devices_do_not_share_a_workspace(pm):
    blk = make(pm)
    step(blk)
    step(blk, device="meta")                         # (data_ptr() of a meta tensor is 0)
    assert pm.lib.steps[0][1] != 0 and pm.lib.steps[1][1] == 0


def test_block_can_be_copied_and_pickled(pm):
    blk = make(pm)
    step(blk)
    for twin in (copy.deepcopy(blk), pickle.loads(pickle.dumps(blk)), copy.copy(blk)):
        step(twin)
        own = {k: getattr(pm.lib.params, k) for k in pm.PARAM_ORDER}
        assert own == {k: v.data_ptr() for k, v in twin.params.items()}
        assert pm.lib.steps[-1][1] != pm.lib.steps[0][1]             # workspaces stay with the object they came from
        assert twin.config == blk.config and pm.lib.config.d_model == 16


def test_edited_configuration_counts(pm):
    blk = make(pm)
    step(blk)
    assert pm.lib.config.rmsnorm_eps == pytest.approx(1e-5)
    blk.config.rmsnorm_eps = 1e-3
    step(blk)
    assert pm.lib.config.rmsnorm_eps == pytest.approx(1e-3)


def calls(pm, kind):
    """A function that makes one call of the kind at a sequence length, and the object that keeps its workspace."""
    blk = make(pm)
    if kind == "block":
        return lambda T: blk.forward(torch.zeros(1, T, 16))
    enc = pm.ContextEncoder(blk.config, [blk.params])
    if kind == "stack":
        return lambda T: enc.forward_checkpointed(torch.zeros(1, T, 16))
    return lambda T: enc.checkpoint_backward(torch.zeros(2, 1, T, 16), torch.zeros(1, T, 16))


@pytest.mark.parametrize("kind", ["block", "stack", "stack backward"])
def test_block_and_stack_workspaces(pm, kind):
    call = calls(pm, kind)
    used = lambda: pm.lib.steps[-1][1:]
    call(8)
    first = used()
    call(4)
    assert used() == first == (first[0], 64 * 8)     # kept, and large enough for less
    held, empty = [], torch.empty
    torch.empty = lambda *a, **k: held.append(empty(*a, **k)) or held[-1]
    try:
        pm.capturing = True
        call(8)
    finally:
        torch.empty, pm.capturing = empty, False
    captured = used()[0]
    assert captured != first[0] and captured in [t.data_ptr() for t in held]
    call(8)
    assert used() == first
    call(16)                                         # grows
    assert used()[1] == 64 * 16 and used()[0] != captured
    pm.on_stream = 9
    call(4)
    assert used()[1] == 64 * 4                       # another stream: not the large one, which stream 7 may still use


def test_block_workspace_on_two_threads(pm):
    call = calls(pm, "block")
    pm.lib.inside = threading.Barrier(2)
    threads = [threading.Thread(target=call, args=(8,)) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert pm.lib.steps[0][1] != pm.lib.steps[1][1]
