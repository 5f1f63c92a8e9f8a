"""Keeping layer activations instead of recomputing them gives the same step (2 gloo ranks, ZeRO-3)."""

import os
import subprocess
import sys


def test_kept_activations_match_recomputation():
    here = os.path.dirname(os.path.abspath(__file__))
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node=2", "--master-addr", "127.0.0.1",
           "--master-port", str(29950 + os.getpid() % 300), os.path.join(here, "_keep_act_worker.py")]
    env = {k: v for k, v in os.environ.items() if k != "VERL_B200_KEEP_ACTIVATION_LAYERS"}
    r = subprocess.run(cmd, capture_output=True, text=True, timeout=600, env=env)
    assert r.returncode == 0 and "KEEP_ACT_OK" in r.stdout, (r.stdout[-2000:], r.stderr[-4000:])


def test_out_of_memory_in_a_training_forward_falls_back_to_recomputation(monkeypatch):
    """Single rank: an OOM raised while layers keep their activations is answered by one repeat of the forward with
    every layer recomputed (and the policy stays off); the step then matches a plain recomputing step."""
    import torch

    from verl_b200.models import preset
    from verl_b200.models.transformer import PackedBatch
    from verl_b200.parallel import zero as zmod
    from verl_b200.workers.engine.native import NativeEngine

    class C(dict):
        __getattr__ = dict.get

    cfg = preset("tiny-qwen2")
    ids = torch.randint(3, cfg.vocab_size, (20,), generator=torch.Generator().manual_seed(0))
    batch = PackedBatch(ids, torch.arange(20), torch.tensor([0, 20], dtype=torch.int32), 20)
    rows, labels = torch.arange(19), ids[1:]

    def step(eng):
        with eng.train_mode():
            eng.optimizer_zero_grad()
            lp, _ = eng.forward_logprob(batch, rows, labels, 1.0)
            (-lp.mean()).backward()
            return eng.zero.grad.clone()

    ref = step(NativeEngine(cfg, C(keep_activation_layers="0"), C(lr=1e-3), device="cpu", seed=1).initialize())
    eng = NativeEngine(cfg, C(keep_activation_layers=str(cfg.num_hidden_layers)), C(lr=1e-3), device="cpu", seed=1).initialize()
    calls = {"n": 0}
    real = zmod._UnitFnKeep.forward

    def boom(ctx, *a):
        calls["n"] += 1
        raise torch.cuda.OutOfMemoryError("fake")

    monkeypatch.setattr(zmod._UnitFnKeep, "forward", staticmethod(boom))
    got = step(eng)
    monkeypatch.setattr(zmod._UnitFnKeep, "forward", real)
    assert calls["n"] == 1 and eng._keep_cap == 0 and eng._layers_to_keep(20) == 0
    torch.testing.assert_close(got, ref)


def test_second_backward_recomputes_a_kept_unit():
    """``retain_graph``: the kept graph of a unit serves one backward, a further one recomputes the unit and adds the same gradient."""
    import torch

    from verl_b200.models import preset
    from verl_b200.models.transformer import PackedBatch
    from verl_b200.workers.engine.native import NativeEngine

    cfg = preset("tiny-qwen2", tie_word_embeddings=False)
    ids = torch.randint(3, cfg.vocab_size, (20,), generator=torch.Generator().manual_seed(0))
    batch = PackedBatch(ids, torch.arange(20), torch.tensor([0, 20], dtype=torch.int32), 20)
    eng = NativeEngine(cfg, {"keep_activation_layers": cfg.num_hidden_layers}, {"lr": 1e-3}, device="cpu", seed=1).initialize()
    with eng.train_mode():
        eng.optimizer_zero_grad()
        lp, ent = eng.forward_logprob(batch, torch.arange(19), ids[1:], 1.0)
        loss = (ent - lp).mean()
        loss.backward(retain_graph=True)
        once = eng.zero.grad.clone()
        loss.backward()
    torch.testing.assert_close(eng.zero.grad, 2 * once)


def test_forwards_that_wait_for_their_backward_count_in_what_is_kept(monkeypatch):
    """Small micro-batches are kept without a look at the memory, but only one at a time: with several forwards before a backward the
    next one asks what is free."""
    import torch

    from verl_b200.models import preset
    from verl_b200.models.transformer import PackedBatch
    from verl_b200.workers.engine.native import NativeEngine

    cfg = preset("tiny-qwen2")
    ids = torch.randint(3, cfg.vocab_size, (20,), generator=torch.Generator().manual_seed(0))
    batch = PackedBatch(ids, torch.arange(20), torch.tensor([0, 20], dtype=torch.int32), 20)
    eng = NativeEngine(cfg, {}, {"lr": 1e-3}, device="cpu", seed=1).initialize()
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device=None: (1 << 30, 180 << 30))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda device=None: 0)
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda device=None: 0)

    def layers_kept():  # as the engine decides on a GPU with 1 GB left
        monkeypatch.setattr(eng, "device", torch.device("cuda", 0))
        n = eng._layers_to_keep(20)
        monkeypatch.setattr(eng, "device", torch.device("cpu"))
        return n

    def forward():
        return -eng.forward_logprob(batch, torch.arange(19), ids[1:], 1.0)[0].mean()

    with eng.train_mode():
        monkeypatch.setattr(eng, "engine_config", {"keep_activation_layers": cfg.num_hidden_layers})
        eng.optimizer_zero_grad()
        losses = [forward()]
        monkeypatch.setattr(eng, "engine_config", {})
        assert layers_kept() == 0
        losses.append(forward())
        losses[0].backward()
        assert layers_kept() == 0  # the second one's head still waits
        losses[1].backward()
        assert layers_kept() == cfg.num_hidden_layers
        forward()  # nobody goes back through it
        assert layers_kept() == 0
        eng.optimizer_zero_grad()
        assert layers_kept() == cfg.num_hidden_layers
