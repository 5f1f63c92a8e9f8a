"""Sanity tier: every module of the package (and its ``verl`` alias) imports on a CPU-only box, public names resolve,
and the native sources carry a binding for every exported entry point that Python calls."""

import importlib
import pkgutil
import re
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_every_module_imports():
    import verl_b200

    failed = []
    for m in pkgutil.walk_packages(verl_b200.__path__, "verl_b200."):
        if m.name.endswith("__main__"):
            continue
        try:
            importlib.import_module(m.name)
        except BaseException as e:  # noqa: BLE001
            failed.append((m.name, repr(e)[:200]))
    assert not failed, failed


def test_alias_covers_every_module():
    import verl  # noqa: F401
    import verl_b200

    for m in pkgutil.walk_packages(verl_b200.__path__, "verl_b200."):
        if m.name.endswith("__main__") or "._" in m.name:
            continue
        alias = importlib.import_module("verl." + m.name[len("verl_b200."):])
        real = importlib.import_module(m.name)
        if alias is not real:  # a package-shaped view (the reference splits this module into sub-modules)
            for k, v in vars(real).items():
                if not k.startswith("_"):
                    assert getattr(alias, k) is v, (m.name, k)


def test_python_calls_only_exported_native_functions():
    """Every ``vb_*`` name used from Python exists as an ``extern "C"`` definition in the native sources."""
    defined = set()
    for src in list((ROOT / "verl_b200" / "csrc").glob("*.cu")) + list((ROOT / "verl_b200" / "csrc").glob("*.cpp")):
        defined |= set(re.findall(r"\b(vb_[a-z0-9_]+)\s*\(", src.read_text()))
    used = set()
    for py in (ROOT / "verl_b200").rglob("*.py"):
        used |= set(re.findall(r"""["'.](vb_[a-z0-9_]+)""", py.read_text()))
    missing = sorted(u for u in used if u not in defined)
    assert not missing, missing


def test_kernels_that_start_early_use_no_read_only_loads():
    """A kernel that waits for the one before it (``pdl_wait``) has begun while that one still writes: what it reads of it may not go
    through loads that promise memory nobody writes. Model weights and position tables, which no such kernel writes, may."""
    constant = {"w", "qw", "kw", "cos_t", "sin_t", "post"}
    found, seen = [], 0
    for name in ("elementwise.cu", "fp8_gemm.cu", "gemm_skinny.cu", "moe_ops.cu", "paged_attention.cu", "paged_attention_mma.cu"):
        src = (ROOT / "verl_b200" / "csrc" / name).read_text()
        for kernel in src.split("__global__")[1:]:
            kernel = kernel.split("\n}\n")[0]
            head, _, body = kernel.partition("{\n")
            if "pdl_wait()" not in body:
                continue
            seen += 1
            params = re.findall(r"const [\w:]+\*\s*__restrict__\s+(\w+)", head)
            found += [(name, head.split("(")[0].split()[-1], p) for p in params if p not in constant]
            if "ld_stream(" in body:
                body += src.split("uint4 ld_stream(")[1].split("\n}\n")[0]
                assert "asm volatile" in body and '"memory"' in body
            found += [(name, w) for w in ("__ldg(", "ld.global.nc") if w in body]
    assert seen >= 12 and not found, (seen, found)


def test_imports_with_a_torch_that_has_no_cuda():
    code = """
import torch
for name in [n for n in vars(torch._C) if n.startswith("_cuda_")]:
    delattr(torch._C, name)
import verl_b200.ops, verl_b200.models
x = torch.randn(3, 8)
assert torch.equal(verl_b200.ops.swiglu(x), torch.nn.functional.silu(x[:, :4]) * x[:, 4:])
"""
    done = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]


def test_short_cuts_are_off_where_something_follows_the_computation():
    import torch
    from torch.autograd import forward_ad

    from verl_b200.ops import _lib

    assert not _lib.plain() and not _lib.followed()
    seen = []
    with torch.no_grad():
        assert _lib.plain()
        torch.jit.trace(lambda x: (seen.append((_lib.plain(), _lib.followed())), x + 1)[1], torch.ones(2), check_trace=False)
        with forward_ad.dual_level():
            seen.append((_lib.plain(), _lib.followed()))
        assert _lib.plain()
    assert seen == [(False, True), (False, True)]


def test_threads_share_one_word_for_refused_indices(monkeypatch):
    """Kernels keep its address: a second one made at the same time would leave the first to the allocator's next user."""
    import threading
    import time

    import torch

    from verl_b200.ops import _lib

    made = []

    def slow_zeros(*size, dtype, pin_memory, _zeros=torch.zeros):
        time.sleep(0.05)
        made.append(_zeros(*size, dtype=dtype))
        return made[-1]

    monkeypatch.setattr(_lib, "_refused", None)
    monkeypatch.setattr(torch, "zeros", slow_zeros)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    got = []
    threads = [threading.Thread(target=lambda: got.append(_lib.refused_word())) for _ in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(made) == 1 and got == [made[0].data_ptr()] * 8
