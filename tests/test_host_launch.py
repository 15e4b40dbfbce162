"""The native launch functions: what they refuse, and operand layouts against contiguous operands (bit for bit)."""
import re
import threading
from pathlib import Path

import pytest
import torch

from torchturbo_b200 import kernels as K


def test_wrong_arguments_are_refused():
    x = torch.zeros(8, 64, dtype=torch.bfloat16)
    with pytest.raises(AssertionError):
        K.gemm(x.float(), x)
    with pytest.raises(AssertionError):
        K.gemm(x, x, out_dtype=torch.float16)
    with pytest.raises(TypeError):
        K.host().rope(x)
    with pytest.raises(TypeError):
        K.host().rmsnorm_fwd(x, None, 1e-6, None, False)
    with pytest.raises(TypeError):
        K.host().rmsnorm_fwd(x, x, "eps", None, False)


def test_declared_once():
    """Both sides of the C interface see one declaration, so that a change of one of them alone does not compile."""
    csrc = Path(K.__file__).parent / "csrc"
    text = {p.name: p.read_text() for p in [*csrc.glob("*.cu"), *csrc.glob("*.cuh"), *csrc.glob("*.h"), *csrc.glob("*.cpp")]}
    assert [name for name, t in text.items() if re.search(r"struct GemmArgs\s*\{", t)] == ["entries.h"]
    assert '#include "entries.h"' in text["common.cuh"] and '#include "entries.h"' in text["host.cpp"]
    declared = set(re.findall(r"\b(ttb_\w+)\(", text["entries.h"]))
    called = set(re.findall(r"return (ttb_\w+)\(", text["host.cpp"]))
    defined = {name for f, t in text.items() if f.endswith(".cu") for name in re.findall(r"^TTB_EXPORT int (ttb_\w+)\(", t, re.M)}
    assert called == declared and declared <= defined and not re.search(r"\bttb_\w+\([^;{]*\);\s*$", text["host.cpp"].split("namespace {")[0], re.M)


@pytest.mark.parametrize("flags", ["NVCC_FLAGS", "FAST_MATH", "HOST_FLAGS", "HOST_LIBS"])
def test_built_again_when_a_flag_changes(flags, monkeypatch):
    from torchturbo_b200.csrc import build

    before = build._digest(build.sources())
    monkeypatch.setattr(build, flags, [*getattr(build, flags), "-DOTHER"])
    assert build._digest(build.sources()) != before
    if flags.startswith("HOST"):
        assert "-DOTHER" in build._host_command()


def _calls(rows, cols):
    g = torch.Generator("cuda").manual_seed(rows)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()                                # noqa: E731
    x, dy, res, w, b = rnd(rows, cols), rnd(rows, cols), rnd(rows, cols), rnd(cols), rnd(cols)
    _, rstd, _ = K.rmsnorm_fwd(x, w, 1e-6)
    _, mean, lstd = K.layernorm_fwd(x, w, b, 1e-6)
    return x, dy, res, {
        "rmsnorm_fwd": lambda x, dy, res: K.rmsnorm_fwd(x, w, 1e-6, res),
        "rmsnorm_bwd": lambda x, dy, res: K.rmsnorm_bwd(dy, x, w, rstd, res, dw_dtype=torch.bfloat16),
        "layernorm_fwd": lambda x, dy, res: K.layernorm_fwd(x, w, b, 1e-6),
        "layernorm_bwd": lambda x, dy, res: K.layernorm_bwd(dy, x, w, mean, lstd),
        "bias_act_fwd": lambda x, dy, res: K.bias_act_fwd(x, b, "gelu_tanh", res),
        "bias_act_bwd": lambda x, dy, res: K.bias_act_bwd(dy, x, b, "gelu_tanh"),
    }


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(1, 64), (61, 2048), (300, 1152)])
def test_layouts(rows, cols):
    """Columns first, rows further apart, one row for all, three dimensions, a side stream and another thread."""
    x, dy, res, calls = _calls(rows, cols)
    forms = {
        "columns": lambda t: t.t().contiguous().t(),
        "apart": lambda t: torch.cat([t, t], 1)[:, :cols],
        "leading": lambda t: t[None],
    }
    for name, call in calls.items():
        want = call(x, dy, res)
        want = want if isinstance(want, tuple) else (want,)

        def same(got, what):
            got = got if isinstance(got, tuple) else (got,)
            for a, b in zip(want, got):
                assert a.dtype == b.dtype and bool((a.reshape(-1) == b.reshape(-1)).all()), (name, what)

        for form, make in forms.items():
            got = call(make(x), make(dy), make(res))
            same(got, form)
            first = got[0] if isinstance(got, tuple) else got
            assert first.shape == make(x).shape and first.is_contiguous()
        row = dy[:1].expand(rows, cols)
        a, b = call(x, row, res), call(x, row.contiguous(), res)
        for u, v in zip(a if isinstance(a, tuple) else (a,), b if isinstance(b, tuple) else (b,)):
            assert bool((u == v).all()), (name, "one row for all")
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            got = call(x, dy, res)
        torch.cuda.current_stream().wait_stream(side)
        same(got, "side stream")
        box = []
        t = threading.Thread(target=lambda: (box.append(call(x, dy, res)), torch.cuda.synchronize()))
        t.start()
        t.join()
        same(box[0], "thread")


@pytest.mark.gpu
def test_tensors_without_storage_are_an_error_and_not_a_crash():
    """Batched gradients have no address: the launch function finds out while it holds no interpreter lock."""
    x = torch.randn(16, 64, device="cuda").bfloat16()
    seen = []

    class Probe(torch.autograd.Function):
        @staticmethod
        def forward(ctx, t):
            return t.float().sum()

        @staticmethod
        def backward(ctx, g):
            with pytest.raises(RuntimeError):
                K.scale(x, g, torch.bfloat16)
            with pytest.raises((RuntimeError, AssertionError)):
                K.gemm(x * g.bfloat16(), x)
            seen.append(True)
            return x * g.bfloat16()

    leaf = x.clone().requires_grad_(True)
    torch.autograd.grad(Probe.apply(leaf), leaf, torch.tensor([1.0, 2.0], device="cuda"), is_grads_batched=True)
    assert seen
    assert K.gemm(x, x).shape == (16, 16)
