"""The layer's autograd node on the CPU, with the library calls replaced by recorders: what each call is handed."""
import pytest
import torch

from cute_mma_b200 import _functional as F
from cute_mma_b200 import _module

M, K, N, GS, RS = 24, 32, 64, 32, 8


@pytest.fixture
def calls(monkeypatch):
    """Plain eager calls on CPU tensors; the kernels return made-up numbers and remember their operands."""
    seen = {"n_dadr": 0}

    def forward(A, B, R, *args, **kw):
        seen["forward"] = dict(A=A, B=B, R=R, **kw)
        return torch.zeros(A.shape[0], B.shape[0], dtype=A.dtype), []

    def dadr(dC, A, B, R, gs, rs, gate, dc_scale, cfg=None, dR_dtype=None, internal_bias=None, **kw):
        assert torch._C._has_storage(dC), "a batch of gradients has no address"
        seen["dadr"] = dict(dC=dC, A=A, B=B, R=R, internal_bias=internal_bias, **kw)
        seen["n_dadr"] += 1
        out = torch.full(A.shape, float(dC.sum())), torch.ones(R.shape)
        return out if internal_bias is None else out + (torch.ones(internal_bias.shape),)

    def db(dC, A, R, gs, rs, gate, dc_scale, cfg=None, dB_dtype=None, internal_bias=None, **kw):
        seen["db"] = dict(dC=dC, A=A, R=R, internal_bias=internal_bias, **kw)
        return torch.ones(dC.shape[1], A.shape[1])

    monkeypatch.setattr(F, "forward", forward)
    monkeypatch.setattr(F, "_backward_dadr", dadr)
    monkeypatch.setattr(F, "_backward_db", db)
    monkeypatch.setattr(F, "bias_grad", lambda dC: dC.sum(0))
    monkeypatch.setattr(F, "cayley", lambda P, rs: P.clone())
    monkeypatch.setattr(F, "cayley_backward", lambda P, dP, rs: dP.clone())
    monkeypatch.setattr(_module, "_plain_eager", lambda *t: True)
    return seen


def _operands():
    return [torch.randn(*s, requires_grad=True) for s in ((M, K), (N, K), (N // GS * RS, K), (N // GS, K))]


def _layer(A, B, R, ib=None, act="silu_gate", cayley=False, seeds=None, p=0.0):
    return _module._layer_eager(A, B, R, None, ib, seeds, GS, RS, act, 1.0, p, None, cayley)


@pytest.mark.parametrize("cayley", [False, True])
def test_unpacked_tensors_reach_the_kernels_in_rows(calls, cayley):
    """Saved-tensor hooks may hand back views of another layout: the kernels take whole rows."""
    A, B, R, ib = _operands()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: torch.stack((t, -t), -1), lambda s: s[..., 0]):
        y = _layer(A, B, R, None if cayley else ib, "" if cayley else "silu_gate", cayley)
    y.sum().backward()
    given = list(calls["dadr"].values()) + list(calls.get("db", {}).values())
    assert all(t.is_contiguous() for t in given if isinstance(t, torch.Tensor))
    for name, t in (("A", A), ("B", B), ("R", R)):
        assert torch.equal(calls["dadr"][name], t.detach())


@pytest.mark.parametrize("which", [0, 1, 2])
def test_strided_operands_are_saved_themselves(calls, which):
    """No copy of a strided operand is kept for the backward, and changing it in between is noticed."""
    base = [t.detach() for t in _operands()[:3]]
    base[which] = base[which].t().contiguous().t()
    ops = [t.requires_grad_() for t in base]
    kept = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: kept.append(t.data_ptr()) or t, lambda t: t):
        _layer(*ops)
    assert {t.data_ptr() for t in ops} <= set(kept)
    y = _layer(*ops)
    with torch.no_grad():
        ops[which].add_(1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()


@pytest.mark.parametrize("cayley", [False, True])
def test_batched_gradients_are_taken_one_by_one(calls, cayley):
    """``is_grads_batched`` after an ordinary forward."""
    A, B, R, ib = _operands()
    ib, act = (None, "") if cayley else (ib, "silu_gate")
    wanted = [A, R] if cayley else [A, B, R, ib]
    dy = torch.randn(3, M, N)
    got = torch.autograd.grad(_layer(A, B, R, ib, act, cayley), wanted, dy, is_grads_batched=True)
    assert [g.shape for g in got] == [(3,) + w.shape for w in wanted] and calls["n_dadr"] == 3
    assert torch.equal(got[0][:, 0, 0], torch.stack([d.sum() for d in dy]))


def test_a_mode_around_the_backward_sees_the_custom_ops(calls, monkeypatch):
    A, B, R, ib = _operands()
    y = _layer(A, B, R, ib)
    monkeypatch.setattr(_module, "_plain_eager", lambda *t: False)   # what it answers under a dispatch mode
    ops = []

    class Seen(torch.utils._python_dispatch.TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            ops.append(func.namespace + "." + func.__name__)
            return func(*args, **(kwargs or {}))

    with Seen():
        torch.autograd.grad(y, A, torch.randn(M, N))
    assert "prism_b200.backward.default" in ops


class _OnGpu(torch.Tensor):
    is_cuda = True


@pytest.mark.parametrize("owner,name", [(torch._C, "_get_tracing_state"), (torch._C, "_len_torch_dispatch_stack"),
                                        (torch._C, "_len_torch_function_stack"), (torch._C._functorch, "peek_interpreter_stack"),
                                        (torch.autograd.forward_ad, "_current_level")])
def test_a_torch_without_a_private_name_runs_the_custom_ops(monkeypatch, owner, name):
    t = torch.zeros(2).as_subclass(_OnGpu)
    monkeypatch.setattr(_module, "_PLAIN_TYPES", (_OnGpu,))   # so that an ordinary call is one on this machine's tensors
    assert _module._plain_eager(t)
    monkeypatch.delattr(owner, name)
    assert not _module._plain_eager(t)


def test_a_torch_without_the_raw_stream_call(monkeypatch):
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device: type("Stream", (), {"cuda_stream": 77}))
    assert F._raw_stream(torch.device("cuda", 0)) == 77


@pytest.mark.parametrize("short", ["mask", "dadr", "db", "both", "always"])
@pytest.mark.parametrize("call", ["layer", "op", "backward"])
def test_backward_with_dropout_where_memory_is_short(calls, built_lib, monkeypatch, short, call):
    """The mask handed from dA+dR to dB is given up where it, or what else the calls need beside it, does not fit; a call
    that does not fit without it fails as before."""
    import weakref
    A, B, R, ib = _operands()
    seeds, masks, given = torch.arange(1, N // GS + 1), [], []
    empty = torch.empty

    def mask_or_not(*shape, **kw):
        if kw.get("dtype") != torch.int32:
            return empty(*shape, **kw)
        if short == "mask":
            raise torch.OutOfMemoryError("no memory")
        t = empty(*shape, **kw)
        masks.append(weakref.ref(t))
        return t

    def needs(name, kernel):
        def f(*args, dropout_mask=None, **kw):
            given.append((name, dropout_mask is not None))
            alive = any(m() is not None for m in masks)
            assert alive == (dropout_mask is not None), "a mask given up is a mask freed"
            if short == "always" or (alive and short in (name, "both")):
                raise torch.OutOfMemoryError("no memory")
            return kernel(*args, **kw)
        return f

    monkeypatch.setattr(torch, "empty", mask_or_not)
    monkeypatch.setattr(F, "_backward_dadr", needs("dadr", F._backward_dadr))
    monkeypatch.setattr(F, "_backward_db", needs("db", F._backward_db))
    if call == "backward":
        monkeypatch.setattr(F, "validate_tensor_params", lambda *a: None)
        run = lambda: F.backward(torch.ones(M, N), A.detach(), B.detach(), R.detach(), GS, RS, activation="silu_gate",   # noqa: E731
                                 dropout_seeds=seeds, dropout_p=0.5)
    elif call == "op":
        run = lambda: _module._prism_backward_op(torch.ones(M, N), A.detach(), B.detach(), R.detach(), GS, RS,   # noqa: E731
                                                 "silu_gate", 1.0, True, False, None, seeds, 0.5)
    else:
        run = lambda: _layer(A, B, R, ib, seeds=seeds, p=0.5).sum().backward()   # noqa: E731
    if short == "always":
        with pytest.raises(torch.OutOfMemoryError):
            run()
        return
    run()
    with_mask, without = True, False
    assert given == {"mask": [("dadr", without), ("db", without)],
                     "dadr": [("dadr", with_mask), ("dadr", without), ("db", without)],
                     "both": [("dadr", with_mask), ("dadr", without), ("db", without)],
                     "db": [("dadr", with_mask), ("db", with_mask), ("db", without)]}[short]


@pytest.mark.parametrize("op", [False, True])
def test_dropout_seeds_reach_the_kernels_as_the_forward_took_them(calls, monkeypatch, op):
    """Seeds given as every second element of a tensor (or on another device): the kernels read them one after the other."""
    A, B, R, ib = _operands()
    seeds = torch.arange(1, 2 * (N // GS) + 1)[::2]
    y = _layer(A, B, R, ib, seeds=seeds, p=0.5)
    if op:
        monkeypatch.setattr(_module, "_plain_eager", lambda *t: False)
    y.sum().backward()
    for name in ("dadr", "db"):
        given = calls[name]["dropout_seeds"]
        assert given.is_contiguous() and given.device == A.device and torch.equal(given, seeds)


def test_seeds_without_dropout_are_not_looked_at(calls):
    """A probability of 0: the forward ignores the seeds, whatever they are, and so does the backward."""
    A, B, R, ib = _operands()
    _layer(A, B, R, ib, seeds=torch.zeros(5), p=0.0).sum().backward()
    assert calls["dadr"]["dropout_mask"] is None and calls["dadr"]["dropout_p"] == 0.0
