"""Which form of the two attention operators a call takes: the registered one, which autograd, modes and
tracers see, or its body called as it is.  The operators themselves are replaced by CPU stand-ins."""
import pytest
import torch

from infllmv2_cuda_impl_b200 import attention


@pytest.fixture
def calls(monkeypatch):
    seen = []

    def forward(name):
        def f(q, k, v, *args):
            seen.append(name)
            return q * 2, q.new_zeros(k.shape[1], q.shape[0] * attention.GROUP), torch.empty(0, dtype=torch.int64)
        return f

    def backward(name):
        def f(dout, q, k, v, *args):
            seen.append(name)
            return dout * 2, torch.zeros_like(k), torch.zeros_like(v)
        return f

    monkeypatch.setattr(attention, "_check_common", lambda *args: None)       # (it refuses CPU tensors)
    monkeypatch.setattr(attention, "_varlen_forward", forward("forward body"))
    monkeypatch.setattr(attention, "_infllmv2_attn_varlen_forward", forward("forward operator"))
    monkeypatch.setattr(attention, "_varlen_backward", backward("backward body"))
    monkeypatch.setattr(attention, "_infllmv2_attn_varlen_backward", backward("backward operator"))
    return seen


def _call():
    q, k, v = (torch.zeros(4, h, 128, dtype=torch.bfloat16, requires_grad=True) for h in (16, 1, 1))
    cu = torch.tensor([0, 4], dtype=torch.int32)
    return q, attention.infllmv2_attn_varlen_func(q, k, v, cu, cu, 4, 4, causal=True)


def test_plain_call_takes_the_bodies(calls):
    q, out = _call()
    torch.autograd.grad(out.sum(), q)
    assert calls == ["forward body", "backward body"]


def test_backward_that_is_differentiated_takes_the_operator(calls):
    q, out = _call()
    torch.autograd.grad(out.sum(), q, create_graph=True)
    assert calls == ["forward body", "backward operator"]


def test_function_modes_and_profilers_see_the_operators(calls):
    from torch.overrides import TorchFunctionMode

    class Pass(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    with Pass():
        _call()
    assert calls == ["forward operator"]
    calls.clear()
    with torch.autograd.profiler.profile(use_kineto=False, use_device=None):
        q, out = _call()
        torch.autograd.grad(out.sum(), q)
    assert calls == ["forward operator", "backward operator"]


@pytest.mark.parametrize("sizes", [(32, 16), (128, 64)])
def test_compressed_lengths_of_a_fake_device_table(sizes):
    # shape propagation and tracing without a device: the lengths are made of tensor operators then
    from torch._subclasses import FakeTensorMode
    from torch.fx.experimental.proxy_tensor import make_fx
    import infllm_v2
    with FakeTensorMode():
        table = torch.empty(6, dtype=torch.int32, device="cuda")
        got = infllm_v2.compressed_lengths(table, *sizes)
        assert got.shape == (6,) and got.dtype == torch.int32 and got.device == table.device
        graph = make_fx(lambda t: infllm_v2.compressed_lengths(t, *sizes))(table)
    assert any("cumsum" in str(n.target) for n in graph.graph.nodes)


@pytest.mark.parametrize("case", ["apart", "neighbours", "onto itself", "swapped", "handed on", "one buffer", "shifted"])
def test_three_copies_in_one_launch_only_when_their_order_does_not_matter(case, monkeypatch):
    """A captured step shows its input buffers, so a caller may pass one of them as another input.  The
    launch is replaced by copies in the opposite order, which differ from the ordered ones if it matters."""
    import contextlib
    import ctypes
    from infllmv2_cuda_impl_b200 import ops
    launched = []

    def launch(name, *args):
        launched.append(name)
        for i in (6, 3, 0):
            ctypes.memmove(args[i + 1], args[i], args[i + 2])

    monkeypatch.setattr(ops._lib, "call", launch)
    monkeypatch.setattr(ops, "_on", lambda device: contextlib.nullcontext())
    monkeypatch.setattr(ops, "_stream", lambda device: 0)
    # (destination, source) offsets of the three copies of 16 elements
    offsets = {"apart": ((0, 64), (16, 96), (32, 128)), "neighbours": ((0, 48), (16, 64), (32, 80)),
               "onto itself": ((0, 0), (16, 96), (32, 32)), "swapped": ((0, 64), (16, 32), (32, 16)),
               "handed on": ((0, 64), (16, 0), (32, 16)), "one buffer": ((0, 64), (0, 96), (32, 128)),
               "shifted": ((0, 8), (32, 96), (64, 128))}[case]
    pairs = lambda buf: [(buf[d:d + 16], buf[s:s + 16]) for d, s in offsets]
    got, exp = (torch.arange(256, dtype=torch.int32) for _ in range(2))
    if case == "shifted":                          # refused by copy_
        with pytest.raises(RuntimeError):
            ops.copy3(pairs(got))
    else:
        ops.copy3(pairs(got))
        for d, s in pairs(exp):
            d.copy_(s)
        assert torch.equal(got, exp)
    assert launched == (["ifv2_copy3"] if case in ("apart", "neighbours") else [])
