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
