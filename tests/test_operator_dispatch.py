"""How the operators are registered: schemas, gradients and tracing, on meta tensors (no kernel runs)."""
import os
import subprocess
import sys

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_COMMON = "Tensor query, Tensor key, Tensor value, Tensor query_offset, Tensor key_offset, "
_SCHEMAS = {
    "": f"({_COMMON}SymInt max_seq_len_q, SymInt max_seq_len_kv, float qk_scale, SymInt activation, SymInt window_size=-1, "
        "bool start_end_offsets=False) -> Tensor",
    "_backward": f"(Tensor do, {_COMMON}SymInt max_seq_len_q, SymInt max_seq_len_kv, float qk_scale, SymInt activation, "
                 "Tensor? out=None, Tensor? lse=None, SymInt window_size=-1, bool start_end_offsets=False) -> (Tensor, Tensor, Tensor)",
    "_softmax": f"({_COMMON}SymInt max_seq_len_q, SymInt max_seq_len_kv, float qk_scale, SymInt window_size=-1, "
                "bool start_end_offsets=False) -> (Tensor, Tensor)",
    "_shared_kv": f"({_COMMON}Tensor kv_seq_index, SymInt max_seq_len_q, SymInt max_seq_len_kv, float qk_scale, SymInt activation, "
                  "SymInt window_size=-1) -> Tensor",
}


def _meta(requires_grad=True):
    q = torch.empty(10, 4, 64, dtype=torch.bfloat16, device="meta", requires_grad=requires_grad)
    k = torch.empty(12, 2, 64, dtype=torch.bfloat16, device="meta", requires_grad=requires_grad)
    v = torch.empty(12, 2, 64, dtype=torch.bfloat16, device="meta", requires_grad=requires_grad)
    off = torch.empty(3, dtype=torch.int64, device="meta")
    return q, k, v, off


def _call(q, k, v, off, activation, **kwargs):
    import ads_model_kernel_library_b200.gdpa as G

    return G.generalized_dot_product_attention(q, k, v, off, off, 5, 6, activation=activation, **kwargs)


@pytest.mark.parametrize("suffix", sorted(_SCHEMAS))
def test_schemas(suffix):
    import ads_model_kernel_library_b200.gdpa  # noqa: F401

    name = f"generalized_dot_product_attention{suffix}"
    op = getattr(torch.ops.gdpa, name).default
    assert str(op._schema) == f"gdpa::{name}{_SCHEMAS[suffix]}"
    assert torch.Tag.pt2_compliant_tag in op.tags


@pytest.mark.parametrize("activation", ["relu", "softmax"])
def test_gradients_of_those_that_ask_for_one(activation):
    q, k, v, off = _meta()
    out = _call(q, k, v, off, activation)
    assert [tuple(g.shape) for g in torch.autograd.grad(out, (q, k, v), torch.empty_like(out))] == [(10, 4, 64), (12, 2, 64), (12, 2, 64)]
    out = _call(q, k.detach(), v, off, activation, window_size=3)
    dq, dv = torch.autograd.grad(out, (q, v), torch.empty_like(out))
    assert dq.shape == q.shape and dv.shape == v.shape
    with torch.no_grad():
        assert not _call(q, k, v, off, activation).requires_grad
    assert not _call(q.detach(), k.detach(), v.detach(), off, activation).requires_grad


@pytest.mark.parametrize("activation", ["relu", "softmax"])
def test_a_second_derivative_raises(activation):
    q, k, v, off = _meta()
    out = _call(q, k, v, off, activation)
    (dq,) = torch.autograd.grad(out, q, torch.empty_like(out), create_graph=True)
    with pytest.raises(RuntimeError, match="no gradient"):
        torch.autograd.grad(dq.sum(), q)


@pytest.mark.parametrize("activation", ["relu", "softmax"])
def test_saved_tensor_hooks_see_what_the_backward_keeps(activation):
    packed = []

    def pack(t):
        packed.append(tuple(t.shape))
        return t

    q, k, v, off = _meta()
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        out = _call(q, k, v, off, activation)
    assert packed[:5] == [(10, 4, 64), (12, 2, 64), (12, 2, 64), (3,), (3,)]
    assert len(packed) == (7 if activation == "softmax" else 5)
    torch.autograd.grad(out, (q, k, v), torch.empty_like(out))


def test_shared_kv_has_no_backward():
    q, k, v, off = _meta()
    out = _call(q, k, v, off, "relu", ad_to_request_offset=torch.empty(2, dtype=torch.int64, device="meta"))
    assert out.requires_grad
    with pytest.raises(NotImplementedError, match="inference path"):
        torch.autograd.grad(out, q, torch.empty_like(out))


@pytest.mark.parametrize("activation", ["relu", "softmax"])
def test_forward_and_backward_trace(activation):
    q, k, v, off = _meta()
    compiled = torch.compile(lambda a, b, c: _call(a, b, c, off, activation) * 2, backend="aot_eager", fullgraph=True)
    out = compiled(q, k, v)
    assert out.shape == q.shape
    assert torch.autograd.grad(out, (k,), torch.empty_like(out))[0].shape == k.shape


def test_gradients_without_the_private_dispatch_guard():
    """A torch without the guard that the gradient kernels use takes the public registration: in a process of its own."""
    code = """
import torch
guard = getattr(torch._C, "_AutoDispatchBelowAutograd", None)
if guard is not None:
    del torch._C._AutoDispatchBelowAutograd
import ads_model_kernel_library_b200.gdpa as G
from ads_model_kernel_library_b200.gdpa import ops
if guard is not None:
    torch._C._AutoDispatchBelowAutograd = guard  # torch's own registration uses it under this name
assert ops._below_autograd is None
q = torch.empty(10, 2, 64, dtype=torch.bfloat16, device="meta", requires_grad=True)
off = torch.empty(3, dtype=torch.int64, device="meta")
for act in ("relu", "softmax"):
    out = G.generalized_dot_product_attention(q, q, q, off, off, 5, 5, activation=act)
    assert torch.autograd.grad(out, q, torch.empty_like(out))[0].shape == q.shape
"""
    subprocess.run([sys.executable, "-c", code], check=True, cwd=ROOT, timeout=300)


_SECOND_LOAD = """
import importlib, sys
import torch
from torch.utils.flop_counter import FlopCounterMode
import ads_model_kernel_library_b200.gdpa as G

NAME = "ads_model_kernel_library_b200"

def tensors():
    q = torch.empty(10, 4, 64, dtype=torch.bfloat16, device="meta", requires_grad=True)
    k = torch.empty(12, 2, 64, dtype=torch.bfloat16, device="meta", requires_grad=True)
    return q, k, torch.empty(3, dtype=torch.int64, device="meta")

def calls(attention, megakernel, fp8):
    q, k, off = tensors()
    for act in ("relu", "softmax"):
        with FlopCounterMode(display=False) as flops:
            out = attention(q, k, k, off, off, 5, 6, activation=act)
            grads = torch.autograd.grad(out, (q, k), torch.empty_like(out))
        assert [g.shape for g in grads] == [q.shape, k.shape]
        assert flops.get_total_flops() == (14 if act == "relu" else 10) * 4 * 64 * 2 * 5 * 6  # the softmax forward has no formula
        with torch.no_grad():
            assert attention(q, k, k, off, off, 5, 6, activation=act).shape == q.shape
    out = attention(q, k, k, off, off, 5, 6, activation="relu", ad_to_request_offset=off[:2])
    try:
        torch.autograd.grad(out, q, torch.empty_like(out))
    except NotImplementedError as e:
        assert "inference path" in str(e)
    else:
        raise AssertionError
    out = megakernel(q, k, k, off, off, 5, 6, activation="relu", fused_rms_norm=True)
    assert out.shape == q.shape and out.requires_grad
    q8 = torch.empty(10, 2, 64, dtype=torch.float8_e4m3fn, device="meta")
    s8 = torch.empty(2, 2, device="meta")
    out = fp8(q8, q8, q8, s8, s8, s8, off, off, off, off, 5, 5)
    assert out.shape == q8.shape and out.dtype == torch.bfloat16

first = G.generalized_dot_product_attention, G.gdpa_megakernel, G.generalized_dot_product_attention_fp8
overload = torch.ops.gdpa.generalized_dot_product_attention.default
calls(*first)
q, k, off = tensors()
pending = {act: first[0](q, k, k, off, off, 5, 6, activation=act) for act in ("relu", "softmax")}
for _ in range(2):
    if HOW == "reload":
        for module in ("ops", "megakernel", "mxfp8"):
            importlib.reload(sys.modules[f"{NAME}.gdpa.{module}"])
        importlib.reload(G)
    else:
        for module in [m for m in sys.modules if m.split(".")[0] == NAME]:
            del sys.modules[module]
        import ads_model_kernel_library_b200.gdpa as G
    assert G.generalized_dot_product_attention is not first[0]
    calls(G.generalized_dot_product_attention, G.gdpa_megakernel, G.generalized_dot_product_attention_fp8)
    calls(*first)
    assert overload(q, k, k, off, off, 5, 6, 1.0, 3).shape == q.shape
for out in pending.values():
    assert torch.autograd.grad(out, k, torch.empty_like(out))[0].shape == k.shape
# a call reaches the functions of the module that was run last
ops = sys.modules[f"{NAME}.gdpa.ops"]
assert torch.ops.gdpa._operators["generalized_dot_product_attention"].functions.impl is ops._gdpa_forward
"""


@pytest.mark.parametrize("how", ["reload", "import"])
def test_operators_outlive_a_second_load_of_their_module(how):
    """importlib.reload, and an import after the package was taken out of sys.modules: calls, gradients, calls through names and
    handles that were taken before, and a backward whose forward ran before.  In a process of its own."""
    subprocess.run([sys.executable, "-c", f"HOW = {how!r}\n{_SECOND_LOAD}"], check=True, cwd=ROOT, timeout=300)


def test_another_schema_of_a_registered_operator_is_refused():
    from ads_model_kernel_library_b200.gdpa import ops

    with pytest.raises(RuntimeError, match="another schema"):
        ops._define_op("generalized_dot_product_attention(Tensor query) -> Tensor", None, None)
    q, k, v, off = _meta()
    assert _call(q, k, v, off, "relu").shape == q.shape


@pytest.mark.parametrize("activation", ["relu", "softmax"])
def test_a_profile_counts_a_call_once(activation):
    """With a gradient and without one, the call and its backward are one event each."""
    q, k, v, off = _meta()
    name = "gdpa::generalized_dot_product_attention"
    forward = name + ("_softmax" if activation == "softmax" else "")
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as trained:
        out = _call(q, k, v, off, activation)
        torch.autograd.grad(out, (q, k, v), torch.empty_like(out), create_graph=True)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as inferred, torch.no_grad():
        _call(q, k, v, off, activation)
    counts = [{e.key: e.count for e in p.key_averages() if e.key.startswith(name)} for p in (trained, inferred)]
    assert counts == [{forward: 1, name + "_backward": 1}, {forward: 1}]


def test_gradients_without_the_private_key_set():
    """As without the dispatch guard: a torch without the set of keys that the gradient kernels pass on takes the public form."""
    code = """
import torch
keys = getattr(torch._C, "_after_autograd_keyset", None)
if keys is not None:
    del torch._C._after_autograd_keyset
from ads_model_kernel_library_b200.gdpa import ops
if keys is not None:
    torch._C._after_autograd_keyset = keys  # torch's own registration uses it under this name
assert ops._keys_below_autograd is None
q = torch.empty(10, 2, 64, dtype=torch.bfloat16, device="meta", requires_grad=True)
off = torch.empty(3, dtype=torch.int64, device="meta")
out = ops.generalized_dot_product_attention(q, q, q, off, off, 5, 5, activation="relu")
assert torch.autograd.grad(out, q, torch.empty_like(out))[0].shape == q.shape
"""
    subprocess.run([sys.executable, "-c", code], check=True, cwd=ROOT, timeout=300)
