"""GPU: the compiled host path of the entry points (csrc/binding.cpp) -- what happens around the kernels."""
import pytest
import torch
from torch.utils.checkpoint import checkpoint

from hdla_impl_b200.synthetic import make_inputs

pytestmark = pytest.mark.gpu
R = 2
NAMES = ("q", "k", "v", "a", "b", "gk")


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    return torch.device("cuda:0")


def leaves(dev, dtype, B=1, T=100, H=2, D=64, seed=0):
    x = make_inputs(B, T, H, D, D, R, seed=seed, dtype=dtype, gk_div=4.0)
    return [x[n].to(dev).requires_grad_(True) for n in NAMES], x["do"].to(dev)


def layer_leaves(dev, B=1, T=100, H=2, D=64):
    g = torch.Generator().manual_seed(3)
    rn = lambda *s: torch.randn(*s, generator=g)
    x = [rn(B, T, H, D), rn(B, T, H, D), rn(B, T, H, D), torch.sigmoid(rn(B, T, H, 1)),
         torch.nn.functional.logsigmoid(rn(B, T, H, D)) / 8, rn(B, T, H * D), 1 + 0.1 * rn(H * D)]
    return [t.to(torch.bfloat16).to(dev).requires_grad_(True) for t in x], rn(B, T, H * D).to(torch.bfloat16).to(dev)


def layer(q, k, v, beta, log_f, gate, weight):
    from hdla_impl_b200.layer_ops import chunk_hdla_delta_rule, rms_norm_fused_gate
    o, _ = chunk_hdla_delta_rule(q, k, v, beta, log_f, normalize_k=True)
    return rms_norm_fused_gate(o.flatten(2), gate, weight)


def chunk(*t):
    import hdla_impl_b200 as HD
    return HD.chunk_hrdplr_delta_rule(*t, R, output_final_state=True)[0]


@pytest.mark.parametrize("what", ["fp32", "bf16", "layer", "operator of the layer"])
def test_non_reentrant_checkpoint_of_the_operator(dev, what):
    """The recomputation ends with an exception from the pack hook of the region's last saved tensor, here one of the
    operator's (or the norm's); the same kernels run on the same inputs, so the gradients are equal bit for bit."""
    if what.startswith("layer"):
        x, do = layer_leaves(dev)
        f = layer
    elif what.startswith("operator"):
        x, do = layer_leaves(dev)
        x, do = x[:5], do.view(x[0].shape)
        from hdla_impl_b200.layer_ops import chunk_hdla_delta_rule
        f = lambda *t: chunk_hdla_delta_rule(*t, normalize_k=True)[0]
    else:
        x, do = leaves(dev, torch.float32 if what == "fp32" else torch.bfloat16)
        f = chunk
    plain = torch.autograd.grad(f(*x), x, do)
    kept = torch.autograd.grad(checkpoint(f, *x, use_reentrant=False), x, do)
    for a, b in zip(plain, kept):
        assert torch.equal(a, b)


@pytest.mark.parametrize("f", ["chunk", "norm"])
def test_a_pack_hooks_exception_arrives_as_itself(dev, f):
    class Mine(Exception):
        pass

    def pack(t):
        raise Mine("from the hook")

    x, _ = layer_leaves(dev) if f == "norm" else leaves(dev, torch.bfloat16)
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        with pytest.raises(Mine, match="from the hook"):
            if f == "norm":
                from hdla_impl_b200.layer_ops import rms_norm_fused_gate
                rms_norm_fused_gate(x[5], x[5], x[6])
            else:
                chunk(*x)


def test_out_of_memory_arrives_as_such(dev):
    x, _ = leaves(dev, torch.bfloat16, T=4096, H=8, D=128)
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(dev).total_memory
    # the inputs are in place; the workspace (hundreds of megabytes here) does not fit into 32 more
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved(dev) + (32 << 20)) / total, dev)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            chunk(*x)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0, dev)
    chunk(*x)


def test_integer_initial_state_and_any_chunk_size(dev):
    """What the entry point took when Python checked its arguments: a state of an integer type is converted, and the
    tensor-core pipeline, which runs at its own chunk, does not look at the chunk size asked for."""
    import hdla_impl_b200 as HD
    x, do = leaves(dev, torch.bfloat16)
    h0 = torch.randint(-1, 2, (1, 2, 64, 64), generator=torch.Generator().manual_seed(1)).to(dev)

    def run(h, c):
        o, ht = HD.chunk_hrdplr_delta_rule(*x, R, initial_state=h, output_final_state=True, chunk_size=c)
        return [o, ht, *torch.autograd.grad(o, x, do)]

    want = run(h0.float(), 64)
    for h, c in ((h0, 64), (h0.to(torch.int32), 64), (h0.float(), None), (h0, 0)):
        for a, b in zip(run(h, c), want):
            assert torch.equal(a, b), (h.dtype, c)
    f32, _ = leaves(dev, torch.float32)
    a = HD.chunk_hrdplr_delta_rule(*f32, R, initial_state=h0, output_final_state=True)
    b = HD.chunk_hrdplr_delta_rule(*f32, R, initial_state=h0.float(), output_final_state=True)
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


def recurrent(*t):
    import hdla_impl_b200 as HD
    return HD.fused_recurrent_dplr_delta_rule(*t, R, output_final_state=True)


@pytest.mark.parametrize("what", ["chunk fp32", "chunk bf16", "recurrent", "layer"])
def test_a_traced_call_runs_on_its_own_inputs(dev, what):
    """torch.jit.trace records the operators as calls: the traced function computes on what it is given, not what it was
    traced with (equal bit for bit to the direct call: the same kernels)."""
    if what == "layer":
        f, (x, _) = layer, layer_leaves(dev)
    else:
        f = recurrent if what == "recurrent" else chunk
        x, _ = leaves(dev, torch.float32 if what == "chunk fp32" else torch.bfloat16)
    x = [t.detach() for t in x]
    y = [t.flip(1) if t.dim() > 1 else t for t in x]
    traced = torch.jit.trace(f, tuple(x), check_trace=False)
    for inputs in (y, x):
        got, want = traced(*inputs), f(*inputs)
        for a, b in zip(got if isinstance(got, tuple) else (got,), want if isinstance(want, tuple) else (want,)):
            assert torch.equal(a, b)


class Sub(torch.Tensor):
    """A tensor subclass without behaviour of its own: such tensors take the Python autograd functions."""


@pytest.mark.parametrize("what", ["chunk fp32", "chunk bf16", "recurrent", "layer"])
def test_tensor_subclasses_take_the_same_kernels(dev, what):
    from hdla_impl_b200 import _lib
    if what == "layer":
        f, (x, do) = layer, layer_leaves(dev)
    else:
        f = recurrent if what == "recurrent" else chunk
        x, do = leaves(dev, torch.float32 if what == "chunk fp32" else torch.bfloat16)
    x = [t.detach() for t in x]

    def run(ts):
        n0 = _lib.kernel_launches()
        if what == "recurrent":
            out = list(f(*ts))
        else:
            ts = [t.requires_grad_(True) for t in ts]
            o = f(*ts)
            out = [o, *torch.autograd.grad(o, ts, do)]
        return out, _lib.kernel_launches() - n0

    (want, n_want), (got, n_got) = run([t.clone() for t in x]), run([t.clone().as_subclass(Sub) for t in x])
    assert n_got == n_want
    for a, b in zip(got, want):
        assert torch.equal(a.as_subclass(torch.Tensor), b)


@pytest.mark.parametrize("f", ["chunk", "norm"])
def test_what_an_unpack_hook_returns_is_looked_at(dev, f):
    """A copy in another layout is as good as the saved tensor; a tensor of another shape, type or device is an error, not
    a pointer for a kernel."""
    if f == "norm":
        from hdla_impl_b200.layer_ops import rms_norm_fused_gate
        x, do = layer_leaves(dev)
        x, op = [x[5], x[5].detach().clone().requires_grad_(True), x[6]], rms_norm_fused_gate
    else:
        x, do = leaves(dev, torch.bfloat16)
        op = chunk

    def grads(unpack):
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t.detach().clone(), unpack):
            o = op(*x)
        return torch.autograd.grad(o, x, do)

    want = torch.autograd.grad(op(*x), x, do)
    strided = lambda t: t.transpose(0, -1).contiguous().transpose(0, -1)
    for a, b in zip(grads(strided), want):
        assert torch.equal(a, b)
    for bad in (lambda t: t.cpu(), lambda t: t.double(), lambda t: t[..., :-1], lambda t: t[:0]):
        with pytest.raises(RuntimeError, match="saved-tensor hook"):
            grads(bad)
    for a, b in zip(grads(lambda t: t), want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_second_backward_recomputes(dev, dtype):
    """The first backward uses up the kept workspace; a second one through the same graph computes it again (the same
    kernels on the same inputs: equal bit for bit), a third after the graph is gone is an error."""
    x, do = leaves(dev, dtype)
    o = chunk(*x)
    first = torch.autograd.grad(o, x, do, retain_graph=True)
    second = torch.autograd.grad(o, x, do)
    for a, b in zip(first, second):
        assert torch.equal(a, b)
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(o, x, do)


def test_threads_on_streams_of_their_own(dev):
    """Four threads, each with its stream and inputs, forward and backward, with a decay history that makes forwards wait
    for their own status words: results as alone."""
    import threading
    import hdla_impl_b200 as HD
    from hdla_impl_b200 import hrdplr
    n, rounds = 4, 40
    inputs = [leaves(dev, torch.bfloat16 if i % 2 else torch.float32, T=100 + 30 * i, seed=i) for i in range(n)]
    want = [torch.autograd.grad(chunk(*x), x, do) for x, do in inputs]
    torch.cuda.synchronize(dev)
    before = hrdplr._status_state(dev)["decay"]
    hrdplr._status_state(dev)["decay"] = 100.0
    wrong = []

    def work(i):
        try:
            x, do = inputs[i]
            with torch.cuda.stream(torch.cuda.Stream(dev)):
                for _ in range(rounds):
                    got = torch.autograd.grad(chunk(*x), x, do)
                torch.cuda.current_stream(dev).synchronize()
            if not all(torch.equal(a, b) for a, b in zip(got, want[i])):
                wrong.append(i)
        except Exception as e:          # noqa: BLE001 -- reported by the main thread
            wrong.append(e)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(n)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    hrdplr._status_state(dev)["decay"] = before
    assert not wrong, wrong
    HD.check_status(dev, wait=True)


@pytest.mark.parametrize("what", ["chunk", "layer"])
def test_transforms_that_the_operator_does_not_support_are_refused(dev, what):
    """Forward-mode gradients and vmap raise; they do not run without the tangent or on a wrapper's memory."""
    import torch.autograd.forward_ad as fwad
    x, _ = layer_leaves(dev) if what == "layer" else leaves(dev, torch.bfloat16)
    f = layer if what == "layer" else chunk
    x = [t.detach() for t in x]
    with fwad.dual_level():
        with pytest.raises(RuntimeError):
            f(fwad.make_dual(x[0], torch.ones_like(x[0])), *x[1:])
    with pytest.raises(RuntimeError):
        torch.vmap(lambda q: f(q, *x[1:]))(torch.stack([x[0], x[0]]))


_FP32_WAIT = """
import ctypes as C, sys, torch
sys.path.insert(0, {root!r})
import hdla_impl_b200 as HD
from hdla_impl_b200 import _lib
from hdla_impl_b200.synthetic import make_inputs
dev = torch.device("cuda:0")
x = make_inputs(1, 40, 2, 64, 64, 2, seed=0)
args = [x[n].to(dev).requires_grad_(True) for n in ("q", "k", "v", "a", "b", "gk")]
step = lambda: torch.autograd.grad(HD.chunk_hrdplr_delta_rule(*args, 2)[0], args, x["do"].to(dev))
for _ in range(100):
    step()
HD.check_status(dev, wait=True)
words = C.c_void_p()
_lib.check(_lib.load().hdla_fp32_status_words(C.byref(words)), "hdla_fp32_status_words")
_lib.check(_lib.load().hdla_debug_wait_timeout(words, C.c_uint64(1000000), _lib.stream_ptr(dev)), "hdla_debug_wait_timeout")
def raised(f):
    try:
        f()
    except RuntimeError as e:
        assert "device-side wait ran out (code 99)" in str(e), e
        return True
    return False
if {how!r} == "check":
    assert raised(lambda: HD.check_status(dev, wait=True))
else:
    def calls():
        for _ in range(64):
            step()
            torch.cuda.synchronize()
    assert raised(calls)
print("reported")
"""


@pytest.mark.parametrize("how", ["check", "calls"])
def test_fp32_pipeline_reports_a_wait_that_ran_out(dev, how):
    """With the fp32 pipeline's words as a kernel's run-out wait leaves them, a check that waits raises, and so does one of
    the next 64 steps.  (The words keep the report for as long as the process lives: a process of its own.)"""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _FP32_WAIT.format(root=root, how=how)], stdout=subprocess.PIPE,
                       stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("reported"), r.stdout
