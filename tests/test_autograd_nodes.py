"""The C++ autograd nodes of linear layers and norms, on the CPU: the kernels are stood in for by PyTorch on the same memory."""
import ctypes
import sysconfig
import time
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path
from types import SimpleNamespace

import pytest
import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from tensor_parallel_b200 import build

pytestmark = pytest.mark.skipif(not (build.LIB_PATH.exists() and build.AUTOGRAD_PATH.exists()), reason="native library not built")

_p, _i, _f = ctypes.c_void_p, ctypes.c_int, ctypes.c_float


def _memory(address, count, dtype):
    size = torch.empty((), dtype=dtype).element_size()
    return torch.frombuffer((ctypes.c_char * (count * size)).from_address(address), dtype=dtype)


def _matrix(address, rows, cols, pitch, dtype=torch.bfloat16):
    return _memory(address, (rows - 1) * pitch + cols, dtype).as_strided((rows, cols), (pitch, 1))


def _plan(tokens, features, k, world, splits, kbox, flags, plan):
    return 0


def _gemm(x, w, out, bias, residual, tokens, features, k, ldx, ldw, ld_out, act, scale, plan, rc, opts, stream):
    from tensor_parallel_b200.ops import native

    o = ctypes.cast(opts, ctypes.POINTER(native.GemmOpts)).contents if opts else native.GemmOpts()
    a = _matrix(x, k, tokens, ldx).t() if o.x_mn else _matrix(x, tokens, k, ldx)
    b = _matrix(w, k, features, ldw).t() if o.w_mn else _matrix(w, features, k, ldw)
    y = a.float() @ b.float().t()
    if bias:
        y = y + _memory(bias, features, torch.bfloat16).float()
    if residual:
        y = y + _matrix(residual, tokens, features, ld_out).float()
    _matrix(out, tokens, features, ld_out).copy_(y)
    return _gemm.code


_gemm.code = 0


def _norm_fwd(x, residual, weight, bias, out, sum_out, rstd, mean, rows, cols, eps, mode, dtype, stream):
    dt = torch.float32 if dtype else torch.bfloat16
    v = _matrix(x, rows, cols, cols, dt).float()
    m = v.mean(-1) if mode else torch.zeros(rows)
    r = ((v - m[:, None]).square().mean(-1) + eps).rsqrt()
    y = (v - m[:, None]) * r[:, None]
    if weight:
        y = y * _memory(weight, cols, dt).float()
    if bias:
        y = y + _memory(bias, cols, dt).float()
    _matrix(out, rows, cols, cols, dt).copy_(y)
    _memory(rstd, rows, torch.float32).copy_(r)
    if mode:
        _memory(mean, rows, torch.float32).copy_(m)
    return 0


def _norm_bwd_parts(rows, cols):
    return 1


def _norm_bwd(dy, x, weight, rstd, mean, dx, part_w, part_b, dw, db, rows, cols, mode, dtype, grad_fp32, stream):
    dt, gt = torch.float32 if dtype else torch.bfloat16, torch.float32 if grad_fp32 else torch.bfloat16
    g, v = _matrix(dy, rows, cols, cols, dt).float(), _matrix(x, rows, cols, cols, dt).float()
    r = _memory(rstd, rows, torch.float32)[:, None]
    xh = (v - _memory(mean, rows, torch.float32)[:, None]) * r if mode else v * r
    gw = g * _memory(weight, cols, dt).float() if weight else g
    c1 = gw.mean(-1, keepdim=True) if mode else 0.0
    _matrix(dx, rows, cols, cols, dt).copy_((gw - c1 - xh * (gw * xh).mean(-1, keepdim=True)) * r)
    if dw:
        _memory(dw, cols, gt).copy_((g * xh).sum(0))
    if db:
        _memory(db, cols, gt).copy_(g.sum(0))
    return 0


def _col_sum_parts(rows, cols):
    return 2


def _col_sum(g, out, partials, rows, cols, fp32, stream):
    _memory(out, cols, torch.float32 if fp32 else torch.bfloat16).copy_(_matrix(g, rows, cols, cols).float().sum(0))
    _col_sum.calls += 1
    return 0


_col_sum.calls = 0


@pytest.fixture
def nodes():
    from tensor_parallel_b200.ops import native

    signatures = dict(tpb_gemm_plan_ex=(_plan, [_i] * 7 + [_p]), tpb_gemm_bf16_ex=(_gemm, [_p] * 5 + [_i] * 7 + [_f] + [_p] * 4),
                      tpb_norm_fwd=(_norm_fwd, [_p] * 8 + [_i, _i, _f, _i, _i, _p]), tpb_norm_bwd=(_norm_bwd, [_p] * 10 + [_i] * 5 + [_p]),
                      tpb_norm_bwd_parts=(_norm_bwd_parts, [_i, _i]), tpb_col_sum_parts=(_col_sum_parts, [_i, _i]),
                      tpb_col_sum=(_col_sum, [_p] * 3 + [_i] * 3 + [_p]))
    stubs = {name: ctypes.CFUNCTYPE(_i, *args)(fn) for name, (fn, args) in signatures.items()}
    context = native.ReduceCtx()
    native.AUTOGRAD.bind({n: ctypes.cast(s, _p).value for n, s in stubs.items()}, native._error_text, lambda index, elems: ctypes.addressof(context))
    yield native
    native._bind_autograd()


@pytest.fixture
def python_nodes(nodes, monkeypatch):
    """The Python autograd functions too run on the stand-ins."""
    types = dict(tpb_gemm_plan_ex=(_plan, [_i] * 7 + [_p]), tpb_gemm_bf16_ex=(_gemm, [_p] * 5 + [_i] * 7 + [_f] + [_p] * 4),
                 tpb_norm_fwd=(_norm_fwd, [_p] * 8 + [_i, _i, _f, _i, _i, _p]), tpb_norm_bwd=(_norm_bwd, [_p] * 10 + [_i] * 5 + [_p]),
                 tpb_norm_bwd_parts=(_norm_bwd_parts, [_i, _i]))
    library = SimpleNamespace(**{name: ctypes.CFUNCTYPE(_i, *args)(fn) for name, (fn, args) in types.items()})
    monkeypatch.setattr(nodes, "LIB", library)
    monkeypatch.setattr(nodes, "gemm_plan", lambda *a, **k: nodes.GemmPlan())
    monkeypatch.setattr(nodes, "device_state", lambda device: SimpleNamespace(ctx=nodes.ReduceCtx()))
    monkeypatch.setattr(nodes, "_stream", lambda: None)
    return nodes


def _close(got, want):
    assert got.dtype == want.dtype and got.shape == want.shape
    assert (got.float() - want.float()).norm() <= 2e-2 * want.float().norm() + 1e-6  # bf16 results of both sides: 2^-8 each, in and out


@pytest.mark.parametrize("with_bias", [False, True])
@pytest.mark.parametrize("frozen", ["", "x", "weight", "bias"])
@pytest.mark.parametrize("form", ["plain", "three dimensions", "strided", "fp32 gradient", "odd pitch"])
def test_linear_node(nodes, with_bias, frozen, form):
    torch.manual_seed(0)
    inputs = 20 if form == "odd pitch" else 24
    x = torch.randn(2, 5, inputs, dtype=torch.bfloat16) if form == "three dimensions" else torch.randn(10, inputs, dtype=torch.bfloat16)
    if form == "strided":
        x = torch.randn(inputs, 10, dtype=torch.bfloat16).t()
    leaves = dict(x=x, weight=torch.randn(16, inputs, dtype=torch.bfloat16) * 0.1, bias=torch.randn(16, dtype=torch.bfloat16) if with_bias else None)
    results = []
    for call in (nodes.linear, F.linear):
        t = {n: None if v is None else v.detach().requires_grad_(n != frozen) for n, v in leaves.items()}
        out = call(t["x"], t["weight"], t["bias"])
        grad = torch.ones_like(out) + torch.arange(16) / 16
        if form == "strided":
            grad = grad.t().contiguous().t()
        if form == "fp32 gradient":
            out.float().backward(grad.float())
        else:
            out.backward(grad.to(out.dtype))
        results.append([out.detach()] + [None if v is None else v.grad for v in t.values()])
    for got, want in zip(*results):
        assert (got is None) == (want is None)
        if want is not None:
            _close(got, want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gradient_of_a_bias_of_its_own_takes_part_in_what_goes_on_around_it(nodes, dtype):
    """The layer's bias alone is trained: its gradient of a batch of gradients, and a graph through it; one gradient takes the kernel."""
    torch.manual_seed(3)
    x, w = torch.randn(10, 24, dtype=torch.bfloat16), torch.randn(16, 24, dtype=torch.bfloat16)
    b = torch.zeros(16, dtype=torch.bfloat16, requires_grad=True)
    out = nodes.linear(x, w, b).to(dtype)
    g = torch.randn(3, 10, 16).to(dtype)
    before = _col_sum.calls
    (batched,) = torch.autograd.grad(out, b, g, is_grads_batched=True, retain_graph=True)
    single = torch.stack([torch.autograd.grad(out, b, t, retain_graph=True)[0] for t in g])
    _close(batched, single)
    assert _col_sum.calls == before + 3
    leaf = g[0].clone().requires_grad_()
    (once,) = torch.autograd.grad(out, b, leaf, create_graph=True)
    (twice,) = torch.autograd.grad(once.float().square().sum(), leaf)
    _close(twice, (2 * once.detach().float()).expand(10, 16).to(dtype))


@pytest.mark.parametrize("frozen", [(), (0,), (1, 3), (2,)])
@pytest.mark.parametrize("unused", [(), (0,), (2,), (0, 1)])
@pytest.mark.parametrize("form", ["plain", "three dimensions", "strided", "fp32 gradient"])
def test_node_of_several_projections(nodes, frozen, unused, form):
    """Against projections with nodes of their own: what an unused one leaves without a gradient, frozen leaves, shapes and strides."""
    torch.manual_seed(0)
    x = torch.randn(2, 5, 24, dtype=torch.bfloat16) if form == "three dimensions" else torch.randn(24, 10, dtype=torch.bfloat16).t()
    if form == "plain":
        x = x.contiguous()
    values = [x] + [torch.randn(n, 24, dtype=torch.bfloat16) * 0.1 for n in (16, 8, 16)]
    results = []
    for call in (lambda x, ws: nodes.AUTOGRAD.linears(x, ws), lambda x, ws: [F.linear(x, w) for w in ws]):
        leaves = [v.detach().requires_grad_(i not in frozen) for i, v in enumerate(values)]
        outs = call(leaves[0], leaves[1:])
        used = [o.float() if form == "fp32 gradient" else o for i, o in enumerate(outs) if i not in unused]
        if any(o.requires_grad for o in used):
            torch.autograd.backward(used, [torch.ones_like(o) + torch.arange(o.shape[-1]) // 4 / 4 for o in used])
        results.append([o.detach() for o in outs] + [t.grad for t in leaves])
    for got, want in zip(*results):
        assert (got is None) == (want is None)
        if want is not None:
            _close(got, want)


def test_modules_that_do_more_than_multiply_are_called_as_they_are(nodes, monkeypatch):
    from tensor_parallel_b200.models import common

    joint = []
    monkeypatch.setattr(common.OF, "linears", lambda x, ws: joint.append(len(ws)) or [F.linear(x, w) for w in ws])

    class Wrapped(common.Linear):
        pass

    def plain():
        return common.Linear(8, 4, bias=False)

    def hooked():
        m = plain()
        m.register_forward_hook(lambda module, args, out: out + 1)
        return m

    def replaced():
        m = plain()
        m.forward = lambda x: F.linear(x, m.weight) * 2
        return m

    x = torch.randn(3, 8)
    for make in (lambda: Wrapped(8, 4, bias=False), lambda: common.Linear(8, 4), lambda: torch.nn.Linear(8, 4, bias=False), hooked, replaced,
                 lambda: torch.nn.utils.parametrizations.weight_norm(plain()), lambda: torch.nn.Sequential(plain())):
        modules = [plain(), make()]
        assert all(torch.equal(a, m(x)) for a, m in zip(common.linears(x, *modules), modules)) and not joint
    handle = torch.nn.modules.module.register_module_forward_pre_hook(lambda module, args: None)
    common.linears(x, plain(), plain())
    handle.remove()
    assert not joint
    modules = [plain(), plain()]
    assert all(torch.equal(a, m(x)) for a, m in zip(common.linears(x, *modules), modules)) and joint == [2]
    monkeypatch.undo()
    assert len(common.linears(x.requires_grad_(), *modules)) == 2  # (on the CPU every module is called)


@pytest.mark.parametrize("use_cache,past", [(False, False), (True, False), (False, True)])
@pytest.mark.parametrize("model", ["llama", "gptj", "t5 encoder", "t5 decoder", "t5 cross-attention"])
def test_cached_keys_and_values_have_graphs_of_their_own(monkeypatch, model, use_cache, past):
    """A backward through cached keys and then one through the values, which left the layer with their graph."""
    from tensor_parallel_b200.models import common, gptj, llama, t5

    joint = []

    class Joint(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x, *ws):
            joint.append(len(ws))
            ctx.save_for_backward(x, *ws)
            return tuple(F.linear(x, w) for w in ws)

        @staticmethod
        def backward(ctx, *gs):
            x, *ws = ctx.saved_tensors
            return (sum(g @ w for g, w in zip(gs, ws)), *(g.flatten(0, 1).t() @ x.flatten(0, 1) for g in gs))

    monkeypatch.setattr(common.OF, "linears", lambda x, ws: Joint.apply(x, *ws))
    torch.manual_seed(0)
    x = torch.randn(2, 5, 32, requires_grad=True)
    before = tuple(torch.randn(2, 2, 3, 16, requires_grad=True) for _ in range(2)) if past and model != "t5 encoder" else None
    positions = torch.arange(5)[None].expand(2, 5)
    if model == "llama":
        layer = llama.LlamaAttention(llama.LlamaConfig(hidden_size=32, num_attention_heads=2, num_key_value_heads=2))
        out, _, present = layer(x, position_ids=positions, past_key_value=before, use_cache=use_cache)
    elif model == "gptj":
        layer = gptj.GPTJAttention(gptj.GPTJConfig(n_embd=32, n_head=2, rotary_dim=8))
        out, present = layer(x, position_ids=positions, layer_past=before, use_cache=use_cache)
    else:
        layer = t5.T5Attention(t5.T5Config(d_model=32, num_heads=2, d_kv=16), True, model != "t5 encoder")
        out, present, _ = layer(x, key_value_states=torch.randn(2, 4, 32, requires_grad=True) if "cross" in model else None, past_key_value=before, use_cache=use_cache)
    escapes = (use_cache or past) and model != "t5 encoder"
    assert joint == ([] if escapes else [2 if "cross" in model else 3])
    if present is not None:
        for t in present:
            if t.requires_grad:
                t.sum().backward()
    else:
        out.sum().backward()


@pytest.mark.parametrize("mode,dtype,wdtype,with_bias,with_weight", [(0, torch.bfloat16, torch.bfloat16, False, True), (0, torch.float32, torch.float32, False, True),
                                                                   (1, torch.bfloat16, torch.bfloat16, True, True), (1, torch.float32, torch.bfloat16, True, True),
                                                                   (1, torch.bfloat16, torch.float32, False, True), (0, torch.bfloat16, None, False, False)])
def test_norm_node(nodes, mode, dtype, wdtype, with_bias, with_weight):
    torch.manual_seed(1)
    x = torch.randn(3, 4, 32, dtype=dtype)
    w = torch.randn(32, dtype=wdtype) if with_weight else None
    b = torch.randn(32, dtype=wdtype) if with_bias else None
    g = torch.randn(3, 4, 32, dtype=dtype)
    leaves = [None if t is None else t.detach().requires_grad_() for t in (x, w, b)]
    refs = [None if t is None else t.detach().double().requires_grad_() for t in (x, w, b)]
    out = nodes.AUTOGRAD.norm(*leaves, 1e-5, mode)
    out.backward(g)
    if mode:
        want = F.layer_norm(refs[0], (32,), refs[1], refs[2], 1e-5)
    else:
        want = refs[0] * (refs[0].square().mean(-1, keepdim=True) + 1e-5).rsqrt() * (1 if w is None else refs[1])
    want.backward(g.double())
    _close(out.detach(), want.detach().to(dtype))
    for leaf, ref in zip(leaves, refs):
        if leaf is not None:
            _close(leaf.grad, ref.grad.to(leaf.dtype))


def _linear_case():
    torch.manual_seed(2)
    return torch.randn(6, 16, dtype=torch.bfloat16, requires_grad=True), torch.randn(8, 16, dtype=torch.bfloat16, requires_grad=True)


def test_saved_tensors_go_through_the_hooks(nodes):
    x, w = _linear_case()
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.data_ptr()) or t.clone(), lambda t: t):
        out = nodes.linear(x, w)
    assert packed == [x.data_ptr(), w.data_ptr()]
    out.sum().backward()
    y = torch.randn(4, 16, requires_grad=True)
    packed.clear()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.data_ptr()) or t.clone(), lambda t: t):
        nodes.rms_norm(y, torch.ones(16), 1e-6)
    assert y.data_ptr() in packed


def test_checkpointed_linear(nodes):
    x, w = _linear_case()
    checkpoint(lambda t: nodes.linear(t, w).relu(), x, use_reentrant=False).sum().backward()
    again, w2 = (t.detach().requires_grad_() for t in (x, w))
    nodes.linear(again, w2).relu().sum().backward()
    assert torch.equal(x.grad, again.grad) and torch.equal(w.grad, w2.grad)


def test_changed_inputs_are_noticed(nodes):
    x, w = _linear_case()
    out = nodes.linear(x, w)
    with torch.no_grad():
        w.add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.sum().backward()


@pytest.mark.parametrize("layer", ["linear", "linears", "norm"])
def test_transforms_are_refused(nodes, layer):
    x, w = _linear_case()
    call = dict(linear=lambda t: nodes.linear(t, w), linears=lambda t: sum(nodes.linears(t, [w, w])),
                norm=lambda t: nodes.rms_norm(t, torch.ones(16, dtype=t.dtype), 1e-6))[layer]
    with pytest.raises(RuntimeError):
        torch.func.vmap(call)(x.detach()[None])
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: call(t).sum())(x.detach())
    with pytest.raises(RuntimeError), torch.autograd.forward_ad.dual_level():
        call(torch.autograd.forward_ad.make_dual(x.detach().requires_grad_(), torch.ones_like(x)))
    out = call(x)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(out, x, torch.ones(3, *out.shape, dtype=out.dtype), is_grads_batched=True)


def test_nothing_is_recorded_without_gradients(nodes):
    x, w = _linear_case()
    with torch.no_grad():
        assert nodes.linear(x, w).grad_fn is None and nodes.rms_norm(x, None, 1e-6).grad_fn is None
    assert nodes.linear(x.detach(), w.detach()).grad_fn is None


def test_an_error_of_a_kernel_reaches_the_caller(nodes, monkeypatch):
    x, w = _linear_case()
    out = nodes.linear(x, w)
    monkeypatch.setattr(_gemm, "code", 6)
    with pytest.raises(RuntimeError, match="tpb_gemm_bf16 failed: reduction workspace too small"):
        nodes.linear(x, w)
    with pytest.raises(RuntimeError, match="tpb_gemm_bf16 failed: reduction workspace too small"):
        out.sum().backward()


class _Layer(torch.nn.Module):
    def __init__(self, nodes, kind, learned, dtype=torch.bfloat16):
        super().__init__()
        self.nodes, self.kind = nodes, kind
        torch.manual_seed(4)
        self.weight = torch.nn.Parameter(torch.randn(*((8, 16) if kind == "linear" else (16,)), dtype=dtype), requires_grad=learned)
        self.bias = torch.nn.Parameter(torch.randn(8 if kind == "linear" else 16, dtype=dtype), requires_grad=learned)

    def forward(self, x):
        if self.kind == "linear":
            return self.nodes.linear(x, self.weight, self.bias)
        if self.kind == "rms":
            return self.nodes.rms_norm(x, self.weight, 1e-6)
        return self.nodes.layer_norm(x, self.weight, self.bias, 1e-6)


@pytest.mark.parametrize("kind", ["linear", "rms", "layer"])
@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("grad_mode", [False, True])
def test_a_traced_layer_computes(python_nodes, kind, learned, grad_mode):
    """On inputs that it was not traced with, and of another number of rows; gradients flow where they did when it was traced."""
    layer = _Layer(python_nodes, kind, learned)
    x = torch.randn(3, 16, dtype=torch.bfloat16)
    with torch.set_grad_enabled(grad_mode):
        traced = torch.jit.trace(layer, x)
        for rows in (3, 5):
            y = torch.randn(rows, 16, dtype=torch.bfloat16)
            assert torch.equal(traced(y), layer(y))
    if grad_mode and learned:
        traced(y).sum().backward()
        grads = [p.grad for p in layer.parameters()]
        layer.zero_grad()
        layer(y).sum().backward()
        for got, p in zip(grads, layer.parameters()):
            assert (got is None) == (p.grad is None) and (got is None or torch.equal(got, p.grad))


def test_the_module_shares_the_cpp_runtime_of_torch():
    """With a runtime of its own, a failed check inside the module ended the process instead of raising."""
    assert b"\0libstdc++.so.6\0" in build.AUTOGRAD_PATH.read_bytes()


@pytest.mark.parametrize("dtype", [torch.float16, torch.float64, torch.int32])
def test_other_types_are_refused_before_a_kernel_is_called(nodes, dtype):
    """The kernels would take 2-byte elements for 4-byte ones, past the end of the tensors."""
    x, w = torch.ones(4, 8).to(dtype), torch.ones(8).to(dtype)
    before = nodes.launch_count
    with pytest.raises(TypeError, match="bf16 or fp32"):
        nodes.rms_norm(x, w, 1e-6)
    with pytest.raises(TypeError, match="bf16 or fp32"):
        nodes.layer_norm(x, None, None, 1e-6)
    with pytest.raises(TypeError, match="bf16 operands"):
        nodes.linear(x, torch.ones(16, 8, dtype=torch.bfloat16))
    with pytest.raises(TypeError, match="bf16 operands"):
        nodes.linear(torch.ones(4, 8, dtype=torch.bfloat16), torch.ones(16, 8).to(dtype))
    assert nodes.launch_count == before


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("weight", [(16, 6), (16, 10), (16,), (1, 16, 8)])
def test_operands_that_do_not_contract_are_refused(nodes, weight, grad):
    before = nodes.launch_count
    with pytest.raises((RuntimeError, IndexError)):
        nodes.linear(torch.ones(4, 8, dtype=torch.bfloat16, requires_grad=grad), torch.ones(*weight, dtype=torch.bfloat16))
    assert nodes.launch_count == before


@pytest.fixture
def compiler(monkeypatch, tmp_path):
    """A module path of its own and a compiler that writes what it was told to, slowly."""
    calls = []

    def run(cmd, **kwargs):
        target = Path(cmd[cmd.index("-o") + 1])
        calls.append(target)
        target.write_bytes(b"half")
        time.sleep(0.1)
        target.write_bytes(b"whole")
        return SimpleNamespace(returncode=run.code, stderr="refused", stdout="")

    run.code = 0
    monkeypatch.setattr(build, "LIB_DIR", tmp_path)
    monkeypatch.setattr(build, "AUTOGRAD_PATH", tmp_path / build.AUTOGRAD_PATH.name)
    monkeypatch.setattr(build.subprocess, "run", run)
    monkeypatch.setattr(build, "_nvcc", lambda: "/usr/local/cuda/bin/nvcc")
    return SimpleNamespace(calls=calls, run=run)


def test_the_module_is_named_after_what_it_fits():
    assert torch.__version__ in build.AUTOGRAD_PATH.name and sysconfig.get_config_var("SOABI") in build.AUTOGRAD_PATH.name


def test_processes_that_build_at_once_take_turns(compiler):
    """No reader sees half a file, and one of them compiles for all.  (The lock of an open file excludes threads as it does processes.)"""
    seen = []
    with ThreadPoolExecutor(4) as pool:
        jobs = [pool.submit(build.build_autograd) for _ in range(4)]
        while not all(j.done() for j in jobs):
            if build.AUTOGRAD_PATH.exists():
                seen.append(build.AUTOGRAD_PATH.read_bytes())
        assert {j.result() for j in jobs} == {build.AUTOGRAD_PATH}
    assert len(compiler.calls) == 1 and compiler.calls[0] != build.AUTOGRAD_PATH
    assert set(seen) <= {b"whole"} and build.AUTOGRAD_PATH.read_bytes() == b"whole"


def test_a_failed_build_leaves_the_module_as_it_was(compiler):
    build.AUTOGRAD_PATH.write_bytes(b"before")
    compiler.run.code = 1
    with pytest.raises(RuntimeError, match="refused"):
        build.build_autograd(force=True)
    assert build.AUTOGRAD_PATH.read_bytes() == b"before" and [p.name for p in build.LIB_DIR.iterdir() if p.suffix == ".part"] == []


def test_a_variant_of_the_library_brings_the_module_up_to_date(compiler, tmp_path):
    build.build(lib_path=tmp_path / "variant" / "libvariant.so")
    assert build.AUTOGRAD_PATH.read_bytes() == b"whole"


def test_without_a_compiler_the_python_nodes_serve(python_nodes, monkeypatch, tmp_path):
    nodes = python_nodes
    results = []
    for module in (nodes.AUTOGRAD, None):
        if module is None:
            monkeypatch.setattr(build, "AUTOGRAD_PATH", tmp_path / "absent.so")
            monkeypatch.setattr(build.subprocess, "run", lambda *a, **k: (_ for _ in ()).throw(FileNotFoundError("g++")))
            monkeypatch.setattr(build, "LIB_DIR", tmp_path)
            with pytest.warns(RuntimeWarning, match="Python autograd functions"):
                monkeypatch.setattr(nodes, "AUTOGRAD", nodes._load_autograd(nodes.LIB))
            assert nodes.AUTOGRAD is None and nodes.launch_count > 0
        x, w = _linear_case()
        bias = torch.linspace(-1, 1, 8, dtype=torch.bfloat16).requires_grad_()
        out = nodes.layer_norm(nodes.linear(x, w, bias), bias, bias, 1e-5)
        out.sum().backward()
        results.append([out.detach(), x.grad, w.grad, bias.grad])
    assert all(torch.equal(a, b) for a, b in zip(*results))


def test_an_import_that_builds_the_library_does_without_the_module(compiler, monkeypatch, tmp_path):
    """Where its headers are missing, the library is built and loaded all the same."""
    from tensor_parallel_b200.ops import native

    monkeypatch.setattr(build, "LIB_PATH", tmp_path / "libnew.so")
    monkeypatch.setattr(build, "OBJ_DIR", tmp_path / "obj")
    monkeypatch.setattr(build, "build_autograd", lambda *a: (_ for _ in ()).throw(RuntimeError("Python.h: No such file")))
    monkeypatch.setattr(native.ctypes, "CDLL", lambda path: path)
    monkeypatch.delenv("TPB_LIB_PATH", raising=False)
    assert native._load() == str(tmp_path / "libnew.so")


def test_a_library_of_another_layout_is_refused(nodes):
    library = SimpleNamespace(tpb_api_layout=ctypes.CFUNCTYPE(ctypes.c_ulonglong)(lambda: nodes.AUTOGRAD.layout() + 1))
    with pytest.raises(RuntimeError, match="rebuild"):
        nodes._load_autograd(library)


def test_the_launch_count_can_be_set(nodes):
    x, w = _linear_case()
    nodes.launch_count = 0
    nodes.linear(x, w)
    assert nodes.launch_count == 1
    nodes.launch_count += 4
    nodes.count_launches(2)
    nodes.linear(x, w)
    assert nodes.launch_count == 8


def test_threads_that_need_the_workspace_at_once(monkeypatch):
    """The nodes run without the interpreter lock, several threads at a time: who finds the workspace large enough finds its address too."""
    from tensor_parallel_b200.ops import native

    state, empty = native.DeviceState(torch.device("cpu")), torch.empty

    def slow(*args, **kwargs):
        time.sleep(0.05)
        return empty(*args, **kwargs)

    monkeypatch.setattr(torch, "empty", slow)

    def reserve(elems):
        state.ensure_slots(elems)
        return state.ctx.slot_stride >= elems and state.ctx.slots[0] == state.slots.data_ptr()

    with ThreadPoolExecutor(4) as pool:
        assert all(pool.map(reserve, [1000] * 4))
        assert all(pool.map(reserve, [1 << 21, 1 << 20, 1 << 21, 1000]))
