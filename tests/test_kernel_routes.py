"""Rules that choose a kernel, checked on the CPU: which GEMM shapes may take the single-rank kernels, how the few-token kernel deals
out its rows, and the relative-position bias by distance against the lookup of every pair."""
import ctypes
import re
import sys
import types

import pytest
import torch

from tensor_parallel_b200 import build
from tensor_parallel_b200.models.t5 import T5Attention, T5Config, relative_position_bucket
from tensor_parallel_b200.ops import functional as OF


def _plan(tokens, features, k, world=1, splits=0, kbox=0, no_swap=0):
    from tensor_parallel_b200.ops import native

    plan = native.GemmPlan()
    native.check(native.LIB.tpb_gemm_plan_ex(tokens, features, k, world, splits, kbox, no_swap, ctypes.byref(plan)), "gemm_plan")
    return plan


needs_library = pytest.mark.skipif(not build.LIB_PATH.exists(), reason="native library not built")


@needs_library
@pytest.mark.parametrize("tokens", [1, 16, 64, 65, 300, 4096, 8192])
@pytest.mark.parametrize("features,k", [(32, 64), (4096, 4096), (12288, 4096), (512, 16384), (1000, 520), (32003, 4096)])
def test_single_rank_kernels_leave_the_other_forms_alone(tokens, features, k):
    plan = _plan(tokens, features, k)
    assert not (plan.pair and plan.stream)
    assert not plan.pair or (not plan.swapped and plan.k_splits == 1 and plan.pair in (128, 256))
    assert not plan.stream or (plan.swapped and tokens <= 64)
    for other in (_plan(tokens, features, k, world=2), _plan(tokens, features, k, splits=1), _plan(tokens, features, k, splits=2)):
        assert other.pair == 0 and other.stream == 0
    assert _plan(tokens, features, k, no_swap=1).stream == 0
    # the fields of the tiled kernels do not depend on the choice
    forced = _plan(tokens, features, k, splits=plan.k_splits)
    assert (plan.swapped, plan.m_tiles, plan.n_tiles) == (forced.swapped, forced.m_tiles, forced.n_tiles)


@needs_library
@pytest.mark.parametrize("features", [1, 32, 33, 1000, 4736, 4737, 4768, 9472, 12288, 22016, 32003, 65024, 151936])
def test_row_ranges_cover_every_row_once_in_even_passes(features, sms=148):
    """The decomposition that the few-token kernel and its launch use: ranges of 32-row units, the same number of passes everywhere, none
    longer than the shared-memory layout or the 128 rows of an accumulator, none shorter than a box."""
    from tensor_parallel_b200.ops import native

    shape, starts = (ctypes.c_int * 5)(), (ctypes.c_int * 64)()

    def rows(cta):
        native.check(native.LIB.tpb_gemm_stream_rows(features, sms, cta, shape, starts, 64), "gemm_stream_rows")
        units, grid, passes, longest, box = shape
        return units, grid, passes, longest, box, list(starts[: passes + 1])

    units, grid, _, longest, box, _ = rows(0)
    assert units == -(-features // 32) and grid == min(units, sms) and 1 <= box <= longest <= 4
    covered = []
    for cta in range(grid):
        *_, at = rows(cta)
        assert all(box <= b - a <= longest for a, b in zip(at, at[1:]))
        covered += list(range(at[0], at[-1]))
    assert covered == list(range(units))


@pytest.mark.parametrize("decoder", [False, True])
@pytest.mark.parametrize("queries,keys", [(1, 1), (1, 40), (7, 12), (130, 130), (5, 300), (0, 0), (0, 4), (4, 0)])
def test_relative_bias_by_distance_equals_the_lookup_of_every_pair(decoder, queries, keys):
    torch.manual_seed(0)
    attention = T5Attention(T5Config(num_heads=3, d_kv=8), True, decoder)
    position = torch.arange(keys - queries, keys)[:, None]
    buckets = relative_position_bucket(torch.arange(keys)[None, :] - position, not decoder, 32, 128)
    want = attention.relative_attention_bias(buckets).permute(2, 0, 1)[None]
    got = attention.compute_bias(queries, keys, "cpu")
    assert torch.equal(got, want)
    g = torch.randn_like(got)
    table = attention.relative_attention_bias.weight
    (a,), (b,) = torch.autograd.grad(got, table, g), torch.autograd.grad(want, table, g)
    torch.testing.assert_close(a, b)


class _Launches:
    """Stands in for the native library: keeps the options of every GEMM that would have been launched."""

    def __init__(self):
        self.early = []

    def tpb_gemm_bf16_ex(self, *args):
        opts = args[15]
        self.early.append(bool(opts is not None and opts._obj.early))
        return 0


@needs_library
@pytest.mark.parametrize("pitch,offset,early", [(104, 0, True), (100, 0, False), (104, 1, False), (104, 8, True)])
def test_a_weight_that_has_to_be_copied_is_not_read_early(monkeypatch, pitch, offset, early):
    """An early launch reads its weights while the previous kernel of the stream runs; the copy of a weight that TMA cannot address
    (a pitch that is no multiple of 8 elements, a base off a 16-byte boundary) is exactly that kernel."""
    from tensor_parallel_b200.ops import native

    lib = _Launches()
    monkeypatch.setattr(native, "LIB", lib)
    monkeypatch.setattr(native, "gemm_plan", lambda *a, **k: native.GemmPlan(stream=1))
    monkeypatch.setattr(native, "device_state", lambda device: type("State", (), {"ctx": native.ReduceCtx()}))
    monkeypatch.setattr(native, "_stream", lambda: 0)
    storage = torch.zeros(64 * 104 + 64, dtype=torch.bfloat16)
    storage = storage[(-storage.data_ptr() % 16) // 2:]
    w = storage[offset:].as_strided((48, 100), (pitch, 1))
    x = torch.zeros(2, 104, dtype=torch.bfloat16)[:, :100]
    native.gemm_nt(x, w, early=True)
    native.gemm_nt(x, w)
    assert lib.early == [early, False]


@pytest.mark.parametrize("file,kernel,inputs", [("attention.cu", "attn_decode_fused_kernel", ["q", "k", "v"]), ("elementwise.cu", "greedy_pick_kernel", ["logits"])])
def test_early_kernels_do_not_call_their_predecessors_output_read_only(file, kernel, inputs):
    """A kernel that starts before its predecessor ends must not promise the compiler that what the predecessor writes is constant
    for the kernel's whole life (``const T* __restrict__`` allows read-only loads that move in front of the wait)."""
    source = (build.CSRC / file).read_text()
    (parameters,) = re.findall(r"\n" + kernel + r"\((.*?)\) \{", source, re.S)
    declared = [d.strip() for d in parameters.replace("\n", " ").split(",")]
    for name in inputs:
        (declaration,) = [d for d in declared if d.split()[-1] == name]
        assert "*" in declaration and "__restrict__" not in declaration


@needs_library
def test_preload_of_a_rank_loads_every_kernel_a_step_may_launch(monkeypatch):
    """A pass of one rank alone runs other GEMM kernels than a step of several ranks does, and one batch size runs only some of them:
    ``preload`` loads all of them by name."""
    from tensor_parallel_b200.engine import DecoderEngine
    from tensor_parallel_b200.ops import native

    loaded = []
    library = types.SimpleNamespace(tpb_gemm_preload=lambda: loaded.append("gemm") or 0, tpb_comm_preload=lambda: loaded.append("comm") or 0)
    monkeypatch.setattr(native, "LIB", library)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
    for comm, want in ((object(), {"gemm", "comm"}), (None, set())):
        engine = types.SimpleNamespace(comm=comm, world=2, head_split="vocab", embed_split=False, max_seq=80, device="cpu", vocab_local=32, x=torch.zeros(1, 8),
                                       logits_local=torch.zeros(1, 32), pos=torch.zeros(1), ids=torch.zeros(1), prefill=lambda ids: None, _decode_body=lambda batch: None)
        loaded.clear()
        DecoderEngine.preload(engine)
        assert set(loaded) == want and engine.comm is comm and engine.world == 2


class _Subclass(torch.Tensor):
    pass


class _Kernel:
    """Stands in for the native module: notes that the relative-bias kernel was chosen."""

    taken = False

    def relative_bias_supported(self, *a):
        return True

    def relative_bias(self, table, buckets, queries, keys):
        self.taken = True
        return torch.zeros(1, table.shape[1], queries, keys)


def _relative_bias_route(monkeypatch, embedding, buckets, queries, keys):
    kernel = _Kernel()
    monkeypatch.setattr(OF, "_native", lambda t: kernel)
    out = OF.relative_bias(embedding, buckets, queries, keys)
    monkeypatch.undo()
    return kernel.taken, out


class _OtherEmbedding(torch.nn.Embedding):
    pass


@pytest.mark.parametrize("kind", ["plain", "subclass", "forward on the instance", "hook", "pre-hook", "hook of all modules", "pre-hook of all modules",
                                  "backward hook of all modules", "padding", "sparse", "weight subclass"])
def test_an_embedding_that_does_more_than_look_up_is_called(monkeypatch, kind):
    embedding = (_OtherEmbedding if kind == "subclass" else torch.nn.Embedding)(8, 3, padding_idx=1 if kind == "padding" else None, sparse=kind == "sparse")
    handle, factor = None, 1.0
    if kind == "forward on the instance":
        embedding.forward = lambda index, plain=embedding.forward: plain(index) * 2
        factor = 2.0
    elif kind.startswith("hook"):
        register = embedding.register_forward_hook if kind == "hook" else torch.nn.modules.module.register_module_forward_hook
        handle = register(lambda module, args, out: out * 2)
        factor = 2.0
    elif kind.startswith("pre-hook"):
        register = embedding.register_forward_pre_hook if kind == "pre-hook" else torch.nn.modules.module.register_module_forward_pre_hook
        handle = register(lambda module, args: None)
    elif kind.startswith("backward"):
        handle = torch.nn.modules.module.register_module_full_backward_hook(lambda module, before, after: None)
    elif kind == "weight subclass":
        embedding.weight = torch.nn.Parameter(embedding.weight.data.as_subclass(_Subclass), requires_grad=False)
    buckets = torch.randint(0, 8, (9,))
    try:
        taken, out = _relative_bias_route(monkeypatch, embedding, buckets, 4, 6)
    finally:
        if handle is not None:
            handle.remove()
    assert taken == (kind == "plain")
    if not taken:
        distance = torch.arange(6)[None, :] - torch.arange(4)[:, None] + 3
        assert torch.equal(torch.as_tensor(out), embedding.weight[buckets[distance]].permute(2, 0, 1)[None] * factor)


@needs_library
@pytest.mark.parametrize("queries,keys,heads,taken", [(1, 1, 1, True), (0, 5, 2, False), (5, 0, 2, False), (0, 0, 2, False), (65535 * 16 + 1, 1, 1, False), (1, 1, 65536, False)])
def test_relative_bias_sizes_that_no_grid_covers_are_looked_up(queries, keys, heads, taken):
    from tensor_parallel_b200.ops import native

    table = torch.zeros(4, heads)
    assert native.relative_bias_supported(table, queries, keys) == taken
    if queries * keys == 0:  # the lookup has always taken these
        assert OF.relative_bias(torch.nn.Embedding(4, heads), torch.zeros(max(0, queries + keys - 1), dtype=torch.int64), queries, keys).shape == (1, heads, queries, keys)


@pytest.mark.parametrize("kind", ["vmap", "grad", "jvp", "forward mode", "trace", "fake tensors"])
def test_a_transformed_lookup_stays_with_pytorch(monkeypatch, kind):
    embedding = torch.nn.Embedding(8, 3)
    buckets = torch.randint(0, 8, (9,))
    kernel = _Kernel()
    monkeypatch.setattr(OF, "_native", lambda t: kernel)

    def bias(table):
        return torch.func.functional_call(_Bias(embedding, buckets), {"embedding.weight": table})

    table, tangent = embedding.weight.detach(), torch.randn(8, 3)
    want = OF.relative_bias_ref(embedding, buckets, 4, 6).detach()
    if kind == "vmap":
        assert torch.equal(torch.func.vmap(bias)(torch.stack([table, 2 * table])), torch.stack([want, 2 * want]))
    elif kind == "grad":
        assert torch.func.grad(lambda t: bias(t).sum())(table).sum() == want.numel()
    elif kind == "jvp":
        out, moved = torch.func.jvp(bias, (table,), (tangent,))
        assert torch.equal(out, want) and moved.shape == want.shape and moved.abs().sum() > 0
    elif kind == "forward mode":
        with torch.autograd.forward_ad.dual_level():
            out = bias(torch.autograd.forward_ad.make_dual(table, tangent))
            assert torch.autograd.forward_ad.unpack_dual(out).tangent is not None
    elif kind == "trace":
        traced = torch.jit.trace(_Bias(embedding, buckets), (), check_trace=False)
        with torch.no_grad():
            embedding.weight.mul_(2)
        assert torch.equal(traced(), 2 * want)
    else:
        from torch._subclasses.fake_tensor import FakeTensorMode

        with FakeTensorMode(allow_non_fake_inputs=True):
            assert OF.relative_bias(embedding, buckets, 4, 6).shape == want.shape
    assert not kernel.taken
    OF.relative_bias(embedding, buckets, 4, 6)
    assert kernel.taken


class _Bias(torch.nn.Module):
    def __init__(self, embedding, buckets):
        super().__init__()
        self.embedding, self.buckets = embedding, buckets

    def forward(self):
        return OF.relative_bias(self.embedding, self.buckets, 4, 6)


def test_table_gradient_of_a_relative_bias():
    embedding = torch.nn.Embedding(8, 3, dtype=torch.float64)
    buckets = torch.randint(0, 8, (9,))
    out = OF.relative_bias_ref(embedding, buckets, 4, 6)
    g = torch.randn_like(out)
    out.backward(g)
    torch.testing.assert_close(OF.relative_bias_table_grad_ref(g, buckets, 8).double(), embedding.weight.grad, atol=1e-5, rtol=1e-5)

    class Lookup(torch.autograd.Function):  # a batch of gradients reaches a backward as one batched tensor
        @staticmethod
        def forward(ctx, table):
            return OF.relative_bias_ref(lambda index: table[index], buckets, 4, 6)

        @staticmethod
        def backward(ctx, grad):
            assert OF.transformed(grad)
            return OF.relative_bias_table_grad_ref(grad, buckets, 8)

    table = embedding.weight.detach().float().requires_grad_()
    (batched,) = torch.autograd.grad(Lookup.apply(table), table, torch.stack([g, 2 * g]).float(), is_grads_batched=True)
    torch.testing.assert_close(batched.double(), torch.stack([embedding.weight.grad, 2 * embedding.weight.grad]), atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("buckets", [torch.zeros(8, dtype=torch.int64), torch.zeros(9), torch.zeros(9, dtype=torch.bool), torch.zeros(9, device="meta", dtype=torch.int64)])
def test_buckets_that_a_lookup_does_not_take_do_not_reach_the_kernel(monkeypatch, buckets):
    """Too few of them, of a type that is no index, on another device: PyTorch's own answer, mostly an error."""
    kernel = _Kernel()
    monkeypatch.setattr(OF, "_native", lambda t: kernel)
    embedding = torch.nn.Embedding(8, 3)
    if buckets.device.type == "meta":
        OF.relative_bias(embedding, buckets, 4, 6)
    else:
        with pytest.raises((IndexError, RuntimeError)):
            OF.relative_bias(embedding, buckets, 4, 6)
    assert not kernel.taken


@needs_library
@pytest.mark.parametrize("code,words", [(0, None), (1, "timed out"), (2, "peer GPU timed out"), (3, "index outside its range"), (9, "status 9")])
def test_a_step_says_what_its_kernels_reported(code, words):
    from tensor_parallel_b200.engine import DecoderEngine
    from tensor_parallel_b200.parallel.collectives import TPCollectiveError

    status = torch.full((4,), code, dtype=torch.int32)
    engine = types.SimpleNamespace(status_host=status.clone(), _status_tensor=lambda: status)
    if words is None:
        DecoderEngine._raise_on_status(engine)
    else:
        with pytest.raises(TPCollectiveError, match=words):
            DecoderEngine._raise_on_status(engine)
    assert int(status.sum()) == 0


@pytest.mark.parametrize("buckets,max_distance,inside", [(32, 128, "vmap"), (32, 128, "grad"), (32, 128, "jvp"), (32, 128, "another device"), (32, 128.0, ""),
                                                         (32, 2 ** 31, ""), (32, 128, "plain")])
def test_relative_buckets_of_a_program_that_transforms_its_functions(monkeypatch, buckets, max_distance, inside):
    """The kernel is asked for only where its result is a plain tensor on the current device, and for numbers that its entry takes."""
    asked = []
    monkeypatch.setitem(sys.modules, "tensor_parallel_b200.ops.native", types.SimpleNamespace(relative_buckets=lambda *a: asked.append(a)))
    import tensor_parallel_b200.ops as ops

    monkeypatch.setattr(ops, "native", sys.modules["tensor_parallel_b200.ops.native"], raising=False)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    device = "cuda:1" if inside == "another device" else "cuda:0"

    def call(t):
        assert OF.relative_buckets(-3, 7, device, True, buckets, max_distance) is None
        return t.sum()

    transform = dict(vmap=torch.vmap, grad=torch.func.grad, jvp=lambda f: lambda t: torch.func.jvp(f, (t,), (t,))).get(inside, lambda f: f)
    transform(call)(torch.ones(2, 3) if inside == "vmap" else torch.ones(3))
    assert len(asked) == (inside == "plain")
