"""Kernels at the sizes where their decompositions change: edges of tiles, remainders, odd strides, the smallest and largest of a
range, each against an fp32 / fp64 PyTorch statement of the same operation.

Tolerances: a bf16 result is half a unit in the last place (2^-9 relative) off its exact value by rounding alone; 2^-8 of the value
leaves room for the fp32 accumulation in front of it, plus an absolute term of a few fp32 roundings of the largest term."""
import ctypes
import math

import pytest
import torch

from tensor_parallel_b200.ops import functional as OF

pytestmark = pytest.mark.gpu


def _native():
    from tensor_parallel_b200.ops import native

    return native


def _close(got, want, terms=1.0):
    err = (got.double() - want).abs()
    bound = want.abs() * 2.0 ** -8 + terms * 2.0 ** -18
    assert bool((err <= bound).all()), f"largest excess {(err - bound).max().item():.3g} at value {want.flatten()[(err - bound).argmax()].item():.3g}"


def _gemm_ref(x, w, bias=None, act=None, residual=None):
    y = x.double() @ w.double().t()
    if bias is not None:
        y = y + bias.double()
    if act == "swiglu16":
        g = y.reshape(y.shape[0], -1, 2, 16)
        y = (torch.nn.functional.silu(g[:, :, 0]) * g[:, :, 1]).reshape(y.shape[0], -1)
    elif act == "gelu":
        y = torch.nn.functional.gelu(y)
    elif act == "relu":
        y = torch.relu(y)
    return y if residual is None else y + residual.double()


# tokens, features, k: whole pair tiles, one row / column / k-block more and less, a ragged last band of token tiles, an odd pitch
PAIR = [(2560, 2048, 256), (2561, 2047, 200), (4000, 1288, 72), (2303, 4100, 136), (8192, 384, 64), (5000, 1000, 1032)]


@pytest.mark.parametrize("tokens,features,k", PAIR)
@pytest.mark.parametrize("x_t,w_t", [(False, False), (False, True), (True, True)])
def test_pair_gemm(tokens, features, k, x_t, w_t):
    nat = _native()
    torch.manual_seed(tokens + features)
    assert nat.gemm_plan(tokens, features, k, no_swap=x_t or w_t).pair in (128, 256)
    x = torch.randn(tokens, k, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(features, k, device="cuda", dtype=torch.bfloat16) / math.sqrt(k)
    bias = torch.randn(features, device="cuda", dtype=torch.bfloat16)
    res = torch.randn(tokens, features, device="cuda", dtype=torch.bfloat16)
    args = (x.t().contiguous() if x_t else x, w.t().contiguous() if w_t else w)
    out = nat.gemm_nt(*args, bias=bias, residual=res, act="gelu", x_t=x_t, w_t=w_t)
    _close(out, _gemm_ref(x, w, bias, "gelu", res), terms=8)
    _close(nat.gemm_nt(*args, x_t=x_t, w_t=w_t), _gemm_ref(x, w), terms=8)
    nat.device_state(x.device).check_status()


@pytest.mark.parametrize("tokens", [2305, 8192])
def test_pair_gemm_gated_into_a_wider_buffer(tokens):
    nat = _native()
    torch.manual_seed(tokens)
    f, k = 1376, 264
    x = torch.randn(tokens, k, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(2 * f, k, device="cuda", dtype=torch.bfloat16) / math.sqrt(k)
    assert nat.gemm_plan(tokens, 2 * f, k).pair
    wide = torch.full((tokens, f + 24), 7.0, device="cuda", dtype=torch.bfloat16)
    nat.gemm_nt(x, w, act="swiglu16", out=wide[:, 16 : 16 + f])
    _close(wide[:, 16 : 16 + f], _gemm_ref(x, w, act="swiglu16"), terms=8)
    assert bool((wide[:, :16] == 7).all()) and bool((wide[:, 16 + f :] == 7).all())


# one unit of 32 rows, a ragged last unit, one unit per SM, one CTA with two, more than one pass of 128 rows per CTA
@pytest.mark.parametrize("features,k", [(32, 64), (40, 136), (1000, 520), (4736, 256), (4768, 1032), (2080, 1400), (4096, 4096), (22016, 264), (32003, 512)])
@pytest.mark.parametrize("tokens", [1, 8, 16, 17, 64])
def test_streamed_few_token_gemm(tokens, features, k):
    nat = _native()
    torch.manual_seed(tokens + features)
    assert nat.gemm_plan(tokens, features, k).stream
    x = torch.randn(tokens, k, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(features, k, device="cuda", dtype=torch.bfloat16) / math.sqrt(k)
    bias = torch.randn(features, device="cuda", dtype=torch.bfloat16)
    res = torch.randn(tokens, features, device="cuda", dtype=torch.bfloat16)
    _close(nat.gemm_nt(x, w, bias=bias, residual=res, act="relu"), _gemm_ref(x, w, bias, "relu", res), terms=8)
    _close(nat.gemm_nt(x, w, act="gelu"), _gemm_ref(x, w, act="gelu"), terms=8)
    if features % 32 == 0:
        _close(nat.gemm_nt(x, w, bias=bias, act="swiglu16"), _gemm_ref(x, w, bias, "swiglu16"), terms=8)
    nat.device_state(x.device).check_status()


@pytest.mark.parametrize("tokens", [1, 16, 40])
def test_early_launch_reads_what_its_predecessor_wrote(tokens):
    """A chain of dependent GEMMs launched ahead of one another gives the bits of the same chain in stream order."""
    nat = _native()
    torch.manual_seed(tokens)
    widths = [512, 4096, 1376, 4768, 512]
    ws = [torch.randn(b, a, device="cuda", dtype=torch.bfloat16) / math.sqrt(a) for a, b in zip(widths, widths[1:])]
    x0 = torch.randn(tokens, widths[0], device="cuda", dtype=torch.bfloat16)

    def chain(early):
        x = x0
        for _ in range(3):
            for w in ws:
                x = nat.gemm_nt(x, w, act="gelu", norm=(1, 1e-6, None), early=early)
        return x

    want = chain(False)
    for _ in range(5):
        assert torch.equal(chain(True), want)


def test_decode_step_with_weights_that_tma_cannot_address():
    """An OPT block of ffn_dim 100 copies its second MLP weight on every step (its pitch is no multiple of 16 bytes): a step with
    early launches gives the bits of a step without them."""
    import tensor_parallel_b200 as tp
    from tensor_parallel_b200.models.opt import OPTConfig, OPTForCausalLM

    nat = _native()
    torch.manual_seed(0)
    cfg = OPTConfig(vocab_size=512, hidden_size=256, num_hidden_layers=2, ffn_dim=100, num_attention_heads=4, max_position_embeddings=128)
    model = OPTForCausalLM(cfg).to("cuda", torch.bfloat16).eval()
    wrapped = tp.tensor_parallel(model, ["cuda:0"])
    wrapped.prefill(torch.randint(0, 512, (2, 9)), max_new_tokens=16)
    engine = wrapped._engine
    engine.use_graph = False
    start = engine.pos.clone()
    plain = nat.gemm_nt

    def steps():
        engine.pos.copy_(start)
        engine.ids[:2] = torch.tensor([3, 5], device="cuda")
        out = []
        for _ in range(5):
            engine.decode_step(2)
            out.append(engine.logits_local[:2].clone())
        return torch.stack(out)

    got = steps()
    try:
        nat.gemm_nt = lambda *a, early=False, **k: plain(*a, **k)
        want = steps()
    finally:
        nat.gemm_nt = plain
    assert torch.equal(got, want)
    engine.check_status()


@pytest.mark.parametrize("hq,hkv,d,splits", [(8, 8, 128, 1), (8, 2, 64, 4), (12, 2, 128, 2)])
def test_early_decode_attention_follows_the_projection(hq, hkv, d, splits):
    nat = _native()
    torch.manual_seed(hq)
    b, smax, hidden = 3, 320, 256
    x = torch.randn(b, hidden, device="cuda", dtype=torch.bfloat16)
    w = torch.randn((hq + 2 * hkv) * d, hidden, device="cuda", dtype=torch.bfloat16) / 16
    kc, vc = (torch.randn(b, hkv, smax, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    for pos in (0, 1, 31, 250, smax - 1):
        at = torch.tensor([pos], device="cuda", dtype=torch.int32)
        torch.cuda.synchronize()
        outs = []
        for early in (False, True, True):
            k2, v2 = kc.clone(), vc.clone()
            qkv = torch.zeros(b, w.shape[0], device="cuda", dtype=torch.bfloat16)
            nat.gemm_nt(x, w, out=qkv, early=early)
            q, k, v = qkv.split([hq * d, hkv * d, hkv * d], dim=1)
            outs.append((nat.attn_decode_fused(q, k, v, k2, v2, at, d, 10000.0, splits=splits, early=early), k2, v2))
        for other in outs[1:]:
            assert all(torch.equal(a, o) for a, o in zip(outs[0], other))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(1, 8), (2, 2048), (295, 2056), (297, 4096), (700, 5120), (61, 8192)])
@pytest.mark.parametrize("mode", ["rms", "layer"])
def test_norm_backward_row_and_column_edges(dtype, rows, cols, mode):
    torch.manual_seed(rows + cols)
    x = (torch.randn(rows, cols, device="cuda") * 2 + 0.1).to(dtype).requires_grad_()
    w = (1 + 0.1 * torch.randn(cols, device="cuda")).to(dtype).requires_grad_()
    b = torch.randn(cols, device="cuda").to(dtype).requires_grad_()
    g = torch.randn(rows, cols, device="cuda").to(dtype)
    xr, wr, br = (t.detach().double().requires_grad_() for t in (x, w, b))
    if mode == "rms":
        OF.rms_norm(x, w, 1e-6).backward(g)
        (xr * (xr.square().mean(-1, keepdim=True) + 1e-6).rsqrt() * wr).backward(g.double())
    else:
        OF.layer_norm(x, w, b, 1e-5).backward(g)
        torch.nn.functional.layer_norm(xr, (cols,), wr, br, 1e-5).backward(g.double())
    rel = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -17  # rounding of the result / of fp32 sums over up to 8192 terms
    for got, want in ((x.grad, xr.grad), (w.grad, wr.grad)) + (((b.grad, br.grad),) if mode == "layer" else ()):
        scale = want.square().mean().sqrt().item()
        err = (got.double() - want).abs()
        assert bool((err <= rel * (want.abs() + 2 * scale) + 1e-6).all()), (err.max().item(), scale)


@pytest.mark.parametrize("vocab", [8, 131, 4096, 5003])
def test_head_loss_rows_at_any_alignment(vocab):
    from tensor_parallel_b200.ops.loss import lm_head_cross_entropy

    torch.manual_seed(vocab)
    rows, hidden = 150, 128
    x = torch.randn(rows, hidden, device="cuda", dtype=torch.bfloat16).requires_grad_()
    w = (torch.randn(vocab, hidden, device="cuda", dtype=torch.bfloat16) * 0.2).requires_grad_()
    labels = torch.randint(0, vocab, (rows,), device="cuda")
    labels[::7] = -100
    loss = lm_head_cross_entropy(x, w, labels)
    loss.backward()
    xr, wr = x.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    want = torch.nn.functional.cross_entropy(xr @ wr.t(), labels)
    want.backward()
    assert abs(loss.item() - want.item()) <= 2e-3 * want.item() + 1e-3  # logits are rounded to bf16
    for got, ref in ((x.grad, xr.grad), (w.grad, wr.grad)):
        assert (got.double() - ref).norm() <= 0.02 * ref.norm()


# (every element by itself below 256 columns, one vector per thread below 8192, four from there on)
@pytest.mark.parametrize("cols", [1, 7, 255, 256, 261, 2049, 8191, 8192, 8203, 17000])
@pytest.mark.parametrize("pad", [0, 3])
def test_loss_kernels_at_the_edges_of_a_row(cols, pad):
    """Labels in the first and last element of each part of a row, outside this slice of the vocabulary, ignored; what lies between
    the rows stays."""
    from tensor_parallel_b200.ops import loss as L

    nat = _native()
    torch.manual_seed(cols + pad)
    rows, start = 24, 100
    wide = (3 * torch.randn(rows, cols + pad, device="cuda")).to(torch.bfloat16)
    logits, before = wide[:, :cols], wide.clone()
    local = torch.randint(0, cols, (rows,), device="cuda")
    local[:6] = torch.tensor([0, cols - 1, min(7, cols - 1), max(0, cols - 8), cols // 8 * 8 % cols, min(2048, cols - 1)])
    labels = local + start
    labels[6], labels[7], labels[8] = -100, start - 1, start + cols
    mine = (labels >= start) & (labels < start + cols)
    exact = logits.double()
    stats = torch.empty(rows, 4, device="cuda")
    nat.check(L.LIB.tpb_ce_stats(logits.data_ptr(), labels.data_ptr(), stats.data_ptr(), rows, cols, cols + pad, start, -100, nat._stream()), "ce_stats")
    lse = exact.logsumexp(-1)
    assert torch.equal(stats[:, 0].double(), exact.amax(-1)) and torch.equal(stats[:, 3] != 0, mine)
    # (the sum of up to 17000 fp32 exponentials: 1 + 2 units each, and a tree of additions of less than 80 levels)
    assert (stats[:, 0].double() + stats[:, 1].double().log() - lse).abs().max().item() <= 2.0 ** -17
    assert torch.equal(stats[mine, 2], exact[mine, local[mine]].float())
    lse, scale = lse.float(), torch.full((1,), 0.5, device="cuda")
    p = (logits.float() - lse[:, None]).double().exp()
    low, high = p * (1 - 2.0 ** -22), p * (1 + 2.0 ** -22)
    at = (torch.arange(rows, device="cuda")[mine], local[mine])
    low[at] -= 1
    high[at] -= 1
    low[6] = high[6] = 0
    nat.check(L.LIB.tpb_ce_grad(logits.data_ptr(), labels.data_ptr(), lse.data_ptr(), rows, cols, cols + pad, start, -100, scale.data_ptr(), nat._stream()), "ce_grad")
    assert _rounded_between(logits, 0.5 * low, 0.5 * high)
    assert torch.equal(wide[:, cols:], before[:, cols:])


def test_loss_statistics_with_infinite_logits():
    """Masked (-inf) logits carry no mass whatever vector, thread or edge they fall into."""
    from tensor_parallel_b200.ops import loss as L

    nat = _native()
    torch.manual_seed(0)
    rows, cols = 40, 4099
    logits = torch.randn(rows, cols, device="cuda", dtype=torch.bfloat16) * 4
    logits[torch.rand(rows, cols, device="cuda") < 0.5] = -math.inf
    logits[3, :4000] = -math.inf
    logits[4, 1:] = -math.inf
    logits[4, 0] = 1.0
    labels = torch.zeros(rows, dtype=torch.int64, device="cuda")
    stats = torch.empty(rows, 4, device="cuda")
    nat.check(L.LIB.tpb_ce_stats(logits.data_ptr(), labels.data_ptr(), stats.data_ptr(), rows, cols, cols, 0, -100, nat._stream()), "ce_stats")
    lse = stats[:, 0].double() + stats[:, 1].double().log()
    assert (lse - logits.double().logsumexp(-1)).abs().max().item() < 1e-5


def _rounded_between(got, low, high):
    """Every bf16 of ``got`` is the rounding of some value from ``low`` to ``high`` (fp64)."""
    low, high = torch.minimum(low, high), torch.maximum(low, high)
    return bool(((got >= low.float().to(torch.bfloat16)) & (got <= high.float().to(torch.bfloat16))).all())


def test_loss_gradient_has_the_accuracy_of_the_fp32_exponential():
    """Probabilities from 1 down to exp(-70), confident labels (p - 1 near 0) among them.  Given the fp32 difference of logit and
    log-sum-exp, the exponential is within 2 units in the last place: what is rounded to bf16 lies in that interval."""
    from tensor_parallel_b200.ops import loss as L

    nat = _native()
    torch.manual_seed(0)
    rows, cols = 1024, 4096
    logits = (-70 * torch.rand(rows, cols, device="cuda")).to(torch.bfloat16)
    labels = torch.randint(0, cols, (rows,), device="cuda")
    at = (torch.arange(rows, device="cuda"), labels)
    logits[at] = 0.0
    lse = torch.logspace(-7, 0, rows, device="cuda")  # (the label has all but 1e-7 .. all but 1 - 1 / e of the mass)
    p = (logits.float() - lse[:, None]).double().exp()
    low, high = p * (1 - 2.0 ** -22), p * (1 + 2.0 ** -22)
    low[at] -= 1
    high[at] -= 1
    scale = torch.ones(1, device="cuda")
    nat.check(L.LIB.tpb_ce_grad(logits.data_ptr(), labels.data_ptr(), lse.data_ptr(), rows, cols, cols, 0, -100, scale.data_ptr(), nat._stream()), "ce_grad")
    assert _rounded_between(logits, low, high)


# (a thread takes one vector of eight below 2^18 of them, two from there on)
@pytest.mark.parametrize("vectors", [5, 1 << 17, (1 << 18) - 1, (1 << 18) + 3])
@pytest.mark.parametrize("gated", [False, True])
def test_silu_has_the_accuracy_of_the_fp32_functions(gated, vectors):
    """On bf16 data too: expf (1 unit in the last place), the sum, the division and the products (half a unit each) stay within 2^-21 of
    the 64-bit value, 2^-20 of the terms of the derivative; what is rounded to bf16 lies in that interval."""
    torch.manual_seed(0)
    x = (160 * torch.rand(vectors, 8, device="cuda") - 80).to(torch.bfloat16).requires_grad_()
    u = (torch.rand(vectors, 8, device="cuda") + 0.5).to(torch.bfloat16).requires_grad_()
    g = torch.randn(vectors, 8, device="cuda").to(torch.bfloat16)
    out = OF.swiglu(x, u) if gated else _native()._ActFn.apply(x, None, 4)
    out.backward(g)
    xd, ud, gd = x.detach().double(), u.detach().double() if gated else 1.0, g.double()
    s = 1 / (1 + (-xd).exp())

    def near(want, terms, eps):
        return want - terms.abs() * eps, want + terms.abs() * eps

    assert _rounded_between(out.detach(), *near(xd * s * ud, xd * s * ud, 2.0 ** -21))
    assert _rounded_between(x.grad, *near(gd * s * (1 + xd * (1 - s)) * ud, gd * s * (1 + xd.abs() * (1 - s)) * ud, 2.0 ** -20))
    if gated:
        assert _rounded_between(u.grad, *near(gd * xd * s, gd * xd * s, 2.0 ** -21))


@pytest.mark.parametrize("heads,tokens", [(1, 3), (3, 700), (12, 65), (33, 2100)])
@pytest.mark.parametrize("interleaved,rotary", [(False, 128), (False, 64), (True, 32)])
def test_rope_head_groups(heads, tokens, interleaved, rotary):
    torch.manual_seed(heads)
    x = torch.randn(1, tokens, heads, 128, device="cuda", dtype=torch.bfloat16)
    pos = torch.randint(0, 4000, (1, tokens), device="cuda")
    got = OF.apply_rope(x, pos, 10000.0, rotary, interleaved)
    want = OF.apply_rope_ref(x.float(), pos, 10000.0, rotary, interleaved)
    # fp32 angles up to 4000 rad are 2.4e-4 rad off between two fp32 evaluations of the frequency
    assert (got.float() - want).abs().max().item() <= 2.0 ** -8 * want.abs().max().item() + 5e-3
    assert torch.equal(got[..., rotary:], x[..., rotary:])


# one head per thread, several, the step between them and rounds of a launch; rows past the end of the cache
@pytest.mark.parametrize("heads,kv,d,rotary,interleaved", [(8, 8, 128, 128, False), (12, 3, 64, 64, False), (9, 1, 128, 32, False), (4, 2, 128, 64, True), (32, 32, 128, 128, False)])
@pytest.mark.parametrize("batch,seq", [(1, 1), (3, 67), (1, 760), (2, 1500), (1, 4000)])
def test_rotary_append_by_head_groups(heads, kv, d, rotary, interleaved, batch, seq):
    nat = _native()
    torch.manual_seed(heads + seq)
    base, room = 5, seq + 3  # (the last two tokens lie past the end of the cache)
    qkv = torch.randn(batch * seq, (heads + 2 * kv) * d, device="cuda", dtype=torch.bfloat16)
    q, k, v = qkv.split([heads * d, kv * d, kv * d], dim=1)
    kc, vc = (torch.full((batch, kv, room, d), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    out = torch.empty(batch * seq, heads * d, device="cuda", dtype=torch.bfloat16)
    nat.qkv_rope_append(q, k, v, out, kc, vc, torch.tensor([base], device="cuda", dtype=torch.int32), batch, seq, rotary, 10000.0, interleaved=interleaved)
    pos = torch.arange(base, base + seq, device="cuda")[None].expand(batch, seq)
    kept = max(0, min(seq, room - base))

    def close(got, x, n):
        x = x.reshape(batch, seq, n, d)
        want = OF.apply_rope_ref(x.float(), pos, 10000.0, rotary, interleaved)[:, :kept]
        # angles up to 4000 rad: 2.4e-4 rad between two fp32 evaluations of the frequency
        assert (got[:, :kept].float() - want).abs().max().item() <= (2.0 ** -8 * want.abs().max().item() + 5e-3 if kept else 0)
        assert torch.equal(got[:, :kept, :, rotary:], x[:, :kept, :, rotary:])

    if kept:
        close(out.view(batch, seq, heads, d), q, heads)
        close(kc[:, :, base : base + kept].transpose(1, 2), k, kv)
        assert torch.equal(vc[:, :, base : base + kept].transpose(1, 2), v.reshape(batch, seq, kv, d)[:, :kept])
    assert bool((kc[:, :, :base] == 7).all()) and bool((vc[:, :, :base] == 7).all())


# (vectors of eight from 2^19 elements on)
@pytest.mark.parametrize("n,offset", [(1, 0), (7, 0), (8, 0), (4099, 0), (4096, 1), ((1 << 19) - 1, 0), (1 << 19, 0), ((1 << 19) + 7, 0), (1 << 19, 1)])
@pytest.mark.parametrize("dtype,gdtype", [(torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float32, torch.float32)])
def test_adamw_remainders_and_alignment(n, offset, dtype, gdtype):
    nat = _native()
    torch.manual_seed(n)

    def make(dt, scale=1.0):
        return (torch.rand(n + offset, device="cuda") * scale).to(dt)[offset:]

    p, g, m, v = make(dtype), make(gdtype, 0.1), make(torch.float32, 0.1), make(torch.float32, 0.01)
    master = p.float().clone() if dtype == torch.bfloat16 else None
    p0, m0, v0 = p.double(), m.double(), v.double()
    nat.adamw_step(p, g, m, v, 3, 1e-2, 0.9, 0.99, 1e-8, 0.1, master=master)
    m1, v1 = 0.9 * m0 + 0.1 * g.double(), 0.99 * v0 + 0.01 * g.double() ** 2
    want = p0 * (1 - 1e-3) - 1e-2 * (m1 / (1 - 0.9 ** 3)) / ((v1 / (1 - 0.99 ** 3)).sqrt() + 1e-8)
    for got, ref in ((m, m1), (v, v1), (p if master is None else master, want)):
        assert (got.double() - ref).abs().max().item() <= 2e-6  # a few fp32 roundings of values below 1 (1 - 0.99f is 1e-6 off)
    if master is not None:
        assert torch.equal(p, master.to(torch.bfloat16))


@pytest.mark.parametrize("cols", [1, 5, 8, 515, 32000, 50257])
def test_greedy_pick_matches_torch_argmax(cols):
    nat = _native()
    torch.manual_seed(cols)
    rows = 9
    logits = torch.randn(rows, cols, device="cuda", dtype=torch.bfloat16)  # bf16: ties are common
    logits[1] = 0.25
    logits[2] = -math.inf
    logits[3, cols // 2] = math.nan
    logits[4, cols // 3 :] = math.nan
    logits[5, -1] = 1000.0
    nxt, ids = torch.zeros(rows, dtype=torch.int64, device="cuda"), torch.zeros(rows, dtype=torch.int64, device="cuda")
    pos = torch.tensor([41], dtype=torch.int32, device="cuda")
    nat.greedy_pick(logits, nxt, ids, pos)
    want = logits.cpu().float().argmax(-1)
    assert torch.equal(nxt.cpu(), want) and torch.equal(ids, nxt) and pos.item() == 42


@pytest.mark.parametrize("sq,sk", [(64, 128), (150, 152), (150, 150), (300, 520)])
@pytest.mark.parametrize("layout", ["dense", "heads_last", "padding", "fp32"])
def test_bias_rows_in_vectors_and_one_by_one(sq, sk, layout):
    torch.manual_seed(sq + sk)
    b, h, d = 3, 4, 64
    q = torch.randn(b, sq, h, d, device="cuda", dtype=torch.bfloat16).requires_grad_()
    k, v = (torch.randn(b, sk, h, d, device="cuda", dtype=torch.bfloat16).requires_grad_() for _ in range(2))
    if layout == "heads_last":
        leaf = torch.randn(sq, sk, h, device="cuda", dtype=torch.bfloat16).requires_grad_()
        bias = leaf.permute(2, 0, 1)[None]
    elif layout == "padding":
        leaf = torch.zeros(b, 1, 1, sk, device="cuda", dtype=torch.bfloat16)
        leaf[1, :, :, sk // 2 :] = -math.inf
        bias = leaf
    else:
        leaf = torch.randn(1, h, sq, sk, device="cuda", dtype=torch.float32 if layout == "fp32" else torch.bfloat16).requires_grad_()
        bias = leaf
    g = torch.randn(b, sq, h, d, device="cuda", dtype=torch.bfloat16)
    OF.attention(q, k, v, False, bias=bias).backward(g)
    ref = [t.detach().double().requires_grad_() for t in (q, k, v, bias)]
    scores = torch.einsum("bqhd,bkhd->bhqk", ref[0], ref[1]) / math.sqrt(d) + ref[3]
    torch.einsum("bhqk,bkhd->bqhd", scores.softmax(-1), ref[2]).backward(g.double())
    got = [q.grad, k.grad, v.grad] + ([] if layout == "padding" else [leaf.grad.permute(2, 0, 1)[None] if layout == "heads_last" else leaf.grad])
    for a, r in zip(got, ref):
        # probabilities and dS pass through bf16 (2^-9 each) on their way into sums that cancel
        assert (a.double() - r.grad).norm() <= 0.02 * r.grad.norm()


# head_dim 128 and 64, causal with several key tiles and with a shift, grouped heads, a bias for each batch or for all heads, ragged tiles
@pytest.mark.parametrize("b,sq,sk,hq,hkv,d,causal,shape", [
    (2, 304, 304, 4, 2, 128, True, (1, 4, 304, 304)), (2, 200, 328, 4, 2, 64, True, (2, 4, 200, 328)), (1, 136, 264, 8, 8, 128, False, (1, 1, 136, 264)),
    (3, 128, 128, 2, 2, 128, False, (3, 2, 128, 128)), (2, 65, 72, 4, 1, 64, True, (1, 4, 65, 72)), (2, 257, 384, 6, 2, 128, True, (2, 1, 257, 384)),
    # rows that no vector fits: element by element
    (1, 301, 303, 4, 2, 128, True, (1, 4, 301, 303)), (2, 150, 260, 2, 2, 64, False, (2, 2, 150, 260))])
def test_dense_bf16_bias(b, sq, sk, hq, hkv, d, causal, shape):
    torch.manual_seed(sq + sk)
    q = torch.randn(b, sq, hq, d, device="cuda", dtype=torch.bfloat16).requires_grad_()
    k, v = (torch.randn(b, sk, hkv, d, device="cuda", dtype=torch.bfloat16).requires_grad_() for _ in range(2))
    bias = torch.randn(shape, device="cuda", dtype=torch.bfloat16)
    bias[..., 1:].masked_fill_(torch.rand(shape, device="cuda")[..., 1:] < 0.1, -math.inf)
    bias.requires_grad_()
    g = torch.randn(b, sq, hq, d, device="cuda", dtype=torch.bfloat16)
    out = OF.attention(q, k, v, causal, bias=bias)
    out.backward(g)
    ref = [t.detach().double().requires_grad_() for t in (q, k, v, bias)]
    keys, values = (t.repeat_interleave(hq // hkv, 2) for t in ref[1:3])
    scores = torch.einsum("bqhd,bkhd->bhqk", ref[0], keys) / math.sqrt(d) + ref[3]
    if causal:
        scores = scores.masked_fill(torch.ones(sq, sk, dtype=torch.bool, device="cuda").triu(sk - sq + 1), -math.inf)
    want = torch.einsum("bhqk,bkhd->bqhd", scores.softmax(-1), values)
    want.backward(g.double())
    # probabilities and dS pass through bf16 (2^-9 each) on their way into sums that cancel
    for a, r in zip((out.detach(), q.grad, k.grad, v.grad, bias.grad), (want.detach(), *(t.grad for t in ref))):
        assert (a.double() - r).norm() <= 0.02 * r.norm()
    _native().device_state(q.device).check_status()


@pytest.mark.parametrize("queries,keys", [(1, 1), (1, 9), (17, 40), (64, 1032), (65, 2100), (512, 512)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_relative_bias_and_its_gradient(queries, keys, dtype):
    torch.manual_seed(queries + keys)
    heads, n = 5, 40
    emb = torch.nn.Embedding(n, heads, device="cuda", dtype=dtype)
    ref = torch.nn.Embedding(n, heads, device="cuda", dtype=torch.float64)
    ref.weight.data.copy_(emb.weight.data)
    buckets = torch.randint(0, n, (queries + keys - 1,), device="cuda")
    out = OF.relative_bias(emb, buckets, queries, keys)
    want = OF.relative_bias_ref(ref, buckets, queries, keys)
    assert out.is_contiguous() and torch.equal(out.double(), want)
    g = torch.randn(1, heads, queries, keys, device="cuda").to(dtype)
    out.backward(g)
    want.backward(g.double())
    rel = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20
    err = (emb.weight.grad.double() - ref.weight.grad).abs()
    assert bool((err <= rel * ref.weight.grad.abs() + 2.0 ** -22 * queries * keys ** 0.5).all())


def test_relative_bias_under_transforms():
    """Second derivative, a batch of output gradients and forward mode, as the lookup itself gives them."""
    torch.manual_seed(0)
    heads, n, queries, keys = 5, 12, 33, 40
    emb = torch.nn.Embedding(n, heads, device="cuda")
    buckets = torch.randint(0, n, (queries + keys - 1,), device="cuda")
    out = OF.relative_bias(emb, buckets, queries, keys)
    want = OF.relative_bias_ref(emb, buckets, queries, keys)
    assert type(out.grad_fn).__name__.startswith("_RelativeBiasFn")
    gs = torch.randn(3, *out.shape, device="cuda")
    (batched,) = torch.autograd.grad(out, emb.weight, gs, is_grads_batched=True, retain_graph=True)
    for got, g in zip(batched, gs):
        torch.testing.assert_close(got, torch.autograd.grad(want, emb.weight, g, retain_graph=True)[0], atol=1e-4, rtol=1e-5)
    g = gs[0].clone().requires_grad_()
    (first,) = torch.autograd.grad(out, emb.weight, g, create_graph=True)
    weights = torch.randn(n, heads, device="cuda")
    (second,) = torch.autograd.grad((first * weights).sum(), g)
    table = torch.nn.Embedding(n, heads, device="cuda", _weight=weights)
    assert torch.equal(second, OF.relative_bias_ref(table, buckets, queries, keys))

    with torch.autograd.forward_ad.dual_level():
        emb.weight.requires_grad_(False)
        stand_in = torch.nn.Embedding(n, heads, device="cuda")
        del stand_in.weight
        stand_in.weight = torch.autograd.forward_ad.make_dual(emb.weight.data, weights)
        moved = torch.autograd.forward_ad.unpack_dual(OF.relative_bias(stand_in, buckets, queries, keys)).tangent
        assert torch.equal(moved, OF.relative_bias_ref(table, buckets, queries, keys))


@pytest.mark.parametrize("bad", [12, -1, 2 ** 32, -(2 ** 32) + 3])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_relative_bias_with_a_bucket_out_of_range(bad, dtype):
    """No row is read for it: its distance is NaN in every head, the status word says so, and its gradient goes nowhere."""
    nat = _native()
    torch.manual_seed(0)
    heads, n, queries, keys = 3, 12, 20, 33
    emb = torch.nn.Embedding(n, heads, device="cuda", dtype=dtype)
    buckets = torch.randint(0, n, (queries + keys - 1,), device="cuda")
    want = OF.relative_bias_ref(emb, buckets, queries, keys).detach()
    distance = torch.arange(keys, device="cuda")[None, :] - torch.arange(queries, device="cuda")[:, None] + queries - 1
    hit = (distance == 30)[None, None].expand_as(want)
    buckets[30] = bad
    out = OF.relative_bias(emb, buckets, queries, keys)
    assert bool(out[hit].isnan().all()) and torch.equal(out[~hit], want[~hit])
    with pytest.raises(RuntimeError, match="index"):
        nat.device_state(out.device).check_status()
    out.backward(hit.to(dtype))
    assert emb.weight.grad.abs().max().item() == 0
    nat.device_state(out.device).check_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 264), (149, 4096), (1200, 256), (700, 5120), (600, 8192), (5, 8200)])
@pytest.mark.parametrize("mode", [0, 1])
def test_norm_forward_in_rings_of_rows(dtype, rows, cols, mode):
    """Fewer rows than CTAs, rings that go round, one warp and 32 per row, and a row too wide for a ring."""
    nat = _native()
    torch.manual_seed(rows + cols)
    x = (torch.randn(rows, cols, device="cuda") * 2 + 0.1).to(dtype)
    w = (1 + 0.1 * torch.randn(cols, device="cuda")).to(dtype)
    bias = torch.randn(cols, device="cuda").to(dtype) if mode else None
    out, rstd, mean = nat.norm_forward(x, w, bias, 1e-6, mode, want_stats=True)
    xd = x.double()
    mu = xd.mean(-1, keepdim=True) if mode else torch.zeros(rows, 1, device="cuda", dtype=torch.double)
    r = ((xd - mu).square().mean(-1, keepdim=True) + 1e-6).rsqrt()
    want = (xd - mu) * r * w.double() + (bias.double() if mode else 0)
    rel = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -18  # rounding of the result / of fp32 sums over up to 8200 terms
    assert bool(((out.double() - want).abs() <= rel * (want.abs() + 1)).all())
    assert bool(((rstd.double() - r[:, 0]).abs() <= 2.0 ** -18 * r[:, 0]).all())
    if mode:
        assert bool(((mean.double() - mu[:, 0]).abs() <= 2.0 ** -20).all())


@pytest.mark.parametrize("rows", [1, 255, 257, 8192, 70001])
@pytest.mark.parametrize("world", [1, 3])
def test_loss_over_the_statistics_of_several_ranks(rows, world):
    """One thread per row, one partial per 256 rows; ignored rows, a slice without a finite logit, no row that counts."""
    _native()
    from tensor_parallel_b200.ops import loss as L

    torch.manual_seed(rows)
    stats = torch.randn(world, rows, 4, device="cuda") * 4
    stats[..., 1] = stats[..., 1].abs() + 1
    labels = torch.randint(0, 100, (rows,), device="cuda")
    labels[::3] = -100
    for ignored in (-100, None):
        if ignored is None:
            labels[:] = -100
        lse, loss, count = torch.empty(rows, device="cuda"), torch.empty((), device="cuda"), torch.empty(1, device="cuda")
        partials = torch.empty(L.LIB.tpb_ce_loss_parts(rows), 2, device="cuda")
        L.check(L.LIB.tpb_ce_loss(stats.data_ptr(), labels.data_ptr(), lse.data_ptr(), partials.data_ptr(), loss.data_ptr(), count.data_ptr(), world, rows, -100,
                                  L.native._stream()), "ce_loss")
        d = stats.double()
        want = torch.logsumexp(d[..., 0] + d[..., 1].log(), dim=0)
        assert bool(((lse.double() - want).abs() <= 2.0 ** -20 * (1 + want.abs())).all())
        valid = labels != -100
        shares = (want - d[..., 2].sum(0)) * valid
        assert count.item() == max(int(valid.sum()), 1)
        # fp32: the shares' own rounding, and a sum of a few hundred terms deep
        assert abs(loss.item() - shares.sum().item() / count.item()) <= 2.0 ** -16 * (shares.abs().sum().item() / count.item() + 1e-6)
    stats[0, 0] = torch.tensor([float("-inf"), float("nan"), 0.0, 0.0])
    L.check(L.LIB.tpb_ce_loss(stats.data_ptr(), labels.data_ptr(), lse.data_ptr(), partials.data_ptr(), loss.data_ptr(), count.data_ptr(), world, rows, -100,
                              L.native._stream()), "ce_loss")
    assert math.isnan(lse[0].item()) and math.isnan(loss.item()) and not lse[1:].isnan().any()


@pytest.mark.parametrize("b,sq,sk,hq,hkv,causal", [(1, 1, 1, 1, 1, True), (2, 127, 129, 2, 1, False), (1, 128, 128, 4, 2, True), (1, 129, 257, 6, 2, True),
                                                   (2, 300, 130, 2, 2, True), (1, 1000, 1000, 3, 1, True), (1, 640, 384, 2, 2, False)])
def test_attention_backward_in_wide_steps(b, sq, sk, hq, hkv, causal):
    """head_dim 128 without a bias, few steps: the launches that stream at least 65 of the last 128 rows take the kernel of 128 rows per step,
    those that end in a first half the one of 64; ragged ends, more rounds than the rings are deep, grouped heads, queries that see no key
    (sq > sk, causal).  (Which launch takes which: test_attention_backward_by_step.)"""
    nat = _native()
    torch.manual_seed(sq + sk)
    q, k, v = (torch.randn(b, s, h, 128, device="cuda", dtype=torch.bfloat16).requires_grad_() for s, h in ((sq, hq), (sk, hkv), (sk, hkv)))
    g = torch.randn(b, sq, hq, 128, device="cuda", dtype=torch.bfloat16)
    nat.attention(q, k, v, causal).backward(g)
    qr, kr, vr = (t.detach().double() for t in (q, k, v))
    for t in (qr, kr, vr):
        t.requires_grad_()
    kh, vh = (t.repeat_interleave(hq // hkv, 2) for t in (kr, vr))
    scores = torch.einsum("bqhd,bkhd->bhqk", qr, kh) / math.sqrt(128)
    if causal:
        hidden = torch.ones(sq, sk, dtype=torch.bool, device="cuda").triu(sk - sq + 1)
        scores = scores.masked_fill(hidden, -1e300)  # (a row without keys becomes uniform, and is removed again)
        probs = scores.softmax(-1).masked_fill(hidden, 0.0)
    else:
        probs = scores.softmax(-1)
    torch.einsum("bhqk,bkhd->bqhd", probs, vh).backward(g.double())
    nat.device_state(q.device).check_status()
    for got, want in ((q.grad, qr.grad), (k.grad, kr.grad), (v.grad, vr.grad)):
        # probabilities, dS and results are rounded to bf16 once each (2^-9 relative, independent errors), the output that delta reads too
        assert (got.double() - want).norm() <= 2.0 ** -7 * want.norm() + 1e-6


@pytest.mark.parametrize("hq,hkv,d", [(4, 1, 128), (10, 2, 64), (16, 1, 64), (34, 2, 128), (12, 3, 128)])
@pytest.mark.parametrize("ctx", [0, 15, 16, 129, 700])
@pytest.mark.parametrize("splits", [1, 3])
def test_decode_attention_of_grouped_heads(hq, hkv, d, ctx, splits):
    """Four and more query heads per KV head: one whole group, several, a remainder in groups of its own; no cached key, a few, rings that
    go round, splits without a key, rows of non-zero data behind the cache's end."""
    nat = _native()
    torch.manual_seed(hq + ctx)
    b, smax = 3, 720
    kc, vc = (torch.randn(b, hkv, smax, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    vc[:, :, ctx + 1:] = float("inf")  # (what lies behind the newest key is never used)
    qkv = torch.randn(b, (hq + 2 * hkv) * d, device="cuda", dtype=torch.bfloat16)
    q, k, v = qkv.split([hq * d, hkv * d, hkv * d], dim=1)
    at = torch.tensor([ctx], device="cuda", dtype=torch.int32)
    out = nat.attn_decode_fused(q, k, v, kc, vc, at, d, 10000.0, splits=splits)
    rot = lambda x, heads: OF.apply_rope_ref(x.reshape(b, 1, heads, d).float(), at.long().view(1, 1).expand(b, 1), 10000.0)[:, 0]
    assert torch.equal(vc[:, :, ctx], v.reshape(b, hkv, d))
    assert bool(((kc[:, :, ctx].double() - rot(k, hkv).double()).abs() <= 2.0 ** -7 * rot(k, hkv).abs() + 1e-3).all())
    qr = rot(q, hq).to(torch.bfloat16).double()
    kd, vd = (t[:, :, : ctx + 1].double().repeat_interleave(hq // hkv, 1) for t in (kc, vc))
    probs = (torch.einsum("bhd,bhnd->bhn", qr, kd) / math.sqrt(d)).softmax(-1)
    want = torch.einsum("bhn,bhnd->bhd", probs, vd)
    # the result's rounding, and that of the rotated query (half a unit of 2^-8, either way) in a handful of its elements
    err = (out.view(b, hq, d).double() - want).abs()
    assert bool((err <= 2.0 ** -7 * want.abs() + 2.0 ** -7 * want.abs().amax(-1, keepdim=True) + 1e-4).all()), err.max()


@pytest.mark.parametrize("hq,hkv,d", [(2, 2, 128), (8, 1, 64), (16, 1, 64), (8, 2, 128)])
@pytest.mark.parametrize("splits", [2, 3])
def test_decode_attention_keeps_its_partial_results_in_32_bits(hq, hkv, d, splits):
    """Scores, probabilities and sums of a split stay fp32: its maximum, sum and unnormalised output, as they lie in the workspace."""
    nat = _native()
    torch.manual_seed(hq + d)
    b, ctx, smax = 2, 1000, 1024
    kc, vc = (torch.randn(b, hkv, smax, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    qkv = torch.randn(b, (hq + 2 * hkv) * d, device="cuda", dtype=torch.bfloat16)
    q, k, v = qkv.split([hq * d, hkv * d, hkv * d], dim=1)
    part_o, part_ml = torch.empty(b, hq, splits, d, device="cuda"), torch.empty(b, hq, splits, 2, device="cuda")
    counters = torch.zeros(b * hq, dtype=torch.int32, device="cuda")
    nat.attn_decode_fused(q, k, v, kc, vc, torch.tensor([ctx], device="cuda", dtype=torch.int32), 0, 10000.0, splits=splits, workspace=(part_o, part_ml, counters))
    kd, vd = (t[:, :, : ctx + 1].double().repeat_interleave(hq // hkv, 1) for t in (kc, vc))
    scores = torch.einsum("bhd,bhnd->bhn", q.reshape(b, hq, d).double(), kd) / math.sqrt(d) * math.log2(math.e)
    chunk = -(-(ctx + 1) // splits)
    for i in range(splits):
        at = slice(i * chunk, (i + 1) * chunk)
        top = scores[..., at].amax(-1)
        p = (scores[..., at] - top[..., None]).exp2()
        assert bool(((part_ml[:, :, i, 0].double() - top).abs() <= 2.0 ** -20 * (1 + top.abs())).all())
        # A score is a sum of d products in fp32: a few roundings of at most 2^-24 of its magnitude (4 or so), independent from key to key, and
        # the same again from the maximum, which is common to all keys: below 1e-6 of both results.  Probabilities of 17 bits exceed it.
        for got, want in ((part_ml[:, :, i, 1], p.sum(-1)), (part_o[:, :, i], torch.einsum("bhn,bhnd->bhd", p, vd[:, :, at]))):
            assert (got.double() - want).norm() <= 1e-6 * want.norm()


@pytest.mark.parametrize("group,d", [(4, 128), (16, 128), (16, 64)])
@pytest.mark.parametrize("outlier", [0, 8, 30, 100])
@pytest.mark.parametrize("ctx", [30, 1000, 2400])
def test_decode_attention_of_grouped_heads_is_as_exact_as_of_single_ones(group, d, outlier, ctx):
    """Outputs before their rounding against 64 bits, from heads that share a KV head and from the same heads two by two, which take a kernel with fp32
    multiplications and additions on the CUDA cores; also where scores are small sums of large products (a few channels of magnitude `outlier`)."""
    nat = _native()
    torch.manual_seed(group + d + outlier)
    b, splits = 4, 2
    kc, vc = (torch.randn(b, 1, ctx + 8, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    qkv = torch.randn(b, (group + 2) * d, device="cuda", dtype=torch.bfloat16)
    for c in (2, 17, 40, 59) if outlier else ():  # two channels whose products with q are each other's negative
        c2 = (c + 21) % d
        qkv.view(b, -1, d)[:, :group, c2] = qkv.view(b, -1, d)[:, :group, c] = outlier * (1 + 0.3 * torch.rand(b, group, device="cuda"))
        kc[..., c] = outlier * (1 + 0.3 * torch.rand(b, 1, ctx + 8, device="cuda"))
        kc[..., c2] = -kc[..., c]
    q, k, v = qkv.split([group * d, d, d], dim=1)
    at = torch.tensor([ctx], device="cuda", dtype=torch.int32)

    def merged(q, heads):
        part_o, part_ml = torch.empty(b, heads, splits, d, device="cuda"), torch.empty(b, heads, splits, 2, device="cuda")
        nat.attn_decode_fused(q, k, v, kc, vc, at, 0, 10000.0, splits=splits, workspace=(part_o, part_ml, torch.zeros(b * heads, dtype=torch.int32, device="cuda")))
        w = (part_ml[..., 0].double() - part_ml[..., 0].double().amax(-1, keepdim=True)).exp2()
        return (part_o.double() * w[..., None]).sum(2) / (part_ml[..., 1].double() * w).sum(2)[..., None]

    got = merged(q, group)
    single = torch.cat([merged(q[:, i * d : (i + 2) * d], 2) for i in range(0, group, 2)], dim=1)
    kd, vd = (t[:, :, : ctx + 1].double().expand(-1, group, -1, -1) for t in (kc, vc))
    want = torch.einsum("bhn,bhnd->bhd", (torch.einsum("bhd,bhnd->bhn", q.reshape(b, group, d).double(), kd) / math.sqrt(d)).softmax(-1), vd)
    assert (got - want).norm() <= (single - want).norm()


@pytest.mark.parametrize("hq,hkv,d", [(4, 1, 128), (16, 1, 64), (2, 2, 64)])
@pytest.mark.parametrize("splits", [1, 3])
def test_decode_attention_of_infinite_values(hq, hkv, d, splits):
    """An infinite cached value gives an infinite element of the output (its probability is above zero), and no NaN anywhere."""
    nat = _native()
    torch.manual_seed(hq + d)
    b, ctx, smax = 2, 300, 320
    kc, vc = (torch.randn(b, hkv, smax, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    vc[:, :, 17, 3] = float("inf")
    vc[:, :, 250, 5] = float("-inf")
    qkv = torch.randn(b, (hq + 2 * hkv) * d, device="cuda", dtype=torch.bfloat16)
    q, k, v = qkv.split([hq * d, hkv * d, hkv * d], dim=1)
    out = nat.attn_decode_fused(q, k, v, kc, vc, torch.tensor([ctx], device="cuda", dtype=torch.int32), d, 10000.0, splits=splits).view(b, hq, d)
    want = torch.zeros_like(out, dtype=torch.float32)
    want[..., 3], want[..., 5] = float("inf"), float("-inf")
    assert torch.equal(out.float().nan_to_num(nan=7.0, posinf=1e9, neginf=-1e9).abs() >= 1e9, want.abs() > 0)
    assert bool((out[..., 3] == float("inf")).all() and (out[..., 5] == float("-inf")).all()) and not out.isnan().any()


@pytest.mark.parametrize("hq,hkv,d", [(4, 1, 128), (16, 1, 64), (23, 1, 64), (1, 1, 128), (2, 1, 64), (3, 1, 128)])
@pytest.mark.parametrize("splits,off", [(1, 0), (3, 0), (3, 1)])
def test_decode_attention_of_grouped_heads_beside_other_keys(hq, hkv, d, splits, off):
    """Masked-out keys (-inf scores), the first of every lane's range among them, and an infinite value change their own sequence only, and leave the others'
    bits alone; the new key at every place of a tile of 16; partial results off a 16-byte boundary."""
    nat = _native()
    torch.manual_seed(hq)
    b, smax = 3, 64
    for ctx in range(30, 50):
        kc, vc = (torch.randn(b, hkv, smax, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        qkv = torch.randn(b, (hq + 2 * hkv) * d, device="cuda", dtype=torch.bfloat16).abs()
        q, k, v = qkv.split([hq * d, hkv * d, hkv * d], dim=1)
        at = torch.tensor([ctx], device="cuda", dtype=torch.int32)
        outs = []
        for bad in (False, True):
            ws = (torch.empty(b * hq * splits * d + off, device="cuda")[off:], torch.empty(b * hq * splits * 2, device="cuda"), torch.zeros(b * hq, dtype=torch.int32, device="cuda"))
            k2, v2 = kc.clone(), vc.clone()
            if bad:
                k2[1, :, [0, 1, 2, 3, 11, 14, 15, 16, 17, 29]] = float("-inf")  # (q is positive: the score is -inf, the probability 0)
                v2[1, :, 7, 3] = float("inf")
            out = nat.attn_decode_fused(q, k, v, k2, v2, at, 0, 10000.0, splits=splits, workspace=ws).view(b, hq, d)
            assert torch.equal(k2[:, :, ctx], k.view(b, hkv, d)) and torch.equal(v2[:, :, ctx], v.view(b, hkv, d))
            kd, vd = (t[:, :, : ctx + 1].double().repeat_interleave(hq // hkv, 1) for t in (k2, v2))
            p = (torch.einsum("bhd,bhnd->bhn", q.reshape(b, hq, d).double(), kd) / math.sqrt(d)).softmax(-1)
            want = torch.einsum("bhn,bhnd->bhd", p, vd)
            outs.append(out)
            assert torch.equal(out.isinf(), want.isinf()) and not out.isnan().any()
            fin = want.isfinite()
            assert bool(((out.double() - want).abs()[fin] <= (2.0 ** -8 * want.abs() + 1e-5)[fin]).all())  # one bf16 rounding
        assert torch.equal(outs[0][[0, 2]], outs[1][[0, 2]])


@pytest.mark.parametrize("group,d", [(1, 64), (2, 128), (8, 64)])
def test_decode_attention_of_a_cache_that_begins_with_masked_keys(group, d):
    nat = _native()
    torch.manual_seed(d)
    b, n, smax = 2, 100, 128
    kc, vc = (torch.randn(b, 1, smax, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    q = torch.randn(b, group, d, device="cuda", dtype=torch.bfloat16).abs()
    kc[:, :, :40] = float("-inf")
    for splits in (1, 4):
        out = nat.attn_decode(q, kc, vc, torch.tensor([n], device="cuda", dtype=torch.int32), 0, splits=splits).view(b, group, d)
        kd, vd = kc[:, :, 40:n].double().expand(-1, group, -1, -1), vc[:, :, 40:n].double().expand(-1, group, -1, -1)
        want = torch.einsum("bhn,bhnd->bhd", (torch.einsum("bhd,bhnd->bhn", q.double(), kd) / math.sqrt(d)).softmax(-1), vd)
        assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all())  # one bf16 rounding


@pytest.mark.parametrize("hq,hkv,d", [(4, 1, 64), (23, 1, 64), (8, 2, 128)])
@pytest.mark.parametrize("off", [1, 2])
def test_decode_attention_with_partials_anywhere(hq, hkv, d, off):
    """Partial results off a 16-byte boundary: the same kernel, one launch, the same bits."""
    nat = _native()
    torch.manual_seed(hq)
    b, splits, ctx, smax = 2, 3, 90, 128
    kc, vc = (torch.randn(b, hkv, smax, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    q, k, v = torch.randn(b, (hq + 2 * hkv) * d, device="cuda", dtype=torch.bfloat16).split([hq * d, hkv * d, hkv * d], dim=1)
    at = torch.tensor([ctx], device="cuda", dtype=torch.int32)
    outs = []
    for o in (0, off):
        ws = (torch.empty(b * hq * splits * d + o, device="cuda")[o:], torch.empty(b * hq * splits * 2, device="cuda"), torch.zeros(b * hq, dtype=torch.int32, device="cuda"))
        outs.append(nat.attn_decode_fused(q, k, v, kc.clone(), vc.clone(), at, 0, 10000.0, splits=splits, workspace=ws))
        assert nat.LIB.tpb_last_launches() == 1
    assert torch.equal(*outs)


@pytest.mark.parametrize("hq,hkv,d", [(2, 2, 128), (2, 1, 64), (4, 1, 128), (8, 1, 64), (6, 2, 128)])
@pytest.mark.parametrize("rotary_dim", [0, 32, None])
@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("table", [False, True])
def test_decode_attention_rotary_forms(hq, hkv, d, rotary_dim, interleaved, table):
    """Partial rotary spans, an untouched rest, interleaved pairs, none at all; angles computed and looked up."""
    nat = _native()
    rotary_dim = d if rotary_dim is None else rotary_dim
    torch.manual_seed(hq + d + rotary_dim)
    b, ctx, smax = 2, 150, 160
    kc, vc = (torch.randn(b, hkv, smax, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    qkv = torch.randn(b, (hq + 2 * hkv) * d, device="cuda", dtype=torch.bfloat16)
    q, k, v = qkv.split([hq * d, hkv * d, hkv * d], dim=1)
    at = torch.tensor([ctx], device="cuda", dtype=torch.int32)
    angles = nat.rope_table(smax, rotary_dim, 10000.0, torch.device("cuda", 0)) if table and rotary_dim else None
    outs = []
    for early in (False, True):
        k2, v2 = kc.clone(), vc.clone()
        torch.cuda.synchronize()
        out = nat.attn_decode_fused(q, k, v, k2, v2, at, rotary_dim, 10000.0, interleaved=interleaved, splits=2, rope_angles=angles, early=early)
        outs.append((out, k2, v2))
    assert all(torch.equal(x, y) for x, y in zip(*outs))
    rot = lambda x, heads: OF.apply_rope_ref(x.reshape(b, 1, heads, d), at.long().view(1, 1).expand(b, 1), 10000.0, rotary_dim, interleaved)[:, 0] if rotary_dim else x.reshape(b, heads, d)
    assert torch.equal(v2[:, :, ctx], v.reshape(b, hkv, d))
    # the angle of position 150 has an fp32 error of a few 2^-17, then one bf16 rounding: half a unit, either way
    assert bool(((k2[:, :, ctx].double() - rot(k, hkv).double()).abs() <= 2.0 ** -7 * rot(k, hkv).double().abs() + 1e-3).all())
    assert torch.equal(k2[:, :, ctx, rotary_dim:], k.reshape(b, hkv, d)[..., rotary_dim:])
    qr = rot(q, hq).double()
    kd, vd = (t[:, :, : ctx + 1].double().repeat_interleave(hq // hkv, 1) for t in (k2, v2))
    want = torch.einsum("bhn,bhnd->bhd", (torch.einsum("bhd,bhnd->bhn", qr, kd) / math.sqrt(d)).softmax(-1), vd)
    err = (out.view(b, hq, d).double() - want).abs()
    # the result's rounding, and that of the rotated query (half a unit of 2^-8, either way) in a handful of its elements
    assert bool((err <= 2.0 ** -7 * want.abs() + 2.0 ** -7 * want.abs().amax(-1, keepdim=True) + 1e-4).all()), err.max()


def _backward_rows(d, bias_mode, streamed, heads, batch):
    return _native().LIB.tpb_attn_backward_step_rows(d, bias_mode, streamed, heads, batch)


# rows per step of the dK / dV launch (which streams the queries) and of the dQ launch (which streams the keys), without a bias
@pytest.mark.parametrize("d,b,sq,sk,hq,hkv,causal,rows", [
    # last wide steps of one row and of 64, more steps than either ring is deep; grouped heads; queries without a key (sq > sk), empty dQ steps
    (128, 1, 1025, 1025, 2, 1, True, (128, 128)), (128, 1, 1088, 1025, 3, 3, False, (128, 128)), (128, 2, 384, 250, 4, 2, True, (128, 128)),
    (128, 1, 512, 100, 2, 2, True, (128, 128)), (128, 1, 65, 385, 2, 1, True, (128, 128)), (128, 2, 448, 449, 2, 2, True, (128, 128)),
    (64, 1, 449, 449, 4, 2, True, (128, 128)), (64, 1, 385, 700, 3, 1, False, (128, 128)), (64, 2, 384, 250, 4, 2, True, (128, 128)),
    (64, 1, 1025, 1088, 2, 2, True, (128, 128)), (64, 2, 100, 128, 2, 1, False, (128, 128)),
    # steps of 64: one short or whole one, a few that end in a first half, one launch of each kind, many heads.  (Two keys at least: with
    # one, the gradients of query and key are zero, and what a kernel returns is the rounding of dP - delta, 2^-24 of its d terms, with no
    # want.grad to hold it against.)
    (128, 2, 1, 33, 2, 1, True, (64, 64)), (128, 1, 300, 129, 4, 2, True, (64, 64)), (128, 2, 64, 200, 2, 2, False, (64, 128)),
    (64, 2, 1, 2, 2, 1, True, (64, 64)), (64, 1, 64, 33, 4, 1, True, (64, 64)), (64, 2, 150, 320, 2, 2, True, (64, 64)), (64, 1, 200, 257, 4, 2, False, (128, 64)),
    (64, 8, 400, 576, 16, 8, True, (64, 64)), (64, 16, 100, 193, 32, 16, True, (64, 64)), (64, 16, 256, 65, 16, 16, True, (64, 64))])
@pytest.mark.parametrize("bias", ["none", "dense", "rows off 16 bytes", "padding"])
def test_attention_backward_by_step(d, b, sq, sk, hq, hkv, causal, rows, bias):
    """Both kernels of the backward against 64 bits, at the edges of their steps and rings, and of the rule that chooses between them."""
    if bias != "none" and b * hq * sq * sk > 1 << 24:
        pytest.skip("the rule for many heads concerns calls without a bias")
    nat = _native()
    torch.manual_seed(sq + sk + d)
    assert rows == (_backward_rows(d, 0, sq, hkv, b), _backward_rows(d, 0, sk, hq, b))
    for mode in (1, 2):
        assert _backward_rows(d, mode, sq, hkv, b) == (64 if d == 128 or sq <= 64 else 128)
    q, k, v = (torch.randn(b, s, h, d, device="cuda", dtype=torch.bfloat16).requires_grad_() for s, h in ((sq, hq), (sk, hkv), (sk, hkv)))
    g = torch.randn(b, sq, hq, d, device="cuda", dtype=torch.bfloat16)
    if bias == "none":
        leaf = added = None
    elif bias == "padding":
        leaf = added = torch.zeros(b, 1, 1, sk, device="cuda", dtype=torch.bfloat16)
        leaf[0, :, :, sk - sk // 3:] = -math.inf
    else:  # rows of a multiple of eight keys travel by TMA, others element by element
        pitch = (sk + 7) // 8 * 8 + (0 if bias == "dense" else 1)
        leaf = torch.randn(1, hq, sq, pitch, device="cuda", dtype=torch.bfloat16)
        added = leaf[..., :sk].detach().requires_grad_()
    nat.attention(q, k, v, causal, added).backward(g)
    ref = [t.detach().double().requires_grad_() for t in (q, k, v)]
    kh, vh = (t.repeat_interleave(hq // hkv, 2) for t in ref[1:])
    scores = torch.einsum("bqhd,bkhd->bhqk", ref[0], kh) / math.sqrt(d)
    if added is not None:
        ref.append(added.detach().double().requires_grad_())
        scores = scores + ref[3]
    hidden = torch.ones(sq, sk, dtype=torch.bool, device="cuda").triu(sk - sq + 1) if causal else torch.zeros(sq, sk, dtype=torch.bool, device="cuda")
    unseen = hidden | (scores.detach() == -math.inf)
    probs = scores.masked_fill(unseen, -1e300).softmax(-1).masked_fill(unseen, 0.0)  # (a row without keys becomes uniform, and is removed again)
    torch.einsum("bhqk,bkhd->bqhd", probs, vh).backward(g.double())
    nat.device_state(q.device).check_status()
    for got, want in zip([q, k, v] + ([added] if added is not None and added.requires_grad else []), ref):
        # probabilities, dS and results are rounded to bf16 once each (2^-9 relative, independent errors), the output that delta reads too
        assert (got.grad.double() - want.grad).norm() <= 2.0 ** -7 * want.grad.norm() + 1e-6


def test_norm_of_as_many_rows_as_an_int_counts():
    """2^31 - 1 narrow rows: the rows fetched ahead of the last ones have numbers that no int holds."""
    rows, cols = 2 ** 31 - 1, 8
    if torch.cuda.mem_get_info()[0] < 80e9:
        pytest.skip("needs 70 GB")
    nat = _native()
    x = torch.empty(rows, cols, device="cuda", dtype=torch.bfloat16)
    x[:-5000] = 1.0
    x[-5000:] = torch.randn(5000, cols, device="cuda")
    out = nat.norm_forward(x, None, None, 1e-6, 1)[0]
    assert bool((out[-5000:].double() - torch.nn.functional.layer_norm(x[-5000:].double(), (cols,), eps=1e-6)).abs().max() <= 2.0 ** -6)  # bf16 results below 4
    assert not bool(out[: 1 << 20].any()) and not bool(out[1 << 30 : (1 << 30) + (1 << 20)].any())
    del x, out
    torch.cuda.empty_cache()


# one share of the rows and several, remainders of 32 rows and of 64 columns, one row, columns that take the sum over tensors
@pytest.mark.parametrize("rows,cols", [(1, 8), (33, 72), (256, 3072), (257, 640), (1000, 520), (4097, 64), (70, 36)])
def test_bias_gradient(rows, cols):
    """Column sums against 64 bits, the same bits every time; a gradient that is not contiguous."""
    nat = _native()
    torch.manual_seed(rows)
    x, w = torch.randn(rows, 64, device="cuda", dtype=torch.bfloat16), torch.randn(cols, 64, device="cuda", dtype=torch.bfloat16)
    for g in (torch.randn(rows, cols, device="cuda", dtype=torch.bfloat16), torch.randn(cols, rows, device="cuda", dtype=torch.bfloat16).t()):
        got = []
        for _ in range(2):
            b = torch.zeros(cols, device="cuda", dtype=torch.bfloat16, requires_grad=True)
            nat.linear(x, w, b).backward(g)
            got.append(b.grad)
        want = g.double().sum(0)
        assert torch.equal(*got) and got[0].dtype == torch.bfloat16
        # one bf16 rounding behind fp32 sums of numbers of magnitude 1
        assert bool(((got[0].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20 * rows).all())


@pytest.mark.parametrize("bidirectional", [False, True])
@pytest.mark.parametrize("buckets,max_distance", [(32, 128), (32, 20), (4, 100), (7, 90), (12, 1000), (64, 100000), (30, 333), (256, 4096)])
def test_relative_buckets_are_those_of_the_tensor_steps(bidirectional, buckets, max_distance):
    from tensor_parallel_b200.models.t5 import relative_position_bucket

    device = torch.device("cuda", 0)
    for first, count in ((-200000, 400001), (-511, 1023), (0, 1), (1, 70), (-(2 ** 40), 300), (2 ** 40, 300)):
        got = OF.relative_buckets(first, count, device, bidirectional, buckets, max_distance)
        assert got is not None
        assert torch.equal(got, relative_position_bucket(torch.arange(first, first + count, device=device), bidirectional, buckets, max_distance))
    for args in ((0, 0, device, bidirectional, buckets, max_distance), (0, 5, "cpu", bidirectional, buckets, max_distance), (0, 5, device, True, 3, 100), (0, 5, device, False, 32, 16)):
        assert OF.relative_buckets(*args) is None


def _attention_double(q, k, v, causal, bias):
    """Output, and what backward needs, of 64-bit attention over leaves of q, k, v and the bias."""
    scores = torch.einsum("bqhd,bkhd->bhqk", q, k.repeat_interleave(q.shape[2] // k.shape[2], 2)) / math.sqrt(q.shape[-1])
    if bias is not None:
        scores = scores + bias
    if causal:
        sq, sk = scores.shape[-2:]
        scores = scores.masked_fill(torch.ones(sq, sk, dtype=torch.bool, device=q.device).triu(sk - sq + 1), -math.inf)
    return torch.einsum("bhqk,bkhd->bqhd", scores.softmax(-1).nan_to_num(0.0), v.repeat_interleave(q.shape[2] // v.shape[2], 2))


# more CTAs than SMs (causal: than two rounds of them) at head_dim 64, and in dQ at head_dim 128: two CTAs per SM.  Lengths off the tiles of 64 and 128, one tile, several, more
# keys than queries; grouped heads.
@pytest.mark.parametrize("b,sq,sk,hq,hkv,causal", [(5, 129, 129, 32, 32, False), (10, 130, 193, 32, 16, True), (5, 200, 72, 32, 32, False), (3, 257, 320, 64, 64, True),
                                                   (2, 1, 64, 160, 160, True), (4, 264, 264, 40, 40, False)])
@pytest.mark.parametrize("d,bias", [(64, "none"), (64, "dense"), (64, "rows off 16 bytes"), (64, "fp32"), (64, "padding"), (128, "none")])
def test_attention_with_two_ctas_per_sm(b, sq, sk, hq, hkv, causal, d, bias):
    nat = _native()
    torch.manual_seed(sq + sk)
    q, k, v = (torch.randn(b, s, h, d, device="cuda", dtype=torch.bfloat16).requires_grad_() for s, h in ((sq, hq), (sk, hkv), (sk, hkv)))
    g = torch.randn(b, sq, hq, d, device="cuda", dtype=torch.bfloat16)
    added = None
    if bias == "padding":
        added = torch.zeros(b, 1, 1, sk, device="cuda", dtype=torch.bfloat16)
        added[0, :, :, sk - sk // 3:] = -math.inf
    elif bias != "none":
        pitch = (sk + 7) // 8 * 8 + (1 if bias == "rows off 16 bytes" else 0)
        added = torch.randn(1, hq, sq, pitch, device="cuda", dtype=torch.float32 if bias == "fp32" else torch.bfloat16)[..., :sk].detach().requires_grad_()
    out = nat.attention(q, k, v, causal, added)
    out.backward(g)
    nat.device_state(q.device).check_status()
    leaves = [t.detach().double().requires_grad_() for t in (q, k, v) + ((added,) if added is not None and added.requires_grad else ())]
    want = _attention_double(*leaves[:3], causal, leaves[3] if len(leaves) > 3 else None if added is None else added.double())
    want.backward(g.double())
    # probabilities, dS and results are rounded to bf16 (2^-9 each, independent from element to element), as in test_attention_backward_by_step
    assert (out.double() - want).norm() <= 0.01 * want.norm()
    for t, ref in zip((q, k, v) + ((added,) if len(leaves) > 3 else ()), leaves):
        assert (t.grad.double() - ref.grad).norm() <= 0.01 * ref.grad.norm() + 1e-6


@pytest.mark.parametrize("bias", ["none", "dense", "fp32", "mask"])
@pytest.mark.parametrize("at", [3, 70, 127])
def test_attention_does_not_round_the_largest_probability_of_the_first_128_keys(bias, at):
    """One key with nearly all of the weight, so that the output is its value, rounded once; tiles of 64 keys at head_dim 64."""
    nat = _native()
    torch.manual_seed(at)
    b, s, h = 10, 140, 16
    scores = torch.full((h, s), -12.0, device="cuda")
    scores[:, 0] = 0.0
    scores[:, at] = 4 + torch.rand(h, device="cuda")  # less than 2^8 above the first key
    scores = scores.bfloat16()
    q, k = (torch.zeros(b, s, h, 64, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    v = torch.randn(b, s, h, 64, device="cuda", dtype=torch.bfloat16)
    added = None
    if bias == "none":
        q[..., 0], k[..., 0] = 8, scores.t()
    elif bias == "mask":
        scores = scores[:1].expand(h, s)
        added = scores[0].view(1, 1, 1, s).repeat(b, 1, 1, 1)
    else:
        added = torch.zeros(1, h, s, 144, device="cuda", dtype=torch.float32 if bias == "fp32" else torch.bfloat16)[..., :s]
        added.copy_(scores[None, :, None])
    out, _ = nat.attention_forward(q, k, v, False, None, want_lse=True, bias=added)
    want = torch.einsum("hk,bkhd->bhd", scores.double().softmax(-1), v.double())[:, None]
    # one bf16 rounding (2^-8 at most); the other keys have 2 % of the weight, each rounded once more, and V is below 5
    assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -8 * 0.02 * 5).all())


# a tile per CTA for the gradient of a shared bias: whole tiles, ragged ones, rows of a multiple of eight, more keys than queries, a plane for all heads
@pytest.mark.parametrize("b,sq,sk,hq,hkv,shared", [(3, 256, 256, 32, 32, False), (1, 240, 248, 30, 15, False), (2, 384, 1000, 6, 6, False), (5, 1152, 1792, 2, 1, True)])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_attention_bias_gradient_by_tiles(b, sq, sk, hq, hkv, shared, causal, dtype):
    """Against 64 bits; the same bits every time; masked pairs contribute nothing, whatever their values."""
    nat = _native()
    torch.manual_seed(sq)
    q, k, v = (torch.randn(b, s, h, 64, device="cuda", dtype=torch.bfloat16) for s, h in ((sq, hq), (sk, hkv), (sk, hkv)))
    g = torch.randn(b, sq, hq, 64, device="cuda", dtype=torch.bfloat16)
    bias = torch.randn(1, 1 if shared else hq, sq, sk, device="cuda", dtype=torch.bfloat16)
    bias[..., 3] = -math.inf
    strides = [0 if n == 1 else st for n, st in zip(bias.shape, bias.stride())]
    assert nat._bias_grad_tiles(b, sq, sk, hq, 64, bias, strides)
    out, lse = nat.attention_forward(q, k, v, causal, None, want_lse=True, bias=bias)
    got = nat.attention_backward(q, k, v, out, g, lse, causal, None, bias=bias, want_dbias=True, dbias_dtype=dtype)[3]
    assert got.dtype == dtype and got.shape == bias.shape and not bool(got[..., 3].any())
    assert torch.equal(got, nat.attention_backward(q, k, v, out, g, lse, causal, None, bias=bias, want_dbias=True, dbias_dtype=dtype)[3])
    leaf = bias.double().requires_grad_()
    _attention_double(q.double(), k.double(), v.double(), causal, leaf).backward(g.double())
    # delta is taken from the rounded output (2^-9, independent over 64 elements); bf16 results are rounded once more
    assert (got.double() - leaf.grad).norm() <= 0.006 * leaf.grad.norm()
    v2 = v.clone()
    v2[:, 3] = math.inf  # dP is not finite where the probability is 0
    inf = nat.attention_backward(q, k, v2, out, g, lse, causal, None, bias=bias, want_dbias=True, dbias_dtype=dtype)[3]
    assert torch.equal(inf, got)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("cols", [8, 264, 776, 1024, 1536, 1544, 1800, 2048, 2568, 3072, 3080, 3584, 4096, 4104, 5120, 6152, 8192])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("with_weight", [False, True])
def test_norm_of_a_row_does_not_depend_on_the_others(dtype, cols, mode, with_weight):
    """The same bits for a row alone, among few, and among as many as take another kernel."""
    nat = _native()
    torch.manual_seed(cols)
    x = (torch.randn(16000, cols, device="cuda") * 2 + 0.1).to(dtype)
    w = torch.randn(cols, device="cuda").to(dtype) if with_weight else None
    b = torch.randn(cols, device="cuda").to(dtype) if with_weight and mode else None
    out, rstd, mean = nat.norm_forward(x, w, b, 1e-6, mode, want_stats=True)
    for first, count in ((0, 1), (5, 20), (3, 148), (9, 149), (100, 700), (7, 1184), (7, 1185), (8, 2048), (1, 8191), (8, 8192)):
        part, r, m = nat.norm_forward(x[first : first + count], w, b, 1e-6, mode, want_stats=True)
        assert torch.equal(part, out[first : first + count]) and torch.equal(r, rstd[first : first + count])
        assert mean is None or torch.equal(m, mean[first : first + count])
    assert (out[:64].double() - _norm_double(x[:64], w, mode) - (0 if b is None else b.double())).norm() <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20) * out[:64].double().norm()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("cols", [1544, 2048, 3080, 4096, 8200, 12296, 16384])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("with_weight", [False, True])
def test_norm_with_a_residual_of_zeros(dtype, cols, mode, with_weight):
    """Rows held as they lie in memory and as sums in fp32: the same numbers, and the same bits where both are added up in the same order."""
    nat = _native()
    torch.manual_seed(cols)
    x = (torch.randn(150, cols, device="cuda") * 2 + 0.1).to(dtype)
    w = torch.randn(cols, device="cuda").to(dtype) if with_weight else None
    b = torch.randn(cols, device="cuda").to(dtype) if with_weight and mode else None
    out, rstd, _ = nat.norm_forward(x, w, b, 1e-6, mode, want_stats=True)
    summed = torch.empty_like(x)
    for kwargs in (dict(), dict(sum_out=summed)):
        other, r, _ = nat.norm_forward(x, w, b, 1e-6, mode, residual=torch.zeros_like(x), want_stats=True, **kwargs)
        if cols > 8192 or (mode == 0 and dtype == torch.bfloat16):
            assert torch.equal(other, out) and torch.equal(r, rstd)
        want = _norm_double(x, w, mode) + (0 if b is None else b.double())
        assert (other.double() - want).norm() <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20) * want.norm()
    assert torch.equal(summed, x)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("batch", [1, 3, 2 ** 20 - 1, 2 ** 20 + 1])
def test_row_sums_of_the_attention_backward(d, batch):
    """Row numbers below and above 2^31 (2048 rows per sequence, sequences that share their memory)."""
    nat = _native()
    torch.manual_seed(d)
    sq, heads = 64, 32
    out, dout = (torch.randn(sq, heads, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    delta = torch.full((batch, heads, sq), math.nan, device="cuda")
    entry = nat.LIB.tpb_attn_bwd_delta  # (only the backward calls it; undeclared pointers would be cut to 32 bits)
    entry.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int] * 4 + [ctypes.c_longlong] * 6 + [ctypes.c_void_p]
    nat.check(entry(out.data_ptr(), dout.data_ptr(), delta.data_ptr(), batch, sq, heads, d, 0, heads * d, d, 0, heads * d, d, nat._stream()),
              "tpb_attn_bwd_delta")
    want = (out.double() * dout.double()).sum(-1).t()
    size = (out.double() * dout.double()).abs().sum(-1).t()
    assert bool(((delta[0].double() - want).abs() <= 2.0 ** -24 * d * size).all())  # (products are exact in fp32, at most d roundings of partial sums)
    assert all(torch.equal(part, delta[:1].expand_as(part)) for part in delta.split(2 ** 16))


def _norm_double(x, w, mode):
    y = x.double()
    if mode:
        y = y - y.mean(-1, keepdim=True)
    y = y * (y.square().mean(-1, keepdim=True) + 1e-6).rsqrt()
    return y if w is None else y * w.double()
