"""GPU tests of the kernels behind the fused nodes (norms, activations, embedding, routing, loss, GEMM with the kept sums) at the
edges of their tiles, against the same operation in 64-bit (or 32-bit) torch.

Tolerances.  u = 2^-8 bounds the relative error of one rounding to bf16.  A result that is worked out in fp32 and rounded
once differs from the exact one by at most u / 2 per element plus the fp32 sums' error, which is far below it: the limit is u
per element relative to the element, plus u / 16 of the result's largest value for elements that cancel.  Where intermediate
results are rounded too (several bf16 operations in a row), the limit is stated with the number of roundings."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

U = 2.0 ** -8


@pytest.fixture(autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device (run the CPU tier with -m 'not gpu')")
    torch.manual_seed(0)


def _bf(*shape, std=1.0, mean=0.0):
    return (torch.randn(*shape, device="cuda") * std + mean).to(torch.bfloat16)


def _close(got, want, roundings=1):
    got, want = got.double(), want.double()
    assert got.shape == want.shape
    err = (got - want).abs()
    limit = roundings * (U * want.abs() + U / 16 * want.abs().max())
    assert torch.isfinite(got).all() and (err <= limit).all(), f"largest excess {(err - limit).max().item():.3g}"


def _comm():
    import mccl_b200 as mccl
    return mccl.Communicator(1, mccl.get_unique_id(), 0, transport="cuda")


@pytest.mark.parametrize("d", [8, 24, 256, 264, 520, 768, 776, 1024, 1032, 2048, 2056, 4096])
@pytest.mark.parametrize("rows", [1, 3, 33, 700])
def test_layer_norm_widths(rows, d):
    from mccl_b200.ops.norm import FusedLayerNorm
    layer = FusedLayerNorm(d).to(device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        layer.weight.copy_(_bf(d, std=0.2, mean=1.0))
        layer.bias.copy_(_bf(d, std=0.1))
    x, dy = _bf(rows, d, std=2.0, mean=0.3).requires_grad_(True), _bf(rows, d)
    y = layer(x)
    got = torch.autograd.grad(y, [x, layer.weight, layer.bias], dy)
    xr, w, b = (t.detach().double().requires_grad_(True) for t in (x, layer.weight, layer.bias))
    want = F.layer_norm(xr, (d,), w, b, layer.eps)
    _close(y, want)
    for g, r in zip(got, torch.autograd.grad(want, [xr, w, b], dy.double())):
        _close(g, r)


def test_layer_norm_of_other_widths_is_torchs_own():
    """Traced without a break and, under autocast, in fp32."""
    from mccl_b200.ops.norm import FusedLayerNorm
    layer, x = FusedLayerNorm(768).to(device="cuda", dtype=torch.bfloat16), _bf(4, 768)
    want = F.layer_norm(x, (768,), layer.weight, layer.bias, layer.eps)
    assert torch.equal(layer(x), want)
    assert torch.equal(torch.compile(layer, backend="eager", fullgraph=True)(x), want)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert layer(x).dtype == torch.float32


@pytest.mark.parametrize("d", [128, 256, 768, 1024])
def test_layer_norm_of_no_rows(d):
    from mccl_b200.ops.norm import FusedLayerNorm
    layer = FusedLayerNorm(d).to(device="cuda", dtype=torch.bfloat16)
    x = torch.empty(0, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    y = layer(x)
    assert y.shape == x.shape
    dx, dw, db = torch.autograd.grad(y, [x, layer.weight, layer.bias], torch.empty_like(y))
    assert dx.shape == x.shape and dw.abs().sum() == 0 and db.abs().sum() == 0


def test_cross_entropy_of_no_rows_is_refused():
    from mccl_b200.ops.loss import fused_cross_entropy
    with pytest.raises(RuntimeError):
        fused_cross_entropy(torch.empty(0, 64, device="cuda", dtype=torch.bfloat16), torch.empty(0, device="cuda", dtype=torch.int64))


def test_cross_entropy_of_targets_on_the_host_is_refused():
    from mccl_b200.ops.loss import fused_cross_entropy
    with pytest.raises(ValueError):
        fused_cross_entropy(_bf(3, 64), torch.zeros(3, dtype=torch.int64))


@pytest.mark.parametrize("n", [1, 7, 8, 4095, 8192, 8200 * 3 + 5])
def test_silu_both(n):
    from mccl_b200 import _ext
    u, dh = _bf(n, std=3.0), _bf(n)
    h, du = _ext.load().silu_both(u, dh)
    ur = u.double().requires_grad_(True)
    want = F.silu(ur)
    _close(h, want)
    _close(du, torch.autograd.grad(want, ur, dh.double())[0])


def test_silu_is_worked_out_in_full_fp32():
    """With a relative error of e before it is rounded, a result rounds apart from the exact one with a probability of 2 e / 2^-8 at
    most.  Arguments where an exponential of the product with log2(e) alone has an error of 2^-19."""
    from mccl_b200 import _ext
    n = 1 << 22
    u, dh = (-80 + 40 * torch.rand(n, device="cuda")).to(torch.bfloat16), _bf(n)
    h, du = _ext.load().silu_both(u, dh)
    ur = u.double().requires_grad_(True)
    want = F.silu(ur)
    g = torch.autograd.grad(want, ur, dh.double())[0]
    for got, exact, e in ((h, want, 2.0 ** -22), (du, g, 2.0 ** -21)):
        assert (got != exact.to(torch.bfloat16)).float().mean().item() <= 2 * e / U


def test_silu_of_every_value_is_rounded_exactly():
    import ctypes as C
    from mccl_b200 import _lib
    x = torch.arange(-32768, 32768, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    up = torch.randn(65536, device="cuda").to(torch.bfloat16)
    y, z = torch.empty_like(x), torch.empty_like(x)
    lib, s = _lib.load(), C.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: C.c_void_p(t.data_ptr())
    assert lib.mcclSiluForward(p(x), p(y), C.c_int64(65536), s) == 0
    assert lib.mcclSwigluForward(p(x), p(up), p(z), C.c_int64(65536), s) == 0
    want = F.silu(x.double()).to(torch.bfloat16)
    library = F.silu(x)                            # beyond 88 the exponential overflows in fp32 and the result is zero
    assert ((y == want) | (y == library) | (y.isnan() & want.isnan())).all()
    assert (y == want)[x.abs() < 80].all()
    ok = torch.isfinite(y)
    assert torch.equal(z[ok], (y * up)[ok])


def test_gelu_of_every_value_is_what_the_tensor_library_rounds_to():
    from mccl_b200 import _ext
    x = torch.arange(-32768, 32768, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    y, want = _ext.load().gelu_forward(x), F.gelu(x, approximate="tanh")
    ok = (y.view(torch.int16) == want.view(torch.int16)) | (y.isnan() & want.isnan())
    assert ok.all(), x[~ok]
    for n in (1, 7, 8, 1021, 8193):                    # a remainder that no 16-byte piece holds
        assert torch.equal(_ext.load().gelu_forward(x[16256:16256 + n].clone()), F.gelu(x[16256:16256 + n], approximate="tanh"))


@pytest.mark.parametrize("rows,d", [(1, 8), (5, 520), (129, 1032), (2000, 4096)])
def test_gelu_gradient_and_its_column_sums(rows, d):
    from mccl_b200 import _ext
    x, dy = _bf(rows, d, std=2.0), _bf(rows, d)
    dx, db = _ext.load().gelu_backward(x, dy)
    xr = x.double().requires_grad_(True)
    want = torch.autograd.grad(F.gelu(xr, approximate="tanh"), xr, dy.double())[0]
    _close(dx, want)
    _close(db, dx.double().sum(0))


def test_gelu_gradient_of_every_value_is_what_the_tensor_library_rounds_to():
    from mccl_b200 import _ext
    x = torch.arange(-32768, 32768, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    for scale in (1.0, 1e-3, 30.0):
        dy = _bf(65536, std=scale)
        dx, _ = _ext.load().gelu_backward(x.view(64, 1024), dy.view(64, 1024))
        want = torch.ops.aten.gelu_backward(dy, x, approximate="tanh")
        ok = (dx.view(-1) == want) | (dx.view(-1).isnan() & x.isnan())
        far = x.abs() >= 2.0 ** 63                     # x^2 overflows in the tensor library's form; here the slope is 1 or 0
        assert ok[~far].all(), x[~far & ~ok]
        assert torch.equal(dx.view(-1)[far], torch.where(x > 0, dy, torch.copysign(torch.zeros_like(dy), dy))[far])


@pytest.mark.parametrize("vocab,d,tokens", [(5, 8, (1, 1)), (3, 64, (2, 300)), (1000, 1024, (4, 129)), (50, 2056, (1, 65)), (70, 4096, (3, 130))])
@pytest.mark.parametrize("with_pos", [True, False])
def test_embedding_adds_repeated_tokens(vocab, d, tokens, with_pos):
    from mccl_b200 import _ext
    idx = torch.randint(0, vocab, tokens, device="cuda")
    table = _bf(vocab, d).requires_grad_(True)
    pos = _bf(tokens[1] + 3, d).requires_grad_(True) if with_pos else None
    y = _ext.load().decoder_embed(idx, table, pos, False)
    dy = _bf(*y.shape)
    ins = [table] + ([pos] if with_pos else [])
    refs = [t.detach().double().requires_grad_(True) for t in ins]
    want = F.embedding(idx, refs[0])
    if with_pos:
        want = want + refs[1][:tokens[1]]
    want = want.reshape(-1, d)
    _close(y, want)
    for g, r in zip(torch.autograd.grad(y, ins, dy), torch.autograd.grad(want, refs, dy.double())):
        _close(g, r)


@pytest.mark.parametrize("tokens,common", [(127, 127), (129, 129), (257, 200), (1024, 512), (4097, 4000), (16384, 16384), (16384, 9000)])
@pytest.mark.parametrize("d", [8, 1024, 2056])
def test_embedding_gradient_of_a_token_that_fills_the_batch(tokens, common, d):
    """Chunks of 128 tokens add up by themselves and meet in token order: the same bits from run to run."""
    from mccl_b200 import _ext
    vocab = 700
    idx = torch.randint(0, vocab, (tokens,), device="cuda")
    idx[torch.randperm(tokens, device="cuda")[:common]] = 11
    table, dy = _bf(vocab, d).requires_grad_(True), _bf(tokens, d)
    runs = [torch.autograd.grad(_ext.load().decoder_embed(idx, table, None, False), table, dy)[0] for _ in range(3)]
    assert torch.equal(runs[0], runs[1]) and torch.equal(runs[0], runs[2])
    want = torch.zeros(vocab, d, device="cuda", dtype=torch.float64).index_add_(0, idx, dy.double())
    _close(runs[0], want)


@pytest.mark.parametrize("tokens", [300, 16384, 16400])
def test_embedding_indices_outside_the_table(tokens):
    """A NaN row forward, no gradient backward: with the kernel and beyond its number of tokens."""
    from mccl_b200 import _ext
    vocab, d = 40, 64
    idx = torch.randint(0, vocab, (tokens,), device="cuda")
    idx[0], idx[7] = vocab, -3
    table = _bf(vocab, d).requires_grad_(True)
    y = _ext.load().decoder_embed(idx, table, None, False)
    assert y[[0, 7]].isnan().all() and not y[1:7].isnan().any()
    dy = _bf(tokens, d)
    ok = (idx >= 0) & (idx < vocab)
    want = torch.zeros(vocab, d, device="cuda", dtype=torch.float64).index_add_(0, idx[ok], dy[ok].double())
    _close(torch.autograd.grad(y, table, dy)[0], want)


@pytest.mark.parametrize("rows,vocab,width", [(1, 50257, 50304), (2, 8, 8), (5, 257, 257), (37, 4096, 4096), (74, 33000, 33001), (300, 1000, 1024), (444, 8192, 8192), (445, 8193, 8193)])
def test_cross_entropy_mean_forms(rows, vocab, width):
    """In the backward pass few rows are shared by several CTAs; an odd width leaves rows unaligned; targets left out."""
    from mccl_b200.ops.loss import fused_cross_entropy
    logits = _bf(rows, width, std=2.0).requires_grad_(True)
    t = torch.randint(0, vocab, (rows,), device="cuda")
    lr = logits.detach()[:, :vocab].double().requires_grad_(True)
    want = F.cross_entropy(lr, t)
    wg = F.pad(torch.autograd.grad(want, lr)[0], (0, width - vocab))
    loss = fused_cross_entropy(logits, t, vocab)
    assert abs(loss.item() - want.item()) <= 1e-5 * max(1.0, abs(want.item()))
    _close(torch.autograd.grad(loss, logits)[0], wg)


@pytest.mark.parametrize("fill", [torch.finfo(torch.bfloat16).min, float("-inf")])
@pytest.mark.parametrize("rows,vocab,lo,hi", [(5, 1000, 0, 64), (3, 4096, 0, 4088), (2, 5000, 8, 4999), (700, 64, 0, 56)])
def test_cross_entropy_of_masked_columns(rows, vocab, lo, hi, fill):
    """Masks of the type's lowest value or of minus infinity, before, around and behind what a thread reads first."""
    from mccl_b200.ops.loss import fused_cross_entropy
    logits = _bf(rows, vocab, std=2.0)
    logits[:, lo:hi] = fill
    t = torch.randint(hi, vocab, (rows,), device="cuda")
    lr = logits.double().requires_grad_(True)
    want = F.cross_entropy(lr, t)
    x = logits.clone().requires_grad_(True)
    loss = fused_cross_entropy(x, t, vocab)
    assert abs(loss.item() - want.item()) <= 1e-5 * max(1.0, abs(want.item()))
    _close(torch.autograd.grad(loss, x)[0], torch.autograd.grad(want, lr)[0])


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_cross_entropy_of_a_row_without_a_maximum_is_nan(bad):
    from mccl_b200.ops.loss import fused_cross_entropy
    for col in (0, 7, 900):
        logits = _bf(2, 1000)
        logits[1, col] = bad
        assert math.isnan(fused_cross_entropy(logits.requires_grad_(True), torch.tensor([3, 5], device="cuda")).item())


@pytest.mark.parametrize("ignored", [0, 5, 17])
def test_head_loss_leaves_ignored_targets_out(ignored):
    from mccl_b200 import _ext
    T, d, V = 17, 64, 96
    h, w = _bf(T, d).requires_grad_(True), _bf(V, d, std=0.2).requires_grad_(True)
    t = torch.randint(0, V, (T,), device="cuda")
    t[:ignored] = -100
    loss = _ext.load().decoder_head_loss(h, w, t, V, True, False)
    logits = (h.detach().double() @ w.detach().double().t()).to(torch.bfloat16).double().requires_grad_(True)
    want = F.cross_entropy(logits, t)
    if ignored == T:
        assert math.isnan(loss.item()) and math.isnan(want.item())
        return
    # a logit may round to the neighbouring bf16 value: u of the largest, 8 at most, in each of the two terms of the loss
    assert abs(loss.item() - want.item()) <= 2 * 8 * U / math.sqrt(T - ignored)
    g = torch.autograd.grad(want, logits)[0]
    dh, dw = torch.autograd.grad(loss, [h, w])
    for a, b in ((dh, g @ w.double()), (dw, g.t() @ h.double())):
        assert (a.double() - b).norm() <= 3 * U * b.norm()       # logits, their gradient and the product: one rounding each
    t[-1] = V                                                     # neither a column nor the value that is left out
    assert math.isnan(_ext.load().decoder_head_loss(h, w, t, V, True, False).item())


def _moe_reference(x, router, w_in, w_out, capacity):
    """The layer in 64 bits on the routing that the bf16 logits give."""
    logits = F.linear(x, router).detach()
    expert = logits.float().softmax(-1).argmax(-1)
    onehot = F.one_hot(expert, router.shape[0])
    slot = (onehot.cumsum(0) * onehot).sum(-1) - 1
    ps = [t.detach().double().requires_grad_(True) for t in (x, router, w_in, w_out)]
    xr, r, wi, wo = ps
    gate = F.linear(xr, r).softmax(-1).gather(1, expert[:, None])
    y = torch.zeros_like(xr)
    for e in range(router.shape[0]):
        rows = ((expert == e) & (slot < capacity)).nonzero().squeeze(1)
        y = y.index_put((rows,), (F.silu(xr[rows] @ wi[e].t()) @ wo[e].t()) * gate[rows])
    return y, ps


@pytest.mark.parametrize("tokens,hidden,ffn,experts,capacity", [(1, 8, 8, 1, 1), (255, 128, 64, 2, 200), (257, 136, 72, 8, 20), (1000, 256, 128, 32, 40),
                                                                (600, 64, 64, 65, 12), (513, 1032, 64, 3, 600)])
def test_moe_layer_on_one_rank(tokens, hidden, ffn, experts, capacity):
    from mccl_b200.parallel.layers import ExpertParallelMoE
    layer = ExpertParallelMoE(_comm(), hidden, ffn, experts, capacity, device="cuda", dtype=torch.bfloat16, fused=True)
    x, dy = _bf(tokens, hidden).requires_grad_(True), _bf(tokens, hidden)
    ins = [x, layer.router.weight, layer.w_in, layer.w_out]
    y = layer(x)
    want, ps = _moe_reference(*ins, capacity)
    got = torch.autograd.grad(y, ins, dy)
    # forward: tokens, pre-activation, activation, expert output, gate and product rounded; backward: the same once more
    assert (y.double() - want).norm() <= 6 * U / math.sqrt(3) * want.norm()
    for g, r in zip(got, torch.autograd.grad(want, ps, dy.double())):
        assert (g.double() - r).norm() <= 12 * U / math.sqrt(3) * r.norm() + 1e-12


@pytest.mark.parametrize("tokens,hidden,ffn", [(128, 64, 64), (256, 128, 192), (384, 320, 512), (1024, 576, 64), (2560, 1024, 3584)])
def test_mlp_keeps_the_sums(tokens, hidden, ffn):
    """Both forms of the GEMM (128-row and 256-row tiles, with and without the split tail) storing two results."""
    from mccl_b200.parallel.tp import FusedTensorParallelMLP
    layer = FusedTensorParallelMLP(_comm(), tokens, hidden, ffn)
    x, dy = _bf(tokens, hidden).requires_grad_(True), _bf(tokens, hidden)
    ins = [x, layer.w_up, layer.w_down]
    y = layer(x)
    xr, wu, wd = (t.detach().double().requires_grad_(True) for t in ins)
    want = F.linear(F.silu(F.linear(xr, wu)), wd)
    assert (y.double() - want).norm() <= 2 * U * want.norm()              # activation and result
    for g, r in zip(torch.autograd.grad(y, ins, dy), torch.autograd.grad(want, [xr, wu, wd], dy.double())):
        assert (g.double() - r).norm() <= 4 * U * r.norm()                # pre-activation, activation, its gradient, result


def test_mlp_on_one_rank_takes_no_memory_that_it_does_not_use():
    from mccl_b200.parallel.tp import FusedTensorParallelMLP
    comm = _comm()
    before = torch.cuda.memory_allocated()
    layer = FusedTensorParallelMLP(comm, 1024, 512, 2048)
    weights = 2 * 2 * 512 * 2048
    assert torch.cuda.memory_allocated() - before <= weights + 4096
    x = _bf(1024, 512)
    y = layer(x)
    with torch.autocast("cuda", dtype=torch.bfloat16):       # the pair of fused kernels, with its buffers
        z = layer(x)
    assert layer.layer.h.shape == (1024, 2048) and (y.float() - z.float()).norm() <= 4 * U * y.float().norm()


@pytest.mark.parametrize("n", [1, 7, 16383, 16384, 16385, 4096 * 16384 + 9])
def test_sum_of_squares_tile_edges(n):
    from mccl_b200.ops.optim import scratch_floats, sum_squares_
    x, out = _bf(n), torch.zeros(1, device="cuda")
    sum_squares_(x, out, torch.zeros(scratch_floats(n), device="cuda"))
    want = x.double().pow(2).sum().item()
    assert abs(out.item() - want) <= 1e-5 * want


@pytest.mark.parametrize("offset", [4, 8])
def test_adamw_on_arrays_off_the_wide_boundary(offset):
    """fp32 arrays on a 16-byte but not a 32-byte boundary (offset 4) take the narrower loads: the same bits."""
    from mccl_b200.ops.optim import fused_adamw_
    n = 2048 + 3
    start = [torch.randn(n, device="cuda"), torch.randn(n, device="cuda") * 1e-3, torch.rand(n, device="cuda") * 1e-5]
    grad = _bf(n, std=1e-2)

    def step(shift):
        st = [torch.zeros(n + shift, device="cuda")[shift:].copy_(t) for t in start]
        p = start[0].to(torch.bfloat16)
        fused_adamw_(p, *st, grad.clone(), lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1, step=3)
        return [p, *st]

    for a, b in zip(step(0), step(offset)):
        assert torch.equal(a, b)
