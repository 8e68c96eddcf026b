"""When the decoders' fused nodes stand for their modules, and that they do nothing else there than the modules would: GPU tests
compare the fused route with the plain one of the same model (a hook on a part sends a block down the plain one)."""
import pytest
import torch
import torch.nn as nn

from mccl_b200.models.gpt2 import GPT2, GPT2Config
from mccl_b200.models.llama import Llama, LlamaConfig
from mccl_b200.utils.fuse import as_made, undisturbed

gpu = pytest.mark.gpu


def test_as_made_sees_replacements_and_hooks():
    m = nn.Linear(4, 4)
    assert as_made(m, nn.Linear)

    class Mine(nn.Linear):
        pass

    assert not as_made(Mine(4, 4), nn.Linear)
    h = m.register_forward_pre_hook(lambda mod, args: None)
    assert not as_made(m, nn.Linear)
    h.remove()
    m.forward = lambda x: x
    assert not as_made(m, nn.Linear)
    w = nn.utils.parametrizations.weight_norm(nn.Linear(4, 4))
    assert not as_made(w, nn.Linear)


def test_as_made_sees_an_embeddings_options_and_weights_of_another_class():
    assert as_made(nn.Embedding(4, 4), nn.Embedding)
    for option in ({"padding_idx": 0}, {"max_norm": 1.0}, {"scale_grad_by_freq": True}, {"sparse": True}):
        assert not as_made(nn.Embedding(4, 4, **option), nn.Embedding)

    class Mine(torch.Tensor):
        pass

    m = nn.Linear(4, 4)
    m._parameters["weight"] = m.weight.detach().as_subclass(Mine)
    assert not as_made(m, nn.Linear)


def test_modes_and_replaced_functions_are_seen(monkeypatch):
    from torch.overrides import TorchFunctionMode

    class Watch(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    assert undisturbed()
    with Watch():
        assert not undisturbed()
    with torch.device("cpu"):                    # where new tensors go is all that this mode says
        assert undisturbed()
    h = nn.modules.module.register_module_forward_hook(lambda mod, args, out: None)
    assert not undisturbed()
    h.remove()
    monkeypatch.setattr(nn.functional, "scaled_dot_product_attention", lambda *a, **k: None)
    assert not undisturbed()


def _comm():
    import mccl_b200 as mccl
    return mccl.Communicator(1, mccl.get_unique_id(), 0, transport="cuda")


def _gpt2(d=128, layers=2, vocab=300, seq=40):
    torch.manual_seed(0)
    cfg = GPT2Config(n_layer=layers, d_model=d, n_head=d // 32, d_ff=4 * d, vocab_size=vocab, seq_len=seq)
    model = GPT2(cfg).to(device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        for n, p in model.named_parameters():
            if n.endswith("bias"):
                p.normal_(std=0.05)
    return model


def _llama(d=128, layers=2, vocab=300, seq=40, heads=None):
    torch.manual_seed(0)
    cfg = LlamaConfig(n_layer=layers, d_model=d, n_head=heads or d // 32, d_ff=3 * d, vocab_size=vocab, seq_len=seq)
    return Llama(cfg, _comm()).to(device="cuda", dtype=torch.bfloat16)


def _batch(vocab=300, b=3, s=37):
    t = torch.randint(0, vocab, (b, s + 1), device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    return t[:, :-1].contiguous(), t[:, 1:].contiguous()


def _grads(model, idx, tgt):
    loss = model(idx, tgt)
    return [loss.detach()] + list(torch.autograd.grad(loss, list(model.parameters())))


def _plain(model):
    """The same model with a hook that does nothing on every part: the fused nodes stand aside."""
    for m in model.modules():
        if m is not model:
            m.register_forward_pre_hook(lambda mod, args: None)
    return model


def _reference(model, idx, tgt):
    """Loss and gradients of the same weights in 64 bits (no kernels take it)."""
    model = _plain(model).double()
    loss = model(idx, tgt)
    return [loss.detach()] + list(torch.autograd.grad(loss, list(model.parameters())))


@gpu
@pytest.mark.parametrize("make,kw", [(_gpt2, {"d": 128}), (_gpt2, {"d": 384}), (_gpt2, {"d": 768}), (_gpt2, {"d": 1056}), (_llama, {"d": 128}), (_llama, {"d": 64, "heads": 4}), (_llama, {"d": 768, "heads": 6}),
                                     (_llama, {"d": 1152, "heads": 9})])
def test_fused_route_is_as_close_to_64_bits_as_the_plain_one(make, kw):
    idx, tgt = _batch()
    fused = _grads(make(**kw), idx, tgt)
    plain = _grads(_plain(make(**kw)), idx, tgt)
    want = _reference(make(**kw), idx, tgt)
    for f, p, w in zip(fused, plain, want):
        scale = w.norm().clamp_min(1e-30)
        ef, ep = (f.double() - w).norm() / scale, (p.double() - w).norm() / scale
        # Two routes of the same roundings in another order: their errors are draws of one distribution.  1.5 x and half a
        # bf16 step (2^-9) cover the spread of the smallest tensors (a bias of 128 values).
        assert ef <= 1.5 * ep + 2.0 ** -9, (tuple(w.shape), ef.item(), ep.item())


@gpu
@pytest.mark.parametrize("bucket", [False, True])
@pytest.mark.parametrize("d", [128, 256, 384, 512, 768, 1024])
def test_fused_gradients_are_the_plain_routes(d, bucket):
    """Whatever a number of the backward pass flows into is the same number on both routes, so models compare with runs of the
    separate operations: the gradients of the matrices are equal.  Sums over tokens (biases, norms, repeated tokens) are taken in another order: a rounding apart."""
    from mccl_b200.parallel.ddp import DistributedDataParallel
    idx, tgt = _batch()

    def grads(model):
        if bucket:
            DistributedDataParallel(model, None)(idx, tgt).backward()
            return [p.grad for p in model.parameters()]
        return _grads(model, idx, tgt)[1:]

    was = torch.backends.cuda.cudnn_sdp_enabled()
    torch.backends.cuda.enable_cudnn_sdp(False)        # the other kernel adds in one order for as few tokens as these
    try:
        fused, again, plain = grads(_gpt2(d)), grads(_gpt2(d)), grads(_plain(_gpt2(d)))
    finally:
        torch.backends.cuda.enable_cudnn_sdp(was)
    for (n, p), f, a, w in zip(_gpt2(d).named_parameters(), fused, again, plain):
        assert torch.equal(f, a), n
        if p.dim() == 2 and n != "wte.weight":
            assert torch.equal(f, w), n
        elif not n.endswith("k.bias"):                 # zero but for rounding
            assert (f.float() - w.float()).norm() <= 2.0 ** -8 * w.float().norm(), n


@gpu
@pytest.mark.parametrize("frozen", [(), ("k.weight",), ("q.bias", "v.weight")])
@pytest.mark.parametrize("d", [128, 1056])
def test_adjacent_projections_are_one_product(d, frozen):
    """In a bucket the three projections' weights lie next to each other; the gradients are those of the separate parameters."""
    from mccl_b200.parallel.ddp import DistributedDataParallel
    idx, tgt = _batch()

    def make():
        m = _gpt2(d)
        for n, p in m.named_parameters():
            p.requires_grad_(not n.endswith(frozen) if frozen else True)
        return m

    apart, packed = make(), make()
    apart(idx, tgt).backward()
    DistributedDataParallel(packed, None)(idx, tgt).backward()
    want = _plain(make()).double()
    want(idx, tgt).backward()
    for (n, a), b, w in zip(apart.named_parameters(), packed.parameters(), want.parameters()):
        assert (b.grad is None) == (not a.requires_grad), n
        if a.requires_grad and not n.endswith("k.bias"):        # the gradient of a key's bias is zero but for rounding
            ea, eb = ((t.grad.double() - w.grad).norm() / w.grad.norm() for t in (a, b))
            assert eb <= 1.5 * ea + 2.0 ** -9, (n, ea.item(), eb.item())


@gpu
@pytest.mark.parametrize("make", [_gpt2, _llama])
def test_hooks_and_replaced_parts_are_called(make):
    idx, tgt = _batch()
    model, seen = make(), []
    getattr(model.blocks[0], "fc" if make is _gpt2 else "o").register_forward_hook(lambda mod, args, out: seen.append("part"))
    model.blocks[1].register_forward_hook(lambda mod, args, out: seen.append(out if isinstance(out, tuple) else out.shape))
    model(idx, tgt).backward()
    assert seen[0] == "part" and isinstance(seen[1], torch.Size) and seen[1][-1] == 128

    class Twice(nn.Module):                      # a part put in the place of another
        def __init__(self, inner):
            super().__init__()
            self.inner, self.weight = inner, inner.weight

        def forward(self, x):
            return 2 * self.inner(x)

    a, b = make(), make()
    name = "fc" if make is _gpt2 else "o"
    setattr(a.blocks[0], name, Twice(getattr(a.blocks[0], name)))
    with torch.no_grad():
        for p in getattr(b.blocks[0], name).parameters():
            p.mul_(2)
    la, lb = a(idx, tgt), b(idx, tgt)
    assert abs(la.item() - lb.item()) <= 2.0 ** -8 * abs(lb.item()) and abs(la.item() - make()(idx, tgt).item()) > 0


@gpu
@pytest.mark.parametrize("hooked", [(1,), (0, 2), (1, 2), (3,)])
def test_blocks_with_hooks_between_fused_ones(hooked):
    """Every gradient, the last bias of each block among them, as without the hooks."""
    idx, tgt = _batch()
    want, model, ref = _grads(_gpt2(layers=4), idx, tgt), _gpt2(layers=4), _reference(_gpt2(layers=4), idx, tgt)
    for i in hooked:
        model.blocks[i].register_forward_hook(lambda mod, args, out: None)
    names = ["loss"] + [n for n, _ in model.named_parameters()]
    for n, a, b, r in zip(names, _grads(model, idx, tgt), want, ref):
        if not n.endswith("k.bias"):                   # zero but for rounding
            ea, eb = ((t.double() - r).norm() / r.norm() for t in (a, b))
            assert ea <= 1.5 * eb + 2.0 ** -9, (n, ea.item(), eb.item())


@gpu
@pytest.mark.parametrize("make", [_gpt2, _llama])
def test_an_embedding_with_a_padding_row(make):
    idx, tgt = _batch()
    model = make()
    name = "wte" if make is _gpt2 else "embed"
    emb = nn.Embedding(*getattr(model, name).weight.shape, padding_idx=int(idx[0, 0])).to(device="cuda", dtype=torch.bfloat16)
    setattr(model, name, emb)
    model(idx, tgt).backward()
    if make is _llama:
        assert emb.weight.grad[idx[0, 0]].abs().sum() == 0 and emb.weight.grad.abs().sum() > 0
        return
    row, got = int(idx[0, 0]), emb.weight.grad.clone()         # GPT-2's weight has the tied projection's gradient as well
    emb.padding_idx = None
    model.zero_grad(set_to_none=True)
    model(idx, tgt).backward()
    other = torch.ones(len(got), dtype=torch.bool, device="cuda")
    other[row] = False
    assert not torch.equal(got[row], emb.weight.grad[row])
    assert (got[other].float() - emb.weight.grad[other].float()).norm() <= 2.0 ** -6 * got.float().norm()


@gpu
def test_input_changed_in_place_is_noticed():
    blk = _gpt2().blocks[0]
    x = torch.randn(2, 8, 128, device="cuda").to(torch.bfloat16).requires_grad_(True)
    h = x * 1
    y = blk(h)
    with torch.no_grad():
        h.add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()


@gpu
@pytest.mark.parametrize("make", [_gpt2, _llama])
def test_frozen_weights_get_no_gradient(make):
    idx, tgt = _batch()
    model = make()
    for blk in model.blocks:
        blk.q.weight.requires_grad_(False)
    model(idx, tgt).backward()
    for n, p in model.named_parameters():
        assert (p.grad is None) == (not p.requires_grad), n


@gpu
def test_gradients_reach_buckets_hooks_and_other_streams():
    from mccl_b200.parallel.ddp import DistributedDataParallel
    idx, tgt = _batch()
    want = [g.clone() for g in _grads(_gpt2(), idx, tgt)[1:]]
    model = _gpt2()
    ddp = DistributedDataParallel(model, None)
    # Attention's gradient may add in another order from run to run: a few roundings of 2^-9, so 2^-6 in all.  The gradient of a
    # key's bias is zero but for rounding and is left out.
    keep = [not n.endswith("k.bias") for n, _ in model.named_parameters()]

    def same(got, ref, k):
        return not k or (got.float() - ref.float()).norm() <= 2.0 ** -6 * ref.float().norm()

    for _ in range(2):
        ddp(idx, tgt).backward()
    for p, w, k in zip(model.parameters(), want, keep):
        assert same(p.grad, 2 * w, k)
        p.grad.zero_()
    # a hook of the user's sees the gradient of its parameter
    seen = []
    model.blocks[0].fc.weight.register_post_accumulate_grad_hook(lambda p: seen.append(p.grad.clone()))
    ddp(idx, tgt).backward()
    fc = [n for n, _ in model.named_parameters()].index("blocks.0.fc.weight")
    assert len(seen) == 1 and torch.equal(seen[0], model.blocks[0].fc.weight.grad)
    assert same(seen[0], want[fc], True)
    for p in model.parameters():
        p.grad.zero_()
    torch.cuda.synchronize()
    # forward on another stream: what the caller's stream reads after backward() is complete
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        loss = ddp(idx, tgt)
    loss.backward()
    got = [p.grad.clone() for p in model.parameters()]
    for g, w, k in zip(got, want, keep):
        assert same(g, w, k)


@gpu
@pytest.mark.parametrize("make", [_gpt2, _llama])
def test_a_retained_graph_is_differentiated_again(make):
    idx, tgt = _batch()
    model = make()
    params = list(model.parameters())
    loss = model(idx, tgt)
    first = torch.autograd.grad(loss, params, retain_graph=True)
    second = torch.autograd.grad(loss, params, retain_graph=True)
    for (n, _), a, b in zip(model.named_parameters(), first, second):      # attention's gradient may add in another order
        if not n.endswith("k.bias"):
            assert (a.float() - b.float()).norm() <= 2.0 ** -6 * a.float().norm(), n


@gpu
@pytest.mark.parametrize("make", [_gpt2, _llama])
def test_second_derivatives_are_not_constants(make):
    """The nodes' gradients raise when differentiated; with attention by products the plain operations answer."""
    from torch.nn.attention import SDPBackend, sdpa_kernel
    idx, tgt = _batch(b=1, s=16)
    model = make()
    w = model.blocks[0].v.weight
    g, = torch.autograd.grad(model(idx, tgt), [w], create_graph=True)
    with pytest.raises(RuntimeError):
        g.float().pow(2).sum().backward()
    if make is _llama:
        with sdpa_kernel(SDPBackend.MATH):
            x = torch.randn(16, 128, device="cuda").to(torch.bfloat16).requires_grad_(True)
            g, = torch.autograd.grad(model.blocks[0](x, 1, 16).float().sum(), [x], create_graph=True)
            assert torch.autograd.grad(g.float().pow(2).sum(), [x])[0].abs().sum() > 0


@gpu
def test_layers_differentiated_twice_match_plain_operations():
    from mccl_b200.ops.norm import FusedLayerNorm
    from mccl_b200.parallel.layers import ExpertParallelMoE
    from mccl_b200.parallel.tp import FusedTensorParallelMLP
    torch.manual_seed(0)

    def twice(f, x):
        g, = torch.autograd.grad(f(x).float().pow(2).sum(), [x], create_graph=True)
        return torch.autograd.grad(g.float().pow(2).sum(), [x])[0].double()

    x = torch.randn(128, 64, device="cuda").to(torch.bfloat16).requires_grad_(True)
    x64 = x.detach().double().requires_grad_(True)

    def twice64(f):
        g, = torch.autograd.grad(f(x64).pow(2).sum(), [x64], create_graph=True)
        return torch.autograd.grad(g.pow(2).sum(), [x64])[0]

    ln = FusedLayerNorm(64).to(device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        ln.weight.normal_(1.0, 0.3)
    mlp = FusedTensorParallelMLP(_comm(), 128, 64, 128)
    wu, wd = mlp.w_up.detach().double(), mlp.w_down.detach().double()
    silu = nn.functional.silu
    moe = ExpertParallelMoE(_comm(), 64, 64, 1, 128, device="cuda", dtype=torch.bfloat16, fused=True)      # one expert: its gate is 1
    wi, wo = moe.w_in.detach().double()[0], moe.w_out.detach().double()[0]
    for f, f64 in ((ln, lambda t: nn.functional.layer_norm(t, (64,), ln.weight.detach().double(), ln.bias.detach().double(), ln.eps)),
                   (mlp, lambda t: silu(t @ wu.t()) @ wd.t()), (moe, lambda t: silu(t @ wi.t()) @ wo.t())):
        want = twice64(f64)
        assert (twice(f, x) - want).norm() <= 0.05 * want.norm()      # about a dozen bf16 roundings of 2^-8 each


@gpu
def test_torch_func_and_tracing_take_the_plain_route():
    idx, tgt = _batch(b=1, s=16)
    model = _llama()
    params = {n: p.detach() for n, p in model.named_parameters()}
    g = torch.func.grad(lambda ps: torch.func.functional_call(model, ps, (idx, tgt)))(params)
    want = _grads(model, idx, tgt)[1:]
    for (n, a), b in zip(g.items(), want):
        assert (a.float() - b.float()).norm() <= 0.05 * b.float().norm(), n      # the two routes round in another order
    model.requires_grad_(False)
    traced = torch.jit.trace(lambda t: model(t), (idx,), check_trace=False)
    other, _ = _batch(b=1, s=16)
    other = (other + 7) % 300
    with torch.no_grad():
        a, b = traced(other), model(other)
    assert (a.float() - b.float()).norm() <= 0.05 * b.float().norm()


@gpu
def test_weights_of_another_class_are_asked():
    from mccl_b200.parallel.layers import ExpertParallelMoE
    seen = []

    class Mine(torch.Tensor):
        @classmethod
        def __torch_function__(cls, func, types, args=(), kwargs=None):
            seen.append(func)
            with torch._C.DisableTorchFunctionSubclass():
                return func(*args, **(kwargs or {}))

    idx, tgt = _batch()
    layer = ExpertParallelMoE(_comm(), 64, 64, 2, 64, device="cuda", dtype=torch.bfloat16, fused=True)
    layer._parameters["w_in"] = layer.w_in.detach().as_subclass(Mine)
    layer(torch.randn(64, 64, device="cuda").to(torch.bfloat16))
    assert seen
    model = _gpt2()
    model.wte._parameters["weight"] = model.wte.weight.detach().as_subclass(Mine)
    seen.clear()
    model(idx, tgt)
    assert any(getattr(f, "__name__", "") == "linear" for f in seen)       # the tied projection


@gpu
def test_moe_subclass_routes_its_own_way():
    from mccl_b200.parallel.layers import ExpertParallelMoE

    class First(ExpertParallelMoE):
        def route(self, x):
            z = torch.zeros(x.shape[0], dtype=torch.int64, device=x.device)
            slot = torch.arange(x.shape[0], device=x.device)
            return z, torch.ones(x.shape[0], dtype=x.dtype, device=x.device), slot, slot < self.capacity

    torch.manual_seed(0)
    layer = First(_comm(), 64, 64, 4, 64, device="cuda", dtype=torch.bfloat16, fused=True)
    x = torch.randn(64, 64, device="cuda").to(torch.bfloat16)
    want = nn.functional.silu(x.double() @ layer.w_in[0].double().t()) @ layer.w_out[0].double().t()
    assert (layer(x).double() - want).norm() <= 4 * 2.0 ** -8 * want.norm()
