"""MoE layer forward/backward on one GPU (EP world of one rank) against a dense PyTorch oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _dense_oracle(x, logits, w1, w2, topk, activation):
    from gpu_data_transfer_profile_b200.models.experts import activate
    from gpu_data_transfer_profile_b200.models.moe_layer import topk_softmax_router
    idx, probs = topk_softmax_router(logits, topk)
    out = torch.zeros_like(x, dtype=torch.float32)
    for k in range(topk):
        for e in range(w1.shape[0]):
            m = idx[:, k] == e
            if m.any():
                h = activate(x[m].float() @ w1[e].float().t(), activation) * probs[m, k][:, None]
                out[m] += h @ w2[e].float().t()
    return out


@pytest.mark.parametrize("mode", ["fused", "deepep"])
@pytest.mark.parametrize("activation", ["swiglu", "gelu"])
def test_moe_layer_forward_backward_matches_dense_oracle(mode, activation):
    from gpu_data_transfer_profile_b200.models import fused_a2a as A
    from gpu_data_transfer_profile_b200.models.moe_layer import MoELayer
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    torch.manual_seed(0)
    T, H, F, E, K = 96, 256, 512, 4, 2
    world = LocalWorld.make(1)[0]
    A.configure_buffer(num_max_tokens_per_rank=128, num_topk=K, num_experts=E, group_by_expert=True)
    try:
        layer = MoELayer(H, F, E, K, None, dtype=torch.float32, activation=activation, expert_backend="torch",
                         dispatcher_mode=mode, world=world)
        x = torch.randn(T, H, device="cuda", requires_grad=True)
        logits = torch.randn(T, E, device="cuda", requires_grad=True)
        out = layer(x, logits)
        ref = _dense_oracle(x, logits, layer.experts.weight1, layer.experts.weight2, K, activation)
        torch.testing.assert_close(out, ref, atol=2e-4, rtol=2e-4)
        g = torch.randn_like(out)
        gx, gl, gw1 = torch.autograd.grad(out, [x, logits, layer.experts.weight1], g, retain_graph=False)
        rx, rl, rw1 = torch.autograd.grad(ref, [x, logits, layer.experts.weight1], g)
        torch.testing.assert_close(gx, rx, atol=2e-4, rtol=2e-4)
        torch.testing.assert_close(gl, rl, atol=2e-4, rtol=2e-3)
        torch.testing.assert_close(gw1, rw1, atol=2e-4, rtol=2e-3)
    finally:
        A.release_buffers()


def test_moe_layer_fused_combine_training_path_gradients():
    """fc2 epilogue performs the combine send in the TRAINING forward; gradients must equal the
    separate-combine path."""
    from gpu_data_transfer_profile_b200.models import fused_a2a as A
    from gpu_data_transfer_profile_b200.models.moe_layer import MoELayer
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    torch.manual_seed(0)
    T, H, F, E, K = 200, 256, 512, 4, 2
    world = LocalWorld.make(1)[0]
    A.configure_buffer(num_max_tokens_per_rank=256, num_topk=K, num_experts=E, group_by_expert=True)
    try:
        layer = MoELayer(H, F, E, K, None, dtype=torch.bfloat16, expert_backend="tcgen05", world=world)
        x0 = torch.randn(T, H, device="cuda").to(torch.bfloat16)
        logits = torch.randn(T, E, device="cuda")
        g = torch.randn(T, H, device="cuda").to(torch.bfloat16)
        res = []
        for fuse in (True, False):
            layer.fuse_combine = fuse
            layer.zero_grad()
            x = x0.clone().requires_grad_(True)
            lg = logits.clone().requires_grad_(True)
            out = layer(x, lg)
            out.backward(g)
            res.append((out.detach().float(), x.grad.float(), lg.grad.float(), layer.experts.weight1.grad.float().clone(),
                        layer.experts.weight2.grad.float().clone()))
        for a, b in zip(*res):
            torch.testing.assert_close(a, b, atol=3e-2, rtol=3e-2)
    finally:
        A.release_buffers()


@pytest.mark.parametrize("fused", [False, True])
def test_moe_layer_tcgen05_experts_bf16(fused):
    """bf16 layer on the tcgen05 grouped GEMMs (separate combine with autograd, and the forward-only
    path whose fc2 epilogue performs the combine send) against the fp32 dense oracle."""
    from gpu_data_transfer_profile_b200.models import fused_a2a as A
    from gpu_data_transfer_profile_b200.models.moe_layer import MoELayer
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    torch.manual_seed(0)
    T, H, F, E, K = 300, 512, 1024, 4, 2
    world = LocalWorld.make(1)[0]
    A.configure_buffer(num_max_tokens_per_rank=512, num_topk=K, num_experts=E, group_by_expert=True)
    try:
        layer = MoELayer(H, F, E, K, None, dtype=torch.bfloat16, activation="swiglu", expert_backend="tcgen05",
                         dispatcher_mode="fused", world=world)
        assert layer.expert_backend == "tcgen05_grouped_gemm"
        x = torch.randn(T, H, device="cuda").to(torch.bfloat16).requires_grad_(not fused)
        logits = torch.randn(T, E, device="cuda")
        ref = _dense_oracle(x.detach().float(), logits, layer.experts.weight1.detach(), layer.experts.weight2.detach(),
                            K, "swiglu")
        if fused:
            with torch.no_grad():
                out = layer(x, logits)
        else:
            out = layer(x, logits)
            out.float().sum().backward()
            assert x.grad is not None and torch.isfinite(x.grad).all()
            assert layer.experts.weight1.grad is not None and torch.isfinite(layer.experts.weight1.grad).all()
        torch.testing.assert_close(out.float(), ref, atol=2e-2, rtol=5e-2)
    finally:
        A.release_buffers()


def test_moe_layer_fp8_inference_path_close_to_bf16():
    """fp8 dispatch (cast fused into the send kernel) feeding the block-scaled fp8 fc1 directly,
    against the same layer's bf16 path: the difference is the e4m3 rounding of rows and weights."""
    from gpu_data_transfer_profile_b200.models import fused_a2a as A
    from gpu_data_transfer_profile_b200.models.moe_layer import MoELayer
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    torch.manual_seed(0)
    T, H, F, E, K = 300, 512, 1024, 4, 2
    world = LocalWorld.make(1)[0]
    A.configure_buffer(num_max_tokens_per_rank=512, num_topk=K, num_experts=E, group_by_expert=True)
    try:
        layer = MoELayer(H, F, E, K, None, dtype=torch.bfloat16, activation="swiglu", expert_backend="tcgen05",
                         dispatcher_mode="fused", world=world, use_fp8=True, fuse_combine=False)
        assert layer.use_fp8
        x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
        logits = torch.randn(T, E, device="cuda")
        with torch.no_grad():
            out8 = layer(x, logits)
            layer.use_fp8 = False
            out16 = layer(x, logits)
        scale = float(out16.float().abs().max())
        torch.testing.assert_close(out8.float(), out16.float(), atol=0.06 * scale, rtol=0.1)
    finally:
        A.release_buffers()


@pytest.mark.parametrize("T,E,H,K", [(1, 3, 8, 1), (7, 8, 264, 2), (64, 64, 2048, 8), (65, 33, 1000, 4), (130, 160, 7168, 6),
                                     (300, 256, 512, 8), (66, 1024, 128, 32), (40, 300, 72, 3)])
def test_router_kernels_against_64_bits(T, E, H, K):
    """Expert ids and weights from bf16 rows and f32 router weights. The logits are f32 sums of H products: their
    error against 64 bits stays within a few ulp times sqrt(H), the ids differ only where two logits are closer."""
    from gpu_data_transfer_profile_b200 import _ext
    C = _ext.load()
    torch.manual_seed(5)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    w = torch.randn(E, H, device="cuda") * 0.02
    idx, prob = C.route(x, w, K)
    logits = x.double() @ w.double().t()
    top, ref = torch.topk(torch.softmax(logits, -1), K, dim=-1)
    eps = 1e-6 * (1 + float(logits.abs().max()))
    picked = logits.gather(1, idx)
    assert bool((picked - logits.gather(1, ref)).abs().max() <= eps)            # as good a choice, rank by rank
    assert all(len(set(r)) == K for r in idx.tolist())
    want = torch.softmax(logits, -1).gather(1, idx)
    torch.testing.assert_close(prob.double(), want / want.sum(-1, keepdim=True), rtol=1e-5, atol=1e-7)
    idx2, prob2 = C.topk_softmax(logits.float().contiguous(), K)
    assert bool((logits.gather(1, idx2) - logits.gather(1, ref)).abs().max() <= eps)
    torch.testing.assert_close(prob2.double().sum(-1), torch.ones(T, dtype=torch.float64, device="cuda"), rtol=1e-5, atol=0)


def test_router_topk_of_masked_infinite_and_nan_logits():
    """Masked experts (-inf, the type's lowest value) are chosen last and weigh nothing; equal logits give distinct
    experts; a row that softmax turns into NaN still names distinct experts in range."""
    from gpu_data_transfer_profile_b200 import _ext
    C = _ext.load()
    E, K, inf = 40, 4, float("inf")
    rows = torch.zeros(7, E)
    rows[0, :] = -inf
    rows[0, [7, 39]] = torch.tensor([1.0, 2.0])                       # two finite, two masked choices
    rows[1, :] = torch.finfo(torch.float32).min
    rows[1, 33] = 0.5
    rows[2, :] = -inf                                                  # nothing but masked: NaN weights
    rows[3, 5] = float("nan")
    rows[4, 6] = inf
    rows[5, 1] = -0.0                                                  # all equal
    rows[6] = torch.linspace(-3, 3, E)
    idx, prob = (t.cpu() for t in C.topk_softmax(rows.cuda(), K))
    assert bool(((idx >= 0) & (idx < E)).all()) and all(len(set(r)) == K for r in idx.tolist())
    assert idx[0, :2].tolist() == [39, 7] and prob[0, 2:].tolist() == [0.0, 0.0]
    torch.testing.assert_close(prob[0, :2], torch.softmax(torch.tensor([2.0, 1.0]), 0))
    assert idx[1, 0] == 33 and prob[1].tolist() == [1.0, 0.0, 0.0, 0.0]
    assert bool(prob[2].isnan().all()) and bool(prob[3].isnan().all()) and bool(prob[4].isnan().all())
    assert prob[5].tolist() == [0.25] * 4 and idx[6].tolist() == [39, 38, 37, 36]


@pytest.mark.parametrize("use_fp8,fuse", [(False, True), (True, True), (True, False)])
@pytest.mark.parametrize("activation", ["swiglu", "silu"])
def test_moe_layer_inference_consumes_rows_in_place(use_fp8, fuse, activation):
    """Two layers of different sizes on one shared buffer, called in turn: the inference path (own router, rows read
    where they arrive, no host read of the counts) gives what the general path gives, and the dispatcher's record of
    the last dispatch is the caller's own."""
    from gpu_data_transfer_profile_b200.models import fused_a2a as A
    from gpu_data_transfer_profile_b200.models.moe_layer import MoELayer, topk_softmax_router
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    torch.manual_seed(0)
    world = LocalWorld.make(1)[0]
    A.configure_buffer(num_max_tokens_per_rank=512, num_topk=4, num_experts=8, group_by_expert=True)
    try:
        layers = [MoELayer(512, 256, 8, 4, None, activation=activation, expert_backend="tcgen05", world=world,
                           use_fp8=use_fp8, fuse_combine=fuse) for _ in range(2)]
        x = torch.randn(301, 512, device="cuda").to(torch.bfloat16)
        with torch.no_grad():
            a = layers[0](x)
            counts, probs = layers[0].dispatcher.tokens_per_expert, layers[0].dispatcher.dispatched_probs
            kept = None if probs is None else probs.clone()
            for _ in range(3):                                       # more dispatches than the region has parities
                b = layers[1](a)
            for layer, inp, got in ((layers[0], x, a), (layers[1], a, b)):
                idx, w = topk_softmax_router(layer.router(inp.float()), 4)
                if use_fp8:
                    rows, tpe, rp = layer.dispatcher.dispatch_fp8(inp, idx, w)
                    y = layer.experts.forward_fp8(rows, tpe, rp)
                else:
                    rows, tpe, rp = layer.dispatcher.dispatch(inp, idx, w)
                    y = layer.experts(rows, tpe, rp)
                want = layer.dispatcher.combine(y)
                # weights differ by f32 rounding of the softmax, rows by one bf16 rounding of it
                torch.testing.assert_close(got.float(), want.float(), rtol=2.0 ** -6, atol=2.0 ** -8 * float(want.abs().max()))
        if not use_fp8:
            assert counts.device.type == "cpu" and int(counts.sum()) == 301 * 4
            assert torch.equal(probs, kept)
        A._BUFFERS[(id(None), id(world))].check_status()
    finally:
        A.release_buffers()


def test_exchange_backward_after_the_index_tensor_is_refilled():
    """A static routing buffer that is refilled between the forward and the backward pass of an exchange."""
    from gpu_data_transfer_profile_b200.models import fused_a2a as A
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    T, H, E, K = 200, 256, 8, 2
    world = LocalWorld.make(1)[0]
    A.configure_buffer(num_max_tokens_per_rank=T, num_topk=K, num_experts=E, group_by_expert=True)
    try:
        g = torch.Generator().manual_seed(0)
        x = torch.randn(T, H, generator=g).to(torch.bfloat16).cuda().requires_grad_(True)
        idx = torch.rand(T, E, generator=g).topk(K, dim=-1).indices.cuda()
        w = torch.rand(T, K, generator=g).cuda().requires_grad_(True)
        dy = torch.randn(T, H, generator=g).to(torch.bfloat16).cuda()
        rows, probs, _, handle = A.FusedDispatchGrouped.apply(x, idx, w, E, None, world)
        out = A.FusedCombineGrouped.apply(rows, None, handle, world)
        idx.fill_(-1)
        (out.float() * dy.float()).sum().add(3 * probs.sum()).backward()
        assert torch.equal(out, 2 * x)
        assert torch.equal(x.grad, 2 * dy) and torch.equal(w.grad, torch.full_like(w, 3.0))
        A._BUFFERS[(id(None), id(world))].check_status()
    finally:
        A.release_buffers()


@pytest.fixture
def small_layer():
    from gpu_data_transfer_profile_b200.models import fused_a2a as A
    from gpu_data_transfer_profile_b200.models.moe_layer import MoELayer
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    torch.manual_seed(0)
    world = LocalWorld.make(1)[0]
    A.configure_buffer(num_max_tokens_per_rank=128, num_topk=2, num_experts=4, group_by_expert=True)
    yield lambda **kw: MoELayer(256, 128, 4, 2, None, expert_backend="tcgen05", world=world, **kw)
    A.release_buffers()


@pytest.mark.parametrize("where", ["input", "logits", "router", "jvp", "vmap"])
def test_moe_layer_inference_refuses_tangents_and_transforms(small_layer, where):
    """Nothing on the way has a forward-mode or batching rule: refused, not dropped."""
    import torch.autograd.forward_ad as fwad
    layer = small_layer()
    x, logits = torch.randn(65, 256, device="cuda").to(torch.bfloat16), torch.randn(65, 4, device="cuda")
    with torch.no_grad():
        want = layer(x)
        if where == "vmap":
            with pytest.raises(RuntimeError):
                torch.vmap(layer)(x[None])
        elif where == "jvp":
            with pytest.raises(RuntimeError):
                torch.func.jvp(layer, (x,), (torch.ones_like(x),))
        else:
            with fwad.dual_level():
                dual = lambda t: fwad.make_dual(t, torch.ones_like(t))
                with pytest.raises(NotImplementedError):
                    if where == "router":
                        torch.func.functional_call(layer, {"router.weight": dual(layer.router.weight.detach())}, (x,))
                    else:
                        layer(dual(x)) if where == "input" else layer(x, dual(logits))
                assert torch.equal(layer(x), want)           # plain tensors inside a dual level: the usual path
        assert torch.equal(layer(x), want)


@pytest.mark.parametrize("use_fp8", [False, True])
def test_moe_layer_inference_calls_replaced_dispatchers_and_experts(small_layer, use_fp8, monkeypatch):
    from gpu_data_transfer_profile_b200.models.experts_tcgen05 import Tcgen05GroupedExperts
    from gpu_data_transfer_profile_b200.models.token_dispatcher import B200TokenDispatcher
    layer = small_layer(use_fp8=use_fp8)
    x = torch.randn(65, 256, device="cuda").to(torch.bfloat16)
    name = "dispatch_fp8" if use_fp8 else "dispatch"
    seen = []

    def noted(fn):
        def f(*a, **k):
            seen.append(fn.__name__)
            return fn(*a, **k)
        return f

    class Sub(B200TokenDispatcher):
        def dispatch(self, *a):
            seen.append("dispatch")
            return super().dispatch(*a)

        def dispatch_fp8(self, *a):
            seen.append("dispatch_fp8")
            return super().dispatch_fp8(*a)

    class Other:                                          # a dispatcher that has nothing but what the general path calls
        def __init__(self, d):
            self.d, self.mode, self.group, self.world = d, d.mode, d.group, d.world
        handle = property(lambda self: self.d.handle, lambda self, v: setattr(self.d, "handle", v))

        def dispatch(self, *a):
            seen.append("dispatch")
            return self.d.dispatch(*a)

        def dispatch_fp8(self, *a):
            seen.append("dispatch_fp8")
            return self.d.dispatch_fp8(*a)

        def combine(self, y):
            return self.d.combine(y)

    class Experts(Tcgen05GroupedExperts):
        def forward_fp8(self, hidden_states, tokens_per_expert, routed_probs, expert_off=None):
            seen.append(sum(int(v) for v in tokens_per_expert))
            return super().forward_fp8(hidden_states, tokens_per_expert, routed_probs, expert_off)

        def forward_fused_combine(self, rows, routed_probs, buffer, handle):
            seen.append(sum(handle.num_recv_tokens_per_expert_list))
            return super().forward_fused_combine(rows, routed_probs, buffer, handle)

    with torch.no_grad():
        want = layer(x)
        own = layer.dispatcher
        for d in (Sub(None, 4, 4, 0, world=own.world), Other(own)):
            layer.dispatcher = d
            # the same rows through the same kernels; the weights come from the same router
            assert torch.equal(layer(x), want) and seen.pop() == name and not seen
        layer.dispatcher = own
        setattr(own, name, noted(getattr(own, name)))                         # wrapped on the instance
        assert torch.equal(layer(x), want) and seen.pop() == name and not seen
        delattr(own, name)
        with monkeypatch.context() as m:                                      # wrapped on the class
            m.setattr(B200TokenDispatcher, name, noted(getattr(B200TokenDispatcher, name)))
            assert torch.equal(layer(x), want) and seen.pop() == name and not seen
        layer.experts.__class__ = Experts
        assert torch.equal(layer(x), want) and seen.pop() == 65 * 2 and not seen


@pytest.mark.parametrize("T,E,K", [(1, 1, 1), (9, 8, 2), (33, 64, 8), (7, 257, 32), (5, 1024, 3)])
def test_training_router_matches_the_torch_form(T, E, K):
    """Choice, renormalised weights and the logits' gradient on this library's kernels against the torch form in f64 (an
    f32 softmax and its gradient: a few units of 2^-24 relative to values of at most one times the incoming gradient), in
    rows with a masked expert, with not-a-number, and through a second derivative."""
    from gpu_data_transfer_profile_b200.models.moe_layer import _TopkSoftmax, topk_softmax_router
    gen = torch.Generator().manual_seed(T * E)
    logits = torch.randn(T, E, generator=gen).cuda() * 3
    if E > K:
        logits[0, 0] = -float("inf")
    gw = torch.randn(T, K, generator=gen).cuda()
    l = logits.clone().requires_grad_(True)
    idx, w = _TopkSoftmax.apply(l, K)
    l64 = logits.double().requires_grad_(True)
    top, idx64 = torch.topk(torch.softmax(l64, -1), K, dim=-1)
    w64 = top / top.sum(-1, keepdim=True)
    assert torch.equal(idx, idx64) and not idx.requires_grad
    torch.testing.assert_close(w.double(), w64, atol=0, rtol=2 ** -19)
    (g,) = torch.autograd.grad(w, l, gw, create_graph=True)
    (g64,) = torch.autograd.grad(w64, l64, gw.double(), create_graph=True)
    bound = dict(atol=2 ** -18 * float(gw.abs().max()), rtol=0)
    torch.testing.assert_close(g.double(), g64, **bound)
    (gg,) = torch.autograd.grad(g.square().sum(), l)
    (gg64,) = torch.autograd.grad(g64.square().sum(), l64)
    torch.testing.assert_close(gg.double(), gg64, atol=2 ** -16 * float(gw.abs().max()) ** 2, rtol=1e-4)
    idx, w = _TopkSoftmax.apply(l, K)
    (g,) = torch.autograd.grad(w, l, gw)                     # the kernel
    torch.testing.assert_close(g.double(), g64, **bound)
    l = logits.clone()
    l[-1] = float("nan")
    l.requires_grad_(True)
    (g,) = torch.autograd.grad(_TopkSoftmax.apply(l, K)[1], l, gw)
    lt = l.detach().clone().requires_grad_(True)
    (gt,) = torch.autograd.grad(topk_softmax_router(lt, K)[1], lt, gw)
    assert bool(g[-1].isnan().all()) and bool(gt[-1].isnan().all()) and not bool(g[:-1].isnan().any())


@pytest.mark.parametrize("use_fp8,fuse", [(False, True), (True, True), (False, False)])
@pytest.mark.parametrize("activation", ["swiglu", "silu"])
def test_moe_layer_without_tokens(use_fp8, fuse, activation):
    """A batch of no tokens between ordinary ones: empty outputs, zero gradients, and calls before and after it agree."""
    from gpu_data_transfer_profile_b200.models import fused_a2a as A
    from gpu_data_transfer_profile_b200.models.moe_layer import MoELayer
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    torch.manual_seed(0)
    world = LocalWorld.make(1)[0]
    A.configure_buffer(num_max_tokens_per_rank=128, num_topk=2, num_experts=4, group_by_expert=True)
    try:
        layer = MoELayer(256, 128, 4, 2, None, activation=activation, expert_backend="tcgen05", world=world,
                         use_fp8=use_fp8, fuse_combine=fuse)
        x = torch.randn(65, 256, device="cuda").to(torch.bfloat16)
        none = x[:0].detach()
        with torch.no_grad():
            want = layer(x)
            assert layer(none).shape == (0, 256)
            assert torch.equal(layer(x), want)
        leaf = none.clone().requires_grad_(True)
        out = layer(leaf)
        assert out.shape == (0, 256)
        out.float().sum().backward()
        assert leaf.grad.shape == (0, 256)
        for w in (layer.router.weight, layer.experts.weight1, layer.experts.weight2):
            assert w.grad.shape == w.shape and not w.grad.any()
        with torch.no_grad():
            assert torch.equal(layer(x), want)
        A._BUFFERS[(id(None), id(world))].check_status()
    finally:
        A.release_buffers()


def test_training_router_gradient_of_batches_and_tangents():
    """A batch of incoming gradients (both forms of it) and one with a tangent, as the torch form takes them."""
    from torch.autograd import forward_ad
    from gpu_data_transfer_profile_b200.models.moe_layer import _TopkSoftmax, topk_softmax_router
    T, E, K, B = 9, 8, 3, 4
    gen = torch.Generator().manual_seed(7)
    logits = torch.randn(T, E, generator=gen).cuda()
    gw = torch.randn(B, T, K, generator=gen).cuda()

    def grads(router):
        l = logits.clone().requires_grad_(True)
        w = router(l, K)[1]
        one = lambda g: torch.autograd.grad(w, l, g, retain_graph=True)[0]
        batch = torch.autograd.grad(w, l, gw, retain_graph=True, is_grads_batched=True)[0]
        mapped = torch.func.vmap(one)(gw)
        with forward_ad.dual_level():
            dual = forward_ad.unpack_dual(one(forward_ad.make_dual(gw[0], gw[1])))
            return torch.stack([one(g) for g in gw]), batch, mapped, dual.primal.clone(), dual.tangent.clone()

    want = grads(topk_softmax_router)
    for got, ref in zip(grads(_TopkSoftmax.apply), want):
        # f32 softmax and its gradient: a few units of 2^-24 relative to the incoming gradient
        torch.testing.assert_close(got, ref, atol=2 ** -18 * float(gw.abs().max()), rtol=0)


@pytest.mark.parametrize("train", [False, True])
@pytest.mark.parametrize("given", [False, True])
def test_moe_layer_calls_a_router_put_in_place_of_its_own(train, given, monkeypatch):
    from gpu_data_transfer_profile_b200.models import fused_a2a as A, moe_layer as M
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    torch.manual_seed(0)
    A.configure_buffer(num_max_tokens_per_rank=128, num_topk=2, num_experts=4, group_by_expert=True)
    seen = []

    def fixed(logits, topk):                                  # the same two experts for every token, one choice masked
        seen.append(tuple(logits.shape))
        idx = torch.arange(topk, device=logits.device).repeat(logits.shape[0], 1)
        idx[0, 1] = -1
        return idx, torch.ones(idx.shape, device=logits.device)

    try:
        layer = M.MoELayer(256, 128, 4, 2, None, expert_backend="tcgen05", world=LocalWorld.make(1)[0])
        x = torch.randn(65, 256, device="cuda").to(torch.bfloat16)
        logits = torch.randn(65, 4, device="cuda") if given else None
        monkeypatch.setattr(M, "topk_softmax_router", fixed)
        with torch.set_grad_enabled(train):
            y = layer(x, logits).detach()
        assert seen == [(65, 4)]
        counts = [65, 64, 0, 0]
        rows = torch.cat([x, x[1:]])
        with torch.no_grad():
            z = layer.experts(rows, counts, torch.ones(129, device="cuda")).float()
        want = z[:65]
        want[1:] += z[65:]
        torch.testing.assert_close(y.float(), want, rtol=2.0 ** -6, atol=2.0 ** -8 * float(want.abs().max()))
    finally:
        A.release_buffers()


@pytest.mark.parametrize("slots", [True, False])
@pytest.mark.parametrize("T,K", [(1, 1), (65, 3)])
def test_dispatch_in_place_keeps_what_a_pulling_combine_reads_in_the_region(slots, T, K):
    """Rows and probabilities of a dispatch in place go back to their tokens without a copy (all that a buffer without
    combine slots can do); the dispatcher's record of the probabilities is a tensor of its own."""
    from gpu_data_transfer_profile_b200.models import fused_a2a as A
    from gpu_data_transfer_profile_b200.models.token_dispatcher import B200TokenDispatcher
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    H, E = 256, 8
    world = LocalWorld.make(1)[0]
    A.configure_buffer(num_max_tokens_per_rank=T, num_topk=K, num_experts=E, group_by_expert=True)
    try:
        buf = Buffer(None, 64 << 20, world=world, timeout_s=2.0, combine_slots=slots)
        A.set_buffer(None, buf, world)
        d = B200TokenDispatcher(None, E, E, 0, world=world)
        g = torch.Generator().manual_seed(T)
        for _ in range(3):
            x = torch.randn(T, H, generator=g).to(torch.bfloat16).cuda()
            idx, w = torch.rand(T, E, generator=g).topk(K, dim=-1).indices.cuda(), torch.rand(T, K, generator=g).cuda()
            rows, probs, handle = d.dispatch_in_place(x, idx, w)
            own = d.dispatched_probs
            order = torch.sort(idx.flatten(), stable=True).indices
            assert torch.equal(rows, x[order // K]) and torch.equal(probs, w.flatten()[order]) and torch.equal(own, probs)
            out, back, _ = buf.combine(rows, handle, topk_weights=probs)
            assert torch.equal(back, w)
            torch.testing.assert_close(out.float(), K * x.float(), rtol=2.0 ** -8, atol=0)
            probs.zero_()
            assert torch.equal(own, w.flatten()[order])
        buf.check_status()
        buf.check_canaries()
    finally:
        A.release_buffers()
