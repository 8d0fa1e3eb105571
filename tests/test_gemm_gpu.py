"""tcgen05 grouped GEMM against a plain PyTorch fp32 reference of the same op."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, w, counts):
    outs, r = [], 0
    for e, c in enumerate(counts):
        outs.append(a[r:r + c].float() @ w[e].float().t())
        r += c
    return torch.cat(outs) if outs else a.new_zeros((0, w.shape[1]), dtype=torch.float32)


# pair=True: the CTA-pair form (cluster of two SMs, 256-row tiles); False: one CTA per 128-row tile
@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("counts,N,K", [([128], 256, 64), ([256, 128], 512, 256), ([100, 0, 333, 7], 256, 320),
                                        ([513], 384, 1024), ([64, 64, 64, 64, 64, 64, 64, 64], 1024, 512),
                                        ([1000, 129, 2300], 768, 448)])
def test_grouped_gemm_plain(counts, N, K, pair):
    from gpu_data_transfer_profile_b200.ops import gemm as G
    torch.manual_seed(0)
    rows = sum(counts)
    a = torch.randn(rows + 5, K, device="cuda").to(torch.bfloat16)        # extra rows must stay untouched
    w = (torch.randn(len(counts), N, K, device="cuda") * 0.1).to(torch.bfloat16)
    off = G.offsets_from_counts(counts, "cuda")
    out = torch.full((rows + 5, N), 7.0, dtype=torch.bfloat16, device="cuda")
    G.grouped_gemm(a, w, off, out=out, pair=pair)
    torch.cuda.synchronize()
    ref = _ref(a[:rows], w, counts)
    torch.testing.assert_close(out[:rows].float(), ref, atol=0.05 * (K ** 0.5) * 0.1, rtol=2e-2)
    assert bool((out[rows:] == 7.0).all())


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("counts,N,K", [([128], 256, 64), ([100, 0, 333, 7], 320, 256), ([513, 31], 384, 1000),
                                        ([1000, 129, 2300], 768, 448)])
def test_grouped_gemm_weights_stored_k_by_n(counts, N, K, pair):
    """out[r] = a[r] @ w[e] with w stored [E, K, N]: the data-gradient form, weights read in place."""
    from gpu_data_transfer_profile_b200.ops import gemm as G
    torch.manual_seed(4)
    rows = sum(counts)
    a = torch.randn(rows, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(len(counts), K, N, device="cuda") * 0.1).to(torch.bfloat16)
    out = G.grouped_gemm(a, w, G.offsets_from_counts(counts, "cuda"), pair=pair, w_kn=True)
    torch.cuda.synchronize()
    ref = _ref(a, w.transpose(1, 2), counts)
    torch.testing.assert_close(out.float(), ref, atol=0.05 * (K ** 0.5) * 0.1, rtol=2e-2)


# edges of the token tiles (one row, a unit of 16 / 32 rows more or less, 256 and beyond, more than 32 experts, most of
# them empty) and of the weight tiles (fewer output columns than a CTA holds, a ragged last tile), short reductions.
# Tolerance: one bf16 rounding of the result (2^-8 of it covers a value at the boundary) plus f32 accumulation noise.
@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("counts", [[1], [15, 16, 17, 31, 32, 33], [255, 256, 257], [511, 513, 800], [5] * 40,
                                    [0] * 10 + [300] + [0] * 30 + [2]])
@pytest.mark.parametrize("N,K", [(8, 8), (136, 72), (264, 200), (640, 328)])
def test_grouped_gemm_token_and_weight_tile_edges(counts, N, K, pair):
    from gpu_data_transfer_profile_b200.ops import gemm as G
    torch.manual_seed(8)
    rows, E = sum(counts), len(counts)
    a = torch.randn(rows + 3, K, device="cuda").to(torch.bfloat16)
    a[rows:] = float("nan")                                # rows after the last expert must not leak
    w = (torch.randn(E, N, K, device="cuda") * 0.1).to(torch.bfloat16)
    off = G.offsets_from_counts(counts, "cuda")
    tol = dict(rtol=2.0 ** -8, atol=1e-4 * K ** 0.5)
    for kn in (False, True):
        out = torch.full((rows + 3, N), 7.0, dtype=torch.bfloat16, device="cuda")
        G.grouped_gemm(a, w.transpose(1, 2).contiguous() if kn else w, off, out=out, pair=pair, w_kn=kn)
        torch.cuda.synchronize()
        torch.testing.assert_close(out[:rows].float(), _ref(a[:rows], w, counts), **tol)
        assert bool((out[rows:] == 7.0).all())
    F = max(128, N // 128 * 128)
    w1 = (torch.randn(E, 2 * F, K, device="cuda") * 0.1).to(torch.bfloat16)
    pre = torch.empty(rows + 3, 2 * F, dtype=torch.bfloat16, device="cuda")
    prob = torch.rand(rows + 3, device="cuda")
    act = G.grouped_gemm_swiglu(a, w1, off, prob, pair=pair, pre_out=pre)
    torch.cuda.synchronize()
    h = _ref(a[:rows], w1, counts)
    torch.testing.assert_close(pre[:rows].float(), h, **tol)
    torch.testing.assert_close(act[:rows].float(), torch.nn.functional.silu(h[:, :F]) * h[:, F:] * prob[:rows, None], rtol=2.0 ** -8, atol=1e-3)


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("counts,F,K", [([128], 128, 128), ([200, 56], 256, 256), ([1, 300], 384, 192),
                                        ([700, 3, 257], 512, 512)])
def test_grouped_gemm_swiglu_prob(counts, F, K, pair):
    from gpu_data_transfer_profile_b200.ops import gemm as G
    torch.manual_seed(1)
    rows = sum(counts)
    a = torch.randn(rows, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(len(counts), 2 * F, K, device="cuda") * 0.1).to(torch.bfloat16)
    prob = torch.rand(rows, device="cuda")
    out = G.grouped_gemm_swiglu(a, w, G.offsets_from_counts(counts, "cuda"), prob, pair=pair)
    torch.cuda.synchronize()
    fc1 = _ref(a, w, counts)
    ref = torch.nn.functional.silu(fc1[:, :F]) * fc1[:, F:] * prob[:, None]
    torch.testing.assert_close(out.float(), ref, atol=0.06, rtol=3e-2)


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("counts,M,N", [([64], 256, 256), ([128, 192], 256, 512), ([100, 0, 333, 7], 256, 320),
                                        ([90, 40], 192, 256), ([70, 0, 130], 200, 136),
                                        ([1], 512, 64), ([513, 63, 65], 768, 264), ([0, 0, 40], 256, 128),
                                        ([1000, 129, 2300], 512, 1024)])
def test_grouped_wgrad(counts, M, N, pair):
    """dW[e] = g_e^T x_e with the reduction over each expert's (ragged) rows; rows after the last
    expert hold NaN and must not leak into any gradient."""
    from gpu_data_transfer_profile_b200.ops import gemm as G
    torch.manual_seed(3)
    rows = sum(counts)
    g = torch.randn(rows + 70, M, device="cuda").to(torch.bfloat16)
    x = torch.randn(rows + 70, N, device="cuda").to(torch.bfloat16)
    g[rows:] = float("nan")
    x[rows:] = float("nan")
    dw = G.grouped_wgrad(g, x, G.offsets_from_counts(counts, "cuda"), pair=pair)
    torch.cuda.synchronize()
    r = 0
    for e, c in enumerate(counts):
        ref = g[r:r + c].float().t() @ x[r:r + c].float()
        torch.testing.assert_close(dw[e].float(), ref, atol=0.05 * max(c, 1) ** 0.5, rtol=2e-2)
        r += c


@pytest.mark.parametrize("counts", [[70] * 12, [1, 65, 130, 3, 0, 200, 64, 129] * 2, [320 + 17] * 5])
def test_grouped_wgrad_many_short_ragged_experts(counts):
    """Several ragged last blocks in the operand ring at once: more output tiles than CTA pairs and
    experts of fewer 64-row blocks than the ring has stages."""
    from gpu_data_transfer_profile_b200.ops import gemm as G
    torch.manual_seed(7)
    rows, M, N = sum(counts), 2560, 2048
    g = torch.randn(rows, M, device="cuda").to(torch.bfloat16)
    x = torch.randn(rows, N, device="cuda").to(torch.bfloat16)
    dw = G.grouped_wgrad(g, x, G.offsets_from_counts(counts, "cuda"), pair=True)
    torch.cuda.synchronize()
    r = 0
    for e, c in enumerate(counts):
        ref = g[r:r + c].float().t() @ x[r:r + c].float()
        torch.testing.assert_close(dw[e].float(), ref, atol=0.05 * max(c, 1) ** 0.5, rtol=2e-2)
        r += c


@pytest.mark.parametrize("pair", [False, True])
def test_grouped_gemm_swiglu_also_stores_pre_activation(pair):
    from gpu_data_transfer_profile_b200.ops import gemm as G
    torch.manual_seed(6)
    counts, F, K = [300, 1, 0, 215], 384, 320
    rows = sum(counts)
    a = torch.randn(rows, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(len(counts), 2 * F, K, device="cuda") * 0.1).to(torch.bfloat16)
    prob = torch.rand(rows, device="cuda")
    pre = torch.full((rows + 3, 2 * F), 5.0, dtype=torch.bfloat16, device="cuda")
    out = G.grouped_gemm_swiglu(a, w, G.offsets_from_counts(counts, "cuda"), prob, pair=pair, pre_out=pre)
    torch.cuda.synchronize()
    fc1 = _ref(a, w, counts)
    torch.testing.assert_close(pre[:rows].float(), fc1, atol=0.06, rtol=2e-2)
    assert bool((pre[rows:] == 5.0).all())
    ref = torch.nn.functional.silu(fc1[:, :F]) * fc1[:, F:] * prob[:, None]
    torch.testing.assert_close(out.float(), ref, atol=0.06, rtol=3e-2)


def test_grouped_gemm_rejects_bad_shapes():
    from gpu_data_transfer_profile_b200.ops import gemm as G
    a = torch.zeros(8, 36, device="cuda", dtype=torch.bfloat16)
    w = torch.zeros(1, 64, 36, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(RuntimeError):
        G.grouped_gemm(a, w, G.offsets_from_counts([8], "cuda"))


def test_swiglu_fwd_bwd_kernels_match_autograd():
    from gpu_data_transfer_profile_b200.ops import gemm as G
    torch.manual_seed(2)
    rows, F = 37, 264
    h = torch.randn(rows, 2 * F, device="cuda").to(torch.bfloat16)
    p = torch.rand(rows, device="cuda")
    dact = torch.randn(rows, F, device="cuda").to(torch.bfloat16)
    hf = h.float().requires_grad_(True)
    pf = p.clone().requires_grad_(True)
    ref = torch.nn.functional.silu(hf[:, :F]) * hf[:, F:] * pf[:, None]
    rdh, rdp = torch.autograd.grad(ref, [hf, pf], dact.float())
    act = G.swiglu_fwd(h, p)
    dh, dp = G.swiglu_bwd(h, p, dact)
    torch.testing.assert_close(act.float(), ref.detach(), atol=2e-2, rtol=2e-2)
    torch.testing.assert_close(dh.float(), rdh, atol=3e-2, rtol=3e-2)
    torch.testing.assert_close(dp, rdp, atol=0.3, rtol=2e-2)


@pytest.mark.parametrize("kind", ["gelu", "silu", "relu"])
def test_ungated_activation_kernels_match_autograd(kind):
    from gpu_data_transfer_profile_b200.models.experts import activate
    from gpu_data_transfer_profile_b200.ops import gemm as G
    torch.manual_seed(2)
    rows, F = 77, 264
    h = (torch.randn(rows, F, device="cuda") * 2).to(torch.bfloat16)
    p = torch.rand(rows, device="cuda")
    d = torch.randn(rows, F, device="cuda").to(torch.bfloat16)
    act = G.act_fwd(h, p, kind)
    hf = h.float().requires_grad_(True)
    pf = p.clone().requires_grad_(True)
    ref = activate(hf, kind) * pf[:, None]
    torch.testing.assert_close(act.float(), ref.detach(), atol=2e-2, rtol=2e-2)
    ref.backward(d.float())
    dh, dp = G.act_bwd(h, p, d, kind)
    torch.testing.assert_close(dh.float(), hf.grad, atol=3e-2, rtol=3e-2)
    torch.testing.assert_close(dp, pf.grad, atol=5e-2, rtol=2e-2)


# one warp per row (many rows) up to eight (few rows), a row of one vector, rows that leave lanes and warps without work.
# Tolerance: dh is one bf16 rounding (2^-8 covers a value at the boundary) of f32 arithmetic, dp an f32 sum of F terms.
@pytest.mark.parametrize("rows,F", [(2500, 264), (2368, 8), (1300, 776), (600, 1416), (37, 2824), (1, 4096), (3, 8)])
@pytest.mark.parametrize("kind", ["swiglu", "gelu", "silu", "relu"])
def test_activation_backward_rows_shared_by_warps(rows, F, kind):
    from gpu_data_transfer_profile_b200.models.experts import activate
    from gpu_data_transfer_profile_b200.ops import gemm as G
    torch.manual_seed(12)
    h = torch.randn(rows, F * (2 if kind == "swiglu" else 1), device="cuda").to(torch.bfloat16)
    p = torch.rand(rows, device="cuda")
    d = torch.randn(rows, F, device="cuda").to(torch.bfloat16)
    hf, pf = h.double().requires_grad_(True), p.double().requires_grad_(True)
    (activate(hf, kind) * pf[:, None]).backward(d.double())
    dh, dp = G.swiglu_bwd(h, p, d) if kind == "swiglu" else G.act_bwd(h, p, d, kind)
    torch.testing.assert_close(dh.double(), hf.grad, rtol=2.0 ** -8, atol=2e-6 * 64)
    torch.testing.assert_close(dp.double(), pf.grad, rtol=1e-5, atol=4e-6 * F ** 0.5)


def test_tcgen05_experts_backward_matches_torch_experts():
    from gpu_data_transfer_profile_b200.models.experts import TorchGroupedExperts
    from gpu_data_transfer_profile_b200.models.experts_tcgen05 import Tcgen05GroupedExperts
    torch.manual_seed(3)
    E, H, F = 3, 256, 384
    counts = [70, 0, 131]
    rows = sum(counts)
    a = Tcgen05GroupedExperts(E, H, F, torch.bfloat16, "swiglu", init_std=0.05)
    b = TorchGroupedExperts(E, H, F, torch.float32, "swiglu")
    with torch.no_grad():
        b.weight1.copy_(a.weight1.float())
        b.weight2.copy_(a.weight2.float())
    x = torch.randn(rows, H, device="cuda")
    p = torch.rand(rows, device="cuda")
    xa, pa = x.to(torch.bfloat16).requires_grad_(True), p.clone().requires_grad_(True)
    xb, pb = x.to(torch.bfloat16).float().requires_grad_(True), p.clone().requires_grad_(True)
    g = torch.randn(rows, H, device="cuda")
    ya = a(xa, counts, pa)
    yb = b(xb, counts, pb)
    ya.backward(g.to(torch.bfloat16))
    yb.backward(g.to(torch.bfloat16).float())
    torch.testing.assert_close(ya.float(), yb, atol=5e-2, rtol=5e-2)
    torch.testing.assert_close(xa.grad.float(), xb.grad, atol=5e-2, rtol=5e-2)
    torch.testing.assert_close(pa.grad, pb.grad, atol=0.5, rtol=5e-2)
    torch.testing.assert_close(a.weight1.grad.float(), b.weight1.grad, atol=0.15, rtol=5e-2)
    torch.testing.assert_close(a.weight2.grad.float(), b.weight2.grad, atol=0.15, rtol=5e-2)


@pytest.mark.parametrize("activation", ["swiglu", "gelu", "silu", "relu"])
def test_tcgen05_expert_mlp_gradients_match_fp32_autograd(activation):
    """Training path of the expert MLP (tcgen05 forward, dgrads reading the weights in place,
    ragged-reduction wgrads, fused activation backward) against fp32 autograd of the same math,
    for every activation the reference's expert MLP offers."""
    from gpu_data_transfer_profile_b200.models.experts import activate
    from gpu_data_transfer_profile_b200.models.experts_tcgen05 import Tcgen05GroupedExperts
    torch.manual_seed(5)
    H, F, counts = 256, 384, [70, 0, 301, 129]
    rows = sum(counts)
    mod = Tcgen05GroupedExperts(len(counts), H, F, init_std=0.05, activation=activation)
    x = torch.randn(rows, H, device="cuda").to(torch.bfloat16).requires_grad_(True)
    p = torch.rand(rows, device="cuda").requires_grad_(True)
    gy = torch.randn(rows, H, device="cuda").to(torch.bfloat16)
    y = mod(x, counts, p)
    y.backward(gy)
    xf = x.detach().float().requires_grad_(True)
    pf = p.detach().clone().requires_grad_(True)
    w1 = mod.weight1.detach().float().requires_grad_(True)
    w2 = mod.weight2.detach().float().requires_grad_(True)
    outs, r = [], 0
    for e, c in enumerate(counts):
        h = xf[r:r + c] @ w1[e].t()
        a = activate(h, activation) * pf[r:r + c, None]
        outs.append(a @ w2[e].t())
        r += c
    yr = torch.cat(outs)
    yr.backward(gy.float())
    torch.testing.assert_close(y.float(), yr.detach(), atol=3e-2, rtol=5e-2)
    torch.testing.assert_close(x.grad.float(), xf.grad, atol=3e-2, rtol=5e-2)
    torch.testing.assert_close(p.grad, pf.grad, atol=5e-2, rtol=5e-2)
    torch.testing.assert_close(mod.weight1.grad.float(), w1.grad, atol=6e-2, rtol=5e-2)
    torch.testing.assert_close(mod.weight2.grad.float(), w2.grad, atol=6e-2, rtol=5e-2)


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("N", [8, 128, 136, 256, 264, 384, 392])
def test_grouped_wgrad_last_tile_columns(N, pair):
    """Widths at which the last tile of columns is fetched 128 or 256 wide, ragged rows, empty experts, more offsets than a
    warp has lanes, against f64: products of bf16 are exact in f32, so a result is off by its own rounding (2^-9) and by
    f32 sums of up to 150 terms (2^-16 of their magnitudes)."""
    from gpu_data_transfer_profile_b200.ops import gemm as G
    torch.manual_seed(N)
    M, counts = 256, [65, 0, 150, 1, 16] + [3] * 30
    g = torch.randn(sum(counts), M, device="cuda").to(torch.bfloat16)
    x = torch.randn(sum(counts), N, device="cuda").to(torch.bfloat16)
    off = G.offsets_from_counts(counts, "cuda")
    out = G.grouped_wgrad(g, x, off, pair=pair).double()
    r = 0
    for e, c in enumerate(counts):
        ge, xe = g[r:r + c].double(), x[r:r + c].double()
        ref = ge.t() @ xe
        assert bool(((out[e] - ref).abs() <= ref.abs() * 2 ** -8 + (ge.abs().t() @ xe.abs()) * 2 ** -16).all()), e
        r += c


def _act_ref(h, activation):
    f = torch.nn.functional
    if activation == "swiglu":
        g, l = h.chunk(2, -1)
        return f.silu(g) * l
    return {"gelu": f.gelu, "silu": f.silu, "relu": f.relu}[activation](h)


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("activation", ["swiglu", "gelu", "silu", "relu"])
@pytest.mark.parametrize("counts,F,H", [([1], 128, 64), ([255, 0, 257], 384, 264), ([16, 33, 0, 300, 7], 256, 512), ([700] + [3] * 39, 640, 128),
                                        ([70, 9], 136, 72), ([40], 8, 64)])
def test_grouped_gemm_activation_epilogues(counts, F, H, activation, pair):
    """fc1 with an ungated activation, and the data gradient of fc2 with the SwiGLU backward, in the epilogue, against
    f64: one row, tiles of 256 and one more, empty experts, an odd number of 128-column blocks (a pair's second CTA has
    none), widths that end inside a block (ungated), more experts than a warp."""
    from gpu_data_transfer_profile_b200.ops import gemm as G
    if activation == "swiglu" and F % 128:
        pytest.skip("swiglu takes multiples of 128")
    torch.manual_seed(5)
    rows, E = sum(counts), len(counts)
    off = G.offsets_from_counts(counts, "cuda")
    spans = [(int(o), int(o) + c) for o, c in zip(off.tolist(), counts)]
    dy = torch.randn(rows, H, device="cuda").to(torch.bfloat16)
    w2 = (torch.randn(E, H, F, device="cuda") * H ** -0.5).to(torch.bfloat16)
    h = torch.randn(rows, 2 * F if activation == "swiglu" else F, device="cuda").to(torch.bfloat16)
    p = torch.rand(rows, device="cuda")
    if activation == "swiglu":
        dh, dp = G.grouped_gemm_dswiglu(dy, w2, off, h, p, pair=pair)
        hf, pf = h.double().requires_grad_(True), p.double().requires_grad_(True)
        dact = torch.cat([dy[a:b].double() @ w2[e].double() for e, (a, b) in enumerate(spans)])
        gh, gp = torch.autograd.grad(_act_ref(hf, activation) * pf[:, None], [hf, pf], dact)
        # one bf16 rounding (2^-9) of f32 results; f32 sums of F terms of order one for the probabilities
        torch.testing.assert_close(dh.double(), gh, atol=1e-4, rtol=2 ** -8)
        torch.testing.assert_close(dp.double(), gp, atol=1e-4 * F ** 0.5, rtol=1e-4)
        dh1, dp1 = G.grouped_gemm_dswiglu(dy, w2, off, h, None, pair=pair)               # no probabilities: all ones
        gh1, = torch.autograd.grad(_act_ref(hf, activation), hf, dact)
        torch.testing.assert_close(dh1.double(), gh1, atol=1e-4, rtol=2 ** -8)
        assert torch.equal(dp1, dp)
    else:
        w1 = (torch.randn(E, F, H, device="cuda") * H ** -0.5).to(torch.bfloat16)
        pre = torch.full((rows, F), 7.0, dtype=torch.bfloat16, device="cuda")
        act = G.grouped_gemm_act(dy, w1, off, p, activation, pair=pair, pre_out=pre)
        ref = torch.cat([dy[a:b].double() @ w1[e].double().t() for e, (a, b) in enumerate(spans)])
        torch.testing.assert_close(pre.double(), ref, atol=1e-4, rtol=2 ** -8)
        torch.testing.assert_close(act.double(), _act_ref(ref, activation) * p.double()[:, None], atol=1e-4, rtol=2 ** -8)
        assert torch.equal(G.grouped_gemm_act(dy, w1, off, p, activation, pair=pair), act)


@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("counts,N,K", [([128], 256, 128), ([200, 0, 57], 384, 512), ([1, 300, 129, 0], 256, 1024),
                                        ([513], 128, 7168),
                                        # more experts than a warp, several tiles per CTA, weight scales of two shuffle rounds
                                        ([5, 0, 140] * 13 + [1], 640, 33 * 128)])
def test_grouped_gemm_fp8_block_scaled(counts, N, K, swiglu):
    """e4m3 rows with 1x128 scales times e4m3 weights with 128x128 scales, against the fp32 matmul
    of the DEQUANTISED operands (the kernel multiplies exactly those numbers, so only the
    accumulation order and the bf16 store differ). Ragged counts with an empty expert."""
    from gpu_data_transfer_profile_b200.ops import gemm as G
    torch.manual_seed(11)
    rows, E = sum(counts), len(counts)
    Nw = 2 * N if swiglu else N
    x = torch.randn(rows + 5, K, device="cuda") * (1 + torch.arange(K, device="cuda") % 7)     # uneven block scales
    w = torch.randn(E, Nw, K, device="cuda") * 0.05
    xq, xs = G.quantize_rows_1x128(x)
    wq, ws = G.quantize_weights_128x128(w)
    p = torch.rand(rows + 5, device="cuda")
    off = G.offsets_from_counts(counts, "cuda")
    out = torch.full((rows + 5, N), 7.0, dtype=torch.bfloat16, device="cuda")
    G.grouped_gemm_fp8(xq, xs, wq, ws, off, swiglu=swiglu, row_prob=p if swiglu else None, out=out)
    xd = (xq.float().view(rows + 5, K // 128, 128) * xs[..., None]).view(rows + 5, K)
    wd = G.dequantize_weights_128x128(wq, ws)
    r = 0
    for e, c in enumerate(counts):
        if c == 0:
            continue
        h = xd[r:r + c] @ wd[e].t()
        ref = torch.nn.functional.silu(h[:, :N]) * h[:, N:] * p[r:r + c, None] if swiglu else h
        torch.testing.assert_close(out[r:r + c].float(), ref, atol=2e-2 * float(ref.abs().max() + 1), rtol=2e-2)
        r += c
    assert bool((out[rows:] == 7.0).all())           # rows beyond the last expert are never written


def test_tcgen05_experts_consume_fp8_dispatch_rows():
    from gpu_data_transfer_profile_b200.models.experts_tcgen05 import Tcgen05GroupedExperts
    from gpu_data_transfer_profile_b200.ops import gemm as G
    torch.manual_seed(3)
    H, F, counts = 512, 256, [90, 0, 200, 33]
    rows = sum(counts)
    mod = Tcgen05GroupedExperts(len(counts), H, F, init_std=0.05, use_fp8=True)
    x = torch.randn(rows, H, device="cuda").to(torch.bfloat16)
    p = torch.rand(rows, device="cuda")
    xq, xs = G.quantize_rows_1x128(x)
    y = mod((xq, xs), counts, p)
    y_ref = mod(x, counts, p)                              # bf16 path on the unquantised rows
    torch.testing.assert_close(y.float(), y_ref.detach().float(), atol=0.08 * float(y_ref.detach().float().abs().max()), rtol=0.1)


def test_grouped_gemms_work_from_a_fresh_thread():
    """The launchers encode TMA descriptors through a driver entry point, which needs a context
    bound to the calling thread; a thread that has made no CUDA runtime call yet (autograd's
    backward workers, user threads) must get one bound by the launcher itself."""
    import threading
    from gpu_data_transfer_profile_b200.ops import gemm as G
    torch.manual_seed(0)
    counts = [70, 0, 130]
    rows, K, N = sum(counts), 256, 384
    off = G.offsets_from_counts(counts, "cuda")
    a = torch.randn(rows, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(len(counts), N, K, device="cuda") * 0.05).to(torch.bfloat16)
    g = torch.randn(rows, N, device="cuda").to(torch.bfloat16)
    out, dx, dw = (torch.empty(rows, N, dtype=torch.bfloat16, device="cuda"),
                   torch.empty(rows, K, dtype=torch.bfloat16, device="cuda"),
                   torch.empty(len(counts), N, K, dtype=torch.bfloat16, device="cuda"))
    torch.cuda.synchronize()
    err = []

    def work():                                    # first CUDA work of this thread
        try:
            G.grouped_gemm(a, w, off, out=out)
            G.grouped_gemm(g, w, off, out=dx, w_kn=True)
            G.grouped_wgrad(g, a, off, out=dw)
            torch.cuda.synchronize()
        except Exception as e:                     # noqa: BLE001
            err.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert not err, err
    r = 0
    for e, c in enumerate(counts):
        if c:
            torch.testing.assert_close(out[r:r + c].float(), a[r:r + c].float() @ w[e].float().t(), atol=3e-2, rtol=3e-2)
            torch.testing.assert_close(dx[r:r + c].float(), g[r:r + c].float() @ w[e].float(), atol=3e-2, rtol=3e-2)
        r += c


@pytest.mark.parametrize("activation", ["swiglu", "gelu"])
def test_experts_without_rows(activation):
    """No rows at all (no tokens, or a rank that none was sent to): empty outputs and zero weight gradients."""
    from gpu_data_transfer_profile_b200.models.experts_tcgen05 import Tcgen05GroupedExperts
    from gpu_data_transfer_profile_b200.ops import gemm as G
    E, H, F = 3, 256, 128
    m = Tcgen05GroupedExperts(E, H, F, activation=activation, use_fp8=True)
    x = torch.empty(0, H, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    p = torch.empty(0, device="cuda", requires_grad=True)
    for pair in (False, True):
        off = G.offsets_from_counts([0] * E, "cuda")
        assert G.grouped_gemm(x.detach(), m.weight1, off, pair=pair).shape == (0, m.weight1.shape[1])
        assert G.grouped_gemm(x.detach(), m.weight2, off, pair=pair, w_kn=True).shape == (0, F)
        dh, dp = G.grouped_gemm_dswiglu(x.detach(), m.weight2, off, torch.empty(0, 2 * F, device="cuda", dtype=torch.bfloat16), None, pair=pair)
        assert dh.shape == (0, 2 * F) and dp.shape == (0,)
    y = m(x, [0] * E, p)
    assert y.shape == (0, H)
    y.float().sum().backward()
    assert x.grad.shape == x.shape and p.grad.shape == p.shape
    for w in (m.weight1, m.weight2):
        assert w.grad.shape == w.shape and not w.grad.any()
    q = torch.empty(0, H, device="cuda").to(torch.float8_e4m3fn)
    assert m((q, torch.empty(0, H // 128, device="cuda")), [0] * E, p.detach()).shape == (0, H)
    torch.cuda.synchronize()


@pytest.mark.parametrize("H,E", [(12, 2), (64, 257)])
def test_grouped_gemm_dswiglu_refuses_bad_shapes(H, E):
    """A width that tensor maps do not take, more experts than the kernel's tables hold: an error that a program can catch."""
    from gpu_data_transfer_profile_b200.ops import gemm as G
    F, rows = 128, 4
    dy = torch.randn(rows, H, device="cuda").to(torch.bfloat16)
    w2 = torch.randn(E, H, F, device="cuda").to(torch.bfloat16)
    h = torch.randn(rows, 2 * F, device="cuda").to(torch.bfloat16)
    off = G.offsets_from_counts([rows] + [0] * (E - 1), "cuda")
    with pytest.raises(RuntimeError, match="invalid arguments"):
        G.grouped_gemm_dswiglu(dy, w2, off, h, None)


@pytest.mark.parametrize("pair", [False, True])
def test_activation_epilogues_divide_where_the_sigmoid_is_subnormal(pair):
    """Gates between -88.7 and -87.4: 1 + exp(-x) lies above 2^126, the sigmoid is a subnormal f32, silu and its
    gradients are ordinary bf16 numbers of about 1e-37. Identity weights bring the values to the epilogues as they are."""
    from gpu_data_transfer_profile_b200.ops import gemm as G
    F, rows = 128, 5
    off = G.offsets_from_counts([rows], "cuda")
    eye = torch.eye(F, device="cuda").to(torch.bfloat16)[None]
    g = torch.tensor([-87.5, -88.0, -88.5, -3.0, 2.0], device="cuda").to(torch.bfloat16)[:, None].expand(rows, F).contiguous()
    one = torch.ones(rows, F, device="cuda", dtype=torch.bfloat16)
    x = g.double()
    silu, sig = x / (1 + (-x).exp()), 1 / (1 + (-x).exp())
    assert bool((silu[:3].abs() > 2.0 ** -126).all()) and bool((sig[:3] < 2.0 ** -126).all())
    # one bf16 rounding, and exp of an argument of 88 from the fast exponential (88 x 2^-22 relative)
    bound = dict(rtol=2.0 ** -8, atol=0)
    torch.testing.assert_close(G.grouped_gemm_act(g, eye, off, None, "silu", pair=pair).double(), silu, **bound)
    dh, dp = G.grouped_gemm_dswiglu(one, eye, off, torch.cat([g, one], 1), None, pair=pair)
    torch.testing.assert_close(dh[:, F:].double(), silu, **bound)
    torch.testing.assert_close(dh[:, :F].double(), sig * (1 + x * (1 - sig)), **bound)
    torch.testing.assert_close(dp.double(), silu.sum(1), rtol=2.0 ** -12, atol=0)


def test_epilogue_sigmoid_is_as_near_as_a_rounded_division():
    """silu of every finite bf16 gate as an f32 number (a row's sum for the gradient of its probability, one term not
    zero), from the epilogue and from the element-wise kernel, which divides."""
    from gpu_data_transfer_profile_b200.ops import gemm as G
    F = 128
    g = torch.arange(1 << 16, device="cuda").to(torch.int32).to(torch.int16).view(torch.bfloat16)
    g = g[g.isfinite()]
    rows = g.numel()
    at = (torch.arange(rows, device="cuda"), torch.arange(rows, device="cuda") % F)
    dy = torch.zeros(rows, F, device="cuda", dtype=torch.bfloat16)
    gate = torch.zeros_like(dy)
    dy[at], gate[at] = 1, g
    h = torch.cat([gate, dy], 1)
    eye = torch.eye(F, device="cuda").to(torch.bfloat16)[None]
    dh, dp = G.grouped_gemm_dswiglu(dy, eye, G.offsets_from_counts([rows], "cuda"), h, None)
    dh1, dp1 = G.swiglu_bwd(h, None, dy)
    # sigmoids within an ulp of each other and a product rounded in both: two ulps, or two of the smallest subnormal times
    # the gate; the gradient of the gate is a bf16 number, 1 + g (1 - sigmoid) cancels near -1.28
    bound = 2.0 ** -22 * dp1.double().abs() + 2.0 ** -148 * g.double().abs()
    assert bool(((dp.double() - dp1.double()).abs() <= bound).all())
    torch.testing.assert_close(dh.float(), dh1.float(), rtol=2.0 ** -7, atol=2.0 ** -20)
    # no further from 64 bits than the division's, down to where exp overflows
    x = g.double()
    silu = x / (1 + (-x).exp())
    normal = (silu.abs() > 2.0 ** -126) & (x > -88.7)
    err = [((d.double() - silu).abs() / silu.abs())[normal] for d in (dp, dp1)]
    assert float(err[0].mean()) <= float(err[1].mean()) * (1 + 2.0 ** -6) and float(err[0].max()) <= float(err[1].max()) + 2.0 ** -23


@pytest.mark.parametrize("activation", ["swiglu", "gelu", "silu", "relu"])
@pytest.mark.parametrize("counts", [[1], [40, 0, 257]])
def test_experts_without_gradients_give_what_those_with_them_give(activation, counts):
    """The pre-activation that a backward needs is written or not: the outputs are the same bits."""
    from gpu_data_transfer_profile_b200.models.experts_tcgen05 import Tcgen05GroupedExperts
    torch.manual_seed(2)
    H, F, rows = 256, 384, sum(counts)
    m = Tcgen05GroupedExperts(len(counts), H, F, activation=activation)
    x, p = torch.randn(rows, H, device="cuda").to(torch.bfloat16), torch.rand(rows, device="cuda")
    want = m(x, counts, p)
    assert want.requires_grad
    for forward in (torch.no_grad, torch.inference_mode):
        with forward():
            assert torch.equal(m(x, counts, p), want)
    for t in m.parameters():
        t.requires_grad_(False)
    got = m(x, counts, p)                                          # nothing that asks for a gradient
    assert torch.equal(got, want) and not got.requires_grad
    probs = p.clone().requires_grad_(True)                         # the probabilities alone ask for one
    y = m(x, counts, probs)
    assert torch.equal(y, want)
    (g,) = torch.autograd.grad(y.float().sum(), probs)
    assert bool(g.isfinite().all()) and bool(g.any())


def test_grouped_gemms_refuse_outputs_and_values_that_their_kernels_cannot_address():
    """Rows that 8-byte stores (16 in fp8 and the weight gradients) would meet unaligned, probabilities on the host or
    with strides, offsets with strides: an error before a launch. What is aligned is taken, with gaps between the rows."""
    from gpu_data_transfer_profile_b200.ops import gemm as G
    E, rows, H, F = 2, 37, 128, 256
    off = G.offsets_from_counts([17, 20], "cuda")
    a = torch.randn(rows, H, device="cuda").to(torch.bfloat16)
    w = (torch.randn(E, F, H, device="cuda") * 0.1).to(torch.bfloat16)
    p = torch.rand(rows, device="cuda")
    new = lambda cols, gap, first: torch.zeros(rows, cols + gap, device="cuda", dtype=torch.bfloat16)[:, first:first + cols]
    q, qs = torch.randn(rows, H, device="cuda").to(torch.float8_e4m3fn), torch.ones(rows, 1, device="cuda")
    wq, ws = torch.randn(E, F, H, device="cuda").to(torch.float8_e4m3fn), torch.ones(E, F // 128, 1, device="cuda")
    calls = {
        "plain": lambda o, p=None, off=off: G.grouped_gemm(a, w, off, out=o),
        "swiglu pre": lambda o, p=p, off=off: G.grouped_gemm_swiglu(a, w, off, p, pre_out=o),
        "act pre": lambda o, p=p, off=off: G.grouped_gemm_act(a, w, off, p, "gelu", pre_out=o),
        "fp8": lambda o, p=None, off=off: G.grouped_gemm_fp8(q, qs, wq, ws, off, out=o),
    }
    for name, call in calls.items():
        vec = 8 if name == "fp8" else 4                              # elements of a store
        want = new(F, 0, 0)
        call(want)
        for gap, first in ((vec, 0), (vec, vec), (2 * vec, vec)):
            got = new(F, gap, first)
            call(got)
            assert torch.equal(got, want) and bool(got.any())
        for gap, first in ((1, 0), (vec, 1), (vec, vec // 2), (2, 0)):
            with pytest.raises(RuntimeError, match="aligned rows"):
                call(new(F, gap, first))
        with pytest.raises(RuntimeError, match="aligned rows"):
            call(torch.zeros(rows, F, dtype=torch.bfloat16))
        with pytest.raises(RuntimeError, match="expert_off"):
            call(want, off=torch.stack([off, off], 1)[:, 0])
        if "pre" in name:
            for bad in (p.cpu(), p[:1].expand(rows), torch.stack([p, p], 1)[:, 0], p[:-1]):
                with pytest.raises(RuntimeError, match="row_prob"):
                    call(want, p=bad)
    flat = torch.zeros(E * H * F + 8, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(rows, F, device="cuda").to(torch.bfloat16)
    assert torch.equal(G.grouped_wgrad(a, x, off, out=flat[8:].view(E, H, F)), G.grouped_wgrad(a, x, off))
    with pytest.raises(RuntimeError, match="aligned"):
        G.grouped_wgrad(a, x, off, out=flat[4:-4].view(E, H, F))
