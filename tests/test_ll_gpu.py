"""Low-latency dispatch/combine on one GPU with virtual ranks, against the PyTorch oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from gpu_data_transfer_profile_b200.ref import cpu_oracle as O


def _inputs(R, T, H, E, K, seed=0):
    xs, idxs, ws = [], [], []
    for r in range(R):
        g = torch.Generator().manual_seed(seed * 100 + r)
        xs.append(torch.randn(T - r, H, generator=g).to(torch.bfloat16))
        i, w = O.make_routing(T - r, E, K, seed * 100 + r)
        i[0, 0] = -1          # a masked choice must be skipped
        idxs.append(i)
        ws.append(w)
    return xs, idxs, ws


def _unpack(src):
    return (src >> 24) & 0xff, (src & 0xffffff) >> 5, src & 31


# signal_mode: 0 = every send CTA adds 1 on every peer's arrival counter, 1 = the last CTA adds the grid size
@pytest.mark.parametrize("signal_mode", [0, 1])
@pytest.mark.parametrize("R,T,H,E,K,fp8", [(1, 16, 256, 4, 2, False), (2, 32, 512, 8, 2, True),
                                           (4, 48, 1024, 16, 4, True), (8, 24, 512, 32, 8, False)])
def test_low_latency_round_trip(R, T, H, E, K, fp8, signal_mode, monkeypatch):
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    from gpu_data_transfer_profile_b200.parallel.local import LocalGroup
    monkeypatch.setattr(Buffer, "ll_signal_mode", signal_mode)
    M = 64
    g = LocalGroup(R, Buffer.get_low_latency_nvl_size_hint(M, H, R, E, K), timeout_s=2.0)
    try:
        xs, idxs, ws = _inputs(R, T, H, E, K)
        cx, ci, cw = [x.cuda() for x in xs], [i.cuda() for i in idxs], [w.cuda() for w in ws]
        El = E // R
        for rep in range(3):     # repeated calls exercise both epoch parities
            outs = g.low_latency_dispatch(cx, ci, M, E, use_fp8=fp8)
            ys = []
            for d in range(R):
                recv, count, handle = outs[d]
                cnt = count.cpu().tolist()
                want = [sum(int((idxs[s] == d * El + e).sum()) for s in range(R)) for e in range(El)]
                assert cnt == want
                src = handle[0].cpu()
                if fp8:
                    q, sc = recv
                    val = (q.float().view(El, R * M, H // 128, 128) * sc[..., None]).view(El, R * M, H).cpu()
                else:
                    val = recv.float().cpu()
                # every (source, token, k) that chose a local expert appears exactly once among its rows
                for e in range(El):
                    keys = src[e, :cnt[e]].tolist()
                    assert len(set(keys)) == len(keys)
                for e in range(El):
                    s_r, s_t, s_k = _unpack(src[e, :cnt[e]])
                    for j in range(cnt[e]):
                        r_, t_, k_ = int(s_r[j]), int(s_t[j]), int(s_k[j])
                        assert int(idxs[r_][t_, k_]) == d * El + e
                        torch.testing.assert_close(val[e, j], xs[r_][t_].float(),
                                                   atol=0.3 if fp8 else 0, rtol=0.07 if fp8 else 0)
                y = torch.zeros((El, R * M, H), dtype=torch.bfloat16, device="cuda")
                for e in range(El):    # "expert" = scale by (1 + global expert id)
                    y[e, :cnt[e]] = (val[e, :cnt[e]] * (1 + d * El + e)).to(torch.bfloat16).cuda()
                ys.append(y)
            comb = g.low_latency_combine(ys, ci, cw, [o[2] for o in outs])
            for s in range(R):
                scale = (torch.where(idxs[s] >= 0, (1 + idxs[s]).float() * ws[s], torch.zeros_like(ws[s]))).sum(1)
                want = xs[s].float() * scale[:, None]
                torch.testing.assert_close(comb[s].float().cpu(), want, atol=0.6 if fp8 else 0.15,
                                           rtol=0.08 if fp8 else 0.03)
        g.check_status()
    finally:
        g.destroy()


# overlap: the kernels are launched with programmatic stream serialisation (captured as such in the graph)
@pytest.mark.parametrize("overlap", [False, True])
def test_low_latency_cuda_graph_replay(overlap, monkeypatch):
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    from gpu_data_transfer_profile_b200.parallel.local import LocalGroup
    monkeypatch.setattr(Buffer, "ll_overlap_launches", overlap)
    R, T, H, E, K, M = 1, 32, 512, 8, 4, 32
    g = LocalGroup(R, Buffer.get_low_latency_nvl_size_hint(M, H, R, E, K), timeout_s=2.0)
    try:
        b = g.buffers[0]
        x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
        idx, w = O.make_routing(T, E, K, 5)
        idx, w = idx.cuda(), w.cuda()
        out = torch.empty((T, H), dtype=torch.bfloat16, device="cuda")

        def step():
            recv, count, handle, _, _ = b.low_latency_dispatch(x, idx, M, E, use_fp8=False)
            b.low_latency_combine(recv, idx, w, handle, out=out)

        step()                      # warm-up outside capture (allocations, module load)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            step()
        for rep in range(4):
            x.copy_(torch.randn(T, H, device="cuda").to(torch.bfloat16))
            out.zero_()
            graph.replay()
            torch.cuda.synchronize()
            torch.testing.assert_close(out.float(), x.float() * w.sum(1, keepdim=True), atol=0.06, rtol=0.03)
        g.check_status()
    finally:
        g.destroy()


@pytest.mark.parametrize("R,T,H,E,K,fp8", [(1, 16, 256, 4, 2, False), (2, 32, 512, 8, 2, True),
                                           (4, 48, 7168, 16, 4, True), (8, 24, 1024, 32, 8, False)])
def test_low_latency_combine_pulls_expert_output_in_place(R, T, H, E, K, fp8):
    """The experts write into the buffer's in-place combine input; combine then loads and reduces
    the K rows of every token straight from the peers' regions. Three rounds with different
    expert scales (both announcement parities, no stale rows)."""
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    from gpu_data_transfer_profile_b200.parallel.local import LocalGroup
    M = 64
    g = LocalGroup(R, Buffer.get_low_latency_nvl_size_hint(M, H, R, E, K), timeout_s=2.0)
    try:
        xs, idxs, ws = _inputs(R, T, H, E, K, seed=3)
        cx, ci, cw = [x.cuda() for x in xs], [i.cuda() for i in idxs], [w.cuda() for w in ws]
        El = E // R
        for rep in range(3):
            outs = g.low_latency_dispatch(cx, ci, M, E, use_fp8=fp8)
            ys = []
            for d in range(R):
                recv, count, handle = outs[d]
                cnt = count.cpu().tolist()
                if fp8:
                    q, sc = recv
                    val = (q.float().view(El, R * M, H // 128, 128) * sc[..., None]).view(El, R * M, H)
                else:
                    val = recv.float()
                y = g.buffers[d].get_next_low_latency_combine_buffer(handle)
                assert g.buffers[d]._ll_is_combine_buffer(y, handle)
                y.fill_(float("nan"))                 # rows that nobody owns must never be read
                for e in range(El):
                    y[e, :cnt[e]] = (val[e, :cnt[e]] * (1 + rep + d * El + e)).to(torch.bfloat16)
                ys.append(y)
            comb = g.low_latency_combine(ys, ci, cw, [o[2] for o in outs])
            for s in range(R):
                scale = (torch.where(idxs[s] >= 0, (1 + rep + idxs[s]).float() * ws[s], torch.zeros_like(ws[s]))).sum(1)
                want = xs[s].float() * scale[:, None]
                torch.testing.assert_close(comb[s].float().cpu(), want, atol=0.8 if fp8 else 0.2,
                                           rtol=0.08 if fp8 else 0.03)
        g.check_status()
    finally:
        g.destroy()


def test_low_latency_pull_combine_under_cuda_graph_replay():
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    from gpu_data_transfer_profile_b200.parallel.local import LocalGroup
    R, T, H, E, K, M = 1, 32, 512, 8, 4, 32
    g = LocalGroup(R, Buffer.get_low_latency_nvl_size_hint(M, H, R, E, K), timeout_s=2.0)
    try:
        b = g.buffers[0]
        x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
        idx, w = O.make_routing(T, E, K, 5)
        idx, w = idx.cuda(), w.cuda()
        out = torch.empty((T, H), dtype=torch.bfloat16, device="cuda")

        def step():
            recv, count, handle, _, _ = b.low_latency_dispatch(x, idx, M, E, use_fp8=False)
            y = b.get_next_low_latency_combine_buffer(handle)
            y.copy_(recv)                                  # identity "expert" writing in place
            b.low_latency_combine(y, idx, w, handle, out=out)

        step()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            step()
        for rep in range(4):
            x.copy_(torch.randn(T, H, device="cuda").to(torch.bfloat16))
            out.zero_()
            graph.replay()
            torch.cuda.synchronize()
            torch.testing.assert_close(out.float(), x.float() * w.sum(1, keepdim=True), atol=0.06, rtol=0.03)
        g.check_status()
    finally:
        g.destroy()


# one rank, through the public calls: several tokens per CTA, rows of more than one batch of loads, more choices than
# are loaded together, masked choices; eager and hook-style completion in turn on the same buffer
@pytest.mark.parametrize("T,H,E,K,fp8", [(1, 1024, 8, 1, True), (7, 4096, 16, 4, False), (300, 512, 8, 8, True),
                                         (131, 264, 32, 9, False), (5, 17408, 16, 3, True), (3, 16640, 8, 2, False)])
@pytest.mark.parametrize("in_place", [False, True])
def test_low_latency_one_rank_public_calls(T, H, E, K, fp8, in_place):
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    buf = Buffer(None, Buffer.get_low_latency_nvl_size_hint(T, H, 1, E, K), 0, low_latency_mode=True,
                 world=LocalWorld.make(1)[0], timeout_s=2.0)
    try:
        for rep in range(5):
            g = torch.Generator().manual_seed(rep)
            x = torch.randn(T, H, generator=g).to(torch.bfloat16).cuda()
            idx, w = O.make_routing(T, E, K, 50 + rep)
            idx[T // 2, K - 1] = -1
            idx_c, w_c = idx.cuda(), w.cuda()
            hook_d, hook_c = rep in (1, 3), rep in (2, 3)
            recv, count, handle, _, hook = buf.low_latency_dispatch(x, idx_c, T, E, use_fp8=fp8, return_recv_hook=hook_d)
            if hook_d:
                recv, count, handle = hook()
            assert count.tolist() == [int((idx == e).sum()) for e in range(E)]
            if fp8:
                y = (recv[0].float().view(E, T, -1, 128) * recv[1][..., None]).view(E, T, H).to(torch.bfloat16)
            else:
                y = recv.clone()
            y = y * (1 + torch.arange(E, device="cuda", dtype=torch.bfloat16))[:, None, None]     # the experts
            for e in range(E):
                y[e, int(count[e]):] = float("nan")                       # rows that nobody owns are never read
            if in_place:
                z = buf.get_next_low_latency_combine_buffer(handle)
                z.copy_(y)
                y = z
            out, _, hook = buf.low_latency_combine(y, idx_c, w_c, handle, return_recv_hook=hook_c)
            if hook_c and out is None:
                out = hook()
            factor = torch.where(idx >= 0, (1 + idx).float() * w, torch.zeros(())).sum(1, keepdim=True)
            # bf16 rounding of the row, of the expert's product and of the result (2^-8 each), e4m3 rows 2^-4
            tol = 2.0 ** -4 if fp8 else 2.0 ** -7
            want = x.float().cpu() * factor
            scale = x.float().abs().amax(1, keepdim=True).cpu() * factor
            assert bool(((out.float().cpu() - want).abs() <= tol * (want.abs() + (scale * 2.0 ** -5 if fp8 else 1e-3))).all())
        buf.check_status()
    finally:
        buf.destroy()


# one buffer that serves several bounds on the tokens of a call, so that the grid of its send kernels changes: powers
# of two and not, fewer tokens than the bound (idle CTAs), odd and even numbers of calls before each change
@pytest.mark.parametrize("signal_mode", [0, 1])
@pytest.mark.parametrize("in_place", [False, True])
def test_low_latency_token_bound_changes_on_one_buffer(signal_mode, in_place, monkeypatch):
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    monkeypatch.setattr(Buffer, "ll_signal_mode", signal_mode)
    H, E, K = 512, 16, 4
    buf = Buffer(None, Buffer.get_low_latency_nvl_size_hint(200, H, 1, E, K), 0, low_latency_mode=True,
                 world=LocalWorld.make(1)[0], timeout_s=2.0)
    try:
        for rep, (M, T) in enumerate([(96, 96), (128, 128), (96, 5), (96, 96), (128, 100), (7, 7), (128, 128), (100, 99),
                                      (7, 3), (1, 1), (200, 200), (128, 128)]):
            g = torch.Generator().manual_seed(rep)
            x = torch.randn(T, H, generator=g).to(torch.bfloat16)
            idx, w = O.make_routing(T, E, K, 90 + rep)
            xc, ic, wc = x.cuda(), idx.cuda(), w.cuda()
            recv, count, handle, _, _ = buf.low_latency_dispatch(xc, ic, M, E, use_fp8=False)
            cnt = count.tolist()
            assert cnt == [int((idx == e).sum()) for e in range(E)]
            src = handle[0].cpu()
            for e in range(E):
                _, s_t, s_k = _unpack(src[e, :cnt[e]])
                assert len(set(src[e, :cnt[e]].tolist())) == cnt[e]
                assert bool((idx[s_t, s_k] == e).all()) and torch.equal(recv[e, :cnt[e]].cpu(), x[s_t])
            y = recv.clone()
            if in_place:
                y = buf.get_next_low_latency_combine_buffer(handle)
                y.copy_(recv)
            out, _, hook = buf.low_latency_combine(y, ic, wc, handle, return_recv_hook=rep % 3 == 0)
            out = hook() if out is None else out
            # one bf16 rounding of a sum whose weights add up to one within f32 rounding
            torch.testing.assert_close(out.float(), xc.float() * wc.sum(1, keepdim=True), atol=1e-6, rtol=2.0 ** -7)
            assert buf._ll_words.view(3, 6)[:, 4].tolist() == [0, 0, 0]       # no count is carried into the next launch
        buf.check_status()
    finally:
        buf.destroy()


@pytest.mark.parametrize("E,M", [(8, 160), (1024, 9), (1032, 9)])
def test_low_latency_counts_of_a_group_of_one(E, M):
    """A group of one counts rows from the choices in a CTA of its own (up to 1024 experts; more take the counters)
    and readies the other parity's row counters: calls that do and calls with a hook in any order, no tokens, one,
    more tokens than CTAs that move rows, masked choices. Rows per expert and the combined rows are exact."""
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    from gpu_data_transfer_profile_b200.parallel.local import LocalGroup
    H, K = 256, 4
    g = LocalGroup(1, Buffer.get_low_latency_nvl_size_hint(M, H, 1, E, K), timeout_s=2.0)
    try:
        b = g.buffers[0]
        gen = torch.Generator().manual_seed(E)
        for rep, (hooked, T) in enumerate([(0, M), (1, M), (1, 3), (0, 1), (0, 0), (0, M), (1, 1), (0, M - 1), (0, M), (1, M), (0, M)]):
            x = torch.randn(T, H, generator=gen).to(torch.bfloat16).cuda()
            idx = torch.stack([torch.randperm(E, generator=gen)[:K] for _ in range(T)]) if T else torch.zeros(0, K, dtype=torch.int64)
            idx[torch.rand(idx.shape, generator=gen) < 0.2] = -1
            idx, keep = idx.cuda(), (idx >= 0)
            if hooked:
                *_, hook = b.low_latency_dispatch(x, idx, M, E, use_fp8=False, return_recv_hook=True)
                recv, count, handle = hook()
            else:
                recv, count, handle, _, _ = b.low_latency_dispatch(x, idx, M, E, use_fp8=False)
            want = torch.bincount(idx[idx >= 0].cpu(), minlength=E)
            assert torch.equal(count.cpu().long(), want), (rep, hooked, T)
            out, _, _ = b.low_latency_combine(recv, idx, torch.ones(T, K, device="cuda"), handle)
            assert torch.equal(out, (x.float() * keep.sum(1, keepdim=True).cuda()).to(torch.bfloat16)), (rep, hooked, T)
        g.check_status()
    finally:
        g.destroy()


@pytest.mark.parametrize("first", ["low latency", "exchange", "both"])
def test_low_latency_shape_after_a_refused_one(first):
    """A shape that is refused (top-k, hidden size, a region too small, too many experts) leaves the buffer as it
    was: what an earlier shape left in the row counters is cleared before another one counts there. Counts, sources
    and combined rows are exact."""
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    from gpu_data_transfer_profile_b200.parallel.local import LocalGroup
    M, H, K, E = 64, 256, 4, 256
    g = LocalGroup(1, Buffer.get_low_latency_nvl_size_hint(M, H, 1, 512, K), timeout_s=2.0)
    gen = torch.Generator().manual_seed(3)

    def inputs(T, experts, k=K, h=H):
        return (torch.randn(T, h, generator=gen).to(torch.bfloat16).cuda(),
                torch.stack([torch.randperm(experts, generator=gen)[:k] for _ in range(T)]).cuda())

    def exchange(b):
        x, idx = inputs(M, 8)
        recv, _, _, _, handle, _ = b.dispatch(x, topk_idx=idx, group_by_expert=True, num_experts=8)
        assert torch.equal(b.combine(recv, handle)[0], 4 * x)

    def low_latency(b, experts):
        x, idx = inputs(M, experts)
        recv, count, handle, _, _ = b.low_latency_dispatch(x, idx, M, experts, use_fp8=False)
        assert torch.equal(count.cpu().long(), torch.bincount(idx.flatten().cpu(), minlength=experts))
        for e in idx.unique().tolist():
            n = int(count[e])
            _, t, k = _unpack(handle[0][e, :n].long())
            assert n == len(set(t.tolist())) and torch.equal(idx[t, k], torch.full_like(t, e)) and torch.equal(recv[e, :n], x[t])
        out, _, _ = b.low_latency_combine(recv, idx, torch.ones(M, K, device="cuda"), handle)
        assert torch.equal(out, 4 * x)

    try:
        b = g.buffers[0]
        if first != "low latency":
            exchange(b)
        for _ in range(2 * (first != "exchange")):
            low_latency(b, 512)
        for _ in range(2):
            x, idx = inputs(2, 64, 33)
            with pytest.raises(RuntimeError):
                b.low_latency_dispatch(x, idx, M, 64, use_fp8=False)
            x, idx = inputs(2, 64, 33)
            with pytest.raises(RuntimeError):
                b.dispatch(x, topk_idx=idx, group_by_expert=True, num_experts=64)
            x, idx = inputs(2, E, K, 100)
            with pytest.raises(RuntimeError):
                b.low_latency_dispatch(x, idx, M, E, use_fp8=False)
            x, idx = inputs(2, E)
            with pytest.raises(ValueError):
                b.low_latency_dispatch(x, idx, 100 * M, E, use_fp8=False)
            with pytest.raises(ValueError):
                b.dispatch(x, topk_idx=idx, group_by_expert=True, num_experts=1 << 20)
        for _ in range(3):
            low_latency(b, E)
        exchange(b)
        low_latency(b, 512)
        b.check_status()
    finally:
        g.destroy()
