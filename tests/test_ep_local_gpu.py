"""Single-GPU checks of the EP data path with several virtual ranks (one kernel set per rank,
phases run in lock step). Every kernel result is compared with the fp32 PyTorch oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from gpu_data_transfer_profile_b200.ref import cpu_oracle as O


def _mk(R, T, H, E, K, dtype=torch.bfloat16, seed=0, zipf=0.0, uneven=False):
    xs, idxs, ws = [], [], []
    for r in range(R):
        t = T + (7 * r if uneven else 0)
        g = torch.Generator().manual_seed(seed * 100 + r)
        xs.append(torch.randn(t, H, generator=g).to(dtype))
        i, w = O.make_routing(t, E, K, seed * 100 + r, zipf)
        idxs.append(i)
        ws.append(w)
    return xs, idxs, ws


def _group(R, nbytes=256 << 20):
    from gpu_data_transfer_profile_b200.parallel.local import LocalGroup
    return LocalGroup(R, nbytes, timeout_s=2.0)


@pytest.mark.parametrize("R,T,H,E,K", [(1, 64, 256, 8, 2), (2, 128, 256, 8, 2), (4, 200, 512, 32, 4),
                                       (8, 96, 1024, 64, 8)])
def test_layout_matches_oracle(R, T, H, E, K):
    xs, idxs, ws = _mk(R, T, H, E, K)
    g = _group(R, 64 << 20)
    try:
        lays = g.get_dispatch_layout([i.cuda() for i in idxs], E)
        for r in range(R):
            pr, pe, inr = O.layout_ref(idxs[r], E, R)
            assert torch.equal(lays[r][0].cpu(), pr)
            assert lays[r][1] is None
            assert torch.equal(lays[r][2].cpu(), pe)
            assert torch.equal(lays[r][3].cpu(), inr)
        g.check_status()
    finally:
        g.destroy()


@pytest.mark.parametrize("R,T,H,E,K,dtype", [
    (1, 64, 256, 8, 2, torch.bfloat16), (2, 128, 256, 8, 2, torch.bfloat16),
    (4, 200, 512, 32, 4, torch.bfloat16), (8, 96, 1024, 64, 8, torch.bfloat16),
    (2, 128, 256, 8, 2, torch.float32), (4, 33, 384, 16, 3, torch.float16)])
def test_dispatch_combine_rank_mode(R, T, H, E, K, dtype):
    xs, idxs, ws = _mk(R, T, H, E, K, dtype, uneven=True)
    g = _group(R)
    try:
        cx = [x.cuda() for x in xs]
        ci = [i.cuda() for i in idxs]
        cw = [w.cuda() for w in ws]
        lays = g.get_dispatch_layout(ci, E)
        outs = g.dispatch(cx, layouts=lays, topk_idx=ci, topk_weights=cw)
        ref = O.dispatch_rank_mode_ref(xs, idxs, ws, E)
        for d in range(R):
            rx, ri, rw, cnt, h = outs[d]
            ex, ei, ew, sr, stok, ecnt = ref[d]
            assert rx.shape == ex.shape
            assert torch.equal(rx.cpu(), ex)
            assert torch.equal(ri.cpu(), ei)
            assert torch.equal(rw.cpu(), ew)
            assert cnt == ecnt
            assert h.n_recv == ex.shape[0]
        # combine with an "expert" that scales by (1 + rank): checks routing of every row
        ys = [(outs[d][0].float() * (1 + d)).to(dtype) for d in range(R)]
        comb = g.combine(ys, [o[4] for o in outs], topk_weights=[o[2] for o in outs])
        cref = O.combine_ref([y.cpu() for y in ys], [r[3] for r in ref], [r[4] for r in ref],
                             [x.shape[0] for x in xs])
        wref = O.combine_ref([r[2] for r in ref], [r[3] for r in ref], [r[4] for r in ref],
                             [x.shape[0] for x in xs])
        tol = 1e-5 if dtype == torch.float32 else 2e-2
        for s in range(R):
            got, got_w = comb[s]
            torch.testing.assert_close(got.cpu().float(), cref[s], atol=tol * 8, rtol=tol)
            torch.testing.assert_close(got_w.cpu(), wref[s], atol=1e-6, rtol=1e-6)
        g.check_status()
        g.check_canaries()
    finally:
        g.destroy()


@pytest.mark.parametrize("R,T,H,E,K", [(1, 64, 256, 8, 2), (2, 128, 256, 8, 2), (4, 100, 512, 32, 4),
                                       (8, 64, 1024, 8, 2)])
def test_dispatch_combine_expert_mode(R, T, H, E, K):
    xs, idxs, ws = _mk(R, T, H, E, K, zipf=1.2)
    g = _group(R)
    try:
        cx = [x.cuda() for x in xs]
        ci = [i.cuda() for i in idxs]
        cw = [w.cuda() for w in ws]
        outs = g.dispatch(cx, topk_idx=ci, topk_weights=cw, group_by_expert=True, num_experts=E)
        ref = O.dispatch_expert_mode_ref(xs, idxs, ws, E)
        for d in range(R):
            rx, _, _, cnt, h = outs[d]
            ex, ep, sr, stok, sk, ecnt = ref[d]
            assert cnt == ecnt
            assert torch.equal(rx.cpu(), ex)
            assert torch.equal(h.recv_prob.cpu(), ep)
        # weighted combine: out[t] = sum_k w[t,k] * x[t]  == x[t] (weights sum to 1)
        comb = g.combine([o[0] for o in outs], [o[4] for o in outs], item_weights=cw)
        for s in range(R):
            torch.testing.assert_close(comb[s][0].cpu().float(), xs[s].float(), atol=3e-2, rtol=2e-2)
        g.check_status()
        g.check_canaries()
    finally:
        g.destroy()


def test_dispatch_fp8_and_cached():
    R, T, H, E, K = 4, 96, 1024, 32, 4
    xs, idxs, ws = _mk(R, T, H, E, K)
    g = _group(R)
    try:
        cx = [x.cuda() for x in xs]
        ci = [i.cuda() for i in idxs]
        cw = [w.cuda() for w in ws]
        lays = g.get_dispatch_layout(ci, E)
        outs = g.dispatch(cx, layouts=lays, topk_idx=ci, topk_weights=cw, use_fp8=True)
        ref = O.dispatch_rank_mode_ref(xs, idxs, ws, E)
        for d in range(R):
            (q, s), _, _, _, h = outs[d]
            eq, es = O.fp8_block_quant_ref(ref[d][0])
            torch.testing.assert_close(s.cpu(), es, rtol=1e-6, atol=0)
            deq = O.fp8_block_dequant_ref(q.cpu(), s.cpu())
            torch.testing.assert_close(deq, ref[d][0].float(), atol=0.3, rtol=0.07)
            assert (q.cpu().view(torch.uint8) != eq.view(torch.uint8)).float().mean() < 0.01
        # cached-handle dispatch of new data reuses the layout
        x2 = [torch.randn_like(x) for x in cx]
        outs2 = g.dispatch(x2, handles=[o[4] for o in outs])
        ref2 = O.dispatch_rank_mode_ref([x.cpu() for x in x2], idxs, ws, E)
        for d in range(R):
            assert torch.equal(outs2[d][0].cpu(), ref2[d][0])
        g.check_status()
    finally:
        g.destroy()


def test_lost_peer_is_an_error_not_a_hang():
    g = _group(1, 8 << 20)
    try:
        assert g.buffers[0].probe_timeout(0.05) == 8
        g.check_status()
    finally:
        g.destroy()


def test_recorded_fault_is_raised_by_the_next_op_without_check_status():
    """A time-out leaves its code in the status word AND in a mapped host word; the next public
    op on the buffer raises it even though nobody called check_status()."""
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer, EpTimeoutError
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    T, H, E, K = 64, 256, 8, 2
    buf = Buffer(None, 32 << 20, world=LocalWorld.make(1)[0], timeout_s=2.0)
    try:
        x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
        idx, w = O.make_routing(T, E, K, 3)
        idx, w = idx.cuda(), w.cuda()
        assert buf.probe_timeout(0.05, clear=False) == 8
        with pytest.raises(EpTimeoutError):
            buf.get_dispatch_layout(idx, E)
        # the fault was consumed: the buffer works again
        pr, _, pe, inr, _ = buf.get_dispatch_layout(idx, E)
        rx, _, _, _, h, _ = buf.dispatch(x, topk_idx=idx, topk_weights=w, is_token_in_rank=inr,
                                         num_tokens_per_expert=pe)
        assert torch.equal(rx, x)
        buf.check_status()
    finally:
        buf.destroy()


def test_cached_dispatch_refuses_a_handle_made_for_another_layout():
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    T, H, E, K = 64, 256, 8, 2
    buf = Buffer(None, 32 << 20, world=LocalWorld.make(1)[0], timeout_s=2.0)
    try:
        x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
        idx, w = O.make_routing(T, E, K, 3)
        idx, w = idx.cuda(), w.cuda()
        pr, _, pe, inr, _ = buf.get_dispatch_layout(idx, E)
        _, _, _, _, h, _ = buf.dispatch(x, topk_idx=idx, topk_weights=w, is_token_in_rank=inr,
                                        num_tokens_per_expert=pe)
        y, _, _, _, _, _ = buf.dispatch(x * 2, handle=h)          # same width: fine
        assert torch.equal(y, x * 2)
        with pytest.raises(ValueError):
            buf.dispatch(x.float(), handle=h)                      # wider rows: other layout, smaller capacity
        buf.check_status()
    finally:
        buf.destroy()


def test_receive_bound_overflow_is_a_status_not_a_fault():
    """`num_max_recv_tokens` caps the receive region; a routing that needs more rows ends in
    status 6 and every out-of-range row is skipped."""
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer, EpStatusError
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    T, H, E, K = 96, 256, 8, 2
    buf = Buffer(None, 32 << 20, world=LocalWorld.make(1)[0], timeout_s=2.0, num_max_recv_tokens=64)
    try:
        x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
        idx, w = O.make_routing(T, E, K, 3)
        idx, w = idx.cuda(), w.cuda()
        pr, _, pe, inr, _ = buf.get_dispatch_layout(idx, E)
        with pytest.raises(EpStatusError):
            buf.dispatch(x, topk_idx=idx, topk_weights=w, is_token_in_rank=inr, num_tokens_per_expert=pe)
            buf.check_status()
        torch.cuda.synchronize()
        try:
            buf.check_status()
        except EpStatusError:
            pass
        # a smaller batch fits
        x2, idx2, w2 = x[:48].contiguous(), idx[:48].contiguous(), w[:48].contiguous()
        pr, _, pe, inr, _ = buf.get_dispatch_layout(idx2, E)
        rx, _, _, _, h, _ = buf.dispatch(x2, topk_idx=idx2, topk_weights=w2, is_token_in_rank=inr,
                                         num_tokens_per_expert=pe)
        assert torch.equal(rx, x2)
        buf.check_status()
        buf.check_canaries()        # the skipped rows of the overflowing call touched no guard band
    finally:
        buf.destroy()


def test_guard_bands_are_checked_and_a_stray_store_is_named():
    """Every region of the carve ends in a painted guard band; `check_canaries` passes after real
    traffic (receive region filled to its last row) and names the region behind which a byte changed."""
    from gpu_data_transfer_profile_b200.parallel.buffer import CANARY, Buffer, EpStatusError
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    T, H, E, K = 64, 256, 8, 2
    buf = Buffer(None, 32 << 20, world=LocalWorld.make(1)[0], timeout_s=2.0, num_max_recv_tokens=T)
    try:
        x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
        idx, w = O.make_routing(T, E, K, 5)
        idx, w = idx.cuda(), w.cuda()
        for _ in range(3):          # both epoch parities; T rows = exactly the capacity
            pr, _, pe, inr, _ = buf.get_dispatch_layout(idx, E)
            rx, _, _, _, h, _ = buf.dispatch(x, topk_idx=idx, topk_weights=w, is_token_in_rank=inr,
                                             num_tokens_per_expert=pe)
            out, _, _ = buf.combine(rx, h)
            assert rx.shape[0] == T == buf._carve.cap
        buf.check_status()
        buf.check_canaries()
        name, parity, off, n = buf._carve.guards[0]
        band = buf.region.view(off, (n,), "uint8")
        assert bool((band == CANARY).all())
        band[7] = 0                 # what a store one row past the region would do
        with pytest.raises(EpStatusError, match=name):
            buf.check_canaries()
        band[7] = CANARY
        buf.check_canaries()
    finally:
        buf.destroy()


@pytest.mark.parametrize("R,T,H,E,K,dtype", [(1, 70, 256, 8, 2, torch.bfloat16), (4, 150, 1024, 32, 4, torch.bfloat16),
                                             (8, 64, 7168, 64, 8, torch.bfloat16), (2, 100, 384, 8, 2, torch.float32)])
def test_pull_combine_reads_rows_in_place_and_matches_the_oracle(R, T, H, E, K, dtype):
    """Zero-copy dispatch output, modified in place by the 'expert', combined by the pull form
    (no slot region): result and reduced side values equal the oracle. Three rounds with
    different data, so a stale cached row from an earlier round would be seen."""
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    xs, idxs, ws = _mk(R, T, H, E, K, dtype, uneven=True, seed=7)
    g = _group(R)
    try:
        ci, cw = [i.cuda() for i in idxs], [w.cuda() for w in ws]
        for rep in range(3):
            cx = [(x.float() * (1 + rep)).to(dtype).cuda() for x in xs]
            ref = O.dispatch_rank_mode_ref([c.cpu() for c in cx], idxs, ws, E)
            lays = g.get_dispatch_layout(ci, E)
            outs = g.dispatch(cx, layouts=lays, topk_idx=ci, topk_weights=cw, zero_copy=True)
            for d in range(R):
                assert g.buffers[d]._use_pull(outs[d][0], outs[d][2])
                outs[d][0].mul_(1 + d)                       # the "expert": in place, inside the region
            ys = [o[0] for o in outs]
            comb = g.combine(ys, [o[4] for o in outs], topk_weights=[o[2] for o in outs])
            cref = O.combine_ref([(r[0].float() * (1 + d)).to(dtype) for d, r in enumerate(ref)],
                                 [r[3] for r in ref], [r[4] for r in ref], [x.shape[0] for x in xs])
            wref = O.combine_ref([r[2] for r in ref], [r[3] for r in ref], [r[4] for r in ref],
                                 [x.shape[0] for x in xs])
            tol = 1e-5 if dtype == torch.float32 else 2e-2
            for s in range(R):
                got, got_w = comb[s]
                torch.testing.assert_close(got.cpu().float(), cref[s], atol=tol * 16 * (1 + rep), rtol=tol)
                torch.testing.assert_close(got_w.cpu(), wref[s], atol=1e-6, rtol=1e-6)
        # forcing the push form on the same tensors gives the same numbers
        old = Buffer.combine_transport
        Buffer.combine_transport = "push"
        try:
            comb2 = g.combine(ys, [o[4] for o in outs], topk_weights=[o[2] for o in outs])
        finally:
            Buffer.combine_transport = old
        for s in range(R):
            assert torch.equal(comb2[s][0], comb[s][0])
        g.check_status()
    finally:
        g.destroy()


def test_pull_combine_expert_mode_with_item_weights():
    R, T, H, E, K = 4, 100, 512, 32, 4
    xs, idxs, ws = _mk(R, T, H, E, K, zipf=1.2)
    g = _group(R)
    try:
        cx, ci, cw = [x.cuda() for x in xs], [i.cuda() for i in idxs], [w.cuda() for w in ws]
        outs = g.dispatch(cx, topk_idx=ci, topk_weights=cw, group_by_expert=True, num_experts=E, zero_copy=True)
        assert all(g.buffers[d]._use_pull(outs[d][0], None) for d in range(R))
        comb = g.combine([o[0] for o in outs], [o[4] for o in outs], item_weights=cw)
        for s in range(R):
            torch.testing.assert_close(comb[s][0].cpu().float(), xs[s].float(), atol=3e-2, rtol=2e-2)
        g.check_status()
        g.check_canaries()
    finally:
        g.destroy()


def test_dispatch_without_host_sync_num_worst_tokens():
    """num_worst_tokens: outputs sized by the caller's bound, true count only on the device."""
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    T, H, E, K = 100, 256, 8, 2
    buf = Buffer(None, 32 << 20, world=LocalWorld.make(1)[0], timeout_s=2.0)
    try:
        x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
        idx, w = O.make_routing(T, E, K, 3)
        idx, w = idx.cuda(), w.cuda()
        pr, _, pe, inr, _ = buf.get_dispatch_layout(idx, E)
        rx, ri, rw, cnt, h, _ = buf.dispatch(x, topk_idx=idx, topk_weights=w, num_tokens_per_rank=pr, is_token_in_rank=inr,
                                            num_tokens_per_expert=pe, num_worst_tokens=256, zero_copy=True)
        assert rx.shape == (256, H) and cnt == [] and h.n_recv == 256
        assert int(h.n_recv_dev.item()) == T
        assert torch.equal(rx[:T], x)
        out, _, _ = buf.combine(rx, h)
        torch.testing.assert_close(out.float(), x.float())
        with pytest.raises(ValueError):
            buf.dispatch(x, topk_idx=idx, topk_weights=w, num_tokens_per_rank=pr, is_token_in_rank=inr,
                         num_tokens_per_expert=pe, num_worst_tokens=1 << 30)
        buf.check_status()
    finally:
        buf.destroy()


def test_dispatch_accepts_caller_quantised_fp8_tuple():
    R, T, H, E, K = 2, 64, 512, 8, 2
    xs, idxs, ws = _mk(R, T, H, E, K)
    g = _group(R, 64 << 20)
    try:
        qs = [O.fp8_block_quant_ref(x) for x in xs]
        ci, cw = [i.cuda() for i in idxs], [w.cuda() for w in ws]
        lays = g.get_dispatch_layout(ci, E)
        outs = g.dispatch([(q.cuda(), s.cuda()) for q, s in qs], layouts=lays, topk_idx=ci, topk_weights=cw)
        ref_q = O.dispatch_rank_mode_ref([q.view(torch.uint8) for q, _ in qs], idxs, ws, E)
        ref_s = O.dispatch_rank_mode_ref([s for _, s in qs], idxs, ws, E)
        for d in range(R):
            (rq, rs), _, _, _, h = outs[d]
            assert rq.dtype == torch.float8_e4m3fn and h.fp8
            assert torch.equal(rq.cpu().view(torch.uint8), ref_q[d][0])
            assert torch.equal(rs.cpu(), ref_s[d][0])
        g.check_status()
    finally:
        g.destroy()


@pytest.mark.parametrize("num_sms", [1, 3, 24, 148])
def test_round_trip_is_independent_of_the_cta_knob(num_sms):
    """Same routing, different numbers of CTAs in the send/reduce kernels: the received rows and the
    combined result must not depend on how the work is cut (shakes out ordering assumptions)."""
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    R, T, H, E, K = 4, 150, 512, 32, 4
    xs, idxs, ws = _mk(R, T, H, E, K, uneven=True, seed=3)
    old = Buffer.num_sms
    Buffer.set_num_sms(num_sms)
    g = _group(R)
    try:
        cx, ci, cw = [x.cuda() for x in xs], [i.cuda() for i in idxs], [w.cuda() for w in ws]
        ref = O.dispatch_rank_mode_ref(xs, idxs, ws, E)
        for rep in range(2):
            lays = g.get_dispatch_layout(ci, E)
            outs = g.dispatch(cx, layouts=lays, topk_idx=ci, topk_weights=cw)
            for d in range(R):
                assert torch.equal(outs[d][0].cpu(), ref[d][0])
                assert torch.equal(outs[d][1].cpu(), ref[d][1])
            comb = g.combine([o[0] for o in outs], [o[4] for o in outs])
            cref = O.combine_ref([r[0] for r in ref], [r[3] for r in ref], [r[4] for r in ref],
                                 [x.shape[0] for x in xs])
            for s in range(R):
                got = comb[s][0] if isinstance(comb[s], tuple) else comb[s]
                torch.testing.assert_close(got.cpu().float(), cref[s], atol=0.16, rtol=2e-2)
        g.check_status()
    finally:
        g.destroy()
        Buffer.set_num_sms(old)


@pytest.mark.parametrize("R", [2, 4])
def test_fc2_epilogue_combine_addresses_every_virtual_rank(R):
    """The fc2 grouped GEMM's combine epilogue stores each output row into its token's slot on the
    SOURCE rank; with several virtual ranks the slots live in different regions, so the peer
    addressing of the epilogue is exercised on one GPU. Oracle: per-expert fp32 matmul of the
    dispatched rows, summed per token by the list-based combine oracle."""
    T, H, F, E, K = 120, 256, 256, 8, 2
    xs, idxs, ws = _mk(R, T, H, E, K, seed=9)
    El = E // R
    g = _group(R)
    try:
        cx, ci, cw = [x.cuda() for x in xs], [i.cuda() for i in idxs], [w.cuda() for w in ws]
        outs = g.dispatch(cx, topk_idx=ci, topk_weights=cw, group_by_expert=True, num_experts=E)
        ref = O.dispatch_expert_mode_ref(xs, idxs, ws, E)
        torch.manual_seed(1)
        w2s = [(torch.randn(El, H, H, device="cuda") * 0.05).to(torch.bfloat16) for _ in range(R)]
        acts = [o[0] for o in outs]                     # stand-in for the fc1 output: F == H here
        comb = g.fused_fc2_combine(acts, w2s, [o[4] for o in outs])
        ys = []
        for d in range(R):
            ex, ep, sr, stok, sk, ecnt = ref[d]
            rows, r0 = [], 0
            for e, c in enumerate(ecnt):
                rows.append(ex[r0:r0 + c].float() @ w2s[d][e].float().cpu().t())
                r0 += c
            ys.append(torch.cat(rows) if rows else torch.zeros(0, H))
        cref = O.combine_ref(ys, [r[2] for r in ref], [r[3] for r in ref], [x.shape[0] for x in xs])
        for s in range(R):
            torch.testing.assert_close(comb[s].cpu().float(), cref[s], atol=6e-2, rtol=3e-2)
        g.check_status()
    finally:
        g.destroy()


def test_buffer_without_combine_slots_pulls_and_refuses_to_push():
    """`combine_slots=False` halves the region: the zero-copy rows are combined by the pull form,
    a tensor outside the region cannot be combined at all, and the size hint shrinks accordingly."""
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    T, H, E, K = 100, 512, 8, 2
    full = Buffer.get_dispatch_config(1, T, K, E).get_nvl_buffer_size_hint(H * 2, 1)
    half = Buffer.get_dispatch_config(1, T, K, E, combine_slots=False).get_nvl_buffer_size_hint(H * 2, 1)
    from gpu_data_transfer_profile_b200.parallel.config import FIXED_BYTES
    assert (half - FIXED_BYTES) < 0.6 * (full - FIXED_BYTES)          # the fixed control area aside
    buf = Buffer(None, half, world=LocalWorld.make(1)[0], timeout_s=2.0, combine_slots=False)
    try:
        x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
        idx, w = O.make_routing(T, E, K, 3)
        idx, w = idx.cuda(), w.cuda()
        pr, _, pe, inr, _ = buf.get_dispatch_layout(idx, E)
        rx, _, _, _, h, _ = buf.dispatch(x, topk_idx=idx, topk_weights=w, is_token_in_rank=inr,
                                         num_tokens_per_expert=pe, zero_copy=True)
        out, _, _ = buf.combine(rx, h)
        torch.testing.assert_close(out.float(), x.float())
        with pytest.raises(ValueError):
            buf.combine(rx.clone(), h)
        buf.check_status()
    finally:
        buf.destroy()


# few tokens with long rows (a row is cut into parts, one warp each), expert counts that are no multiple of
# a warp, one rank (no flags) and two
@pytest.mark.parametrize("R,T,H,E,K,dtype,fp8", [(1, 1, 7168, 160, 8, torch.bfloat16, False), (1, 37, 7168, 33, 4, torch.bfloat16, True),
                                                 (2, 5, 4096 + 8, 96, 6, torch.float32, False), (2, 300, 3200, 8, 2, torch.bfloat16, True),
                                                 (1, 1100, 2176, 64, 3, torch.float16, False)])
@pytest.mark.parametrize("grouped", [False, True])
def test_dispatch_rows_cut_into_parts_and_receive_tables(R, T, H, E, K, dtype, fp8, grouped):
    xs, idxs, ws = _mk(R, T, H, E, K, dtype=dtype, seed=11, zipf=0.7)
    g = _group(R, 768 << 20)
    El = E // R
    try:
        cx, ci, cw = [x.cuda() for x in xs], [i.cuda() for i in idxs], [w.cuda() for w in ws]
        lays = None if grouped else g.get_dispatch_layout(ci, E)
        outs = g.dispatch(cx, layouts=lays, topk_idx=ci, topk_weights=cw, use_fp8=fp8, group_by_expert=grouped, num_experts=E)
        ref = (O.dispatch_expert_mode_ref if grouped else O.dispatch_rank_mode_ref)(xs, idxs, ws, E)
        for d in range(R):
            h, cnt = outs[d][4], ref[d][5]
            n = ref[d][0].shape[0]
            meta = h.meta.cpu().tolist()
            assert meta[0] == n == h.n_recv and meta[2:2 + El] == list(cnt) == list(outs[d][3])
            off = h.meta[2 + El:2 + El + El + 1].cpu().tolist()
            assert off == [sum(cnt[:q]) for q in range(El + 1)]
            if fp8:
                q, sc = outs[d][0]
                torch.testing.assert_close(sc.cpu(), O.fp8_block_quant_ref(ref[d][0])[1], rtol=1e-6, atol=0)
                torch.testing.assert_close(O.fp8_block_dequant_ref(q.cpu(), sc.cpu()), ref[d][0].float(), atol=0.3, rtol=0.07)
            else:
                assert torch.equal(outs[d][0].cpu(), ref[d][0])
            if grouped:
                assert torch.equal(h.recv_prob.cpu(), ref[d][1])
            else:
                assert torch.equal(outs[d][1].cpu(), ref[d][1]) and torch.equal(outs[d][2].cpu(), ref[d][2])
        again = g.dispatch(cx, handles=[o[4] for o in outs], use_fp8=fp8)     # the cached form writes the same rows
        for d in range(R):
            a, b = again[d][0], outs[d][0]
            assert torch.equal(a[0].view(torch.uint8), b[0].view(torch.uint8)) if fp8 else torch.equal(a, b)
        g.check_status()
        g.check_canaries()
    finally:
        g.destroy()


# own rows are reduced where they lie, peers' rows from their slots; few tokens: rows cut into up to 16 parts
@pytest.mark.parametrize("R,T,H,E,K,dtype", [(1, 3, 7168, 16, 8, torch.bfloat16), (2, 9, 7168, 16, 4, torch.bfloat16),
                                             (4, 2, 4104, 8, 2, torch.float32), (2, 700, 520, 8, 8, torch.float16)])
@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("weighted", [False, True])
def test_push_combine_reads_own_rows_in_place(R, T, H, E, K, dtype, grouped, weighted):
    xs, idxs, ws = _mk(R, T, H, E, K, dtype=dtype, seed=21)
    idxs[0][0, 0] = -1                                    # an empty choice contributes nothing
    g = _group(R, 512 << 20)
    try:
        cx, ci, cw = [x.cuda() for x in xs], [i.cuda() for i in idxs], [w.cuda() for w in ws]
        for rep in range(3):
            lays = None if grouped else g.get_dispatch_layout(ci, E)
            outs = g.dispatch(cx, layouts=lays, topk_idx=ci, topk_weights=cw, group_by_expert=grouped, num_experts=E)
            ys = [(o[0].float() * (rep + 1 + d)).to(dtype) for d, o in enumerate(outs)]       # tensors of their own: push
            side = [o[4].recv_prob if grouped else o[2] for o in outs]
            J = K if grouped else R
            iw = [torch.rand(T, J, device="cuda", generator=torch.Generator("cuda").manual_seed(r)) for r in range(R)] if weighted else None
            comb = g.combine(ys, [o[4] for o in outs], topk_weights=side, item_weights=iw)
            for r in range(R):
                valid = idxs[r] >= 0
                dest = torch.where(valid, idxs[r] // (E // R), torch.zeros_like(idxs[r]))
                if grouped:
                    factor = torch.where(valid, rep + 1.0 + dest, torch.zeros(()))
                else:
                    hit = torch.zeros(T, R, dtype=torch.bool)
                    hit[torch.arange(T)[:, None].expand_as(dest)[valid], dest[valid]] = True
                    factor = hit * (rep + 1.0 + torch.arange(R))
                if weighted:
                    factor = factor * iw[r].cpu()
                got, got_w = comb[r]
                tol = dict(atol=1e-5, rtol=1e-5) if dtype == torch.float32 else dict(atol=0.08, rtol=2e-2)
                torch.testing.assert_close(got.cpu().float(), xs[r].float() * factor.sum(1, keepdim=True), **tol)
                torch.testing.assert_close(got_w.cpu(), torch.where(valid, ws[r], torch.zeros(())), atol=1e-6, rtol=1e-6)
        g.check_status()
        g.check_canaries()
    finally:
        g.destroy()


def test_clone_views_copies_every_byte_of_every_buffer():
    """Sizes around a vector, a CTA's chunk and the grid; an empty buffer between others."""
    from gpu_data_transfer_profile_b200 import _ext
    C = _ext.load()
    g = torch.Generator("cuda").manual_seed(1)
    sizes = [1, 0, 15, 16, 17, 16384 - 1, 16384 + 33, 16384 * 148 * 8 + 16384 + 5]
    src = [torch.randint(0, 256, (n,), generator=g, device="cuda", dtype=torch.uint8) for n in sizes]
    for part in (src, src[:1], src[1:2], []):
        out = C.clone_views(part)
        assert len(out) == len(part)
        for a, b in zip(out, part):
            assert torch.equal(a, b) and (a.numel() == 0 or a.data_ptr() != b.data_ptr())
    x = torch.randn(37, 5, 3, device="cuda").to(torch.float8_e4m3fn)
    y = C.clone_views([x])[0]
    assert y.dtype == x.dtype and y.shape == x.shape and torch.equal(y.view(torch.uint8), x.view(torch.uint8))
    with pytest.raises(RuntimeError):
        C.clone_views([src[4][1:]])                     # not 16-byte aligned
    with pytest.raises(RuntimeError):
        C.clone_views(src + src[:1])


# a group of one: owned outputs are written where they are owned, and equal the views of the region; T = 0, every
# choice masked, more items than rows, few and all choices masked
@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("form", ["plain", "fp8", "tuple"])
@pytest.mark.parametrize("T,masked", [(0, 0.0), (1, 0.0), (33, 1.0), (130, 0.4), (257, 0.0)])
def test_owned_outputs_of_a_group_of_one_equal_the_region_views(T, masked, form, grouped):
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    H, E, K = 256, 8, 3
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, H, generator=g).to(torch.bfloat16).cuda()
    idx = torch.rand(T, E, generator=g).topk(K, dim=-1).indices
    idx[torch.rand(T, K, generator=g) < masked] = -1
    idx, w = idx.cuda(), torch.rand(T, K, generator=g).cuda()
    if form == "tuple":
        x = (x.to(torch.float8_e4m3fn), torch.rand(T, H // 128, generator=g).cuda())
    raw = lambda t: t.contiguous().view(torch.uint8) if t.dtype == torch.float8_e4m3fn else t
    buf = Buffer(None, 32 << 20, world=LocalWorld.make(1)[0], timeout_s=2.0)
    try:
        lay = {} if grouped else dict(zip(("num_tokens_per_rank", "is_token_in_rank"),
                                          (lambda l: (l[0], l[3]))(buf.get_dispatch_layout(idx, E))))
        kw = dict(topk_idx=idx, topk_weights=w, num_experts=E, group_by_expert=grouped, use_fp8=form == "fp8", **lay)

        def flat(out):
            rx, ri, rw, cnt, h, _ = out
            ts = [*(rx if isinstance(rx, tuple) else (rx,)), ri, rw, h.recv_prob, h.recv_meta, h.send_row[:T], h.send_slot[:T]]
            return [t for t in ts if t is not None], cnt, h

        own, own_cnt, h = flat(buf.dispatch(x, **kw))
        view, cnt, _ = flat(buf.dispatch(x, zero_copy=True, **kw))
        want = [t.clone() for t in view]
        for _ in range(2):                                     # both parities of the region are written over
            buf.dispatch((x[0], x[1] + 1) if form == "tuple" else x + 1, zero_copy=True, **kw)
        again = buf.dispatch(x, handle=h, use_fp8=form == "fp8")[0]
        again = list(again) if isinstance(again, tuple) else [again]
        assert own_cnt == cnt and len(own) == len(want)
        assert h.n_recv == int((idx >= 0).sum() if grouped else (idx >= 0).any(1).sum())
        for a, b in zip(own, want):
            assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(raw(a), raw(b))
        assert own[0]._base is None                            # its own tensor, not a view of a larger one
        for a, b in zip(again, want):
            assert a.shape == b.shape and torch.equal(raw(a), raw(b))
        if form == "plain" and T:
            back = buf.combine(own[0], h)[0]
            n = (idx >= 0).sum(1) if grouped else (idx >= 0).any(1)
            torch.testing.assert_close(back.float(), (x.float() * n[:, None]).to(torch.bfloat16).float())
        buf.check_status()
    finally:
        buf.destroy()


# the count exchange as one CTA (T <= 256), as one cluster (several chunks per CTA, a last CTA with none, few and many
# buckets) and as a grid with an arrival counter (histograms beyond a cluster's shared memory); choices above eight
@pytest.mark.parametrize("R,T,E,K", [(1, 256, 8, 2), (1, 257, 8, 8), (2, 300, 64, 9), (1, 2047, 64, 8), (2, 4096, 256, 8),
                                     (4, 1025, 16, 3), (1, 60000, 256, 2), (2, 33, 32, 1)])
def test_row_order_of_the_count_exchange(R, T, E, K):
    H = 8
    g = torch.Generator().manual_seed(T)
    idxs = [torch.rand(T, E, generator=g).topk(K, dim=-1).indices for _ in range(R)]
    idxs[0][T // 3] = -1                                      # a token without choices
    grp = _group(R, 256 << 20)
    El = E // R
    try:
        # a row says who sent it: (rank, token) in two exact bf16 pairs of bytes
        xs = []
        for r in range(R):
            x = torch.zeros(T, H)
            x[:, 0], x[:, 1], x[:, 2] = r, torch.arange(T) // 256, torch.arange(T) % 256
            xs.append(x.to(torch.bfloat16).cuda())
        ci = [i.cuda() for i in idxs]
        for grouped in (True, False):
            lays = None if grouped else grp.get_dispatch_layout(ci, E)
            outs = grp.dispatch(xs, layouts=lays, topk_idx=ci, group_by_expert=grouped, num_experts=E)
            for d in range(R):
                src, tok = [], []
                if grouped:
                    for e in range(d * El, (d + 1) * El):
                        for r in range(R):
                            t = (idxs[r] == e).any(1).nonzero().flatten()
                            src.append(torch.full_like(t, r))
                            tok.append(t)
                else:
                    for r in range(R):
                        t = ((idxs[r] >= d * El) & (idxs[r] < (d + 1) * El)).any(1).nonzero().flatten()
                        src.append(torch.full_like(t, r))
                        tok.append(t)
                src, tok = torch.cat(src), torch.cat(tok)
                got = outs[d][0].float().cpu().long()
                assert got.shape[0] == src.numel()
                assert torch.equal(got[:, 0], src) and torch.equal(got[:, 1] * 256 + got[:, 2], tok)
        grp.check_status()
        grp.check_canaries()
    finally:
        grp.destroy()


# the handle alone says where a row went: the caller may refill the index tensor after dispatch (static buffers under graph
# replay, interleaved micro-batches), whether the choices are masked or name experts of another rank by then
@pytest.mark.parametrize("R", [1, 2, 4])
@pytest.mark.parametrize("pull", [False, True])
@pytest.mark.parametrize("change", ["masked", "moved"])
def test_combine_and_cached_dispatch_after_the_index_tensor_is_refilled(R, pull, change):
    T, H, E, K = 130, 256, 8, 3
    xs, idxs, ws = _mk(R, T, H, E, K, seed=31)
    for i in idxs:
        i[i == E - 1] = -1                                # an expert without rows: the last of the last rank
        i[0] = -1
    g = _group(R)
    try:
        cx, ci, cw = [x.cuda() for x in xs], [i.cuda() for i in idxs], [w.cuda() for w in ws]
        outs = g.dispatch(cx, topk_idx=ci, topk_weights=cw, group_by_expert=True, num_experts=E, zero_copy=pull)
        rows = [o[0].clone() for o in outs]
        for i in ci:
            i.copy_(torch.full_like(i, -1) if change == "masked" else (i + max(1, E // R)) % E)
        handles = [o[4] for o in outs]
        ys = [o[0].mul_(1 + d) if pull else o[0] * (1 + d) for d, o in enumerate(outs)]
        comb = g.combine(ys, handles, topk_weights=[h.recv_prob for h in handles])
        for r in range(R):
            valid = idxs[r] >= 0
            factor = torch.where(valid, 1.0 + idxs[r] // (E // R), torch.zeros(())).sum(1, keepdim=True)
            # factors up to 12 and bf16 rows: one rounding of the row's product, one of the sum
            torch.testing.assert_close(comb[r][0].cpu().float(), xs[r].float() * factor, rtol=2.0 ** -7, atol=1e-6)
            assert torch.equal(comb[r][1].cpu(), torch.where(valid, ws[r], torch.zeros(())))
        again = g.dispatch(cx, handles=handles)
        for d in range(R):
            assert torch.equal(again[d][0], rows[d])
        g.check_status()
        g.check_canaries()
    finally:
        g.destroy()


def _side_stream_buffer(nbytes, **kw):
    """A group of one whose asynchronous calls run on a communication stream, as those of a process group do."""
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    world = LocalWorld.make(1)[0]
    world.local = False
    return Buffer(None, nbytes, world=world, timeout_s=2.0, **kw)


@pytest.mark.parametrize("grouped", [False, True])
def test_asynchronous_calls_hold_what_their_kernels_read(grouped):
    T, H, E, K = 64, 256, 8, 2
    (x,), (idx,), (w,) = _mk(1, T, H, E, K)
    x, idx, w = x.cuda(), idx.cuda(), w.cuda()
    buf = _side_stream_buffer(32 << 20)
    held = lambda ev: {t.data_ptr() for t in ev.extra_tensors if isinstance(t, torch.Tensor)}
    try:
        _, _, per_expert, in_rank, ev = (None,) * 5 if grouped else buf.get_dispatch_layout(idx, E, async_finish=True)
        rx, _, rw, _, h, ev = buf.dispatch(x, topk_idx=idx, topk_weights=w, is_token_in_rank=in_rank, num_tokens_per_expert=per_expert,
                                           num_experts=E, group_by_expert=grouped, async_finish=True, previous_event=ev)
        read = [x, idx, w, h.send_row, h.send_slot, h.meta] + ([] if grouped else [in_rank, per_expert])
        assert {t.data_ptr() for t in read} <= held(ev)
        side = h.recv_prob if grouped else rw
        iw = torch.rand(T, K if grouped else 1, device="cuda")
        bias = torch.ones(T, H, dtype=torch.bfloat16, device="cuda")
        out, out_w, ev = buf.combine(rx, h, topk_weights=side, item_weights=iw, bias=bias, async_finish=True)
        read = [rx, side, iw, bias, h.send_row, h.send_slot, h.meta, h.recv_meta]
        assert {t.data_ptr() for t in read} <= held(ev)
        ev.current_stream_wait()
        want = x.float() * iw.sum(1, keepdim=True)
        torch.testing.assert_close(out.float(), want.to(torch.bfloat16).float() + 1, rtol=2.0 ** -7, atol=2.0 ** -7)
        assert torch.equal(out_w, w)
        buf.check_status()
    finally:
        buf.destroy()


def test_outgrown_scratch_is_kept_for_the_communication_stream():
    """Scratch made by a synchronous call and used by an asynchronous one: when a larger call replaces it while the
    communication stream still has work, the allocator may not hand the old blocks out on the caller's stream."""
    H, E, K = 256, 8, 2
    inputs = []
    for T in (64, 4096):
        (x,), (idx,), _ = _mk(1, T, H, E, K)
        inputs.append((x.cuda(), idx.cuda()))
    buf = _side_stream_buffer(96 << 20)
    kw = dict(num_experts=E, group_by_expert=True, zero_copy=True)
    pending = lambda: sum(b["state"] == "active_pending_free" for s in torch.cuda.memory_snapshot() for b in s["blocks"])
    try:
        (x, idx), (big, big_idx) = inputs
        keep = [buf.get_dispatch_layout(idx, E), buf.dispatch(x, topk_idx=idx, num_worst_tokens=64 * K, **kw)]
        torch.cuda.synchronize()
        before = pending()
        torch.cuda._sleep(1 << 29)                            # about a quarter of a second; the communication stream follows it
        keep.append(buf.dispatch(x, topk_idx=idx, num_worst_tokens=64 * K, async_finish=True, **kw))
        keep.append(buf.dispatch(big, topk_idx=big_idx, num_worst_tokens=4096 * K, async_finish=True, **kw))
        held_back = pending()
        keep[-1][5].current_stream_wait()
        torch.cuda.synchronize()
        assert held_back >= before + 2                        # item positions and chunk counts of the small call
        rows = torch.sort(big_idx.flatten(), stable=True).indices // K
        assert torch.equal(keep[-1][0], big[rows])
        buf.check_status()
    finally:
        buf.destroy()


@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("masked", [0.0, 0.4, 1.0])
def test_owned_outputs_hold_no_more_memory_than_their_rows(masked, grouped):
    from gpu_data_transfer_profile_b200.parallel.buffer import Buffer
    from gpu_data_transfer_profile_b200.parallel.symm import LocalWorld
    T, H, E, K = 300, 256, 8, 3
    g = torch.Generator().manual_seed(0)
    idx = torch.rand(T, E, generator=g).topk(K, dim=-1).indices
    idx[torch.rand(T, generator=g) < masked] = -1
    x, idx, w = torch.randn(T, H, generator=g).to(torch.bfloat16).cuda(), idx.cuda(), torch.rand(T, K, generator=g).cuda()
    buf = Buffer(None, 32 << 20, world=LocalWorld.make(1)[0], timeout_s=2.0)
    try:
        lay = {} if grouped else dict(zip(("num_tokens_per_rank", "is_token_in_rank"),
                                          (lambda l: (l[0], l[3]))(buf.get_dispatch_layout(idx, E))))
        for fp8 in (False, True):
            rx, ri, rw, _, h, _ = buf.dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E, group_by_expert=grouped,
                                               use_fp8=fp8, **lay)
            for t in [*(rx if fp8 else (rx,)), ri, rw, h.recv_prob, h.recv_meta]:
                if t is not None:
                    assert t.shape[0] == h.n_recv and t._base is None and t.untyped_storage().nbytes() == t.nbytes
        buf.check_status()
    finally:
        buf.destroy()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("R,pull", [(1, True), (1, False), (2, True), (2, False)])
@pytest.mark.parametrize("K", [1, 2, 3, 5, 9, 17, 32])
def test_combine_sums_in_order_whatever_the_number_of_contributors(K, R, pull, dtype):
    """Bit by bit the f32 sum over the choices in ascending order, rounded once: every form of the reduction, with rows
    read where they lie and from slots, some choices masked, a token without any, a row that ends inside a step."""
    T, H, E = 37, 264, 32
    g = torch.Generator().manual_seed(K)
    idxs = [torch.rand(T, E, generator=g).topk(K, dim=-1).indices for _ in range(R)]
    for i in idxs:
        i[torch.rand(T, K, generator=g) < 0.25] = -1
        i[3] = -1
    ws = [torch.rand(T, K, generator=g) for _ in range(R)]
    grp = _group(R, 64 << 20)
    try:
        outs = grp.dispatch([torch.randn(T, H, generator=g).to(dtype).cuda() for _ in range(R)], topk_idx=[i.cuda() for i in idxs],
                            topk_weights=[w.cuda() for w in ws], group_by_expert=True, num_experts=E, zero_copy=pull)
        handles = [o[4] for o in outs]
        values = [torch.randn(o[0].shape, generator=g).to(dtype) for o in outs]
        ys = [o[0].copy_(v) if pull else v.cuda() for o, v in zip(outs, values)]
        comb = grp.combine(ys, handles, topk_weights=[h.recv_prob for h in handles])
        got = [(c[0].cpu(), c[1].cpu()) for c in comb]
        rows = [h.send_row[:T].cpu() for h in handles]
        grp.check_status()
        grp.check_canaries()
    finally:
        grp.destroy()
    for r in range(R):
        acc = torch.zeros(T, H)
        for k in range(K):
            for d in range(R):
                t = (idxs[r][:, k] >= 0) & (idxs[r][:, k] // (E // R) == d)
                acc[t] += values[d][rows[r][t, k].long()].float()
        assert torch.equal(got[r][0], acc.to(dtype))
        assert torch.equal(got[r][1], torch.where(idxs[r] >= 0, ws[r], torch.zeros(())))


@pytest.mark.parametrize("zero_copy", [False, True])
@pytest.mark.parametrize("R", [2, 4])
def test_fc2_epilogue_combine_where_a_rank_receives_nothing(R, zero_copy):
    """All tokens go to experts of rank 0: the others' GEMMs have no rows and still tell their peers that they are done."""
    T, H, E, K = 70, 256, 8, 1
    El = E // R
    xs, idxs, ws = _mk(R, T, H, E, K, seed=4)
    idxs = [i % El for i in idxs]
    torch.manual_seed(1)
    g = _group(R, 64 << 20)
    try:
        w2s = [(torch.randn(El, H, H) * 0.05).to(torch.bfloat16) for _ in range(R)]
        for _ in range(3):                                    # both parities of the combine region, and one again
            outs = g.dispatch([x.cuda() for x in xs], topk_idx=[i.cuda() for i in idxs], topk_weights=[w.cuda() for w in ws],
                              group_by_expert=True, num_experts=E, zero_copy=zero_copy)
            assert [o[0].shape[0] for o in outs] == [R * T] + [0] * (R - 1)
            comb = g.fused_fc2_combine([o[0] for o in outs], [w.cuda() for w in w2s], [o[4] for o in outs])
            got = [c.cpu().float() for c in comb]
            g.check_status()
            for r in range(R):
                want = torch.einsum("th,tfh->tf", xs[r].float(), w2s[0][idxs[r][:, 0]].float())
                torch.testing.assert_close(got[r], want, atol=2e-3, rtol=2.0 ** -7)
        g.check_canaries()
    finally:
        g.destroy()
