"""Edges of the exchange kernels: the fused cast at ragged row widths on one and on two ranks, and the kernels that move rows directly when
there is a single rank.  Everything is compared bitwise."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rows(T, H, seed):
    """N(0, 1) rows with the values a cast or a sum can trip over: zeros of both signs, subnormals, infinities, NaN, extremes."""
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(T, H, generator=g).bfloat16()
    special = torch.tensor([0.0, -0.0, 1e-40, -1e-40, 3.3e38, -3.3e38, float('inf'), float('-inf'), float('nan')]).bfloat16()
    at = torch.randint(0, T * H, (T * H // 97 + 9,), generator=g)
    x.view(-1)[at] = special[torch.arange(at.numel()) % special.numel()]
    x[T // 2, :128] = 0.0                                  # a scale group of zeros
    x[T - 1, -16:] = float('nan')
    return x.cuda()


def _routing(T, E, K, seed):
    g = torch.Generator().manual_seed(seed)
    idx = torch.rand(T, E, generator=g).topk(K, dim=-1).indices
    idx[torch.rand(T, K, generator=g) < 0.2] = -1
    idx[T // 3] = -1                                       # a token that goes nowhere
    return idx.cuda(), torch.rand(T, K, generator=g).cuda()


@pytest.mark.parametrize('R', [1, 2])
@pytest.mark.parametrize('T,H,sms', [(1, 128, 3), (3, 1024, 5), (37, 1152, 2), (64, 2048, 3), (90, 2176, 1), (41, 4096, 8), (130, 7168, 4)])
@pytest.mark.parametrize('mode', ['cast', 'fp8_in', 'bf16'])
@pytest.mark.parametrize('do_expand', [False, True])
def test_dispatch_rows_at_the_edges_of_a_batch(R, T, H, sms, mode, do_expand):
    """Rows of less than, exactly and more than one block (1024 channels) and one batch (2048) of the cast, whole and cut units of one
    rank's rows, fewer tokens than SMs and many per SM.  The cast is that of ``per_token_cast_to_fp8`` (another kernel)."""
    from deepep_ascend_b200.backends.emulated import EmulatedWorld
    from deepep_ascend_b200.ops import gemm as G
    from deepep_ascend_b200.utils import refs
    E, K, A = 8, 3, 4 if do_expand else 1
    world = EmulatedWorld(R, num_max_tokens_per_rank=T, hidden=H, num_topk=K, use_fp8_dispatch=mode != 'bf16', enable_expand=do_expand,
                          num_experts=E, expert_alignment=A)
    try:
        xs = [_rows(T, H, 10 * T + r) for r in range(R)]
        idxs, ws = zip(*[_routing(T, E, K, T + r) for r in range(R)])
        cast = [G.per_token_cast_to_fp8(x) for x in xs]
        ins = cast if mode == 'fp8_in' else xs
        for handles in (None, 'cached'):
            if handles is not None:
                outs = world.dispatch(ins, [None] * R, ws, E, num_sms=sms, handles=[o[3] for o in outs])
            else:
                outs = world.dispatch(ins, idxs, ws, E, num_sms=sms, expert_alignment=A, do_expand=do_expand)
            torch.cuda.synchronize()
            expect = refs.dispatch_all([q if mode != 'bf16' else x for (q, _), x in zip(cast, xs)],
                                       [sf for _, sf in cast] if mode != 'bf16' else None, list(idxs), list(ws), E, T, do_expand, A)
            for r, (x, idx, w, handle) in enumerate(outs):
                world.buffers[r].check_status()
                e, valid = expect[r], expect[r]['valid']
                x, sf = x if mode != 'bf16' else (x, None)
                assert torch.equal(x.cpu().view(torch.uint8)[valid], e['x'].cpu().view(torch.uint8)[valid])
                if sf is not None:
                    assert torch.equal(sf.cpu()[valid], e['sf'].cpu()[valid])
                if not do_expand:
                    assert torch.equal(idx.cpu(), e['idx'])
                assert torch.equal(w.cpu()[valid], e['w'][valid])
                assert torch.equal(handle.recv_src_metadata.cpu()[valid], e['meta'][valid])
    finally:
        world.destroy()


@pytest.mark.parametrize('fp8', [False, True])
def test_dispatch_with_every_number_of_warps(fp8):
    """1 to 20 warps on one rank, where 20 is the default; more are refused, and more than 12 with several ranks."""
    from deepep_ascend_b200 import ElasticBuffer
    from deepep_ascend_b200.backends.emulated import EmulatedWorld
    T, H, E, K = 45, 2176, 8, 3
    buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K, use_fp8_dispatch=fp8)
    try:
        x = _rows(T, H, 3)
        idx, w = _routing(T, E, K, 3)
        results = []
        for warps in (0, 20, 19, 13, 12, 7, 1):
            buf.set_dispatch_tuning(warps, 4 if warps == 7 else 0)
            rx, ri, rw, handle, _ = buf.dispatch(x, idx, w, num_experts=E, num_sms=3)
            results.append([t.clone().view(torch.uint8) for t in (*(rx if fp8 else (rx,)), ri.contiguous(), rw.contiguous(), handle.plan)])
        torch.cuda.synchronize()
        buf.check_status()
        for r in results[1:]:
            assert all(torch.equal(a, b) for a, b in zip(r, results[0]))
        with pytest.raises(AssertionError):
            buf.set_dispatch_tuning(21)
    finally:
        buf.destroy()
    world = EmulatedWorld(2, num_max_tokens_per_rank=T, hidden=H, num_topk=K)
    try:
        world.buffers[0].set_dispatch_tuning(12)
        with pytest.raises(AssertionError):
            world.buffers[0].set_dispatch_tuning(13)
    finally:
        world.destroy()


@pytest.mark.parametrize('T,H,sms', [(1, 128, 3), (5, 256, 2), (37, 1168, 1), (64, 2048, 3), (90, 4112, 7), (41, 7168, 64), (300, 7168, 4)])
def test_combine_of_one_rank_is_the_sum_of_one_row(T, H, sms):
    """Non-expand layout on one rank: every token has its row or none; the result has the bits of an fp32 sum that starts at zero
    (-0 becomes 0), and the carried weights come back.  With a bias the general kernel takes over on the same buffer."""
    from deepep_ascend_b200 import ElasticBuffer
    E, K = 8, 3
    buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K)
    try:
        idx, w = _routing(T, E, K, T)
        bias = torch.randn(T, H, device='cuda').bfloat16()
        for seed in (1, 2):
            _, _, rw, handle, _ = buf.dispatch(torch.zeros(T, H, dtype=torch.bfloat16, device='cuda'), idx, w, num_experts=E, num_sms=sms)
            y = _rows(max(1, handle.num_rows), H, seed)[:handle.num_rows]
            out, out_w, _ = buf.combine(y, handle, topk_weights=rw, num_sms=sms)
            with_bias, _, _ = buf.combine(y, handle, bias=bias, num_sms=sms)
            torch.cuda.synchronize()
            buf.core.check_status()
            sent = (idx >= 0).any(1)
            want = torch.zeros(T, H, device='cuda')
            want[sent] += y.float()
            for got, ref in ((out, want.bfloat16()), (with_bias, (want + bias.float()).bfloat16())):
                nan = ref.isnan()
                assert torch.equal(got.isnan(), nan)
                assert torch.equal(got.view(torch.int16)[~nan], ref.view(torch.int16)[~nan])
            assert torch.equal(out_w[idx >= 0], w[idx >= 0])
    finally:
        buf.destroy()


@pytest.mark.parametrize('T,H,E,K,sms', [(0, 256, 8, 2, 4), (1, 128, 4, 1, 148), (7, 1040, 8, 3, 148), (40, 7168, 256, 8, 0), (128, 2176, 1024, 16, 0),
                                         (300, 512, 24, 6, 5), (1024, 256, 16, 8, 0), (1100, 256, 16, 8, 0)])
@pytest.mark.parametrize('use_fp8', [False, True])
def test_low_latency_rows_of_one_rank(T, H, E, K, sms, use_fp8):
    """Rows cut into column parts (few tokens), several tokens per CTA, the most ids that are counted (8192) and more (slot claims).  Counted
    rows are in token order.  The combine in one launch has the bits of the two halves, which go through the slabs."""
    from deepep_ascend_b200 import ElasticBuffer
    from deepep_ascend_b200.ops import gemm as G
    M = T + 2
    buf = ElasticBuffer(None, num_max_tokens_per_rank=M, hidden=H, num_topk=K,
                        extra_bytes=ElasticBuffer.get_low_latency_size_hint(M, H, 1, E, K) + (1 << 20))
    try:
        x = torch.randn(T, H, device='cuda').bfloat16()
        idx, w = _routing(T, E, K, T) if T else (torch.zeros(0, K, dtype=torch.int64, device='cuda'), torch.zeros(0, K, device='cuda'))
        stats = torch.zeros(E, dtype=torch.int32, device='cuda')
        recv, count, handle, _, _ = buf.low_latency_dispatch(x, idx, M, E, stats, use_fp8=use_fp8, num_sms=sms)
        torch.cuda.synchronize()
        buf.core.check_status()
        t, k = (idx >= 0).nonzero(as_tuple=True)
        e = idx[t, k]
        want = torch.bincount(e, minlength=E)
        assert torch.equal(count.long(), want) and torch.equal(stats.long(), want)
        order = torch.sort(e * (T * K + 1) + t * K + k).indices                      # by expert, then in token order
        slot = torch.cat([torch.arange(int(n), device='cuda') for n in want]) if e.numel() else e
        rows, (t, k) = e[order] * M + slot, (t[order], k[order])
        info = handle[0].view(-1)[rows]
        if T * K > 8192:                                                              # claimed: any order inside an expert
            assert torch.equal(torch.sort(info).values, torch.sort((k << 20 | t).int()).values)
            t, k = info & 0xfffff, info >> 20
        assert torch.equal(info, (k << 20 | t).int())
        if use_fp8:
            q, sf = G.per_token_cast_to_fp8(x) if T else (x.to(torch.float8_e4m3fn), torch.zeros(0, H // 128, device='cuda'))
            assert torch.equal(recv[0].view(E * M, H)[rows].view(torch.uint8), q[t.long()].view(torch.uint8))
            assert torch.equal(recv[1].reshape(E * M, -1)[rows], sf[t.long()])
        else:
            assert torch.equal(recv.view(E * M, H)[rows], x[t.long()])
        y = torch.randn(E, M, H, device='cuda').bfloat16()
        out, _, _ = buf.low_latency_combine(y, idx, w, handle, num_sms=sms)
        split, _, hook = buf.low_latency_combine(y, idx, w, handle, return_recv_hook=True)
        hook()
        torch.cuda.synchronize()
        buf.core.check_status()
        assert torch.equal(out, split)
        exact = torch.zeros(T, H, dtype=torch.float64, device='cuda')
        exact.index_add_(0, t.long(), w[t.long(), k.long()].double()[:, None] * y.view(E * M, H)[rows].double())
        # one rounding to bf16 (2^-9 of the result) and up to 16 fp32 sums of terms below 1 * 6
        assert bool(((out.double() - exact).abs() <= exact.abs() * 2.0**-8 + 16 * 6 * 2.0**-23).all())
    finally:
        buf.destroy()


@pytest.mark.parametrize('sms', [1, 7, 148])
@pytest.mark.parametrize('use_fp8', [False, True])
def test_low_latency_expert_with_too_many_selections(sms, use_fp8):
    """Tokens that name an expert twice give it more selections than the rows it has.  The failure is reported while other CTAs start and
    end; whatever each of them sees of it, nothing is written outside the call's tensors."""
    from deepep_ascend_b200 import ElasticBuffer
    T, H, E, K = 96, 1024, 8, 4
    guards = [torch.full((1 << 22,), 0x5A, dtype=torch.uint8, device='cuda') for _ in range(4)]
    for attempt in range(4):
        buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K,
                            extra_bytes=ElasticBuffer.get_low_latency_size_hint(T, H, 1, E, K) + (1 << 20))
        try:
            idx = torch.arange(T * K, device='cuda').view(T, K) % E
            idx[:, 1] = idx[:, 0]                            # 0, 0, 2, 3 / 4, 4, 6, 7: experts 0 and 4 get T selections, T rows each: fits
            x = torch.randn(T, H, device='cuda').bfloat16()
            buf.low_latency_dispatch(x, idx, T, E, use_fp8=use_fp8, num_sms=sms)
            torch.cuda.synchronize()
            buf.core.check_status()
            idx[attempt, 2] = idx[attempt, 0]                # one more: does not fit
            buf.low_latency_dispatch(x, idx, T, E, use_fp8=use_fp8, num_sms=sms)
            torch.cuda.synchronize()
            code, _, peer, expected, observed, rank = buf.core.read_status()
            assert (code, peer, expected, rank) == (2, 0, T, 0) and observed >= T
            with pytest.raises(RuntimeError):
                buf.core.check_status()
            assert all(bool((g == 0x5A).all()) for g in guards)
        finally:
            buf.destroy()


@pytest.mark.parametrize('why', ['too_many_selections', 'failed_before'])
def test_low_latency_dispatch_that_gives_up_counts_nothing(why):
    """Work that is queued behind a call takes the counts before the host can look at the status: they are zero if the call gave up."""
    from deepep_ascend_b200 import ElasticBuffer
    T, H, E, K = 64, 512, 16, 4
    buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K, num_gpu_timeout_secs=0.2,
                        extra_bytes=ElasticBuffer.get_low_latency_size_hint(T, H, 1, E, K) + (1 << 20))
    try:
        idx = torch.arange(T * K, device='cuda').view(T, K) % E
        if why == 'too_many_selections':
            idx[:, 1] = 5
            idx[3] = 5
        x = torch.randn(T, H, device='cuda').bfloat16()
        stats = torch.full((E,), 3, dtype=torch.int32, device='cuda')
        with torch.cuda.stream(buf.comm_stream):             # what the call's small tensors will be made of
            old = [torch.full((n,), 77, dtype=torch.int32, device='cuda') for n in (E, E, 2 * E, E * T) for _ in range(4)]
        torch.cuda.synchronize()
        del old
        if why == 'failed_before':
            buf.core.wait_flag_test(7)                       # ends after 0.2 s with a failure; the call is queued behind it
        _, count, handle, _, _ = buf.low_latency_dispatch(x, idx, T, E, stats, num_sms=7)
        torch.cuda.synchronize()
        assert buf.core.read_status()[0] != 0
        assert not count.any() and not handle[1].any() and bool((stats == 3).all())
    finally:
        buf.destroy()


@pytest.mark.parametrize('T,H,E,K', [(1536, 128, 16, 4), (1537, 128, 16, 4), (2048, 256, 8, 4), (1024, 128, 8, 9), (1025, 512, 32, 2), (1536, 2048, 4, 1),
                                     (1537, 2048, 4, 1)])
@pytest.mark.parametrize('use_fp8', [False, True])
def test_low_latency_batches_on_both_sides_of_the_rules(T, H, E, K, use_fp8):
    """One launch (counted or claimed positions, searched or indexed rows) against the two halves, which go through the slabs."""
    from deepep_ascend_b200 import ElasticBuffer
    buf = ElasticBuffer(None, num_max_tokens_per_rank=2 * T, hidden=H, num_topk=K,
                        extra_bytes=ElasticBuffer.get_low_latency_size_hint(2 * T, H, 1, E, K) + (1 << 20))
    try:
        x = torch.randn(T, H, device='cuda').bfloat16()
        g = torch.Generator().manual_seed(T)
        idx = torch.randint(-1, E, (T, K), generator=g).cuda()             # an expert may be named twice
        idx[:, 0] = torch.where(torch.arange(T, device='cuda') % 3 == 0, 0, idx[:, 0])
        w = torch.rand(T, K, generator=g).cuda()
        packed = []
        for halves in (False, True):
            stats = torch.zeros(E, dtype=torch.int32, device='cuda')
            recv, count, handle, _, hook = buf.low_latency_dispatch(x, idx, 2 * T, E, stats, use_fp8=use_fp8, return_recv_hook=halves)
            if halves:
                hook()
            torch.cuda.synchronize()
            buf.core.check_status()
            assert torch.equal(count, stats) and torch.equal(handle[1].view(-1), count.long())
            rows = torch.arange(2 * T, device='cuda')[None] < count[:, None]
            info = torch.where(rows, handle[0], 1 << 30)
            order = info.sort(1).indices                                   # every expert's rows by (lane, token)
            data = [t.view(torch.uint8) if t.dtype == torch.float8_e4m3fn else t for t in (recv if use_fp8 else (recv,))]
            packed.append([count, info.gather(1, order)] + [d[torch.arange(E, device='cuda')[:, None], order][rows] for d in data])
            last = handle
        for a, b in zip(*packed):
            assert torch.equal(a, b)
        y = torch.randn(E, 2 * T, H, device='cuda').bfloat16()
        out, _, _ = buf.low_latency_combine(y, idx, w, last)
        split, _, hook = buf.low_latency_combine(y, idx, w, last, return_recv_hook=True)
        hook()
        torch.cuda.synchronize()
        buf.core.check_status()
        assert torch.equal(out, split)
    finally:
        buf.destroy()


@pytest.mark.parametrize('T,H,E,K', [(40, 256, 8, 4), (3000, 1024, 4, 2), (3000, 2048, 4, 4)])
def test_low_latency_on_more_sms_than_there_are(T, H, E, K):
    """160 SMs may be asked for with any batch; the kernels of large batches take what the GPU has."""
    from deepep_ascend_b200 import ElasticBuffer
    buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K,
                        extra_bytes=ElasticBuffer.get_low_latency_size_hint(T, H, 1, E, K) + (1 << 20))
    try:
        idx, w = _routing(T, E, K, T)
        x = torch.randn(T, H, device='cuda').bfloat16()
        outs = []
        for sms in (0, 160):
            recv, count, handle, _, _ = buf.low_latency_dispatch(x, idx, T, E, use_fp8=False, num_sms=sms)
            outs.append((count, buf.low_latency_combine(recv, idx, w, handle, num_sms=sms)[0]))
        torch.cuda.synchronize()
        buf.core.check_status()
        assert all(torch.equal(a, b) for a, b in zip(*outs))
    finally:
        buf.destroy()


@pytest.mark.parametrize('how', ['one_launch', 'halves'])
def test_low_latency_wait_statistics(how):
    """Waiting is added up where there is any: never in the one launch of a small batch, whose kernels wait for nobody."""
    from deepep_ascend_b200 import ElasticBuffer
    T, H, E, K = 16, 256, 8, 2
    buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K,
                        extra_bytes=ElasticBuffer.get_low_latency_size_hint(T, H, 1, E, K) + (1 << 20))
    try:
        idx, w = _routing(T, E, K, 4)
        sent, back = (torch.full((1,), 1000, dtype=torch.int64, device='cuda') for _ in range(2))
        x, halves = torch.randn(T, H, device='cuda').bfloat16(), how == 'halves'
        recv, _, handle, _, hook = buf.low_latency_dispatch(x, idx, T, E, dispatch_wait_recv_cost_stats=sent, use_fp8=False, return_recv_hook=halves)
        if halves:
            hook()
        _, _, hook = buf.low_latency_combine(recv, idx, w, handle, combine_wait_recv_cost_stats=back, return_recv_hook=halves)
        if halves:
            hook()
        torch.cuda.synchronize()
        buf.core.check_status()
        for stat in (sent, back):
            assert 1000 <= int(stat) < 10**9 if halves else int(stat) == 1000
    finally:
        buf.destroy()


def test_threads_with_streams_of_their_own():
    """Every thread has a buffer and a current stream; all share the communication stream and the code that orders streams against it."""
    import threading
    from deepep_ascend_b200 import ElasticBuffer
    T, H, E, K, n = 64, 1024, 16, 4, 3
    errors = []
    gate = threading.Barrier(n)

    def work(i):
        try:
            torch.cuda.set_device(0)
            with torch.cuda.stream(torch.cuda.Stream()):
                buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K)
                idx, w = _routing(T, E, K, i)
                sent = (idx >= 0).any(1)
                x = torch.zeros(T, H, dtype=torch.bfloat16, device='cuda')
                torch.cuda.current_stream().synchronize()
                gate.wait()
                for step in range(40):
                    x.fill_(100 * i + step)              # the dispatch has to wait for this, and this for the combine before it
                    y, _, _, handle, _ = buf.dispatch(x, idx, w, num_experts=E)
                    out, _, _ = buf.combine(y, handle)
                    if not bool((out == torch.where(sent, 100 * i + step, 0)[:, None]).all()):
                        errors.append((i, step))
                torch.cuda.current_stream().synchronize()
                buf.destroy()
        except Exception as e:                           # noqa: BLE001 (reported by the main thread)
            gate.abort()
            errors.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(n)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:5]
