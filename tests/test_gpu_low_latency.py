"""Low-latency dispatch / combine on one GPU with virtual ranks, against a plain PyTorch statement of the result."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(R, T, H, E, K, seed):
    g = torch.Generator().manual_seed(seed)
    xs = [(torch.randn(T - r, H, generator=g) * (1 + r)).bfloat16().cuda() for r in range(R)]
    idxs = []
    for r in range(R):
        idx = torch.rand(T - r, E, generator=g).topk(K, dim=-1).indices
        idx[torch.rand(idx.shape, generator=g) < 0.1] = -1
        idxs.append(idx.cuda())
    ws = [torch.rand(T - r, K, generator=g).cuda() for r in range(R)]
    return xs, idxs, ws


@pytest.mark.parametrize('R,T,H,E,K', [(2, 16, 256, 8, 2), (4, 33, 2048, 32, 4), (8, 32, 7168, 64, 8)])
@pytest.mark.parametrize('mode', ['bf16', 'fp8', 'fp8_round', 'ue8m0'])
@pytest.mark.parametrize('split', [False, True])
def test_low_latency_roundtrip(R, T, H, E, K, mode, split):
    from deepep_ascend_b200.backends.emulated import EmulatedWorld
    from deepep_ascend_b200.buffers.elastic import ElasticBuffer
    from deepep_ascend_b200.utils.math import per_token_cast_back, per_token_cast_to_fp8
    M = T + 3
    extra = ElasticBuffer.get_low_latency_size_hint(M, H, R, E, K)
    world = EmulatedWorld(R, num_max_tokens_per_rank=M, hidden=H, num_topk=K, extra_bytes=extra, num_gpu_timeout_secs=5)
    try:
        El = E // R
        for it in range(3):     # several calls: both buffer sets and the epoch tags get exercised
            xs, idxs, ws = _inputs(R, T, H, E, K, seed=it)
            use_fp8 = mode != 'bf16'
            stats = [torch.zeros(El, dtype=torch.int32, device='cuda') for _ in range(R)]
            outs = world.low_latency_dispatch(xs, idxs, M, E, use_fp8=use_fp8, round_scale=(mode == 'fp8_round'),
                                              use_ue8m0=(mode == 'ue8m0'), stats=stats, split_phases=split)
            torch.cuda.synchronize()
            for b in world.buffers:
                b.check_status()
            if use_fp8:
                ref = [per_token_cast_to_fp8(x.cpu(), round_scale=(mode == 'fp8_round'), use_ue8m0=(mode == 'ue8m0')) for x in xs]
            ys = []
            for d in range(R):
                recv, count, handle = outs[d]
                src_info, layout_range = handle[0].cpu(), handle[1].cpu()
                rx, rsf = (recv[0].cpu(), recv[1].cpu()) if use_fp8 else (recv.cpu(), None)
                y = torch.zeros(El, R * M, H, dtype=torch.bfloat16)
                for j in range(El):
                    e = d * El + j
                    total = 0
                    for s in range(R):
                        n, begin = int(layout_range[j, s]) & 0xffffffff, int(layout_range[j, s]) >> 32
                        want = sorted((idxs[s].cpu() == e).any(dim=1).nonzero().flatten().tolist())
                        info = src_info[j, begin:begin + n]
                        got_t, got_k = (info & 0xfffff).tolist(), (info >> 20).tolist()
                        assert sorted(got_t) == want, (d, j, s)
                        assert begin == total
                        total += n
                        for i, (t, k) in enumerate(zip(got_t, got_k)):
                            assert int(idxs[s][t, k]) == e
                            row = begin + i
                            if use_fp8:
                                assert torch.equal(rx[j, row].view(torch.uint8), ref[s][0][t].view(torch.uint8))
                                assert torch.equal(rsf[j, row], ref[s][1][t])
                                val = per_token_cast_back(ref[s][0][t:t + 1], ref[s][1][t:t + 1])[0]
                            else:
                                assert torch.equal(rx[j, row], xs[s][t].cpu())
                                val = xs[s][t].cpu()
                            y[j, row] = (val.float() * (1 + 0.25 * (e % 3))).bfloat16()
                    assert int(count[j]) == total and int(stats[d][j]) == total
                ys.append(y.cuda())
            res = world.low_latency_combine(ys, idxs, ws, [o[2] for o in outs], split_phases=split)
            torch.cuda.synchronize()
            for b in world.buffers:
                b.check_status()
            for s in range(R):
                x = xs[s].cpu()
                if use_fp8:
                    x = per_token_cast_back(*ref[s])
                idx, w = idxs[s].cpu(), ws[s].cpu()
                want = torch.zeros(x.shape[0], H)
                for k in range(K):
                    m = idx[:, k] >= 0
                    yk = (x[m].float() * (1 + 0.25 * (idx[m, k] % 3)).unsqueeze(1)).bfloat16().float()
                    want[m] += w[m, k].unsqueeze(1) * yk
                torch.testing.assert_close(res[s].cpu().float(), want.bfloat16().float(), atol=3e-2, rtol=2e-2)
    finally:
        world.destroy()


@pytest.mark.parametrize('R,T,H,E,K', [(2, 16, 256, 8, 2), (4, 33, 2048, 32, 4), (8, 32, 7168, 64, 8)])
@pytest.mark.parametrize('split', [False, True])
def test_low_latency_combine_logfmt(R, T, H, E, K, split):
    """Combine with LogFMT-10 rows on the wire: the result is the weighted sum of the CODED rows (stated in plain PyTorch by
    ``logfmt10_roundtrip``) and stays within the accuracy the reference asks of this mode (calc_diff against the exact
    sum, tests/legacy/test_low_latency.py:178-181).  Zero rows and rows of one repeated value are coded exactly."""
    from deepep_ascend_b200.backends.emulated import EmulatedWorld
    from deepep_ascend_b200.buffers.elastic import ElasticBuffer
    from deepep_ascend_b200.utils.math import calc_diff, logfmt10_roundtrip
    M = T + 1
    extra = ElasticBuffer.get_low_latency_size_hint(M, H, R, E, K)
    world = EmulatedWorld(R, num_max_tokens_per_rank=M, hidden=H, num_topk=K, extra_bytes=extra, num_gpu_timeout_secs=5)
    try:
        for it in range(3):
            xs, idxs, ws = _inputs(R, T, H, E, K, seed=40 + it)
            for x in xs:
                x[0] = 0                 # an all-zero row
                x[1, :128] = -1.5        # a group with a single magnitude
            outs = world.low_latency_dispatch(xs, idxs, M, E, use_fp8=False, split_phases=split)
            res = world.low_latency_combine([o[0] for o in outs], idxs, ws, [o[2] for o in outs], split_phases=split, use_logfmt=True)
            torch.cuda.synchronize()
            for r in range(R):
                world.buffers[r].check_status()
                wsum = (ws[r].cpu() * (idxs[r].cpu() >= 0)).sum(dim=1, keepdim=True)
                coded = logfmt10_roundtrip(xs[r].cpu()) * wsum
                exact = xs[r].cpu().float() * wsum
                got = res[r].cpu().float()
                assert bool(torch.isfinite(got).all())
                assert calc_diff(got, exact) < 2e-5, calc_diff(got, exact)
                torch.testing.assert_close(got, coded, atol=3e-2, rtol=3e-2)
                assert bool((got[0] == 0).all())
                torch.testing.assert_close(got[1, :128], (-1.5 * wsum[1]).expand(128).bfloat16().float(), atol=0, rtol=1e-2)
    finally:
        world.destroy()


@pytest.mark.parametrize('T,H,E,K', [(1, 128, 4, 1), (33, 2048, 32, 4), (128, 7168, 64, 8)])
@pytest.mark.parametrize('mode', ['bf16', 'fp8', 'ue8m0'])
@pytest.mark.parametrize('split', [False, True])
def test_one_rank_moves_rows_once(T, H, E, K, mode, split):
    """One rank: both halves in one launch place and reduce the rows directly, the split halves go through the slabs; same contract,
    and an output over the expert rows still reads all of them first."""
    test_low_latency_roundtrip(1, T, H, E, K, mode, split)
    from deepep_ascend_b200 import ElasticBuffer
    M = T + 3
    buf = ElasticBuffer(None, num_max_tokens_per_rank=M, hidden=H, num_topk=K,
                        extra_bytes=ElasticBuffer.get_low_latency_size_hint(M, H, 1, E, K) + (1 << 20))
    try:
        xs, idxs, ws = _inputs(1, T, H, E, K, seed=9)
        recv, _, handle, _, hook = buf.low_latency_dispatch(xs[0], idxs[0], M, E, use_fp8=False, return_recv_hook=split)
        if split:
            hook()
        want, _, hook = buf.low_latency_combine(recv, idxs[0], ws[0], handle, return_recv_hook=split)
        if split:
            hook()
        over = recv.view(-1, H)[:T]
        got, _, hook = buf.low_latency_combine(recv, idxs[0], ws[0], handle, out=over, return_recv_hook=split)
        if split:
            hook()
        torch.cuda.synchronize()
        buf.check_status()
        assert torch.equal(got, want)
    finally:
        buf.destroy()


def test_tensors_of_an_asynchronous_call_live_until_it_has_run():
    """With ``async_finish`` the kernels may still be waiting for the communication stream when the caller drops its inputs and allocates again."""
    from deepep_ascend_b200 import ElasticBuffer
    T, H, E, K = 32, 1024, 8, 2
    buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K,
                        extra_bytes=ElasticBuffer.get_low_latency_size_hint(T, H, 1, E, K) + (1 << 20))
    try:
        x0, idx0, w0 = torch.randn(T, H, device='cuda').bfloat16(), torch.rand(T, E, device='cuda').topk(K, dim=-1).indices, torch.rand(T, K, device='cuda')

        def run(late):
            tensors = [t.clone() for t in (x0, idx0, w0)]
            torch.cuda.synchronize()
            if late:
                with torch.cuda.stream(buf.comm_stream):
                    torch.cuda._sleep(20_000_000)                          # about 10 ms
            recv, count, handle, event, _ = buf.low_latency_dispatch(tensors[0], tensors[1], T, E, use_fp8=False, async_finish=late)
            del event
            tensors[0] = None
            later = [torch.full_like(x0, 7)]                               # where the rows lay, if their memory is free
            if late:
                with torch.cuda.stream(buf.comm_stream):
                    torch.cuda._sleep(20_000_000)
            out, event, _ = buf.low_latency_combine(recv, tensors[1], tensors[2], handle, async_finish=late)
            shapes = [(t.shape, t.dtype) for t in (recv, tensors[1], tensors[2], *handle[:2])]
            del event, recv, handle
            tensors.clear()
            later += [torch.full(shape, 1, dtype=dtype, device='cuda') for shape, dtype in shapes]
            torch.cuda.synchronize()
            buf.core.check_status()
            return out.clone(), count.clone()
        want = run(False)
        for _ in range(3):
            assert all(torch.equal(a, b) for a, b in zip(run(True), want))
    finally:
        buf.destroy()
