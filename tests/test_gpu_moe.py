"""Fused MoE layer (dispatch -> FP8 grouped GEMM -> SwiGLU -> FP8 grouped GEMM -> weighted combine) and its
backward pass on one GPU (a group of one rank), against a plain fp32 PyTorch statement of the layer."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('copy_rows,chunks,local_expand', [(False, 1, True), (True, 1, True), (True, 2, True), (True, 4, True),
                                                          (False, 1, False), (True, 1, False), (True, 2, False)])
@pytest.mark.parametrize('T,H,I,E,K', [(200, 256, 128, 4, 2), (512, 1024, 512, 8, 4)])
def test_fused_moe_forward_backward(T, H, I, E, K, copy_rows, chunks, local_expand):
    from deepep_ascend_b200 import ElasticBuffer
    from deepep_ascend_b200.models.moe import FusedMoE, moe_reference
    from deepep_ascend_b200.utils.math import calc_diff
    torch.manual_seed(0)
    buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K, enable_expand=True, num_experts=E,
                        expert_alignment=128)
    try:
        layer = FusedMoE(buf, E, H, I, init_std=0.05, num_sms=16, copy_saved_rows=copy_rows, num_chunks=chunks, local_expand=local_expand)
        x = torch.randn(T, H, device='cuda').bfloat16().requires_grad_(True)
        scores = torch.softmax(torch.randn(T, E, device='cuda'), dim=-1)
        w, idx = scores.topk(K, dim=-1)
        idx[::7, 0] = -1
        w = w.clone().requires_grad_(True)
        out = layer(x, idx, w)
        g = torch.randn_like(out)
        out.backward(g)
        torch.cuda.synchronize()
        buf.check_status()

        xr = x.detach().float().requires_grad_(True)
        wr = w.detach().clone().requires_grad_(True)
        w13 = layer.w13.detach().float().requires_grad_(True)
        w2 = layer.w2.detach().float().requires_grad_(True)
        ref = moe_reference(xr, idx, wr, w13, w2)
        ref.backward(g.float())
        assert calc_diff(out.float(), ref) < 3e-3, calc_diff(out.float(), ref)
        assert calc_diff(x.grad.float(), xr.grad) < 3e-3, calc_diff(x.grad.float(), xr.grad)
        assert calc_diff(w.grad, wr.grad) < 3e-3, calc_diff(w.grad, wr.grad)
        assert calc_diff(layer.w2.grad.float(), w2.grad) < 3e-3, calc_diff(layer.w2.grad.float(), w2.grad)
        assert calc_diff(layer.w13.grad.float(), w13.grad) < 3e-3, calc_diff(layer.w13.grad.float(), w13.grad)
    finally:
        buf.destroy()


@pytest.mark.parametrize('T,H,I,E,K,chunks', [(200, 256, 128, 4, 2, 1), (512, 1024, 512, 8, 4, 2)])
def test_fused_moe_fp8_backward(T, H, I, E, K, chunks):
    """``fp8_backward=True``: the data-gradient GEMMs and the dispatch of the output gradient run in e4m3 with block scales.
    The gradients stay within the accuracy of an FP8 pipeline (calc_diff against the fp32 layer), and the forward
    result is the same as without the option."""
    from deepep_ascend_b200 import ElasticBuffer
    from deepep_ascend_b200.models.moe import FusedMoE, moe_reference
    from deepep_ascend_b200.utils.math import calc_diff
    torch.manual_seed(1)
    buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K, enable_expand=True, num_experts=E,
                        expert_alignment=128)
    try:
        layer = FusedMoE(buf, E, H, I, init_std=0.05, num_sms=16, num_chunks=chunks, fp8_backward=True)
        x = torch.randn(T, H, device='cuda').bfloat16().requires_grad_(True)
        w, idx = torch.softmax(torch.randn(T, E, device='cuda'), dim=-1).topk(K, dim=-1)
        idx[::5, 1] = -1
        w = w.clone().requires_grad_(True)
        out = layer(x, idx, w)
        g = torch.randn_like(out)
        out.backward(g)
        torch.cuda.synchronize()
        buf.check_status()
        layer.fp8_backward = False
        with torch.no_grad():
            assert torch.equal(layer(x, idx, w), out)
        xr, wr = x.detach().float().requires_grad_(True), w.detach().clone().requires_grad_(True)
        w13, w2 = layer.w13.detach().float().requires_grad_(True), layer.w2.detach().float().requires_grad_(True)
        moe_reference(xr, idx, wr, w13, w2).backward(g.float())
        diffs = dict(dx=calc_diff(x.grad.float(), xr.grad), dw=calc_diff(w.grad, wr.grad),
                     dw2=calc_diff(layer.w2.grad.float(), w2.grad), dw13=calc_diff(layer.w13.grad.float(), w13.grad))
        assert all(v < 5e-3 for v in diffs.values()), diffs
    finally:
        buf.destroy()


@pytest.mark.parametrize('rows,H,I', [(128, 256, 128), (640, 1024, 512)])
def test_backward_elementwise_kernels(rows, H, I):
    """The three element-wise kernels of the backward pass (row-major and transposed outputs) vs PyTorch."""
    from deepep_ascend_b200.ops import gemm as G
    from deepep_ascend_b200.utils.math import per_token_cast_to_fp8, per_token_cast_back
    torch.manual_seed(rows)
    valid = torch.rand(rows, device='cuda') > 0.2
    g = torch.randn(rows, H, device='cuda').bfloat16()
    y = torch.randn(rows, H, device='cuda').bfloat16()
    w = torch.rand(rows, device='cuda')
    dy, dy_t, dot = G.moe_bwd_prep(g, y, w, valid)
    vm = valid.unsqueeze(1)
    ref_dy = torch.where(vm, (g.float() * w.unsqueeze(1)).bfloat16(), torch.zeros_like(g))
    assert torch.equal(dy, ref_dy)
    assert torch.equal(dy_t, ref_dy.t().contiguous())
    ref_dot = torch.where(valid, (g.float() * y.float()).sum(1), torch.zeros_like(w))
    torch.testing.assert_close(dot, ref_dot, rtol=1e-4, atol=1e-3)

    d_act = torch.randn(rows, I, device='cuda').bfloat16()
    h = torch.randn(rows, 2 * I, device='cuda').bfloat16()
    dh, dh_t, act_t = G.swiglu_bwd(d_act, h, valid)
    gate, up, d = h[:, :I].float(), h[:, I:].float(), d_act.float()
    sig = torch.sigmoid(gate)
    ref_dh = torch.cat([d * up * sig * (1 + gate * (1 - sig)), d * gate * sig], dim=1)
    ref_dh = torch.where(vm, ref_dh, torch.zeros_like(ref_dh))
    ref_act = torch.where(vm, gate * sig * up, torch.zeros_like(gate))
    torch.testing.assert_close(dh.float(), ref_dh, rtol=2e-2, atol=2e-2)
    assert torch.equal(dh_t, dh.t().contiguous())
    torch.testing.assert_close(act_t.float(), ref_act.t(), rtol=2e-2, atol=2e-2)

    dh2, dh2_t, act2_t, dot2 = G.swiglu_bwd(d_act, h, valid, row_weight=w)
    ref_dh2 = torch.where(vm, ref_dh * w.unsqueeze(1), torch.zeros_like(ref_dh))
    torch.testing.assert_close(dh2.float(), ref_dh2, rtol=2e-2, atol=2e-2)
    assert torch.equal(dh2_t, dh2.t().contiguous()) and torch.equal(act2_t, act_t)
    ref_dot2 = torch.where(valid, (d * act_t.t().float()).sum(1), torch.zeros_like(w))
    torch.testing.assert_close(dot2, ref_dot2, rtol=1e-3, atol=1e-2)
    gw_t = G.weighted_transpose(g, w, valid)
    assert torch.equal(gw_t, ref_dy.t().contiguous())

    x = torch.randn(rows, H, device='cuda').bfloat16()
    q, sf = per_token_cast_to_fp8(x)
    x_t = G.dequant_transpose(q, sf, valid)
    ref_x = torch.where(vm, per_token_cast_back(q, sf).bfloat16(), torch.zeros_like(x))
    assert torch.equal(x_t, ref_x.t().contiguous())


def test_two_layers_share_one_buffer():
    """Two layers on ONE buffer, both forwards before any backward (what gradient accumulation and pipeline micro-batches
    do): the rows a layer keeps for its backward pass must survive the other layer's dispatches."""
    from deepep_ascend_b200 import ElasticBuffer
    from deepep_ascend_b200.models.moe import FusedMoE, moe_reference
    from deepep_ascend_b200.utils.math import calc_diff
    T, H, I, E, K = 256, 512, 256, 4, 2
    torch.manual_seed(3)
    buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K, enable_expand=True, num_experts=E, expert_alignment=128)
    try:
        layers = [FusedMoE(buf, E, H, I, init_std=0.05, num_sms=8) for _ in range(2)]
        xs, ws, idxs, outs, gs = [], [], [], [], []
        for layer in layers:
            x = torch.randn(T, H, device='cuda').bfloat16().requires_grad_(True)
            w, idx = torch.softmax(torch.randn(T, E, device='cuda'), dim=-1).topk(K, dim=-1)
            w = w.clone().requires_grad_(True)
            outs.append(layer(x, idx, w))
            xs.append(x), ws.append(w), idxs.append(idx), gs.append(torch.randn(T, H, device='cuda').bfloat16())
        for out, g in zip(outs, gs):
            out.backward(g)
        torch.cuda.synchronize()
        buf.check_status()
        for layer, x, w, idx, g in zip(layers, xs, ws, idxs, gs):
            xr, wr = x.detach().float().requires_grad_(True), w.detach().clone().requires_grad_(True)
            w13, w2 = layer.w13.detach().float().requires_grad_(True), layer.w2.detach().float().requires_grad_(True)
            moe_reference(xr, idx, wr, w13, w2).backward(g.float())
            assert calc_diff(x.grad.float(), xr.grad) < 3e-3 and calc_diff(w.grad, wr.grad) < 3e-3
            assert calc_diff(layer.w13.grad.float(), w13.grad) < 3e-3 and calc_diff(layer.w2.grad.float(), w2.grad) < 3e-3
    finally:
        buf.destroy()


@pytest.mark.parametrize('R', [2, 4])
def test_moe_forward_on_virtual_ranks(R):
    """The forward data flow of the layer across several ranks on one GPU (every collective of the virtual ranks is one
    cooperative launch): expand-layout FP8 dispatch -> grouped FP8 GEMMs with SwiGLU -> fused weighted combine, against the
    plain PyTorch layer that holds all experts."""
    from deepep_ascend_b200.backends.emulated import EmulatedWorld
    from deepep_ascend_b200.models.moe import moe_reference
    from deepep_ascend_b200.ops import gemm as G
    from deepep_ascend_b200.utils.math import calc_diff
    T, H, I, K = 160, 512, 256, 4
    E = 4 * R
    El = E // R
    torch.manual_seed(R)
    world = EmulatedWorld(R, num_max_tokens_per_rank=T, hidden=H, num_topk=K, use_fp8_dispatch=True, enable_expand=True,
                          num_experts=E, expert_alignment=128)
    try:
        w13 = (torch.randn(E, 2 * I, H, device='cuda') * 0.05).bfloat16()
        w2 = (torch.randn(E, H, I, device='cuda') * 0.05).bfloat16()
        xs = [torch.randn(T - r, H, device='cuda').bfloat16() for r in range(R)]
        tk = [torch.softmax(torch.randn(T - r, E, device='cuda'), dim=-1).topk(K, dim=-1) for r in range(R)]
        ws, idxs = [t[0].contiguous() for t in tk], [t[1].contiguous() for t in tk]
        outs = world.dispatch(xs, idxs, ws, E, num_sms=6, expert_alignment=128, do_expand=True)
        ys, handles = [], []
        for r, ((rx, rsf), _, recv_w, handle) in enumerate(outs):
            q13, s13 = G.quantize_weight_blocks(w13[r * El:(r + 1) * El].float())
            q2, s2 = G.quantize_weight_blocks(w2[r * El:(r + 1) * El].float())
            tile_group, _ = G.expert_tile_groups(handle.psum_num_recv_tokens_per_expert, handle.num_rows)
            h = G.grouped_gemm_nt(rx, q13, tile_group, sfa=rsf, sfb=s13, buffer=world.buffers[r])
            a2, sf2 = G.swiglu_quant(h)
            y = world.buffers[r].get_combine_buffer(handle)
            G.grouped_gemm_nt(a2, q2, tile_group, out=y, sfa=sf2, sfb=s2, buffer=world.buffers[r])
            ys.append(y)
            handles.append(handle)
        res = world.combine(ys, handles, weighted=True, num_sms=6)
        torch.cuda.synchronize()
        for r in range(R):
            world.buffers[r].check_status()
            ref = moe_reference(xs[r].float(), idxs[r], ws[r], w13.float(), w2.float())
            d = calc_diff(res[r][0].float(), ref)
            assert d < 3e-3, (r, d)
    finally:
        world.destroy()


def test_expert_segments_kernel_matches_its_pytorch_statement():
    """Tile groups, row validity and segment boundaries of the expand layout: the one-launch kernel against plain PyTorch."""
    from deepep_ascend_b200.ops import gemm as G
    torch.manual_seed(11)
    for trial in range(30):
        num_experts = int(torch.randint(1, 70, (1,)))
        alignment = 128 * int(torch.randint(1, 3, (1,)))
        counts = torch.randint(0, 700, (num_experts,))
        counts[torch.rand(num_experts) < 0.3] = 0
        ends, start = [], 0
        for c in counts.tolist():
            ends.append(start + c)
            start = (start + c + alignment - 1) // alignment * alignment
        rows = start + (64 if trial % 3 == 0 else 0)        # also a row count that is not a multiple of the tile
        ends_t = torch.tensor(ends, dtype=torch.int32, device='cuda')
        got = G.expert_segments(ends_t, rows, alignment)
        want = G.expert_segments_ref(ends_t, rows, alignment)
        for g, w in zip(got, want):
            assert g.dtype == w.dtype and torch.equal(g, w)
        assert torch.equal(G.segment_offsets(ends_t, alignment), want[2])


@pytest.mark.parametrize('rows,I', [(5, 128), (77, 384), (300, 2048), (40, 4352)])
def test_swiglu_quant_kernel(rows, I):
    """SwiGLU fused with the 1 x 128 e4m3 cast against plain PyTorch (I = 4352 takes more than 16 steps per row, I = 384
    ends in a half step)."""
    from deepep_ascend_b200.ops import gemm as G
    from deepep_ascend_b200.utils.math import calc_diff, per_token_cast_back
    torch.manual_seed(rows + I)
    h = (torch.randn(rows, 2 * I, device='cuda') * 2).bfloat16()
    h[0, :I] = -60.0                      # sigmoid underflows: the activation is 0 and the scale is clamped
    q, sf, act = G.swiglu_quant(h, keep_bf16=True)
    gate, up = h[:, :I].float(), h[:, I:].float()
    ref = (torch.nn.functional.silu(gate) * up)
    assert act.dtype == torch.bfloat16 and q.dtype == torch.float8_e4m3fn and sf.shape == (rows, I // 128)
    torch.testing.assert_close(act.float(), ref.bfloat16().float(), rtol=1.6e-2, atol=1e-6)
    # the scales are exactly amax / 448 of the bf16 activation the kernel produced, and the codes are its cast
    # (stated on the CPU: CUDA PyTorch turns a division by a constant into a multiplication by its reciprocal)
    act_c = act.float().cpu().view(rows, I // 128, 128)
    amax = act_c.abs().amax(dim=2).clamp(1e-4)
    assert torch.equal(sf.cpu(), amax / 448.0)
    want_q = (act_c * (448.0 / amax).unsqueeze(2)).view(rows, I).to(torch.float8_e4m3fn)
    assert torch.equal(q.cpu().view(torch.uint8), want_q.view(torch.uint8))
    assert calc_diff(per_token_cast_back(q, sf), ref) < 1e-3
    q2, sf2 = G.swiglu_quant(h)
    assert torch.equal(q2.view(torch.uint8), q.view(torch.uint8)) and torch.equal(sf2, sf)


@pytest.mark.parametrize('rows,K,El,H,idx_dtype', [(37, 2, 4, 256, torch.int64), (900, 8, 32, 1024, torch.int64), (513, 4, 7, 7168, torch.int32)])
def test_local_expand_and_reduce_kernels(rows, K, El, H, idx_dtype):
    """The (token, rank) -> (token, expert) expansion on the expert rank and its inverse, against plain PyTorch: positions
    ordered by received row inside 128-aligned expert segments, row / scale / weight copies, weighted and plain reductions."""
    from deepep_ascend_b200.ops import gemm as G
    g = torch.Generator().manual_seed(rows + K)
    # every row picks up to K distinct local experts; the other lanes (experts of other ranks) are -1
    idx = torch.full((rows, K), -1, dtype=torch.int64)
    for r in range(rows):
        n = int(torch.randint(0, min(K, El) + 1, (1,), generator=g))
        lanes = torch.randperm(K, generator=g)[:n]
        idx[r, lanes] = torch.randperm(El, generator=g)[:n]
    counts = torch.stack([(idx == e).sum() for e in range(El)])
    aligned = (counts + 127) // 128 * 128
    psum = aligned.cumsum(0).to(torch.int32)
    starts = psum - aligned.to(torch.int32)
    total = int(psum[-1])
    want_pos = torch.full((rows, K), -1, dtype=torch.int32)
    for e in range(El):
        rr, kk = torch.nonzero(idx == e, as_tuple=True)          # row-major order = received order
        want_pos[rr, kk] = starts[e] + torch.arange(len(rr), dtype=torch.int32)
    # the index tensor as dispatch returns it: rows with a pitch (a view into wider records)
    wide = torch.full((rows, K + 3), 77, dtype=idx_dtype, device='cuda')
    wide[:, :K] = idx.to(idx_dtype).cuda()
    pos, seg_end = G.local_expand_plan(wide[:, :K], psum.cuda())
    assert torch.equal(pos.cpu(), want_pos)
    assert torch.equal(seg_end.cpu(), (starts + counts.to(torch.int32)))

    x = torch.randn(rows, H, generator=g).bfloat16().cuda()
    sf = torch.rand(rows, H // 128, generator=g).cuda()
    w = torch.rand(rows, K, generator=g).cuda()
    x_e, sf_e, w_e = G.local_expand_copy(pos, x, total, sf=sf, w=w)
    valid = pos >= 0
    src_row = torch.nonzero(valid, as_tuple=True)[0]
    at = pos[valid].long()
    assert torch.equal(x_e[at], x[src_row]) and torch.equal(sf_e[at], sf[src_row]) and torch.equal(w_e[at], w[valid])
    q = x.view(torch.uint8)[:, :H].contiguous().view(torch.float8_e4m3fn)       # a one-byte element type takes the same path
    assert torch.equal(G.local_expand_copy(pos, q, total)[0][at].view(torch.uint8), q[src_row].view(torch.uint8))

    y = torch.zeros(total, H, dtype=torch.bfloat16, device='cuda')
    y[at] = torch.randn(len(at), H, device='cuda').bfloat16()
    for weights in (None, w_e):
        got = G.local_reduce(pos, y, w=weights)
        want = torch.zeros(rows, H, device='cuda')
        for k in range(K):
            m = valid[:, k]
            rowsel = y[pos[m, k].long()].float()
            want[m] += rowsel if weights is None else rowsel * weights[pos[m, k].long()].unsqueeze(1)
        torch.testing.assert_close(got.float(), want.bfloat16().float(), rtol=1.6e-2, atol=1e-3)
        assert bool((got[~valid.any(dim=1)] == 0).all())
    out = torch.empty(rows, H, dtype=torch.bfloat16, device='cuda')
    assert G.local_reduce(pos, y, w=w_e, out=out).data_ptr() == out.data_ptr()


def test_fused_moe_on_a_buffer_without_expand_regions():
    """With ``local_expand`` (the default) the layer only uses the (token, rank) layout of the buffer, so a buffer built without
    ``enable_expand`` serves it; without ``local_expand`` the constructor asks for the expand-capable buffer."""
    from deepep_ascend_b200 import ElasticBuffer
    from deepep_ascend_b200.models.moe import FusedMoE, moe_reference
    from deepep_ascend_b200.utils.math import calc_diff
    T, H, I, E, K = 300, 512, 256, 8, 4
    torch.manual_seed(21)
    buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K)      # rows sized for the bf16 gradients of the backward pass
    try:
        with pytest.raises(AssertionError, match='enable_expand'):
            FusedMoE(buf, E, H, I, local_expand=False)
        layer = FusedMoE(buf, E, H, I, init_std=0.05, num_sms=16)
        x = torch.randn(T, H, device='cuda').bfloat16().requires_grad_(True)
        w, idx = torch.softmax(torch.randn(T, E, device='cuda'), dim=-1).topk(K, dim=-1)
        w = w.clone().requires_grad_(True)
        out = layer(x, idx, w)
        g = torch.randn_like(out)
        out.backward(g)
        torch.cuda.synchronize()
        buf.check_status()
        xr, wr = x.detach().float().requires_grad_(True), w.detach().clone().requires_grad_(True)
        w13, w2 = layer.w13.detach().float().requires_grad_(True), layer.w2.detach().float().requires_grad_(True)
        ref = moe_reference(xr, idx, wr, w13, w2)
        ref.backward(g.float())
        assert calc_diff(out.float(), ref) < 3e-3 and calc_diff(x.grad.float(), xr.grad) < 3e-3
        assert calc_diff(layer.w13.grad.float(), w13.grad) < 3e-3 and calc_diff(w.grad, wr.grad) < 3e-3
    finally:
        buf.destroy()


@pytest.mark.parametrize('G,N,K', [(1, 128, 128), (3, 8, 8), (2, 129, 136), (2, 384, 2056), (1, 127, 7168)])
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float32])
def test_weight_block_cast_matches_pytorch(G, N, K, dtype):
    """The one-pass cast has the bits of the PyTorch statement: ragged edge blocks, an all-zero block (clamped amax), a block
    with an infinity, one with a NaN, and subnormal values."""
    from deepep_ascend_b200.ops import gemm as ops
    torch.manual_seed(N + K)
    w = (torch.randn(G, N, K, device='cuda') * 0.02).to(dtype)
    w[0, :128, :128] = 0
    w[-1, -1, -1] = 1e-39
    cases = [w]
    for special in (float('inf'), float('nan'), -float('inf')):
        v = w.clone()
        v[0, N // 2, K // 2] = special
        cases.append(v)
    for v in cases:
        q, sf = ops.quantize_weight_blocks(v)
        q_ref, sf_ref = ops.quantize_weight_blocks_ref(v.float())
        assert q.shape == q_ref.shape and sf.shape == sf_ref.shape
        assert torch.equal(q.view(torch.uint8), q_ref.view(torch.uint8))
        assert torch.equal(sf.view(torch.int32), sf_ref.view(torch.int32))


@pytest.mark.parametrize('rows,I,H', [(1, 128, 128), (67, 136, 144), (256, 2048, 7168)])
def test_row_major_backward_kernels(rows, I, H):
    """The row-major SwiGLU gradient and dequantisation against the transposing kernels' PyTorch statement: ragged rows, masked rows
    with NaN payloads give exact zeros."""
    from deepep_ascend_b200.ops import gemm as ops
    torch.manual_seed(rows)
    valid = torch.rand(rows, device='cuda') > 0.2
    vm = valid.unsqueeze(1)
    d_act, h = torch.randn(rows, I, device='cuda').bfloat16(), torch.randn(rows, 2 * I, device='cuda').bfloat16()
    w = torch.rand(rows, device='cuda')
    d_act[~valid], h[~valid] = float('nan'), float('nan')
    dh, act, dot = ops.swiglu_bwd_rows(d_act, h, valid, w)
    gate, up, d = h[:, :I].double(), h[:, I:].double(), d_act.double()
    sig = torch.sigmoid(gate)
    wd = w.double().unsqueeze(1)
    ref_dh = torch.where(vm, torch.cat([wd * d * up * sig * (1 + gate * (1 - sig)), wd * d * gate * sig], dim=1), 0.0)
    ref_act = torch.where(vm, gate * sig * up, 0.0)
    # one rounding to bf16 (2^-9 of the value) and the fp32 expression around __expf (a few 2^-22 relative)
    torch.testing.assert_close(dh.double(), ref_dh, rtol=2.0 ** -8, atol=1e-5)
    torch.testing.assert_close(act.double(), ref_act, rtol=2.0 ** -8, atol=1e-5)
    act16 = (gate * sig * up).float().bfloat16().double()
    ref_dot = torch.where(valid, (d * act16).sum(1), 0.0)
    scale = torch.where(valid, (d * act16).abs().sum(1), 0.0)
    assert bool(((dot.double() - ref_dot).abs() <= scale * 2.0 ** -8 + 1e-6).all())
    x = torch.randn(rows, H, device='cuda').bfloat16()
    q, sf = ops.per_token_cast_to_fp8(x)
    sf[~valid] = float('nan')
    out = ops.dequant_rows(q, sf, valid)
    ref = (q.float().view(rows, -1) * sf.repeat_interleave(128, dim=1)[:, :H]).bfloat16()
    assert torch.equal(out, torch.where(vm, ref, torch.zeros_like(ref)))
    out = ops.dequant_rows(q, sf, valid, row_weight=w)
    ref = (q.float().view(rows, -1) * (sf * w.unsqueeze(1)).repeat_interleave(128, dim=1)[:, :H]).bfloat16()
    assert torch.equal(out, torch.where(vm, ref, torch.zeros_like(ref)))
    x[~valid] = float('nan')
    ref = (x.float() * w.unsqueeze(1)).bfloat16()
    assert torch.equal(ops.weighted_rows(x, w, valid), torch.where(vm, ref, torch.zeros_like(ref)))


@pytest.mark.parametrize('rows,I', [(1, 128), (67, 384), (300, 1920), (256, 2048)])
def test_swiglu_backward_with_cast(rows, I):
    """The SwiGLU gradient that also leaves in e4m3: the bits of the kernel without and of the stand-alone cast of its result (whole and
    half steps of 256 channels, masked rows with NaN payloads, a row of zeros)."""
    from deepep_ascend_b200.ops import gemm as ops
    torch.manual_seed(rows + I)
    valid = torch.rand(rows, device='cuda') > 0.2
    d_act, h = torch.randn(rows, I, device='cuda').bfloat16(), torch.randn(rows, 2 * I, device='cuda').bfloat16()
    w = torch.rand(rows, device='cuda')
    w[0] = 0.0
    d_act[~valid], h[~valid] = float('nan'), float('nan')
    want = ops.swiglu_bwd_rows(d_act, h, valid, w)
    want = (*want, *ops.per_token_cast_to_fp8(want[0]))
    for got, ref in zip(ops.swiglu_bwd_rows_fp8(d_act, h, valid, w), want):
        assert got.shape == ref.shape and got.dtype == ref.dtype and torch.equal(got.view(torch.uint8), ref.view(torch.uint8))


@pytest.mark.parametrize('K', [1, 6, 8, 16])
def test_expand_copy_of_few_scale_columns(K):
    """Scale rows whose last 32-column step has fewer columns than there are top-k lanes (hidden 512 .. 5120)."""
    from deepep_ascend_b200.ops import gemm as ops
    torch.manual_seed(K)
    for G in (1, 4, 5, 31, 32, 33, 39, 40):
        rows = 50
        pos = torch.randperm(rows * K, device='cuda').to(torch.int32).view(rows, K)
        x, sf = torch.randn(rows, 64, device='cuda').bfloat16(), torch.randn(rows, G, device='cuda')
        out, sf_out = ops.local_expand_copy(pos, x, rows * K, sf=sf)
        for k in range(K):
            assert torch.equal(sf_out[pos[:, k].long()], sf) and torch.equal(out[pos[:, k].long()], x)


@pytest.mark.parametrize('rows', [1, 9, 64])
@pytest.mark.parametrize('H,I', [(64, 16), (1032, 272), (7168, 2048)])
def test_few_rows_are_split_by_columns(rows, H, I):
    """With few rows the element-wise kernels give several warps one row: the bits are those of the unsplit kernel, which the same
    rows take inside a tall tensor."""
    from deepep_ascend_b200.ops import gemm as ops
    torch.manual_seed(rows + H)
    K, tall = 8, 8 * 600
    h = torch.randn(tall, 2 * I, device='cuda').bfloat16()
    q, sf, act = ops.swiglu_quant(h, keep_bf16=True)
    q1, sf1, act1 = ops.swiglu_quant(h[:rows].contiguous(), keep_bf16=True)
    assert torch.equal(q1.view(torch.uint8), q[:rows].view(torch.uint8)) and torch.equal(sf1, sf[:rows]) and torch.equal(act1, act[:rows])
    pos = torch.randperm(tall * K, device='cuda').to(torch.int32).view(tall, K)[:, :K].contiguous()
    pos[torch.rand(tall, K, device='cuda') < 0.3] = -1
    y = torch.randn(tall * K, H, device='cuda').bfloat16()
    w = torch.rand(tall * K, device='cuda')
    assert torch.equal(ops.local_reduce(pos[:rows].contiguous(), y, w=w), ops.local_reduce(pos, y, w=w)[:rows])
    x, xs, xw = torch.randn(rows, H, device='cuda').bfloat16(), torch.randn(rows, (H + 127) // 128, device='cuda'), torch.rand(rows, K, device='cuda')
    out, s_out, w_out = ops.local_expand_copy(pos[:rows].contiguous(), x, tall * K, sf=xs, w=xw)
    r, k = torch.nonzero(pos[:rows] >= 0, as_tuple=True)
    at = pos[r, k].long()
    assert torch.equal(out[at], x[r]) and torch.equal(s_out[at], xs[r]) and torch.equal(w_out[at], xw[r, k])


@pytest.mark.parametrize('rows,K,El', [(0, 4, 8), (1, 1, 1), (511, 2, 3), (128, 8, 32), (128, 8, 512), (129, 8, 32), (64, 8, 513), (513, 16, 40), (20000, 8, 256), (300, 8, 1024)])
def test_expand_plan_over_many_ctas(rows, K, El):
    """Pairs over 1 to 148 CTAs, more experts than fit the default shared memory, ids outside the local range."""
    from deepep_ascend_b200.ops import gemm as ops
    torch.manual_seed(rows + El)
    idx = torch.randint(-1, El + 1, (rows, K), device='cuda')
    counts = torch.bincount(idx[(idx >= 0) & (idx < El)].flatten(), minlength=El)
    psum = ((counts + 127) // 128 * 128).cumsum(0).to(torch.int32)
    pos, seg_end = ops.local_expand_plan(idx, psum)
    want_pos, want_end = ops.local_expand_plan_ref(idx.cpu(), psum.cpu())
    assert torch.equal(pos.cpu(), want_pos) and torch.equal(seg_end.cpu(), want_end)
    # plan and segments together: one launch up to 1024 pairs and 512 experts, three otherwise
    for got, want in zip(ops.local_expand_layout(idx, psum, int(psum[-1])), ops.local_expand_layout(idx.cpu(), psum.cpu(), int(psum[-1]))):
        assert torch.equal(got.cpu(), want)


@pytest.mark.parametrize('rows,K,El', [(0, 2, 3), (1, 1, 1), (5, 3, 2), (64, 8, 32), (700, 6, 5)])
def test_weights_of_alignment_rows_are_zero(rows, K, El):
    """With `valid_row` the copy itself fills them, for rows that are split by columns and whole ones, with fewer and with more
    alignment rows than threads; without it, a launch in front does."""
    from deepep_ascend_b200.ops import gemm as ops
    torch.manual_seed(rows)
    idx = torch.stack([torch.randperm(max(K, El), device='cuda')[:K] for _ in range(rows)]) if rows else torch.empty(0, K, dtype=torch.int64, device='cuda')
    counts = torch.bincount(idx[idx < El].flatten(), minlength=El)
    psum = ((counts + 127) // 128 * 128).cumsum(0).to(torch.int32)
    num = int(psum[-1])
    pos, _, _, valid, _, _ = ops.local_expand_layout(idx, psum, num)
    x, w = torch.randn(rows, 256, device='cuda').bfloat16(), torch.rand(rows, K, device='cuda') + 1
    junk = torch.full((max(1, num),), float('nan'), device='cuda')         # what the allocator hands out next
    del junk
    x1, w1 = ops.local_expand_copy(pos, x, num, w=w, valid_row=valid)
    x0, w0 = ops.local_expand_copy(pos, x, num, w=w)
    assert torch.equal(w1, w0) and torch.equal(x1[valid], x0[valid]) and bool((w1[~valid] == 0).all()) and bool((w1[valid] >= 1).all())


@pytest.mark.parametrize('rows,K', [(0, 3), (1, 1), (85, 3), (5000, 8), (40000, 7)])
def test_local_gather(rows, K):
    """Less than a block, ragged blocks, more than the grid covers at once; a NaN in a row nobody asks for stays out."""
    from deepep_ascend_b200.ops import gemm as ops
    torch.manual_seed(rows)
    v = torch.randn(max(1, rows * K), device='cuda')
    v[0] = float('nan')
    pos = torch.randint(-1, v.numel(), (rows, K), device='cuda', dtype=torch.int32)
    pos[pos == 0] = -1
    assert torch.equal(ops.local_gather(pos, v), torch.where(pos >= 0, v[pos.clamp(min=0).long()], torch.zeros((), device='cuda')))


@pytest.mark.parametrize('counts', [[1, 31, 32, 33], [64, 0, 65, 96, 97], [127, 128, 129, 300, 0]])
def test_thin_tiles_are_read_and_stored_by_rows(counts):
    """Tiles with few token rows: results of those rows are those of the whole-tile product, other rows of the output and of the
    activation keep what they held."""
    from deepep_ascend_b200.ops import gemm as ops
    torch.manual_seed(len(counts))
    E, N, K = len(counts), 264, 384
    cnt = torch.tensor(counts)
    aligned = (cnt + 127) // 128 * 128
    ends = (aligned.cumsum(0) - aligned + cnt).to(torch.int32)
    rows = int(aligned.sum())
    tile_group, valid, seg_off, tile_rows = ops.expert_tiles(ends.cuda(), rows)
    for got, want in zip((tile_group, valid, seg_off, tile_rows), ops.expert_tiles(ends, rows)):
        assert torch.equal(got.cpu(), want)
    x = torch.randn(rows, K, device='cuda').bfloat16()
    q, sf = ops.per_token_cast_to_fp8(x)
    w, sw = ops.quantize_weight_blocks(torch.randn(E, N, K, device='cuda').bfloat16())
    want = ops.grouped_gemm_nt(q, w, tile_group, sfa=sf, sfb=sw)
    # rows without a token hold NaN in both operands' buffers
    q.view(torch.uint8)[~valid] = 0x7f
    sf[~valid] = float('nan')
    out = torch.full((rows, N), 7.0, dtype=torch.bfloat16, device='cuda')
    for num_sms in (0, 1, 3):
        ops.grouped_gemm_nt(q, w, tile_group, out=out, sfa=sf, sfb=sw, num_sms=num_sms, tile_rows=tile_rows)
        assert torch.equal(out[valid], want[valid]) and bool((out[~valid] == 7.0).all())
    h = torch.randn(rows, 512, device='cuda').bfloat16()
    a, s = ops.swiglu_quant(h)
    h[~valid] = float('nan')
    a1, s1 = ops.swiglu_quant(h, valid_row=valid)
    assert torch.equal(a1.view(torch.uint8)[valid], a.view(torch.uint8)[valid]) and torch.equal(s1[valid], s[valid])


@pytest.mark.parametrize('G,N,K,num_sms', [(64, 264, 1168, 0), (64, 264, 1168, 37), (8, 2056, 640, 0), (3, 1000, 6912, 5), (13, 2048, 16, 0), (16, 256, 128, 148)])
def test_products_that_stream_the_weights(G, N, K, num_sms):
    """Thin tiles, at most one per expert: the bits of the 256-column kernel (which takes the product when no tile_rows are given), with every
    number of token rows at which the kernel changes its way, idle tiles, two tiles of one group, a ragged last tile, odd K blocks,
    columns that end inside a tile, last waves that are cut and whole, and scales in either order; a count of the rows that rules the
    kernel out, or none, changes nothing."""
    from deepep_ascend_b200 import _native
    from deepep_ascend_b200.ops import gemm as ops
    gen = torch.Generator(device='cuda').manual_seed(N)
    edges = [1, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 96, 127, 128, 0, 40]
    tiles = min(G, 48)
    rows = torch.tensor([edges[(5 * t + G) % len(edges)] for t in range(tiles)], dtype=torch.int32, device='cuda')
    M = tiles * 128 - 72                                          # the last tile has 56 rows in the tensor
    rows[-1] = 128
    group = torch.arange(tiles, dtype=torch.int32, device='cuda') * G // tiles
    group[1] = group[0]
    group[2] = -1

    def e4m3(*shape):
        b = torch.randint(0, 256, shape, dtype=torch.uint8, device='cuda', generator=gen)
        return torch.where((b & 0x7f) == 0x7f, 0, b).to(torch.uint8).view(torch.float8_e4m3fn)
    a, w = e4m3(M, K), e4m3(G, N, K)
    sa = torch.rand(M, (K + 127) // 128, device='cuda', generator=gen) + 0.5
    sb = torch.rand(G, (N + 127) // 128, (K + 127) // 128, device='cuda', generator=gen) + 0.5
    want = ops.grouped_gemm_nt(a, w, group, sfa=sa, sfb=sb, num_sms=num_sms)
    at = torch.arange(M, device='cuda')
    valid = (at % 128 < rows[at // 128]) & (group[at // 128] >= 0)
    a.view(torch.uint8)[~valid] = 0x7f
    streams = _native.load().gemm_streams_weights
    for scales, bound in ((sa, 0), (sa, M), (sa.t().contiguous().t(), 1), (sa, 1)):
        assert streams(M, N, num_groups=G, total_rows=bound) == (bound == 1)
        out = torch.full((M, N + 8), 7.0, dtype=torch.bfloat16, device='cuda')
        ops.grouped_gemm_nt(a, w, group, out=out[:, :N], sfa=scales, sfb=sb, num_sms=num_sms, tile_rows=rows, total_rows=bound)
        assert torch.equal(out[valid, :N], want[valid]) and bool((out[~valid] == 7.0).all()) and bool((out[:, N:] == 7.0).all())
    # and the product itself (the streaming kernel's, of the last pass), in 64 bits: sums of K products in 32 bits and one rounding to bf16 (2^-8)
    k_scale = lambda s: s.repeat_interleave(128, dim=-1)[..., :K]    # noqa: E731
    for t in range(tiles):
        e, r = int(group[t]), min(int(rows[t]), M - t * 128)
        if e < 0 or r == 0:
            continue
        at = slice(t * 128, t * 128 + r)
        x = a[at].double() * k_scale(sa[at]).double()
        y = w[e].double() * k_scale(sb[e].repeat_interleave(128, dim=0)[:N]).double()
        exact = x @ y.t()
        bound = exact.abs() * 2.0**-8 + (x.abs() @ y.abs().t()) * K * 2.0**-24
        assert bool(((out[at, :N].double() - exact).abs() <= bound).all()), t


@pytest.mark.parametrize('local_expand', [True, False])
@pytest.mark.parametrize('tokens,K,streams', [(40, 2, True), (448, 1, True), (512, 2, False), (1024, 1, False)])
def test_the_layer_streams_weights_for_thin_tiles_only(monkeypatch, tokens, K, streams, local_expand):
    """Both layouts tell the products how many rows there are, forward and backward: 10 and 56 rows per expert are thin tiles, 128 are not."""
    from deepep_ascend_b200 import ElasticBuffer, _native
    from deepep_ascend_b200.models.moe import FusedMoE
    from deepep_ascend_b200.ops import gemm as ops
    E, H, I = 8, 512, 256
    routes, product, choice = [], ops.grouped_gemm_nt, _native.load().gemm_streams_weights

    def watched(a, b, tile_group, tile_rows=None, total_rows=0, **kw):
        counted = int(tile_rows[tile_group >= 0].sum())
        assert total_rows == counted == tokens * K                    # one rank, nothing dropped
        routes.append(choice(a.shape[0], b.shape[1], num_groups=E, total_rows=total_rows))
        return product(a, b, tile_group, tile_rows=tile_rows, total_rows=total_rows, **kw)
    monkeypatch.setattr(ops, 'grouped_gemm_nt', watched)
    buf = ElasticBuffer(None, num_max_tokens_per_rank=tokens, hidden=H, num_topk=K, enable_expand=not local_expand, num_experts=E,
                        expert_alignment=1 if local_expand else 128)
    try:
        layer = FusedMoE(buf, E, H, I, fp8_backward=True, local_expand=local_expand)
        x = torch.randn(tokens, H, device='cuda').bfloat16().requires_grad_(True)
        at = torch.arange(tokens, device='cuda').unsqueeze(1)
        idx = (at + torch.arange(K, device='cuda')) % E               # the same number of rows for every expert
        layer(x, idx, torch.full((tokens, K), 1.0 / K, device='cuda')).sum().backward()
    finally:
        buf.destroy()
    assert routes == [streams] * 4


@pytest.mark.parametrize('rows,H,I', [(128, 128, 128), (384, 7168, 384), (2048, 1024, 2048)])
@pytest.mark.parametrize('captured', [False, True])
def test_kernels_that_start_before_the_one_before_has_ended(rows, H, I, captured):
    """A chain of launches that may overlap, each reading what the one before it writes (one tile up to several waves, in a stream and in a
    CUDA graph): every pass gives the bytes that it gives when the host waits after each kernel.  Copies part the passes."""
    from deepep_ascend_b200.ops import gemm as ops
    torch.manual_seed(rows + I)
    passes = 12
    q0, s0 = ops.per_token_cast_to_fp8(torch.randn(passes * rows, H, device='cuda').bfloat16())
    w1, sw1 = ops.quantize_weight_blocks(torch.randn(1, 2 * I, H, device='cuda').bfloat16() * 0.1)
    w2, sw2 = ops.quantize_weight_blocks(torch.randn(1, H, I, device='cuda').bfloat16() * 0.1)
    group = torch.zeros(rows // 128, dtype=torch.int32, device='cuda')
    pos = torch.randperm(rows, device='cuda').view(rows // 2, 2).to(torch.int32)
    x = torch.empty(rows, H, dtype=q0.dtype, device='cuda')
    sf = torch.empty(rows, s0.shape[1], device='cuda')
    h, y = (torch.empty(rows, n, dtype=torch.bfloat16, device='cuda') for n in (2 * I, H))

    def run(pause):
        outs = []
        for i in range(passes):
            x.view(torch.uint8).copy_(q0[i * rows:(i + 1) * rows].view(torch.uint8))
            sf.copy_(s0[i * rows:(i + 1) * rows])
            ops.grouped_gemm_nt(x, w1, group, out=h, sfa=sf, sfb=sw1)
            pause()
            a, sa = ops.swiglu_quant(h)
            pause()
            ops.grouped_gemm_nt(a, w2, group, out=y, sfa=sa, sfb=sw2)
            pause()
            outs.append(ops.local_reduce(pos, y))
            pause()
            outs.append(ops.local_expand_copy(pos, outs[-1], rows)[0])
            pause()
        return outs
    want = run(torch.cuda.synchronize)
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = run(lambda: None)
        graph.replay()
        torch.cuda.synchronize()
    else:
        got = run(lambda: None)
    for g, w in zip(got, want):
        assert torch.equal(g.view(torch.int16), w.view(torch.int16))


@pytest.mark.parametrize('M,N,sms', [(128, 256, (0,)), (512, 1024, (0, 3)), (1024, 512, (2, 1)), (1024, 512, (1, 2, 0)), (2048, 2048, (148, 8))])
@pytest.mark.parametrize('captured', [False, True])
def test_launches_that_overwrite_what_the_one_before_reads(M, N, sms, captured):
    """Products and reductions write each other's operands in turn, so every launch overwrites what the one before it reads, without anything between
    them.  The numbers of SMs give products on both sides of the eight waves up to which launches overlap."""
    from deepep_ascend_b200.ops import gemm as ops
    torch.manual_seed(M + N)
    passes = 24
    x0 = torch.randn(M, N, device='cuda').bfloat16()
    w = (torch.randn(N, N, device='cuda') * N**-0.5).bfloat16()
    pos = torch.randperm(M, device='cuda').view(-1, 1).to(torch.int32)
    x, y = torch.empty_like(x0), torch.empty_like(x0)

    def run(pause):
        x.copy_(x0)
        for i in range(passes):
            ops.gemm_nt(x, w, out=y, num_sms=sms[i % len(sms)])
            pause()
            if i % 3 == 2:
                ops.gemm_nt(y, w, out=x, num_sms=sms[i % len(sms)])
            else:
                ops.local_reduce(pos, y, out=x)
            pause()
    run(torch.cuda.synchronize)
    want = x.clone()
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run(lambda: None)
        graph.replay()
    else:
        run(lambda: None)
    torch.cuda.synchronize()
    assert bool(want.any()) and torch.equal(x.view(torch.int16), want.view(torch.int16))


def _assert_a_dispatch_fits_beside(product):
    """`product` (about a millisecond on 16 SMs) with a kernel behind it, and a dispatch that is issued meanwhile: it ends long before they do."""
    from deepep_ascend_b200 import ElasticBuffer
    from deepep_ascend_b200.ops import gemm as ops
    T, H, E, K = 256, 1024, 16, 4
    y = torch.randn(1 << 17, 256, device='cuda').bfloat16()
    pos = torch.randperm(1 << 17, device='cuda').view(-1, 1).to(torch.int32)
    x, idx = torch.randn(T, H, device='cuda').bfloat16(), torch.rand(T, E, device='cuda').topk(K, dim=-1).indices
    buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K)
    side = torch.cuda.Stream()
    try:
        for attempt in range(3):
            start, sent, end = (torch.cuda.Event(enable_timing=True) for _ in range(3))
            torch.cuda.synchronize()
            start.record()
            product()
            ops.local_reduce(pos, y)
            end.record()
            with torch.cuda.stream(side):
                buf.dispatch(x, idx, num_experts=E, num_sms=24, do_cpu_sync=False)
                sent.record()
            torch.cuda.synchronize()
            times = start.elapsed_time(sent), start.elapsed_time(end)
            assert attempt == 0 or times[0] < 0.6 * times[1], times                         # the first pass may load code
    finally:
        buf.destroy()


def test_a_product_of_few_sms_leaves_the_others_to_an_exchange():
    """The kernel behind a product is launched early, but not so early that its waiting CTAs take the SMs that the product leaves free."""
    from deepep_ascend_b200.ops import gemm as ops
    a, b = (torch.randn(2048, 32768, device='cuda').bfloat16() for _ in range(2))           # 128 tiles: eight waves of 16 CTAs, over a millisecond
    out = torch.empty(2048, 2048, dtype=torch.bfloat16, device='cuda')
    _assert_a_dispatch_fits_beside(lambda: ops.gemm_nt(a, b, out=out, num_sms=16))


def test_a_product_of_few_sms_in_parts_leaves_the_others_to_an_exchange():
    """The same for a product whose K blocks are shared out, with the kernel that adds the parts behind it."""
    from deepep_ascend_b200 import _native
    from deepep_ascend_b200.ops import gemm as ops
    a, b = torch.randn(256, 1 << 20, device='cuda').bfloat16(), torch.randn(128, 1 << 20, device='cuda').bfloat16()     # 2 tiles in 8 parts
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert _native.load().gemm_split_plan(256, 128, 1 << 20, num_sms=16, device_sms=sms)[0] == 8
    _assert_a_dispatch_fits_beside(lambda: ops.gemm_nt(a, b, num_sms=16))


def test_a_product_of_few_sms_that_streams_weights_leaves_the_others_to_an_exchange():
    """The same for thin tiles: 128 tiles of 16 token rows, eight waves of 16 CTAs, 268 MB of weights."""
    from deepep_ascend_b200 import _native
    from deepep_ascend_b200.ops import gemm as ops
    G, N, K = 32, 512, 16384
    assert _native.load().gemm_streams_weights(G * 128, N, num_groups=G, total_rows=G * 16)
    a, w = torch.zeros(G * 128, K, dtype=torch.uint8, device='cuda'), torch.zeros(G, N, K, dtype=torch.uint8, device='cuda')
    sa, sb = torch.ones(G * 128, K // 128, device='cuda'), torch.ones(G, N // 128, K // 128, device='cuda')
    group, rows = torch.arange(G, dtype=torch.int32, device='cuda'), torch.full((G,), 16, dtype=torch.int32, device='cuda')
    _assert_a_dispatch_fits_beside(lambda: ops.grouped_gemm_nt(a.view(torch.float8_e4m3fn), w.view(torch.float8_e4m3fn), group, sfa=sa, sfb=sb, num_sms=16,
                                                               tile_rows=rows, total_rows=G * 16))


@pytest.mark.parametrize('rows,I', [(768, 2032), (1024, 2048), (1029, 1040), (1152, 2064), (4090, 1808), (4099, 4096), (12300, 2320)])
@pytest.mark.parametrize('masked', [False, True])
def test_swiglu_of_rows_that_are_split(rows, I, masked):
    """Single steps, two and more of them, chains that are halved, last pieces that are not whole: the bits of the same rows in small
    launches that are cut differently."""
    from deepep_ascend_b200 import _native
    from deepep_ascend_b200.ops import gemm as ops
    torch.manual_seed(rows + I)
    h = torch.randn(rows, 2 * I, device='cuda').bfloat16()
    valid = torch.rand(rows, device='cuda') > 0.5 if masked else None
    chunk = _native.load().swiglu_quant_col_chunk
    part = next(p for p in (40, 600) if chunk(p, I) != chunk(rows, I))
    at = torch.arange(rows, device='cuda')[valid] if masked else slice(None)
    got = ops.swiglu_quant(h, keep_bf16=True, valid_row=valid)
    want = [ops.swiglu_quant(h[r:r + part], keep_bf16=True) for r in range(0, rows, part)]
    for g, w in zip(got, (torch.cat(t) for t in zip(*[(q.view(torch.uint8), s, a) for q, s, a in want]))):
        assert torch.equal((g.view(torch.uint8) if g.dtype == torch.float8_e4m3fn else g)[at], w[at])


@pytest.mark.parametrize('rows,I', [(0, 128), (4, 0), (0, 0)])
@pytest.mark.parametrize('masked', [False, True])
def test_swiglu_of_nothing(rows, I, masked):
    """No rows or no channels: empty results and no launch."""
    from deepep_ascend_b200.ops import gemm as ops
    h = torch.empty(rows, 2 * I, dtype=torch.bfloat16, device='cuda')
    valid = torch.ones(rows, dtype=torch.bool, device='cuda') if masked else None
    q, sf, act = ops.swiglu_quant(h, keep_bf16=True, valid_row=valid)
    torch.cuda.synchronize()
    assert q.shape == act.shape == (rows, I) and sf.shape == (rows, (I + 127) // 128)


def _off_by_one(t):
    """The same values at a storage offset of one element."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    flat.view(torch.uint8)[t.element_size():].copy_(t.contiguous().view(-1).view(torch.uint8))
    return flat[1:].view(t.shape)


@pytest.mark.parametrize('name', ['swiglu_bwd_rows d_act', 'swiglu_bwd_rows h', 'weighted_rows', 'dequant_rows', 'swiglu_bwd d_act', 'swiglu_bwd h',
                                  'moe_bwd_prep g', 'moe_bwd_prep y', 'weighted_transpose', 'dequant_transpose', 'swiglu_quant',
                                  'swiglu_quant pitch', 'per_token_cast_to_fp8'])
def test_operands_off_their_alignment_are_refused(name):
    """Contiguous tensors that start (or whose rows start) between the kernel's vectors: an error on the host, no launch."""
    from deepep_ascend_b200.ops import gemm as ops
    rows, I, off = 64, 128, _off_by_one
    d, h, w = (torch.randn(rows, n, device='cuda').bfloat16() for n in (I, 2 * I, I))
    q, sf = ops.per_token_cast_to_fp8(d)
    rw, valid = torch.rand(rows, device='cuda'), torch.ones(rows, dtype=torch.bool, device='cuda')
    pitched = torch.randn(rows, 2 * I + 1, device='cuda').bfloat16()[:, :2 * I]
    call = {
        'swiglu_bwd_rows d_act': lambda: ops.swiglu_bwd_rows(off(d), h, valid, rw),
        'swiglu_bwd_rows h': lambda: ops.swiglu_bwd_rows(d, off(h), valid, rw),
        'weighted_rows': lambda: ops.weighted_rows(off(d), rw, valid),
        'dequant_rows': lambda: ops.dequant_rows(off(q), sf, valid),
        'swiglu_bwd d_act': lambda: ops.swiglu_bwd(off(d), h, valid),
        'swiglu_bwd h': lambda: ops.swiglu_bwd(d, off(h), valid),
        'moe_bwd_prep g': lambda: ops.moe_bwd_prep(off(d), w, rw, valid),
        'moe_bwd_prep y': lambda: ops.moe_bwd_prep(d, off(w), rw, valid),
        'weighted_transpose': lambda: ops.weighted_transpose(off(d), rw, valid),
        'dequant_transpose': lambda: ops.dequant_transpose(off(q), sf, valid),
        'swiglu_quant': lambda: ops.swiglu_quant(off(h)),
        'swiglu_quant pitch': lambda: ops.swiglu_quant(pitched),
        'per_token_cast_to_fp8': lambda: ops.per_token_cast_to_fp8(off(d)),
    }[name]
    with pytest.raises(RuntimeError):
        call()
    torch.cuda.synchronize()
    # a single row has no pitch
    got, want = ops.swiglu_quant(pitched[:1]), ops.swiglu_quant(pitched[:1].clone())
    assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(got, want))


@pytest.mark.parametrize('fp8_backward', [False, True])
@pytest.mark.parametrize('layout', ['odd offset', 'transposed storage'])
def test_layer_on_weights_that_are_views(layout, fp8_backward):
    """Weights inside a flat buffer (starting between two 16-byte pieces) or stored with other strides: forward and every gradient
    have the bits of the layer on ordinary weights."""
    from deepep_ascend_b200 import ElasticBuffer
    from deepep_ascend_b200.models.moe import FusedMoE
    T, H, I, E, K = 200, 256, 128, 4, 2
    torch.manual_seed(4)
    buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K)
    try:
        layer = FusedMoE(buf, E, H, I, init_std=0.05, num_sms=16, fp8_backward=fp8_backward)
        x, g = torch.randn(T, H, device='cuda').bfloat16().requires_grad_(True), torch.randn(T, H, device='cuda').bfloat16()
        w, idx = torch.softmax(torch.randn(T, E, device='cuda'), dim=-1).topk(K, dim=-1)
        w = w.clone().requires_grad_(True)

        def step():
            out = layer(x, idx, w)
            return (out.detach().clone(), *torch.autograd.grad(out, [x, w, layer.w13, layer.w2], g))
        want = step()
        for name in ('w13', 'w2'):
            p = getattr(layer, name)
            p.data = _off_by_one(p.data) if layout == 'odd offset' else p.data.transpose(1, 2).contiguous().transpose(1, 2)
            assert p.data_ptr() % 16 != 0 or not p.is_contiguous()
        got = step()
        torch.cuda.synchronize()
        buf.check_status()
        for a, b in zip(got, want):
            assert torch.equal(a, b)
    finally:
        buf.destroy()
