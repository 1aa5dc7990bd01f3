"""tcgen05 GEMM kernels against fp32 PyTorch references."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _C():
    from deepep_ascend_b200 import _native
    return _native.load()


@pytest.mark.parametrize('M,N,K', [(128, 128, 64), (128, 128, 256), (256, 384, 512), (1000, 520, 1096), (4096, 2048, 7168),
                                   (1024, 896, 1024), (2048, 7168, 512), (18944, 896, 64), (130, 1000, 1096)])
def test_bf16_gemm(M, N, K):
    """Shapes that take each of the three tile widths (128, 224 and 256 columns; the launcher picks by tile count)."""
    C = _C()
    g = torch.Generator(device='cuda').manual_seed(M + N)
    a = torch.randn(M, K, device='cuda', generator=g).bfloat16()
    b = torch.randn(N, K, device='cuda', generator=g).bfloat16()
    c = C.gemm_nt(a, b)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    ref = a.float() @ b.float().t()
    err = (c.float() - ref).abs().max().item()
    assert err <= 2e-2 * ref.abs().max().item() + 1e-2, err


def _quant_b(b):
    """[G, N, K] -> e4m3 with one fp32 scale per 128 x 128 block."""
    G, N, K = b.shape
    nb, kb = (N + 127) // 128, (K + 127) // 128
    bp = torch.zeros(G, nb * 128, kb * 128, device=b.device)
    bp[:, :N, :K] = b
    blocks = bp.view(G, nb, 128, kb, 128)
    amax = blocks.abs().amax(dim=(2, 4)).clamp(1e-4)
    q = (blocks * (448.0 / amax)[:, :, None, :, None]).to(torch.float8_e4m3fn).view(G, nb * 128, kb * 128)[:, :N, :K].contiguous()
    return q, (amax / 448.0).contiguous()


@pytest.mark.parametrize('M,N,K,G', [(128, 128, 128, 1), (256, 256, 512, 1), (512, 384, 1024, 4), (1024, 2048, 7168, 8)])
def test_fp8_blockscaled_grouped_gemm(M, N, K, G):
    from deepep_ascend_b200.utils.math import per_token_cast_back
    C = _C()
    g = torch.Generator(device='cuda').manual_seed(K + G)
    a = torch.randn(M, K, device='cuda', generator=g).bfloat16()
    b = torch.randn(G, N, K, device='cuda', generator=g) * 0.1
    qa, sfa = C.per_token_cast_to_fp8(a, False, False)
    qb, sfb = _quant_b(b)
    tiles = (M + 127) // 128
    tile_group = (torch.arange(tiles, device='cuda', dtype=torch.int32) % G).contiguous()
    if tiles > 2:
        tile_group[1] = -1
    c = torch.full((M, N), 7.0, device='cuda', dtype=torch.bfloat16)
    C.gemm_nt(qa, qb, sfa, sfb, tile_group, c)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    a_deq = per_token_cast_back(qa, sfa).float()
    kb = (K + 127) // 128
    for t in range(tiles):
        rows = slice(t * 128, min(M, (t + 1) * 128))
        grp = int(tile_group[t])
        if grp < 0:
            assert bool((c[rows] == 7.0).all())
            continue
        b_deq = qb[grp].float().view(N, -1) * sfb[grp].repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)[:, :K]
        ref = a_deq[rows] @ b_deq.t()
        err = (c[rows].float() - ref).abs().max().item()
        assert err <= 2e-2 * ref.abs().max().item() + 1e-2, (t, err)


@pytest.mark.parametrize('M,N,segs', [(128, 128, [64, 0, 192]), (384, 520, [128, 256, 0, 0, 640]), (2048, 7168, [1152, 1024, 0, 1280])])
def test_k_grouped_gemm(M, N, segs):
    """out[e] = a_t[:, seg_e] @ b_t[:, seg_e]^T (weight gradients of a grouped layer); empty segments give zeros."""
    from deepep_ascend_b200.ops import gemm as G
    C = _C()
    g = torch.Generator(device='cuda').manual_seed(M + N)
    K = sum(segs)
    a_t = torch.randn(M, K, device='cuda', generator=g).bfloat16()
    b_t = torch.randn(N, K, device='cuda', generator=g).bfloat16()
    off = torch.tensor([0] + list(torch.tensor(segs).cumsum(0)), dtype=torch.int32, device='cuda')
    out = G.gemm_kgrouped(a_t, b_t, off)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    assert out.shape == (len(segs), M, N)
    k0 = 0
    for e, n in enumerate(segs):
        ref = a_t[:, k0:k0 + n].float() @ b_t[:, k0:k0 + n].float().t()
        err = (out[e].float() - ref).abs().max().item()
        assert err <= 2e-2 * max(ref.abs().max().item(), 1.0) + 1e-2, (e, err)
        if n == 0:
            assert out[e].abs().max().item() == 0
        k0 += n


@pytest.mark.parametrize('M,N,K,G', [(128, 128, 64, 1), (256, 256, 128, 2), (300, 520, 72, 3), (640, 136, 200, 4), (1000, 1032, 1096, 2)])
def test_grouped_gemm_reads_mn_major_weights(M, N, K, G):
    """a [M, K] @ b[group] [K, N] without a transposed copy: edge tiles in M, N and K, skipped tiles.  A K tail must not pick up the
    next group's rows: the last group is followed by nothing, the others by NaN-free but different weights."""
    from deepep_ascend_b200.ops import gemm as ops
    C = _C()
    g = torch.Generator(device='cuda').manual_seed(M + N + K)
    a = torch.randn(M, K, device='cuda', generator=g).bfloat16()
    b = torch.randn(G, K, N, device='cuda', generator=g).bfloat16()
    tiles = (M + 127) // 128
    tile_group = torch.tensor([t % (G + 1) - 1 for t in range(tiles)], dtype=torch.int32, device='cuda')
    out = torch.full((M, N), 7.0, dtype=torch.bfloat16, device='cuda')
    ops.grouped_gemm_nn(a, b, tile_group, out=out)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0
    for t in range(tiles):
        rows, grp = slice(t * 128, min(M, (t + 1) * 128)), int(tile_group[t])
        if grp < 0:
            assert bool((out[rows] == 7.0).all())
            continue
        ref = a[rows].double() @ b[grp].double()
        # fp32 sums rounded once to bf16: half an ulp (2^-9) of the value plus K fp32 roundings of the summed magnitudes
        bound = ref.abs() * 2.0 ** -8 + (a[rows].double().abs() @ b[grp].double().abs()) * K * 2.0 ** -24 + 1e-6
        assert bool(((out[rows].double() - ref).abs() <= bound).all()), t


@pytest.mark.parametrize('M,N,segs', [(128, 128, [64, 0, 192]), (384, 520, [128, 256, 0, 0, 640]), (136, 264, [64]), (2048, 7168, [1152, 1024, 0, 1280])])
def test_k_grouped_gemm_on_row_major_operands(M, N, segs):
    """out[e] = a[seg_e]^T @ b[seg_e]; empty segments give zeros; strided rows."""
    from deepep_ascend_b200.ops import gemm as ops
    C = _C()
    g = torch.Generator(device='cuda').manual_seed(M + N)
    K = sum(segs)
    a = torch.randn(K, M + 8, device='cuda', generator=g).bfloat16()[:, :M]
    b = torch.randn(K, N, device='cuda', generator=g).bfloat16()
    off = torch.tensor([0] + list(torch.tensor(segs).cumsum(0)), dtype=torch.int32, device='cuda')
    out = ops.gemm_kgrouped_tn(a, b, off)
    torch.cuda.synchronize()
    assert C.gemm_error(0) == 0 and out.shape == (len(segs), M, N)
    k0 = 0
    for e, n in enumerate(segs):
        ref = a[k0:k0 + n].double().t() @ b[k0:k0 + n].double()
        bound = ref.abs() * 2.0 ** -8 + (a[k0:k0 + n].double().abs().t() @ b[k0:k0 + n].double().abs()) * max(n, 1) * 2.0 ** -24 + 1e-6
        assert bool(((out[e].double() - ref).abs() <= (bound if n else 0)).all()), e
        k0 += n


@pytest.mark.parametrize('M,N,K,num_sms', [(64, 128, 8000, 0), (130, 264, 2056, 0), (74, 832, 5704, 0), (300, 256, 7168, 13), (512, 1024, 5000, 0), (1, 8, 1600, 0),
                                           (129, 1032, 5000, 40)])
@pytest.mark.parametrize('captured', [False, True])
def test_products_whose_k_blocks_are_shared_out(M, N, K, num_sms, captured):
    """Few tiles and a long K: parts of uneven length, a last K block that is not whole, ragged tiles; the same bits on every pass, in a stream and
    from a CUDA graph, with the products following one another closely (their workspaces are reused)."""
    from deepep_ascend_b200.ops import gemm as ops
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert _C().gemm_split_plan(M, N, K, num_sms=num_sms or sms, device_sms=sms)[0] > 1
    gen = torch.Generator(device='cuda').manual_seed(M + N + K)
    a, b = torch.randn(M, K, device='cuda', generator=gen).bfloat16(), torch.randn(N, K, device='cuda', generator=gen).bfloat16()
    first = ops.gemm_nt(a, b, num_sms=num_sms)
    exact = a.double() @ b.double().t()
    # fp32 sums rounded once to bf16: half an ulp (2^-9) of the value plus K fp32 roundings of the summed magnitudes
    bound = exact.abs() * 2.0 ** -8 + (a.double().abs() @ b.double().abs().t()) * K * 2.0 ** -24 + 1e-6
    assert bool(((first.double() - exact).abs() <= bound).all())

    def passes():
        return [ops.gemm_nt(a * s, b, num_sms=num_sms) for s in (1.0, 2.0, 4.0, 1.0)]
    if captured:
        graph = torch.cuda.CUDAGraph()
        passes()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            results = passes()
        for _ in range(3):
            graph.replay()
    else:
        results = passes()
    for got, s in zip(results, (1.0, 2.0, 4.0, 1.0)):        # powers of two: the same roundings
        assert torch.equal(got, first * s)


@pytest.mark.parametrize('M,N,K', [(64, 128, 8000), (130, 264, 2056), (512, 1024, 5000), (1, 8, 1600), (300, 256, 7168)])
def test_products_into_given_memory_are_summed_in_one_chain(M, N, K):
    """Shapes whose K blocks are shared out otherwise: with `out` nothing is allocated, and the bits of a row are those of the same row
    among others, on any number of SMs and in a result with a pitch."""
    from deepep_ascend_b200 import _native
    from deepep_ascend_b200.ops import gemm as ops
    assert _native.load().gemm_split_plan(M, N, K, num_sms=148, device_sms=148)[0] > 1
    gen = torch.Generator(device='cuda').manual_seed(M + N + K)
    b = torch.randn(N, K, device='cuda', generator=gen).bfloat16()
    a = torch.randn(20000, K, device='cuda', generator=gen).bfloat16()
    many = torch.empty(20000, N, dtype=torch.bfloat16, device='cuda')
    ops.gemm_nt(a, b, out=many)
    full = torch.empty(M + 1, N + 8, dtype=torch.bfloat16, device='cuda')
    for num_sms in (0, 24, 100, 1):
        full.fill_(7.0)
        out, rows = full[:M, :N], a[:M]
        before = torch.cuda.memory_stats()['allocation.all.allocated']
        ops.gemm_nt(rows, b, out=out, num_sms=num_sms)
        assert torch.cuda.memory_stats()['allocation.all.allocated'] == before
        assert torch.equal(out, many[:M]) and bool((full[M] == 7.0).all()) and bool((full[:, N:] == 7.0).all())


@pytest.mark.parametrize('M,N,K,num_sms', [(128, 256, 128, 0), (300, 264, 256, 0), (513, 520, 1152, 2), (200, 1032, 384, 1),
                                           (130, 256, 128, 1), (200, 1000, 384, 1), (513, 504, 1152, 2), (300, 1016, 256, 2)])
@pytest.mark.parametrize('fp8', [False, True])
def test_output_rows_leave_through_shared_memory(M, N, K, num_sms, fp8):
    """Ragged last rows and columns of 256-column tiles, several tiles per CTA, an output with a row pitch whose padding must not be
    touched.  bf16 takes tiles of 256 columns in the last four cases; in the others those of 224 columns, stored directly, cost less."""
    from deepep_ascend_b200.ops import gemm as ops
    from deepep_ascend_b200.utils.math import per_token_cast_to_fp8
    gen = torch.Generator(device='cuda').manual_seed(M + N)
    a = torch.randn(M, K, device='cuda', generator=gen).bfloat16()
    w = torch.randn(1, N, K, device='cuda', generator=gen).bfloat16()
    tile_group = torch.zeros((M + 127) // 128, dtype=torch.int32, device='cuda')
    full = torch.full((M + 1, N + 24), 7.0, dtype=torch.bfloat16, device='cuda')
    out = full[:M, :N]
    if fp8:
        q, sf = per_token_cast_to_fp8(a)
        qw, sw = ops.quantize_weight_blocks(w)
        ops.grouped_gemm_nt(q, qw, tile_group, out=out, sfa=sf, sfb=sw, num_sms=num_sms)
        a = q.double() * sf.double().repeat_interleave(128, 1)[:, :K]
        w = qw.double() * sw.double().repeat_interleave(128, 1)[:, :N].repeat_interleave(128, 2)[:, :, :K]
    else:
        ops.grouped_gemm_nt(a, w, tile_group, out=out, num_sms=num_sms)
    torch.cuda.synchronize()
    assert _C().gemm_error(0) == 0
    a, b_t = a.double(), w[0].double().t()
    ref = a @ b_t
    # fp32 sums (and, for e4m3, one fp32 product with the scales per 128 channels) rounded once to bf16
    bound = ref.abs() * 2.0 ** -8 + (a.abs() @ b_t.abs()) * K * 2.0 ** -24 + 1e-6
    assert bool(((out.double() - ref).abs() <= bound).all())
    assert bool((full[M:] == 7.0).all()) and bool((full[:, N:] == 7.0).all())


@pytest.mark.parametrize('M,N,K', [(128, 128, 128), (512, 768, 1024), (1300, 512, 512)])
@pytest.mark.parametrize('named', [False, True])
def test_rows_announced_by_flags(M, N, K, named):
    """A product whose row tiles are announced by flags, all of them set before the launch, with other kernels of the library in front of and behind it."""
    from deepep_ascend_b200 import _native
    from deepep_ascend_b200.ops import gemm as G
    C = _native.load()
    torch.manual_seed(M)
    a, b = torch.randn(M, K, device='cuda').bfloat16(), torch.randn(N, K, device='cuda').bfloat16()
    tiles = (M + 127) // 128
    flags = torch.full((2 * tiles,), 4, dtype=torch.int64, device='cuda')
    of_tile = torch.arange(2 * tiles - 1, tiles - 1, -1, dtype=torch.int32, device='cuda') if named else None
    flags[(of_tile if named else torch.arange(tiles, device='cuda')).long()] = 5
    pos = torch.randperm(M, device='cuda')[:M // 2 * 2].view(-1, 2).to(torch.int32)
    want = G.gemm_nt(a, b)
    torch.cuda.synchronize()
    reduced = G.local_reduce(pos, want)
    for _ in range(3):
        copy = G.local_expand_copy(torch.arange(M, device='cuda', dtype=torch.int32)[:, None], a, M)[0]
        out = C.gemm_nt(copy, b, None, None, None, None, 0, flags, 5, of_tile, None, None)
        again = G.local_reduce(pos, out)
        assert torch.equal(out, want) and torch.equal(again, reduced)
    assert C.gemm_error(0) == 0
