"""Edges of the exchange kernels that move rows directly when there is a single rank.  Everything is compared bitwise."""
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
