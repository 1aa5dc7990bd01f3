"""What the GEMM launcher chooses from sizes alone (host code of the native module, no GPU needed)."""
import pytest


def _C():
    from deepep_ascend_b200 import _native
    return _native.load()


@pytest.mark.parametrize('num_sms', [13, 16, 40, 124, 147, 148, 200])
@pytest.mark.parametrize('M,N,K', [(300, 256, 7168), (64, 128, 8000), (512, 1024, 20000), (1, 8, 1600)])
def test_the_parts_of_a_product_are_added_on_its_own_sms(M, N, K, num_sms):
    """A product of few SMs: its second kernel has no more CTAs than that, and none of them waits for the product on another SM."""
    splits, ctas, threads, beside_product = _C().gemm_split_plan(M, N, K, num_sms=num_sms, device_sms=148)
    if num_sms < 148:
        assert ctas <= num_sms and not beside_product
    else:
        assert beside_product
    assert splits * ((M + 127) // 128) * ((N + 127) // 128) <= num_sms or splits == 1
    assert 1 <= ctas <= (M * N // 8 + threads - 1) // threads and ctas <= 8 * 148 and threads % 32 == 0 and threads <= 1024
