"""What the GEMM and SwiGLU launchers choose from sizes alone (host code of the native module, no GPU needed)."""
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


@pytest.mark.parametrize('tiles,N,groups,total_rows,streams', [
    (32, 4096, 32, 0, False),                   # nothing known: the tiles may be full
    (32, 4096, 32, 32 * 16, True), (32, 7168, 32, 32 * 56, True), (1, 256, 1, 1, True), (13, 512, 32, 13 * 56, True),
    (32, 7168, 32, 32 * 56 + 1, False), (32, 4096, 32, 32 * 128, False), (33, 4096, 32, 33, False), (32, 248, 32, 32, False)])
def test_thin_tiles_stream_the_weights_where_the_rows_are_known(tiles, N, groups, total_rows, streams):
    for M in (128 * tiles, 128 * tiles - 127):
        assert _C().gemm_streams_weights(M, N, num_groups=groups, total_rows=total_rows) == streams


@pytest.mark.parametrize('inter', [8, 256, 264, 512, 768, 1024, 1408, 2048, 3072, 4096])
@pytest.mark.parametrize('rows', [1, 128, 512, 767, 768, 1024, 1536, 2048, 4096, 6016, 8192, 9400, 12000, 1 << 20])
def test_rows_of_swiglu_are_cut_where_that_pays(rows, inter):
    """The split for the row mask comes on top of the one of small launches and ends where full rows got slower: single steps of 256 columns on few or
    on many CTAs (512 x 2048 2.7 -> 3.2 us, 8192 x 512 5.7 -> 6.8), two steps on more than 1536 (8192 x 1024 9.0 -> 9.9)."""
    ctas, steps = (rows + 7) // 8, (inter + 255) // 256
    plain_steps = -(-steps // max(1, min(steps, -(-296 // ctas))))          # of a warp, as in the other kernels
    chunk = _C().swiglu_quant_col_chunk(rows, inter)
    per = chunk // 256
    assert chunk % 256 == 0 and 1 <= per <= plain_steps
    if per < plain_steps:
        assert ctas >= 96
        if per == 1:
            assert 768 <= ctas * steps <= 1152
        else:
            assert ctas >= 128 and (ctas * -(-steps // per) <= 1536 or (plain_steps > 8 and 4 < per <= 8))
