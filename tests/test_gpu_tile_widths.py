"""GPU: shapes whose rounds of tiles take the 192-column tiles of the tensor-core GEMM (and neighbours that do not), ragged
in every dimension, against the CUDA-core kernel.  Integer operands: every sum is exact, so the outputs are equal bit for
bit."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# two rounds, ragged columns and depth, ragged rows, columns of one and a half tiles; the last keeps 256 columns
SHAPES = [(1000, 6144, 320), (1000, 6136, 136), (1025, 4400, 192), (2432, 2048, 128), (2400, 2040, 200), (1913, 4096, 320)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("mode,group_k", [(0, 0), (2, 64), (2, 128)])
def test_equal_to_the_cuda_core_kernel(M, N, K, mode, group_k):
    import hbq_b200 as H
    from hbq_b200.gemm import gemm
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randint(-4, 5, (M, K), device="cuda", generator=g).half()
    w = torch.randint(-3, 4, (N, K), device="cuda", generator=g).half()
    bias = torch.randint(-8, 9, (N,), device="cuda", generator=g).half()
    for b in (None, bias):
        got = gemm(a, w, mode, group_k, bias=b, b_is_nk=True)
        want = gemm(a, w, mode, group_k, bias=b, b_is_nk=True, force_simt=True)
        assert torch.equal(got, want)
    assert H.gemm_status() == 0


@pytest.mark.parametrize("mode,group_k", [(0, 0), (2, 128)])
@pytest.mark.parametrize("rows", [[500, 0, 613, 401, 7, 128, 129, 250], [256] * 8])
def test_grouped_products(mode, group_k, rows):
    from hbq_b200.gemm import gemm, gemm_grouped
    K, N, E = 256, 4096, len(rows)
    g = torch.Generator(device="cuda").manual_seed(sum(rows))
    off = torch.tensor([0] + rows, device="cuda").cumsum(0).int()
    a = torch.randint(-4, 5, (sum(rows), K), device="cuda", generator=g).half()
    ws = [torch.randint(-3, 4, (N, K), device="cuda", generator=g).half() for _ in rows]
    out = torch.empty((sum(rows), N), device="cuda", dtype=torch.float16)
    gemm_grouped(a, off, ws, [out] * E, range(E), mode, group_k)
    r0 = 0
    for n, w in zip(rows, ws):
        if n:
            assert torch.equal(out[r0:r0 + n], gemm(a[r0:r0 + n].contiguous(), w, mode, group_k, b_is_nk=True, force_simt=True))
        r0 += n


def test_width_follows_the_sms_that_are_left():
    """1000 x 6144: 192 tiles of 256 columns or 256 of 192, two rounds either way on 128 SMs and more; on fewer the
    narrower tiles take a third round."""
    import hbq_b200 as H
    from hbq_b200 import _lib
    from hbq_b200.gemm import gemm
    L = _lib.lib()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    a = torch.randint(-4, 5, (1000, 320), device="cuda").half()
    w = torch.randint(-3, 4, (6144, 320), device="cuda").half()
    want = gemm(a, w, 0, b_is_nk=True)
    prev = H.gemm_reserve_sms(0)
    try:
        for left, columns in ((148, 192), (128, 192), (127, 256), (100, 256), (96, 256)):
            H.gemm_reserve_sms(sms - left)
            assert L.hbq_gemm_tile_columns(1000, 6144, 0, 0) == columns == L.hbq_gemm_tile_columns(1000, 6144, 0, left)
            assert torch.equal(gemm(a, w, 0, b_is_nk=True), want)
    finally:
        H.gemm_reserve_sms(prev)
