"""spmm_dia_device with element or column numbers beyond 32 bits, and just within."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,R,offs", [(40, (1 << 31) + 5, 1, [0, (1 << 31) - 20, -7, 1 << 31]),   # columns past 2^31
                                        (3, 2, (1 << 30) + 33, [0, -1, 1]),                        # elements past 2^31
                                        (40, (1 << 31) - 41, 1, [0, (1 << 31) - 60, -7]),          # rows + columns 2^31 - 1
                                        (2, 2, (1 << 30) - 1, [1, 0])])                            # 2^31 - 2 elements
def test_beyond_32_bits(native, M, K, R, offs):
    """Sums of at most three float64 products, against torch on the device."""
    import torch

    capi, _ = native
    torch.cuda.empty_cache()
    off = torch.tensor(offs, dtype=torch.int64, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(3)
    V = torch.randn(len(offs), M, generator=g, device="cuda", dtype=torch.float64)
    B = torch.randn(K, R, generator=g, device="cuda", dtype=torch.float64)
    C = torch.full((M, R), float("nan"), device="cuda", dtype=torch.float64)
    capi.check(capi.lib().diaq_spmm_dia_device(off.data_ptr(), V.data_ptr(), len(offs), M, K, B.data_ptr(), R, C.data_ptr(),
                                               0, torch.cuda.current_stream().cuda_stream))
    for r in range(M):
        want = torch.zeros(R, device="cuda", dtype=torch.float64)
        for k, o in enumerate(offs):
            if 0 <= r + o < K:
                want += V[k, r] * B[r + o]
        assert float((C[r] - want).abs().max()) < 1e-13, r
    del B, C, want
    torch.cuda.empty_cache()
