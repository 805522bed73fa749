"""The reduction of few K splits (2 to 16) against an unsplit product in the same order: small integers, so that every
sum is exact and every association gives the same bits."""
import pytest

pytestmark = pytest.mark.gpu


# splits = min(K / 512, 296 / tiles), of 64-wide K blocks
@pytest.mark.parametrize("M,N,K", [(128, 64, 1024), (1152, 128, 1536), (4608, 512, 2048), (300, 40, 3584), (1024, 1024, 4096),
                                   (1024, 1024, 8192), (136, 264, 8192)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_few_splits(gpu, M, N, K, accumulate):
    import torch
    from vortexlab_b200 import warmstart as WS
    g = torch.Generator(device="cuda").manual_seed(M + K)
    a = torch.randint(-3, 4, (M, K), generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randint(-3, 4, (N, K), generator=g, device="cuda").to(torch.bfloat16)
    out = torch.randint(-9, 10, (M, N + 8), generator=g, device="cuda").float()
    want = out.clone()
    want[:, :N] = (out[:, :N].double() if accumulate else 0.0) + a.double() @ b.double().T
    err = WS._Err()
    WS.gemm(a, K, b, K, M, N, K, out, N + 8, WS.EPI_ACCUM if accumulate else 0, None, err)
    assert int(err.t.item()) == 0 and torch.equal(out, want)
