"""The float32 product on the tensor cores: edges of its tiles and panels against 64 bits, and numbers that are not finite."""
import pytest
import torch

from test_kernels_gpu import dev, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 15, 16, 17, 31, 33, 63, 64, 65, 449])
@pytest.mark.parametrize("N,K", [(127, 32), (128, 33), (129, 36), (300, 64), (1024, 65), (19000, 68), (257, 1000), (64, 5000)])
def test_edges_against_64_bits(M, N, K):
    """An addition to the running sum rounds by 2^-24 of it, once for 32 terms; the tensor cores cut the two sums of 16 off at
    2^-23 of what they hold by then, and so the ten small products before them; parts below 2^-24 of a product are left out."""
    from xinfer_b200 import kernels
    a, w = rnd(M, K, seed=1), rnd(N, K, seed=2)
    a[:, ::7] *= 100.0
    w[::3] *= 1e-3
    out = torch.full((M, N), float("nan"), device=dev())
    err = torch.zeros(1, dtype=torch.int32, device=dev())
    kernels.gemm_plain(out, a, w, err)
    x, y = a.double(), w.double()
    bound = ((K + 31) // 32 + 8) * 2.0 ** -24 * (x.abs() @ y.abs().t())
    assert int(err) == 0 and ((out.double() - x @ y.t()).abs() <= bound).all()


@pytest.mark.parametrize("M,K", [(3, 70), (40, 128)])
def test_infinities_and_overflow_give_what_float32_gives(M, K):
    from xinfer_b200 import kernels
    N = 200
    a, w = rnd(M, K, seed=3), rnd(N, K, seed=4)
    a[0, 5] = float("inf")
    a[1, K - 1] = float("nan")
    w[7, 5] = -float("inf")
    a[:, 0] = 0.5
    w[9, 0], a[2, 0] = 3e38, 2.0          # the product overflows, in this row alone
    w[11, 3] = 0.5                         # (one part of it is zero: an infinity there is still an infinity)
    out = torch.empty(M, N, device=dev())
    kernels.gemm_plain(out, a, w)
    ref = (a.double() @ w.double().t()).float()
    assert torch.equal(torch.isnan(out), torch.isnan(ref))
    assert torch.equal(out[torch.isinf(ref)], ref[torch.isinf(ref)])
    fine = torch.isfinite(ref)
    # every row but the two with an infinity and no number, every column but 7 and, in row 2, 9
    assert torch.isfinite(out[fine]).all() and fine.sum() == (M - 2) * (N - 1) - 1
