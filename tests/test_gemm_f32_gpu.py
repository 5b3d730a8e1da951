"""The float32 product on the tensor cores: edges of its tiles and panels against 64 bits, and numbers that are not finite."""
import pytest
import torch

from test_kernels_gpu import dev, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 15, 16, 17, 31, 33, 63, 64, 65, 449])
@pytest.mark.parametrize("N,K", [(127, 32), (128, 33), (129, 36), (300, 64), (1024, 65), (19000, 68), (257, 1000), (64, 5000)])
def test_edges_against_64_bits(M, N, K):
    """An addition to the running sum rounds by 2^-24 of it, once for 32 terms.  The rest is 8 of them: the products of parts that are
    left out, the addition of a block's large and small products, and what the tensor cores cut off each of 16 products, 2^-25 of
    the largest of them, mostly far from all in one direction."""
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


@pytest.mark.parametrize("e", [0, -100, -112, -118, -124, -140])
def test_small_operands_keep_all_their_digits(e):
    """Single products: 2^-24 of one for its rounding, 2^-24 for the products of parts that are left out and 2^-29 for what tensor
    memory cuts off the sum of the small ones; of an operand below 2^-126 what is left out may reach its last digit, 2^-149."""
    from xinfer_b200 import kernels
    M, N, K = 17, 300, 64
    for first in (True, False):
        a, w = torch.zeros(M, K, device=dev()), torch.zeros(N, K, device=dev())
        a[:, 5], w[:, 5] = rnd(M, seed=8), rnd(N, seed=9)
        small, large = (a, w) if first else (w, a)
        small *= 2.0 ** (e // 2)
        small *= 2.0 ** (e - e // 2)
        large *= 2.0 ** min(-e, 60)
        out = torch.empty(M, N, device=dev())
        kernels.gemm_plain(out, a, w)
        x, y = a.double().abs()[:, 5, None], w.double().abs()[None, :, 5]
        ref = a.double() @ w.double().t()
        assert ((out.double() - ref).abs() <= (2.0 ** -23 + 2.0 ** -29) * ref.abs() + 2.0 ** -149 * (x if large is a else y)).all()


@pytest.mark.parametrize("kind,K", [("normal", 64), ("small", 64), ("normal", 1024), ("positive", 1024), ("one term of 30", 1024),
                                    ("one term of 1000", 1024), ("small", 1024), ("normal", 3072)])
def test_error_is_no_larger_than_that_of_float32_multiply_adds(kind, K):
    """In 2-norm over many outputs, against float32's own: 16 terms by fused multiply-adds, these sums added up."""
    from xinfer_b200 import kernels
    M, N = 64, 512
    a, w = rnd(M, K, seed=10), rnd(N, K, seed=11)
    if kind == "positive":
        a, w = a.abs(), w.abs()
    elif kind.startswith("one"):
        a[:, K // 3] *= float(kind.split()[-1])
    elif kind == "small":
        a *= 2.0 ** -118
    x, y = a.double(), w.double()
    acc = torch.zeros(M, N, device=dev())
    for k0 in range(0, K, 16):
        part = torch.zeros(M, N, device=dev())
        for k in range(k0, k0 + 16):
            part = (part.double() + x[:, k, None] * y[None, :, k]).float()
        acc += part
    out = torch.empty(M, N, device=dev())
    kernels.gemm_plain(out, a, w)
    ref = x @ y.t()
    assert (out.double() - ref).norm() <= (acc.double() - ref).norm()


@pytest.mark.parametrize("M,N,K", [(449, 4100, 200), (1, 24577, 130), (70, 19000, 65)])
def test_tiles_of_every_size_form_the_same_bits(M, N, K):
    """Tiles of 16, 32 and 64 tokens and of any number of rows of W: a row, and some of the columns, as they are alone."""
    from xinfer_b200 import kernels
    a, w = rnd(M, K, seed=12), rnd(N, K, seed=13)
    out = torch.full((M, N), float("nan"), device=dev())
    kernels.gemm_plain(out, a, w)
    for rows, cols in (([M // 2], slice(0, N)), (slice(0, min(M, 33)), slice(N - 200, N)), (slice(0, M), slice(88, 130))):
        x, y = a[rows].contiguous(), w[cols].contiguous()
        part = torch.full((x.shape[0], y.shape[0]), float("nan"), device=dev())
        kernels.gemm_plain(part, x, y)
        assert torch.equal(part, out[rows][:, cols])


def test_the_largest_operands_whose_leading_part_rounds_to_infinity():
    from xinfer_b200 import kernels
    a, w = rnd(20, 80, seed=16), rnd(150, 80, seed=17) * 2.0 ** -30
    a[3, 7], a[5, 64] = 3.4028234663852886e38, -3.4e38
    out = torch.empty(20, 150, device=dev())
    kernels.gemm_plain(out, a, w)
    x, y = a.double(), w.double()
    # term by term in those rows: 16 multiply-adds, five sums
    assert ((out.double() - x @ y.t()).abs() <= 21 * 2.0 ** -24 * (x.abs() @ y.abs().t())).all()


def test_no_terms_give_zeros():
    from xinfer_b200 import kernels
    out = torch.full((3, 5), float("nan"), device=dev())
    kernels.gemm_plain(out, torch.empty(3, 0, device=dev()), torch.empty(5, 0, device=dev()))
    assert torch.count_nonzero(out) == 0 and torch.isfinite(out).all()


def test_the_word_of_calls_without_one_is_looked_at():
    """Also where the first such calls are captured: the word is no part of a graph's memory."""
    from xinfer_b200 import kernels
    from xinfer_b200.parts import gemm_backend
    a, w = rnd(3, 64, seed=14), rnd(40, 64, seed=15)
    out, want = torch.empty(3, 40, device=dev()), torch.empty(3, 40, device=dev())
    kernels.gemm_plain(want, a, w, torch.zeros(1, dtype=torch.int32, device=dev()))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        kernels.gemm_plain(out, a, w)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    y = torch.empty(3, 40, dtype=torch.bfloat16, device=dev())
    for call in (lambda: kernels.gemm_plain(out, a, w), lambda: gemm_backend.try_fast(y, a.bfloat16(), w.bfloat16())):
        kernels.own_err_word().value.value = kernels.ERR_WAIT
        with pytest.raises(kernels.KernelError, match="bounded wait"):
            call()
        call()                  # said once
        torch.cuda.synchronize()
        assert kernels.own_err_word().value.value == 0
