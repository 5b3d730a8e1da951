"""Talking heads of single tokens with keys and values in registers: against 64 bits, over key ranges, windows, sinks, groups of
heads and pages, and the values that no query sees."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("nh,nkv,d,contexts,ps,window,sink,parts", [
    (16, 8, 128, [1, 16, 17, 31, 300], 16, None, False, 1), (16, 2, 128, [5, 129], 8, None, True, 3), (32, 8, 128, [64, 65, 1000], 16, None, True, 8),
    (32, 4, 128, [40, 700, 3], 32, 50, False, 2), (16, 8, 128, [15, 513], 4, 16, True, 64), (32, 5 - 1, 128, [1], 16, None, True, 2),
    (16, 8, 64, [1, 33, 300], 16, None, False, 1), (8, 8, 128, [17, 400], 16, None, True, 4), (8, 1, 64, [700, 2], 16, None, False, 5),
    (24, 8, 128, [65, 500], 16, None, False, 3), (20, 5, 64, [31, 129], 8, 40, True, 2), (64, 8, 128, [300, 16], 16, None, True, 2),
    (40, 8, 64, [90], 16, None, False, 1), (1, 1, 64, [47], 16, None, True, 2), (32, 8, 64, [1000], 16, None, False, 8)])
def test_single_tokens_against_64_bits(nh, nkv, d, contexts, ps, window, sink, parts):
    from xinfer_b200 import kernels as k
    g = torch.Generator().manual_seed(nh + len(contexts))
    T = len(contexts)
    assert k.attn_talking_decode_takes(nh, nkv, d, d)
    per = max(contexts) // ps + 1
    table = torch.randperm(T * per, generator=g).int().view(T, per)
    kc = torch.full((T * per, nkv, ps, d), float("nan")).bfloat16()      # what is not a request's own is never part of a result
    vc = torch.full((T * per, nkv, ps, d), float("nan")).bfloat16()
    ks, vs = [], []
    for b, n in enumerate(contexts):
        ks.append(torch.randn(n, nkv, d, generator=g).bfloat16())
        vs.append(torch.randn(n, nkv, d, generator=g).bfloat16())
        for i in range(n):
            kc[table[b, i // ps], :, i % ps], vc[table[b, i // ps], :, i % ps] = ks[b][i], vs[b][i]
    q = torch.randn(T, nh, d, generator=g).bfloat16()
    talk = torch.randn(nh, nh, generator=g) / math.sqrt(nh)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    out = torch.zeros(T, nh * d, dtype=torch.bfloat16, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    po = torch.zeros(T * parts * nh * d, device=DEV)
    pml = torch.zeros(T * parts * nh * 2, device=DEV)
    scale = d ** -0.5
    starts = i32([n - 1 for n in contexts])
    args = (kc.to(DEV), vc.to(DEV), talk.to(DEV), i32(list(range(T + 1))), starts, T, table.to(DEV), per, window, scale, sink, 0.5, 1, err, parts, po, pml)
    k.attn_talking_mma(out, q.to(DEV), *args)
    assert int(err) == 0
    for b, n in enumerate(contexts):
        lo = max(0, n - window) if window else 0
        s = torch.einsum("hd,khd->hk", q[b].double(), ks[b][lo:].double().repeat_interleave(nh // nkv, 1)) * scale
        s = talk.double() @ s
        if sink:
            s = torch.cat([s, torch.zeros(nh, 1, dtype=torch.float64)], 1)
        w = torch.softmax(s, 1)[:, : n - lo]
        ref = 0.5 * torch.einsum("hk,khd->hd", w, vs[b][lo:].double().repeat_interleave(nh // nkv, 1))
        # a rounding to bfloat16 (eight digits) is up to 2^-8 of a number: of the weights in the sum of values (of every term) and in
        # their own sum (of the result), and of the result; 2^-16 of every term for scores, mix and exponentials in float32
        terms = 0.5 * torch.einsum("hk,khd->hd", w, vs[b][lo:].double().abs().repeat_interleave(nh // nkv, 1))
        bound = (2.0 ** -8 + 2.0 ** -16) * terms + 2.0 ** -7 * ref.abs()
        assert ((out[b].double().cpu().view(nh, d) - ref).abs() <= bound).all(), (b, n)


def test_a_token_of_no_request_and_a_bad_page():
    from xinfer_b200 import kernels as k
    nh, nkv, d, ps = 16, 8, 128, 16
    kc = torch.zeros(4, nkv, ps, d, dtype=torch.bfloat16, device=DEV)
    q = torch.ones(2, nh, d, dtype=torch.bfloat16, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    out = torch.full((2, nh * d), 3.0, dtype=torch.bfloat16, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    table = i32([[0, 9]])
    run = lambda start: k.attn_talking_mma(out, q, kc, kc, None, i32([0, 1]), i32([start]), 1, table, 2, None, 1.0, False, 1.0, 1, err)
    run(3)
    assert int(err) == 0 and torch.count_nonzero(out[0]) == 0 and (out[1] == 3.0).all()
    run(20)
    assert int(err) == k.ERR_BAD_PAGE and torch.isfinite(out).all()


@pytest.mark.parametrize("what", ["key", "value"])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_numbers_that_are_not_finite_reach_what_they_reach_in_the_tiled_kernel(what, bad):
    """Scratch that is not aligned keeps to the kernel with tiles."""
    from xinfer_b200 import kernels as k
    nh, nkv, d, ps, n, parts, T = 16, 4, 64, 16, 200, 2, 2
    g = torch.Generator().manual_seed(4)
    kc, vc = (torch.randn(2 * 13, nkv, ps, d, generator=g).bfloat16().to(DEV) for _ in range(2))
    (kc if what == "key" else vc)[5, 2, 3, 7] = bad            # the first request's key 83
    q = torch.randn(T, nh, d, generator=g).bfloat16().to(DEV)
    talk = (torch.randn(nh, nh, generator=g) / 4).to(DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    table = torch.arange(26, dtype=torch.int32, device=DEV).view(2, 13)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    outs = []
    for shift in (0, 1):
        po, pml = torch.zeros(T * parts * nh * d + 4, device=DEV), torch.zeros(T * parts * nh * 2 + 4, device=DEV)
        out = torch.zeros(T, nh * d, dtype=torch.bfloat16, device=DEV)
        k.attn_talking_mma(out, q, kc, vc, talk, i32([0, 1, 2]), i32([n - 1, n - 1]), 2, table, 13, None, 0.1, True, 1.0, 1, err, parts, po[shift:], pml[shift:])
        outs.append(out.float())
    a, b = outs
    assert int(err) == 0 and torch.isfinite(a[1]).all() and not torch.isfinite(a[0]).all()
    assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.isinf(a), torch.isinf(b))
    fine = torch.isfinite(a)
    assert (a[fine] - b[fine]).abs().max() <= 2.0 ** -7 * (1 + b[fine].abs().max())
