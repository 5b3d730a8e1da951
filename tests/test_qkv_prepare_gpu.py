"""Heads of many tokens, a warp per token: the same as by the block-per-token kernel, which the same tokens take in small steps."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("nh,nkv,d,dv,rot,interleaved,mode,bias,temp,tokens", [
    (32, 8, 128, 128, 128, False, 2, False, None, 65), (3, 1, 128, 64, 128, False, 1, True, (0.3, 7), 200),
    (8, 8, 64, 128, 0, False, 1, False, None, 130), (16, 2, 112, 48, 56, True, 0, True, None, 129),
    (5, 5, 48, 48, 48, False, 0, False, (0.1, 3), 1000), (1, 1, 16, 16, 16, True, 2, False, None, 66),
    (3, 1, 128, 64, 64, False, 1, True, (0.3, 7), 200)])
def test_many_tokens_as_by_small_steps(nh, nkv, d, dv, rot, interleaved, mode, bias, temp, tokens):
    from xinfer_b200 import kernels as k
    g = torch.Generator().manual_seed(d + nh)
    rnd = lambda *s: torch.randn(*s, generator=g)
    width, ps = (nh + nkv) * d + nkv * dv, 16
    qkv = (rnd(tokens, width) * 2).bfloat16().to(DEV)
    first = tokens // 3
    pos = torch.tensor([11 + i for i in range(first)] + list(range(tokens - first)), dtype=torch.int32, device=DEV)
    req = torch.tensor([0] * first + [1] * (tokens - first), dtype=torch.int32, device=DEV)
    req[tokens - 2:] = -1                                  # padding
    per = (tokens + 11) // ps + 1
    table = torch.randperm(2 * per, generator=g).int().view(2, per).to(DEV)
    qw, kw = (rnd(d).abs().to(DEV) if mode == 1 else None for _ in range(2))
    freq = (rnd(rot // 2).abs() * 0.1).to(DEV) if rot else None
    b = rnd(width).to(DEV) if bias else None
    err = torch.zeros(1, dtype=torch.int32, device=DEV)

    def run(step):
        q = torch.zeros(tokens, nh, d, dtype=torch.bfloat16, device=DEV)
        kc = torch.full((2 * per, nkv, ps, d), 7.0, dtype=torch.bfloat16, device=DEV)
        vc = torch.full((2 * per, nkv, ps, dv), 7.0, dtype=torch.bfloat16, device=DEV)
        for a in range(0, tokens, step):
            e = min(a + step, tokens)
            k.qkv_prepare(q[a:e], kc, vc, qkv[a:e], qw, kw, freq, pos[a:e].contiguous(), req[a:e].contiguous(), table, per, nh, nkv, d, dv, rot,
                          interleaved, mode, 1e-5, True, err, rot_magnitude=1.25, bias=b, q_temp=temp)
        return q, kc, vc

    for x, y in zip(run(tokens), run(50)):
        # one rounding to bfloat16 of values that differ by a few float32 roundings
        assert (x.float() - y.float()).abs().max() <= 2.0 ** -7 * float(y.float().abs().max())
        assert (x != y).float().mean() <= 0.01
    assert int(err) == 0
    table[0, 0] = 2 * per
    run(tokens)
    assert int(err) == (k.ERR_BAD_PAGE if first > 5 else 0)
