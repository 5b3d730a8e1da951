"""Heads of many tokens, a warp per token: the same as by the block-per-token kernel, which the same tokens take in small steps, and
against 64 bits."""
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

    # in 64 bits: bias, norm before or after the rotation, rotation (its angles are formed in float32), temperature
    x = qkv.double().cpu() + (b.double().cpu() if bias else 0.0)
    heads = x[:, : (nh + nkv) * d].view(tokens, nh + nkv, d).clone()
    p = pos.cpu()

    def norm(h):
        h = h * torch.rsqrt((h * h).mean(-1, keepdim=True) + 1e-5)
        return h * torch.cat([w.double().cpu().expand(n, d) if w is not None else torch.ones(n, d).double() for w, n in ((qw, nh), (kw, nkv))])
    if mode == 1:
        heads = norm(heads)
    if rot:
        angle = (p[:, None].float() * freq.cpu()[None]).double()[:, None]
        cs, sn = torch.cos(angle) * 1.25, torch.sin(angle) * 1.25
        i, j = (slice(0, rot, 2), slice(1, rot, 2)) if interleaved else (slice(0, rot // 2), slice(rot // 2, rot))
        u, v = heads[..., i].clone(), heads[..., j].clone()
        heads[..., i], heads[..., j] = u * cs - v * sn, v * cs + u * sn
    if mode == 2:
        heads = norm(heads)
    if temp:
        heads[:, :nh] *= 1.0 + temp[0] * torch.log((p[:, None, None] + 1) // temp[1] + 1.0).double()
    values = x[:, (nh + nkv) * d:].view(tokens, nkv, dv)
    q, kc, vc = (t.double().cpu() for t in run(tokens))
    live = req.cpu() >= 0
    rows = table.cpu()[req.cpu().clamp(min=0).long(), p.long() // ps].long(), p.long() % ps
    for got, ref in ((q, heads[:, :nh]), (kc[rows[0], :, rows[1]][live], heads[live, nh:]), (vc[rows[0], :, rows[1]][live], values[live])):
        # the rounding of the result to bfloat16 (eight digits), and 2^-18 of the largest for norm, sine, cosine and rotation in float32
        assert ((got - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -18 * ref.abs().max()).all()
    for x, y in zip(run(tokens), run(50)):
        # one rounding to bfloat16 of values that differ by a few float32 roundings
        assert (x.float() - y.float()).abs().max() <= 2.0 ** -7 * float(y.float().abs().max())
        assert (x != y).float().mean() <= 0.01
    assert int(err) == 0
    table[0, 0] = 2 * per
    run(tokens)
    assert int(err) == (k.ERR_BAD_PAGE if first > 5 else 0)
