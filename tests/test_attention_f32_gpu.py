"""The tiled float32 attention: every change of scores and mask against 64 bits, tiles that hold several requests, and the
same bits for a token whatever runs beside it."""
import math

import numpy as np
import pytest
import torch

from test_kernels_gpu import dev, err_word, make_cache, meta, rnd

pytestmark = pytest.mark.gpu


def reference(q, k, v, start, scale, window=None, keep_first=0, chunk=None, sink=None, softcap=None, slope_exponent=None, out_scale=1.0):
    n, nh, _ = q.shape
    out = torch.zeros(n, nh, v.shape[2], dtype=torch.float64)
    for i in range(n):
        p = start + i
        lo = max(0, p - window + 1) if window else 0
        if chunk:
            lo = max(lo, p // chunk * chunk)
        seen = [j for j in range(p + 1) if j >= lo or j < keep_first]
        for h in range(nh):
            g = h // (nh // k.shape[1])
            s = (k[seen, g] @ q[i, h]) * scale
            if softcap:
                s = softcap * torch.tanh(s / softcap)
            if slope_exponent:
                s = s - 2.0 ** (-slope_exponent * (h + 1) / nh) * (p - torch.tensor(seen, dtype=torch.float64))
            if sink is not None:
                s = torch.cat([s, sink[h:h + 1]])
            w = torch.softmax(s, 0)[: len(seen)]
            out[i, h] = out_scale * (w @ v[seen, g])
    return out


# nh, nkv, d, dv, page, entries, what changes
CASES = [
    (16, 8, 128, 128, 16, [(0, 45), (31, 1), (32, 1), (0, 1), (95, 33)], {}),
    (6, 2, 100, 36, 8, [(0, 7), (64, 9)], dict(softcap=3.0)),
    (20, 1, 4, 8, 16, [(0, 34), (63, 2)], dict(sink=True)),
    (8, 8, 64, 128, 4, [(130, 40), (0, 3)], dict(window=37, keep_first=5)),
    (8, 8, 64, 64, 16, [(130, 40), (5, 3)], dict(window=3, keep_first=70)),
    (4, 2, 32, 32, 16, [(60, 70), (0, 1)], dict(chunk=48, slope_exponent=8.0)),
    (12, 4, 80, 80, 32, [(200, 1), (0, 19)], dict(window=33, out_scale=0.5)),
]


@pytest.mark.parametrize("nh,nkv,d,dv,ps,entries,kw", CASES)
def test_tiles_against_64_bits_and_one_token_alone(nh, nkv, d, dv, ps, entries, kw):
    from xinfer_b200 import kernels
    pages = sum((s + c + ps - 1) // ps for s, c in entries) + 3
    pos, req, table, stride, table_np = meta(entries, ps, pages, 3)
    kc, _ = make_cache(pages, nkv, ps, d, torch.float32)
    vc, _ = make_cache(pages, nkv, ps, dv, torch.float32)
    kc.fill_(float("nan"))       # keys that nobody has written, and values that a mask hides, reach no sum
    vc.fill_(float("nan"))
    T = sum(c for _, c in entries)
    q = rnd(T, nh, d, seed=9)
    ks, vs = [], []
    for b, (s, c) in enumerate(entries):
        ks.append(rnd(s + c, nkv, d, seed=20 + b))
        vs.append(rnd(s + c, nkv, dv, seed=40 + b))
        for j in range(s + c):
            kc[table_np[b, j // ps], :, j % ps] = ks[b][j]
            vc[table_np[b, j // ps], :, j % ps] = vs[b][j]
    scale, e = 1.0 / math.sqrt(d), err_word()
    args = dict(kw)
    if args.pop("sink", None):
        args["sink"] = rnd(nh, seed=7)

    def run(rows):
        out = torch.full((len(rows), nh, dv), float("nan"), device=dev())
        window = args.get("window")
        kernels.attention_plain(out, q[rows].contiguous(), kc, vc, pos[rows].contiguous(), req[rows].contiguous(), table, stride,
                                window, scale, e, **{k: v for k, v in args.items() if k != "window"})
        return out

    out = run(list(range(T)))
    assert int(e) == 0
    t0 = 0
    for b, (s, c) in enumerate(entries):
        ref = reference(q[t0:t0 + c].double().cpu(), ks[b].double().cpu(), vs[b].double().cpu(), s, scale,
                        **{k: v.double().cpu() if isinstance(v, torch.Tensor) else v for k, v in args.items()})
        diff = (out[t0:t0 + c].double().cpu() - ref).abs().max().item()
        assert diff <= 2e-5, (b, diff)       # (the bound of the plain kernel's own test)
        t0 += c
    for t in sorted({0, T // 2, T - 1}):
        assert torch.equal(run([t])[0], out[t]), "a token's bits changed with what ran beside it"


def test_a_padding_token_gives_zeros_and_a_bad_page_is_reported():
    from xinfer_b200 import kernels
    nh, nkv, d, ps = 4, 2, 32, 16
    kc, vc = make_cache(4, nkv, ps, d, torch.float32)
    q = rnd(3, nh, d)
    table = torch.tensor([[0, 9], [1, 2]], dtype=torch.int32, device=dev())     # page 9 does not exist
    out = torch.full((3, nh, d), float("nan"), device=dev())
    e = err_word()
    kernels.attention_plain(out, q, kc, vc, torch.tensor([3, 5, 0], dtype=torch.int32, device=dev()),
                            torch.tensor([0, 1, -1], dtype=torch.int32, device=dev()), table, 2, None, 0.2, e)
    assert int(e) == 0 and torch.isfinite(out).all() and torch.count_nonzero(out[2]) == 0
    kernels.attention_plain(out, q, kc, vc, torch.tensor([20, 5, 0], dtype=torch.int32, device=dev()),
                            torch.tensor([0, 1, -1], dtype=torch.int32, device=dev()), table, 2, None, 0.2, e)
    assert int(e) == kernels.ERR_BAD_PAGE and torch.isfinite(out).all()


def test_tokens_of_a_request_that_are_not_neighbours():
    """Tokens of two requests in turn: each as it is alone."""
    from xinfer_b200 import kernels
    nh, nkv, d, ps = 4, 4, 32, 16
    kc, vc = rnd(6, nkv, ps, d, seed=1), rnd(6, nkv, ps, d, seed=2)
    table = torch.tensor([[0, 1, 2], [3, 4, 5]], dtype=torch.int32, device=dev())
    pos = torch.tensor([5, 3, 40, 41, 17, 0], dtype=torch.int32, device=dev())
    req = torch.tensor([0, 1, 0, 0, 1, 0], dtype=torch.int32, device=dev())
    q, e = rnd(6, nh, d, seed=3), err_word()

    def run(rows):
        out = torch.full((len(rows), nh, d), float("nan"), device=dev())
        kernels.attention_plain(out, q[rows].contiguous(), kc, vc, pos[rows].contiguous(), req[rows].contiguous(), table, 3, None, 0.2, e)
        return out

    out = run(list(range(6)))
    for t in range(6):
        assert torch.equal(run([t])[0], out[t]), t
        keys = lambda c: c[table[req[t]].long()].transpose(1, 2).reshape(48, nkv, d)[: int(pos[t]) + 1].double()
        w = torch.softmax(torch.einsum("hd,khd->hk", q[t].double(), keys(kc)) * 0.2, 1)
        assert (out[t].double() - torch.einsum("hk,khd->hd", w, keys(vc))).abs().max() <= 2e-5      # (as above)
    assert int(e) == 0


def test_a_model_with_head_sizes_on_both_sides_of_the_tiled_kernels():
    """Layers with heads of 96 and of 160 channels: the float32 logits have the same bits however the tokens are cut into steps."""
    from xinfer_b200.engine.runner import ModelRunner, StepInput
    layer = lambda dim, vdim: dict(type="attention", mlp=dict(kind="dense", ff=96), mixer=dict(
        heads=4, kv_heads=2, dim=dim, vdim=vdim, scale=dim ** -0.5, mask=dict(size=50), rot=dict(dims=16, base=1000.0)))
    cfg = dict(architecture="Dufitar", vocab=101, width=64, norm=dict(eps=1e-5), residual_mult=0.7, embedding=dict(scale=1.5),
               layers=[layer(96, 64), layer(160, 144), layer(160, 32), layer(128, 128)])
    rng = np.random.default_rng(3)
    a, b = (rng.integers(0, 101, size=n, dtype=np.int32) for n in (90, 41))

    def run(script):
        r = ModelRunner.random(cfg, 5, dtype="f32", block_size=16, num_blocks=32, max_num_seqs=2, max_model_len=128)
        slots, at, rows = [r.open_request(), r.open_request()], [0, 0], [[], []]
        for step in script:
            parts = [(i, (a, b)[i][at[i]:at[i] + n]) for i, n in step]
            logits = r.step([StepInput(slots[i], t, range(len(t))) for i, t in parts], allow_graph=False)
            for i, t in parts:
                rows[i].append(logits[:len(t)].clone())
                logits = logits[len(t):]
                at[i] += len(t)
        r.check_errors()
        return [torch.cat(x) for x in rows]

    whole = run([[(0, 90), (1, 41)]])
    cut = run([[(0, 33)], [(1, 20), (0, 1)], [(0, 55), (1, 20)], [(0, 1), (1, 1)]])
    for x, y in zip(whole, cut):
        assert torch.isfinite(x).all() and torch.equal(x, y)
