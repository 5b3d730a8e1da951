"""Attention with talking heads in steps of many tokens, the mixed scores passed through memory: the work lists (CPU), the
pair of kernels against plain float64 attention, and a model with and without them."""
import math

import numpy as np
import pytest
import torch

from xinfer_b200 import kernels

DEV = "cuda:0"


@pytest.mark.parametrize("counts,starts,window,heads,kv_heads,cap,ctas", [
    ([1], [0], None, 8, 4, 1 << 16, 148), ([2048], [0], None, 32, 8, 1 << 16, 148), ([2048], [0], None, 32, 8, 5000, 148),
    ([300, 1, 129, 4, 128], [7, 900, 0, 0, 64], None, 16, 16, 3000, 20), ([700], [1000], 100, 16, 8, 700, 7), ([64, 65], [63, 64], 16, 8, 8, 64, 148),
])
def test_the_work_lists_hold_every_score_and_every_head_once(counts, starts, window, heads, kv_heads, cap, ctas, monkeypatch):
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda t: t)
    host, chunks, most = kernels.talk_work(counts, starts, window, heads, kv_heads, cap, max_ctas=ctas)
    w = host.numpy()
    first_key = lambda p: max(0, p - window + 1) if window else 0
    qn, rep = 512 // heads, heads // kv_heads
    scored, summed, worst = set(), set(), 0

    def items(at, n):
        offs = w[at:at + n + 1]
        assert offs[0] == 0 and (np.diff(offs) >= 1).all() and n <= ctas
        return w[at + n + 1:at + n + 1 + 4 * offs[-1]].reshape(-1, 4)
    for blocks_at, one, two, c1, c2 in chunks:
        blocks = w[blocks_at:one].reshape(-1, 6)
        at = 0
        for b, first, kb0, nkb, tile0, _ in blocks:
            assert tile0 == at and kb0 % 4 == 0 and nkb % 4 == 0
            at += nkb * heads
        worst = max(worst, at)
        assert at <= cap
        for i, qt, kt, n in items(one, c1):
            b, first, kb0, nkb = blocks[i][:4]
            assert n >= 1 and kb0 <= 4 * kt and 4 * (kt + n) <= kb0 + nkb        # the tiles it writes are the block's
            for t in range(kt, kt + n):
                assert (b, first, qt, t) not in scored
                scored.add((int(b), int(first), int(qt), int(t)))
        for i, h0, nh, _ in items(two, c2):
            b, first, kb0, nkb = blocks[i][:4]
            rows = min(128, counts[b] - first)
            assert nh in (1, 2) and h0 // rep == (h0 + nh - 1) // rep
            lo, hi = first_key(starts[b] + first) // 64, (starts[b] + first + rows - 1) // 64
            assert 2 * lo >= kb0 and 2 * hi + 2 <= kb0 + nkb                        # and so are those it reads
            for h in range(h0, h0 + nh):
                assert (b, first, h) not in summed
                summed.add((int(b), int(first), h))
    assert worst == most
    assert summed == {(b, f, h) for b, n in enumerate(counts) for f in range(0, n, 128) for h in range(heads)}
    want = set()
    for b, n in enumerate(counts):
        for p in range(0, n):       # every tile that some query of a query tile sees
            f, qt = p // 128 * 128, p % 128 // qn
            for t in range(first_key(starts[b] + p) // 128, (starts[b] + p) // 128 + 1):
                want.add((b, f, qt, t))
    assert scored == want


def test_a_block_with_more_tiles_than_the_scratch_holds_is_refused(monkeypatch):
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda t: t)
    assert kernels.talk_work([5], [4000], None, 32, 8, 4000) is None


def _plain(q, k, v, talk, start, window, scale, sink):
    n, H, _ = q.shape
    end, G, _ = k.shape
    k, v = (t.repeat_interleave(H // G, 1) for t in (k, v))
    s = torch.einsum("hg,gij->hij", talk, torch.einsum("ihd,jhd->hij", q, k) * scale)
    far = torch.arange(start, end)[:, None] - torch.arange(end)[None]
    s = s.masked_fill((far < 0) | (far >= window if window else far < 0), -math.inf)
    if sink:
        s = torch.cat([s, torch.zeros(H, n, 1, dtype=s.dtype)], -1)
    return torch.einsum("hij,jhd->ihd", torch.softmax(s, -1)[..., :end], v)


@pytest.mark.gpu
@pytest.mark.parametrize("H,G,d,dv,ps", [(32, 8, 128, 128, 16), (16, 8, 128, 64, 8), (16, 16, 64, 128, 64), (8, 4, 64, 64, 128),
                                         (8, 8, 128, 128, 256), (32, 4, 64, 64, 32), (32, 16, 128, 128, 16)])
@pytest.mark.parametrize("counts,starts,window,sink,cap", [
    ([1, 5], [0, 9], None, True, 1 << 14), ([127, 1, 129], [0, 340, 0], None, True, 1 << 14), ([128, 256, 257], [64, 0, 63], None, False, 600),
    ([300, 6], [777, 130], 100, True, 1 << 14), ([64, 500], [3, 0], 33, False, 1 << 14), ([17], [1], 1, False, 1 << 14),
])
def test_the_pair_of_kernels_agrees_with_plain_attention(H, G, d, dv, ps, counts, starts, window, sink, cap):
    g = torch.Generator().manual_seed(H + d + sum(counts))
    bf = lambda *s: torch.randn(*s, generator=g).bfloat16()
    i32 = lambda a: torch.tensor(np.asarray(a), dtype=torch.int32, device=DEV)
    B, T = len(counts), sum(counts)
    ks, vs, q = [bf(s + c, G, d) for s, c in zip(starts, counts)], [bf(s + c, G, dv) for s, c in zip(starts, counts)], bf(T, H, d)
    talk = torch.randn(H, H, generator=g) * H ** -0.5
    per = max(-(-k.shape[0] // ps) for k in ks)
    table = torch.full((B, per), -1, dtype=torch.int32)
    order = torch.randperm(B * per + 1, generator=g).tolist()
    kc, vc = torch.full((B * per + 1, G, ps, d), float("nan")).bfloat16(), torch.full((B * per + 1, G, ps, dv), float("nan")).bfloat16()
    for b, k in enumerate(ks):
        gone = max(0, starts[b] - window + 1) // ps if window else 0        # pages in front of the window were given back
        for p in range(gone, -(-k.shape[0] // ps)):
            table[b, p] = order[b * per + p]
            n = min(ps, k.shape[0] - p * ps)
            kc[table[b, p], :, :n] = k[p * ps:p * ps + n].transpose(0, 1)
            vc[table[b, p], :, :n] = vs[b][p * ps:p * ps + n].transpose(0, 1)
    cap = max(cap, 4 * H * (-(-max(s + c for s, c in zip(starts, counts)) // 128) + 1))
    host, chunks, tiles = kernels.talk_work(counts, starts, window, H, G, cap)
    scores = torch.full((tiles * kernels.TALK_TILE_FLOATS,), float("nan"), device=DEV)
    buf = torch.zeros(T, H * dv + 24, dtype=torch.bfloat16, device=DEV)     # the output lies inside wider rows
    out, err = buf[:, 8:8 + H * dv], i32([0])
    kernels.attn_talking_tc(out, q.to(DEV), kc.to(DEV), vc.to(DEV), talk, scores, host.to(DEV), chunks,
                            i32(np.concatenate([[0], np.cumsum(counts)])), i32(starts), table.to(DEV), per, window, d ** -0.5, sink, 0.75, err)
    torch.cuda.synchronize()
    assert int(err) == 0 and not buf[:, :8].any() and not buf[:, 8 + H * dv:].any()
    at = 0
    for b, (c, s) in enumerate(zip(counts, starts)):
        ref = 0.75 * _plain(q[at:at + c].double(), ks[b].double(), vs[b].double(), talk.double(), s, window, d ** -0.5, sink)
        got = out[at:at + c].double().cpu().view(c, H, dv)
        # scores are float32; the probabilities (of a row whose weighted values are of the size of its result, or 1) and the
        # result are each rounded once to bfloat16, whose unit roundoff is 2^-8
        assert (got - ref).abs().max() <= 2 * 2 ** -8 * max(1.0, ref.abs().max()), (b, (got - ref).abs().max())
        at += c


@pytest.mark.gpu
def test_a_model_gives_the_same_logits_both_ways_and_for_mixed_steps(monkeypatch):
    from xinfer_b200.engine.runner import ModelRunner, StepInput
    from xinfer_b200.parts import talking_attention as part
    left = dict(heads=8, kv_heads=4, dim=64, vdim=64, scale=0.125, rot=dict(dims=64, base=1000.0))
    layer = dict(type="parallel", mixer=dict(left=left, left_scale=0.5, right=dict(width=64), right_scale=1.0), mlp=dict(kind="dense", ff=128))
    cfg = dict(architecture="Tidarax", vocab=300, width=128, norm=dict(eps=1e-6), layers=[layer, layer])
    ids = np.random.default_rng(1).integers(0, 300, size=400)

    def logits(on, nbytes):
        monkeypatch.setattr(part, "USE_SCORES", on)
        monkeypatch.setattr(part, "SCORES_BYTES", nbytes)
        monkeypatch.setattr(part, "SCORES_MIN_US", 0.0)
        r = ModelRunner.random(cfg, 3, block_size=16, num_blocks=128, max_num_seqs=4, max_model_len=512)
        before = kernels.launch_counts().get("attn_talking_tc", 0)
        a, b = r.open_request(), r.open_request()
        out = [r.step([StepInput(a, ids[:200], [7, 199])]).clone()]
        out.append(r.step([StepInput(a, ids[200:201], [0]), StepInput(b, ids[:333], [332])]).clone())      # one token beside a prompt
        out.append(r.step([StepInput(b, ids[333:400], [66]), StepInput(a, ids[201:204], [2])]).clone())     # portions behind cached tokens
        r.check_errors()
        return torch.cat(out).double(), kernels.launch_counts().get("attn_talking_tc", 0) - before
    want, none = logits(False, 0)
    got, some = logits(True, 1 << 28)
    again, more = logits(True, 128 * 16384)       # a block or two per chunk
    assert none == 0 and some == 12 and more > some
    # two bfloat16 computations of the same numbers
    assert (got - want).norm() <= 0.02 * want.norm() and (again - got).norm() <= 1e-3 * got.norm()


@pytest.mark.parametrize("heads,counts,starts,window,pays", [
    (32, [100] * 8, [0] * 8, None, False), (32, [400, 400], [0, 0], None, True), (16, [400, 400], [0, 0], None, True),
    (16, [100] * 8, [0] * 8, None, False), (32, [20], [0], None, False), (32, [2048], [0], None, True), (32, [2048], [0], 64, True),
    (32, [64, 1], [0, 3000], None, True), (32, [64, 1], [0, 3000], 64, False), (8, [5], [0], None, False)])
def test_short_steps_stay_on_the_kernel_that_holds_all_heads(heads, counts, starts, window, pays):
    from types import SimpleNamespace as N
    from xinfer_b200.parts.talking_attention import TalkingAttention
    layer = N(spec=N(num_heads=heads, window=window))
    ctx = N(max_context=max(a + b for a, b in zip(counts, starts)), real_tokens=sum(counts), real_entries=len(counts),
            h_q_start=np.concatenate([[0], np.cumsum(counts)]), h_start_pos=np.asarray(starts))
    assert TalkingAttention._scores_pay(layer, ctx) == pays


def _prompt(T, H, G, d, dv, g, vary=1.0):
    """A prompt of T tokens on pages of 16: (q, keys, values, table, work lists, scratch, the rest of the arguments)."""
    bf = lambda *s: torch.randn(*s, generator=g).bfloat16()
    i32 = lambda a: torch.tensor(np.asarray(a), dtype=torch.int32, device=DEV)
    n = -(-T // 16)
    host, chunks, tiles = kernels.talk_work([T], [0], None, H, G, 1 << 16)
    scores = torch.empty(tiles * kernels.TALK_TILE_FLOATS, device=DEV)
    return ((vary * bf(T, H, d)).to(DEV), bf(n, G, 16, d).to(DEV), bf(n, G, 16, dv).to(DEV), i32([range(n)]), (host.to(DEV), chunks), scores,
            (i32([0, T]), i32([0])), i32([0]))


@pytest.mark.gpu
@pytest.mark.parametrize("key", [0, 3, 7, 38, 63, 64, 130])
def test_a_key_that_is_not_a_number_shows_in_every_query_that_sees_it(key):
    T, H, G, d, dv = 200, 8, 4, 64, 64
    g = torch.Generator().manual_seed(key)
    q, k, v, table, (work, chunks), scores, (q_start, start_pos), err = _prompt(T, H, G, d, dv, g)
    k[key // 16, :, key % 16] = float("nan")
    talk = torch.randn(H, H, generator=g)
    out = torch.zeros(T, H * dv, dtype=torch.bfloat16, device=DEV)
    kernels.attn_talking_tc(out, q, k, v, talk, scores, work, chunks, q_start, start_pos, table, table.shape[1], None, d ** -0.5, True, 1.0, err)
    bad = torch.isnan(out)
    assert int(err) == 0 and bad[key:].all() and not bad[:key].any()


@pytest.mark.gpu
@pytest.mark.parametrize("key,channel,value", [(0, 0, math.nan), (63, 5, math.inf), (64, 63, -math.inf), (130, 8, math.nan), (190, 17, math.inf),
                                               (199, 40, math.nan)])
@pytest.mark.parametrize("window", [None, 70])
@pytest.mark.parametrize("H,G,dv", [(16, 8, 128), (8, 8, 64)])
def test_a_value_that_is_not_finite_reaches_only_the_queries_that_see_it(H, G, dv, window, key, channel, value):
    T, d = 200, 64
    g = torch.Generator().manual_seed(key)
    q, k, v, table, _, _, (q_start, start_pos), err = _prompt(T, H, G, d, dv, g)
    host, chunks, tiles = kernels.talk_work([T], [0], window, H, G, 1 << 16)
    work, scores = host.to(DEV), torch.empty(tiles * kernels.TALK_TILE_FLOATS, device=DEV)
    talk = torch.randn(H, H, generator=g) * H ** -0.5

    def run():
        out = torch.zeros(T, H, dv, dtype=torch.bfloat16, device=DEV)
        kernels.attn_talking_tc(out.view(T, H * dv), q, k, v, talk, scores, work, chunks, q_start, start_pos, table, table.shape[1], window,
                                d ** -0.5, True, 1.0, err)
        return out
    v[key // 16, 1, key % 16, channel] = 0
    want = run()
    v[key // 16, 1, key % 16, channel] = value
    got = run()
    sees = torch.zeros_like(want, dtype=torch.bool)
    sees[key:key + (window or T), H // G: 2 * (H // G), channel] = True
    # (a query of a tile that every query sees whole may turn a weight too small for bfloat16 times infinity into no number)
    assert int(err) == 0 and not torch.isfinite(got[sees]).any() and torch.equal(got[~sees], want[~sees])
    if value == value:
        assert not (got[sees] == -value).any()


@pytest.mark.gpu
def test_weights_are_divided_by_their_own_sum():
    # Values that are all one: the result is the sum of the rounded weights over what it is divided by, times the factor.  The
    # factor lies 2^-14 above the middle between two bfloat16 numbers, so that a quotient that is off by more than that rounds to
    # the lower one (weights that are summed before they are rounded: by up to 2^-9); float32 sums of 200 terms are off by 2^-20.
    T, H, G, d, dv = 200, 8, 4, 64, 64
    g = torch.Generator().manual_seed(5)
    q, k, v, table, (work, chunks), scores, (q_start, start_pos), err = _prompt(T, H, G, d, dv, g, vary=2.0)
    out = torch.zeros(T, H * dv, dtype=torch.bfloat16, device=DEV)
    factor = 1.0 + 2.0 ** -8 + 2.0 ** -14
    kernels.attn_talking_tc(out, q, k, torch.ones_like(v), torch.eye(H), scores, work, chunks, q_start, start_pos, table, table.shape[1], None,
                            d ** -0.5, False, factor, err)
    assert int(err) == 0 and (out == 1.0 + 2.0 ** -7).all()


@pytest.mark.gpu
def test_scratch_and_work_lists_that_are_too_short_are_refused():
    T, H, G, d, dv = 300, 8, 4, 64, 64
    q, k, v, table, (work, chunks), scores, (q_start, start_pos), err = _prompt(T, H, G, d, dv, torch.Generator().manual_seed(2))
    out = torch.zeros(T, H * dv, dtype=torch.bfloat16, device=DEV)

    def run(work=work, chunks=chunks, scores=scores):
        kernels.attn_talking_tc(out, q, k, v, torch.eye(H), scores, work, chunks, q_start, start_pos, table, table.shape[1], None, 0.1, True, 1.0, err)
    for bad in (dict(work=work[:-1].contiguous()), dict(scores=scores[:-1].contiguous()), dict(chunks=list(chunks))):
        with pytest.raises(kernels.KernelError):
            run(**bad)
    run()
    assert int(err) == 0
