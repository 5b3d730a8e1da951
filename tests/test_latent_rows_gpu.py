"""Attention of long portions over a cached latent through keys and values formed for the step: the work list (CPU), the
kernels against plain float64 attention, and the choice between the two ways inside a layer."""
import math

import numpy as np
import pytest
import torch

from xinfer_b200 import kernels

DEV = "cuda:0"


@pytest.mark.parametrize("counts,starts,window,heads,ctas", [
    ([1], [0], None, 4, 148), ([5], [0], None, 1, 148), ([2048], [0], None, 32, 148), ([300, 1, 129, 4, 128], [7, 90, 0, 0, 64], None, 3, 20),
    ([700], [1000], 100, 2, 7), ([64, 65], [63, 64], 16, 5, 148),
])
def test_the_work_list_holds_every_query_of_every_head_once(counts, starts, window, heads, ctas, monkeypatch):
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda t: t)
    host, n, rows, at = kernels.latent_prefill_work(counts, starts, 4, window, heads, max_ctas=ctas)
    long = [b for b, c in enumerate(counts) if c > 4]
    assert (n == 0) == (not long) and n <= ctas
    if not long:
        assert rows == 0
        return
    w = host.numpy()
    items = w[n + 1:at].reshape(-1, 4)
    runs = w[at:].reshape(-1, 2)
    assert w[0] == 0 and w[n] == len(items) and (np.diff(w[:n + 1]) >= 1).all() and len(runs) * 64 == rows
    row_of = {(int(b), int(j)): i * 64 for i, (b, j) in enumerate(runs)}
    seen = set()
    for b, first, hn, row0 in items:
        h, nt = int(hn) & 0xffff, int(hn) >> 16
        assert nt in (1, 2) and counts[b] - first > (nt - 1) * 128
        for i in range(nt):
            assert (b, first + 128 * i, h) not in seen
            seen.add((b, first + 128 * i, h))
            p = starts[b] + first + 128 * i
            last = p + min(128, counts[b] - first - 128 * i) - 1
            lo = max(0, p - window + 1) if window else 0
            for kt in range(lo // 64, last // 64 + 1):          # every key tile the kernel reads is a run of this portion
                assert row_of[(int(b), kt * 64)] == row0 + kt * 64
    assert seen == {(b, q, h) for b in long for q in range(0, counts[b], 128) for h in range(heads)}


def _plain(q, rows, w_kv, heads, d, rd, dv, rank, start, window, scale, sink):
    """float64: q [n, H, d + rd], rows [start + n, width]."""
    n, end = q.shape[0], rows.shape[0]
    k = (rows[:, :rank] @ w_kv[:heads * d].T).view(end, heads, d)
    v = (rows[:, :rank] @ w_kv[heads * d:].T).view(end, heads, dv)
    k = torch.cat([k, rows[:, None, rank:rank + rd].expand(end, heads, rd)], -1)
    s = torch.einsum("ihd,jhd->hij", q, k) * scale
    far = torch.arange(start, end)[:, None] - torch.arange(end)[None]
    s = s.masked_fill((far < 0) | (far >= window if window else far < 0), -math.inf)
    if sink is not None:
        s = torch.cat([s, sink[:, None, None].expand(heads, n, 1)], -1)
    return torch.einsum("hij,jhd->ihd", torch.softmax(s, -1)[..., :end], v)


@pytest.mark.gpu
@pytest.mark.parametrize("d,rd,dv,rank,tail", [(128, 64, 128, 512, 0), (128, 32, 128, 256, 0), (128, 0, 128, 64, 32), (64, 64, 64, 128, 0),
                                               (64, 0, 64, 72, 0), (64, 8, 128, 64, 0), (128, 0, 64, 64, 0)])
@pytest.mark.parametrize("counts,starts,window,heads,sink", [
    ([5], [0], None, 1, False), ([127, 1, 129], [0, 40, 0], None, 3, True), ([128, 256, 257], [64, 0, 63], None, 2, False),
    ([300, 6], [777, 130], 100, 2, True), ([64, 700], [3, 0], 64, 1, False), ([130], [1], 1, 2, False),
])
def test_rows_attention_agrees_with_plain_attention(d, rd, dv, rank, tail, counts, starts, window, heads, sink):
    g = torch.Generator().manual_seed(d + 3 * rd + sum(counts))
    bf = lambda *s: torch.randn(*s, generator=g).bfloat16()
    i32 = lambda a: torch.tensor(np.asarray(a), dtype=torch.int32, device=DEV)
    width, ps, B, T = rank + rd + tail, 16, len(counts), sum(counts)
    seqs = [bf(s + c, width) for s, c in zip(starts, counts)]
    w_kv = (bf(heads * (d + dv), rank).float() * rank ** -0.5).bfloat16()
    q_row = heads * (d + rd) + 8                                # queries in front of something else
    q = bf(T, q_row)
    per = max(-(-r.shape[0] // ps) for r in seqs)
    table = torch.full((B, per), -1, dtype=torch.int32)
    pages = torch.full((B * per + 1, ps, width), float("nan")).bfloat16()
    order = torch.randperm(B * per + 1, generator=g).tolist()
    for b, r in enumerate(seqs):
        # pages that lie wholly in front of the window have been given back
        gone = max(0, starts[b] - window + 1) // ps if window else 0
        for p in range(gone, -(-r.shape[0] // ps)):
            table[b, p] = order[b * per + p]
            part = r[p * ps:(p + 1) * ps]
            pages[table[b, p], :len(part)] = part
    q_start, start_pos, err = i32(np.concatenate([[0], np.cumsum(counts)])), i32(starts), i32([0])
    sinks = torch.randn(heads, generator=g) if sink else None
    host, ctas, rows_n, at = kernels.latent_prefill_work(counts, starts, 4, window, heads)
    work = host.to(DEV)
    rows = torch.full((rows_n, width), float("nan"), dtype=torch.bfloat16, device=DEV)
    kernels.latent_gather(rows, pages.to(DEV), work, at, q_start, start_pos, table.to(DEV), per, window, err)
    kv = rows[:, :rank] @ w_kv.to(DEV).t()
    out = torch.full((T, heads * dv), float("nan"), dtype=torch.bfloat16, device=DEV)
    scale = (d + rd) ** -0.5
    kernels.attn_rows_tc(out, q.to(DEV), q_row, kv, rows, work, ctas, q_start, start_pos, heads, d, rd, dv, rank, window, scale,
                         sinks.to(DEV) if sink else None, err)
    torch.cuda.synchronize()
    assert int(err) == 0
    at = 0
    for b, (c, s) in enumerate(zip(counts, starts)):
        got = out[at:at + c].double().cpu().view(c, heads, dv)
        if c <= 4:
            assert torch.isnan(got).all()                       # left to the kernel of the small portions
        else:
            ref = _plain(q[at:at + c, :heads * (d + rd)].double().view(c, heads, d + rd), seqs[b].double(), w_kv.double(), heads, d, rd,
                         dv, rank, s, window, scale, sinks.double() if sink else None)
            # keys, values, probabilities and the result are rounded to 8 bits: scores of size 1 move by 2^-9 each key
            # channel's share, the result by 2^-9 of the largest value a few times over
            assert (got - ref).abs().max() <= 4 * 2 ** -8 * max(1.0, ref.abs().max()), (b, (got - ref).abs().max())
        at += c


@pytest.mark.gpu
@pytest.mark.parametrize("design", ["dufitar", "napuzen"])
def test_a_model_gives_the_same_logits_both_ways_and_for_mixed_steps(design, monkeypatch):
    from xinfer_b200.engine.runner import ModelRunner, StepInput
    from xinfer_b200.parts import latent_attention as part
    d, H, rot = 64, 2, dict(dims=32, base=1000.0)
    dense = dict(kind="dense", ff=128, limit=7.0)
    if design == "dufitar":
        m = dict(heads=H, dim=d, rot_dim=32, vdim=d, kv_rank=64, scale=0.1, mask=dict(size=150), rot=rot)
        layers = [dict(type="latent_attention", mixer=m, mlp=dense), dict(type="latent_attention", mixer=dict(m, kv_from=0), mlp=dense)]
        cfg = dict(architecture="Dufitar", vocab=300, width=128, norm=dict(eps=1e-6), residual_mult=0.5, embedding=dict(scale=2.0), layers=layers)
    else:
        one = dict(type="latent_attention", mlp=dense, mixer=dict(heads=H, dim=d, rot_dim=32, vdim=d, q_rank=96, kv_rank=64, scale=0.1, rot=rot))
        two = dict(type="latent_attention_2", mlp=dense, mixer=dict(heads=H, dim=d, vdim=d, kv_rank=64, scale=0.1, mask=dict(size=100)))
        cfg = dict(architecture="Napuzen", vocab=300, width=128, norm=dict(eps=1e-6), canon=dict(taps=4), logit_scale=0.8, layers=[one, two])
    ids = np.random.default_rng(1).integers(0, 300, size=400)

    def logits(rates):
        monkeypatch.setattr(part, "ROWS_RATES", rates)
        r = ModelRunner.random(cfg, 3, block_size=16, num_blocks=128, max_num_seqs=4, max_model_len=512)
        before = kernels.launch_counts().get("attn_rows_tc", 0)
        a, b = r.open_request(), r.open_request()
        out = [r.step([StepInput(a, ids[:200], [7, 199])]).clone()]
        out.append(r.step([StepInput(a, ids[200:201], [0]), StepInput(b, ids[:333], [332])]).clone())      # one token beside a prompt
        out.append(r.step([StepInput(b, ids[333:400], [66]), StepInput(a, ids[201:204], [2])]).clone())     # portions behind cached tokens
        r.check_errors()
        return torch.cat(out).double(), kernels.launch_counts().get("attn_rows_tc", 0) - before
    want, none = logits((1e30, 1.0, 1.0, 1e30, 1e30))         # attention over the rows themselves
    got, some = logits((1e-9, 1e30, 1e30, 0.0, 0.0))         # on formed keys and values wherever they may be
    assert none == 0 and some == 6
    # two bfloat16 computations of the same numbers
    assert (got - want).norm() <= 0.02 * want.norm()


@pytest.mark.parametrize("counts,starts,window,most", [([1], [0], None, 4), ([5, 4, 300], [7, 900, 40], None, 4), ([5, 4, 300, 1], [7, 900, 40, 0], 33, 4),
                                                       ([2, 2], [9, 9], 1, 0)])
def test_the_sums_over_portions(counts, starts, window, most):
    got = kernels.portion_sums(np.concatenate([[0], np.cumsum(counts)]), starts, len(counts), most, window)
    for part, at in ((lambda n: n > most, 0), (lambda n: n <= most, 5)):
        them = [(n, s if not window else min(s, window)) for n, s in zip(counts, starts) if part(n)]
        pairs = [n * s + n * (n + 1) / 2 for n, s in them]
        if window:
            pairs = [min(p, n * window) for p, (n, _) in zip(pairs, them)]
        assert got[at:at + 5] == [len(them), sum(n for n, _ in them), sum(n + s for n, s in them), sum(pairs),
                                  max([n + s for n, s in them], default=0)]


# What was measured as steps of four layers: which way was the faster one (heads, rank; portions; requests that decode at a context).
@pytest.mark.parametrize("heads,rank,prompts,live,context,pays", [
    (32, 512, [(0, 2048)], 0, 0, True), (32, 512, [(3000, 300)], 0, 0, True), (32, 512, [(2000, 16)], 0, 0, True), (16, 256, [(3000, 300)], 0, 0, True),
    (32, 512, [(0, 1275), (0, 632)], 0, 0, True), (16, 256, [(0, 100)] * 8, 0, 0, False), (32, 512, [(0, 30)], 32, 1000, False),
    (32, 512, [(0, 512)], 4, 500, False), (32, 512, [(0, 512)], 16, 1000, False), (32, 512, [(0, 200)], 24, 2000, False),
    (32, 512, [(0, 512)], 48, 3000, False), (32, 512, [(0, 100)], 8, 4000, False), (32, 512, [(1000, 40)] * 3, 4, 200, False),
    (32, 512, [(0, 2048)], 4, 500, True), (32, 512, [(0, 6)], 8, 1000, False)])
def test_the_way_that_was_measured_to_be_faster_is_taken(heads, rank, prompts, live, context, pays):
    from types import SimpleNamespace as N
    from xinfer_b200.parts.latent_attention import rows_pay
    counts, starts = [1] * live + [n for _, n in prompts], [context] * live + [s for s, _ in prompts]
    ctx = N(max_context=max(a + b for a, b in zip(counts, starts)), real_tokens=sum(counts), real_entries=len(counts),
            h_q_start=np.concatenate([[0], np.cumsum(counts)]), h_start_pos=np.asarray(starts))
    got = rows_pay(ctx, heads, 128, rank // 8, 128, rank, rank + rank // 8, None)
    assert got == (live if pays else None)


def _one_portion(T, heads, d, dv, rank, g):
    """What ``attn_rows_tc`` takes for a prompt of T tokens: (work, CTAs, q, kv, rows, q_start, start_pos, err)."""
    host, ctas, n, _ = kernels.latent_prefill_work([T], [0], 4, None, heads)
    bf = lambda *s: torch.randn(*s, generator=g).bfloat16().to(DEV)
    i32 = lambda *a: torch.tensor(a, dtype=torch.int32, device=DEV)
    return host.to(DEV), ctas, bf(T, heads * d), bf(n, heads * (d + dv)), bf(n, rank), i32(0, T), i32(0), i32(0)


@pytest.mark.gpu
@pytest.mark.parametrize("key", [0, 3, 7, 38, 63, 64, 130])
def test_a_key_that_is_not_a_number_shows_in_every_query_that_sees_it(key):
    T, H, d, dv, rank = 200, 2, 64, 64, 64
    work, ctas, q, kv, rows, q_start, start_pos, err = _one_portion(T, H, d, dv, rank, torch.Generator().manual_seed(key))
    out = torch.zeros(T, H * dv, dtype=torch.bfloat16, device=DEV)
    kv[key, :H * d] = float("nan")           # the keys of both heads; the values stay numbers
    kernels.attn_rows_tc(out, q, H * d, kv, rows, work, ctas, q_start, start_pos, H, d, 0, dv, rank, None, d ** -0.5, None, err)
    bad = torch.isnan(out)
    assert int(err) == 0 and bad[key:].all() and not bad[:key].any()


@pytest.mark.gpu
def test_a_full_device_keeps_to_the_rows_and_a_growing_context_moves_its_scratch_rarely(monkeypatch):
    from xinfer_b200.engine.runner import ModelRunner, StepInput
    from xinfer_b200.parts import latent_attention as part
    from xinfer_b200.parts.base import Workspace
    m = dict(heads=2, dim=64, rot_dim=32, vdim=64, kv_rank=64, scale=0.1, rot=dict(dims=32, base=1000.0))
    cfg = dict(architecture="Dufitar", vocab=300, width=128, norm=dict(eps=1e-6), residual_mult=0.5, embedding=dict(scale=2.0),
               layers=[dict(type="latent_attention", mixer=m, mlp=dict(kind="dense", ff=128, limit=7.0))])
    ids = np.random.default_rng(1).integers(0, 300, size=1000)
    monkeypatch.setattr(part, "ROWS_RATES", (1e-9, 1e30, 1e30, 0.0, 0.0))

    def logits():
        r = ModelRunner.random(cfg, 3, block_size=16, num_blocks=128, max_num_seqs=4, max_model_len=1024)
        before, a, out, places = kernels.launch_counts().get("attn_rows_tc", 0), r.open_request(), [], []
        for at in range(0, 1000, 40):
            out.append(r.step([StepInput(a, ids[at:at + 40], [39])]).clone())
            buf = r.workspace._bufs.get("latent.kv")
            places.append(None if buf is None else (buf.data_ptr(), buf.numel()))
        r.check_errors()
        return torch.cat(out).double(), kernels.launch_counts().get("attn_rows_tc", 0) - before, places
    got, some, places = logits()
    assert some == 25 and len(set(places)) == 5                 # 64, 128, 256, 512 and 1,024 rows
    monkeypatch.setattr(Workspace, "reserve", lambda *a: False)
    want, none, places = logits()
    assert none == 0 and set(places) == {None}
    assert (got - want).norm() <= 0.02 * want.norm()             # two bfloat16 computations of the same numbers


@pytest.mark.gpu
def test_a_work_list_that_was_cut_off_is_refused():
    T, H, d, dv, rank = 300, 2, 64, 64, 64
    work, ctas, q, kv, rows, q_start, start_pos, err = _one_portion(T, H, d, dv, rank, torch.Generator().manual_seed(1))
    _, _, n, at = kernels.latent_prefill_work([T], [0], 4, None, H)
    out = torch.zeros(T, H * dv, dtype=torch.bfloat16, device=DEV)

    def run(work, kv=kv, rows=rows, at=at):
        kernels.attn_rows_tc(out, q, H * d, kv, rows, work, ctas, q_start, start_pos, H, d, 0, dv, rank, None, 0.1, None, err, at)
    for bad in (dict(work=work[:-1].contiguous()), dict(work=work[:ctas + 1].contiguous()), dict(work=work[:-4].contiguous()),
                dict(work=work, kv=kv[:-64].contiguous(), rows=rows[:-64].contiguous(), at=None), dict(work=work[:-1].contiguous(), at=None)):
        with pytest.raises(kernels.KernelError):
            run(**bad)
    run(work)
    run(work, at=None)
    assert int(err) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("key,channel,value", [(0, 0, math.nan), (100, 71, math.inf), (127, 3, -math.inf), (128, 8, math.nan), (190, 70, math.nan),
                                               (250, 9, math.inf), (449, 5, math.nan)])
@pytest.mark.parametrize("window", [None, 70])
def test_a_row_that_is_not_finite_reaches_only_the_queries_that_see_it(key, channel, value, window):
    H, d, rd, dv, rank, ps, start, n = 3, 64, 8, 64, 72, 16, 150, 300
    g = torch.Generator().manual_seed(key)
    i32 = lambda *a: torch.tensor(a, dtype=torch.int32, device=DEV)
    end, width = start + n, rank + rd
    rows_in, q = torch.randn(end, width, generator=g).bfloat16(), torch.randn(n, H * (d + rd), generator=g).bfloat16().to(DEV)
    w_kv = (torch.randn(H * (d + dv), rank, generator=g) * rank ** -0.5).bfloat16().to(DEV)
    per = -(-end // ps)
    host, ctas, total, at = kernels.latent_prefill_work([n], [start], 4, window, H)
    work, q_start, start_pos, err, table = host.to(DEV), i32(0, n), i32(start), i32(0), torch.arange(per, dtype=torch.int32, device=DEV).view(1, per)

    def run(rows_in):
        pages = torch.zeros(per * ps, width, dtype=torch.bfloat16)
        pages[:end] = rows_in
        rows, bad = torch.empty(total, width, dtype=torch.bfloat16, device=DEV), torch.full((total // 32,), -1, dtype=torch.int32, device=DEV)
        kernels.latent_gather(rows, pages.to(DEV).view(per, ps, width), work, at, q_start, start_pos, table, per, window, err, rank=rank, bad=bad)
        out = torch.zeros(n, H * dv, dtype=torch.bfloat16, device=DEV)
        kernels.attn_rows_tc(out, q, H * (d + rd), rows[:, :rank] @ w_kv.t(), rows, work, ctas, q_start, start_pos, H, d, rd, dv, rank, window,
                             (d + rd) ** -0.5, None, err, at, bad)
        assert int(err) == 0
        return out.cpu(), bad.cpu()
    clean, none = run(rows_in)
    assert not none.any() and torch.isfinite(clean).all()
    rows_in[key, channel] = value
    got, bad = run(rows_in)
    first = max(0, start - window + 1) if window else 0
    assert sum(bin(int(b) & 0xFFFFFFFF).count("1") for b in bad) == (1 if key >= first else 0)
    sees = torch.tensor([key <= start + i and (window is None or key > start + i - window) for i in range(n)])
    assert torch.isnan(got[sees]).all() and torch.equal(got[~sees], clean[~sees])


@pytest.mark.gpu
@pytest.mark.parametrize("rank,parts,shift", [(8, 2, 0), (72, 64, 0), (512, 18, 0), (512, 65, 0), (512, 130, 0), (136, 3, 2), (512, 70, 2)])
def test_merge_of_key_ranges_against_64_bits(rank, parts, shift):
    """Vectors of four columns and single ones (scratch that starts on an 8-byte boundary only), factors for more than 64 ranges, ranges
    without keys.  Scratch that starts off an 8-byte boundary, where the ranges' sums cannot be stored, is refused by the host."""
    from xinfer_b200 import kernels as k
    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(rank + parts)
    nh, ps, contexts = 3, 16, [700, 1, 130]
    dk, T = rank + (-rank % 16) + 16, 3
    per = 700 // ps + 1
    rows = torch.randn(T * per, ps, dk, generator=g).bfloat16()
    q = (torch.randn(T, nh, dk, generator=g) / math.sqrt(dk)).bfloat16()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    table = torch.arange(T * per, dtype=torch.int32, device=dev).view(T, per)
    out = torch.full((T, nh, rank), float("nan"), dtype=torch.bfloat16, device=dev)
    po = torch.full((T * nh * parts * rank + 6,), float("nan"), device=dev)[shift:]
    pml = torch.full((T * nh * parts * 2,), float("nan"), device=dev)
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    args = (out, q.to(dev), rows.to(dev), i32([0, 1, 2, 3]), i32([n - 1 for n in contexts]), T, table, per, None, 1.0, None, err)
    k.attn_latent_mma(*args, parts=parts, part_o=po, part_ml=pml)
    with pytest.raises(k.KernelError):
        k.attn_latent_mma(*args, parts=parts, part_o=po[1:], part_ml=pml)
    assert int(err) == 0
    for b, n in enumerate(contexts):
        keys = rows[b * per:(b + 1) * per].reshape(-1, dk)[:n].double()
        w = torch.softmax(q[b].double() @ keys.t(), 1)
        ref, terms = w @ keys[:, :rank], w @ keys[:, :rank].abs()
        # as for any attention with weights in bfloat16: 2^-8 of every term and of their sum, 2^-8 of the result, float32 for the rest
        assert ((out[b].double().cpu() - ref).abs() <= (2.0 ** -8 + 2.0 ** -16) * terms + 2.0 ** -7 * ref.abs()).all(), (b, n)
