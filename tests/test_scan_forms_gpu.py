"""The scans take the tokens of a step one by one where no request brings many, else in groups of four; what they compute does not
depend on it, nor on what the caller says of the longest request."""
import numpy as np
import pytest
import torch

from xinfer_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("H,d,dv", [(2, 16, 6), (3, 64, 64), (2, 100, 130), (1, 130, 33), (2, 512, 40)])
@pytest.mark.parametrize("counts", [[1], [1, 1, 1], [16, 2, 0, 5], [17, 1], [70, 3]])
def test_both_forms_give_the_same(H, d, dv, counts):
    g = torch.Generator().manual_seed(d + dv + sum(counts))
    rn = lambda *s: torch.randn(*s, generator=g).to(DEV)
    i32 = lambda a: torch.tensor(np.asarray(a), dtype=torch.int32, device=DEV)
    B, T = len(counts), sum(counts)
    q_start, slots, start = i32(np.concatenate([[0], np.cumsum(counts)])), i32(range(B)), i32([0] * B)
    qkv, ag, proj, vec, bias = rn(T, H * (2 * d + dv)), rn(T, H * d), rn(T, H), rn(H), rn(H * d)
    xbc, alpha, gates = rn(T, H * dv + 2 * d), torch.rand(T, H * d, generator=g).to(DEV), rn(T, H * (2 * d + dv) + 2 * H)
    first = rn(B, H, d, dv)

    def run(longest):
        out = []
        for one in ("selective", "linear", "memory", "delta"):
            o, S = torch.full((T, H * dv), float("nan"), device=DEV), first.clone()
            if one == "selective":
                kernels.selective_scan(o, xbc, proj, 0, vec, vec, vec, S, q_start, slots, B, H, dv, d, 1, longest)
            elif one == "linear":
                kernels.linear_scan(o, qkv, alpha, S, q_start, slots, B, H, d, dv, d ** -0.5, longest)
            elif one == "memory":
                div, state = torch.empty(T, H, device=DEV), dict(S=S, n=torch.zeros(B, H, d, device=DEV), m=torch.zeros(B, H, 2, 2, device=DEV))
                kernels.matrix_memory(o, div, gates, H * (2 * d + dv), vec, vec, 9.0, state, q_start, start, slots, B, H, d, dv, d ** -0.5,
                                      1e-3, longest)
                out += [div, state["n"], state["m"]]
            else:
                kernels.delta_rule(o, qkv, proj, 0, ag, bias, vec, S, q_start, slots, B, H, H, d, dv, longest=longest)
            out += [o, S]
        return out
    few, many = run(1), run(1000)
    for a, b in zip(few[:-2], many[:-2]):
        assert torch.equal(a, b)
    # The two forms of the delta rule add the same terms in another order: a sum over d rows is rounded at most 16 + 5 times, a
    # state and a group's figures a few times per token; the terms of a sum of d random signs are together sqrt(d) times the sum.
    tol = (24 + max(counts)) * 2.0 ** -24 * d ** 0.5
    for a, b in zip(few[-2:], many[-2:]):
        assert torch.isfinite(a).all() and (a - b).abs().max() <= 2 * tol * (1 + b.abs().max())


def test_a_full_device_takes_the_tokens_of_the_delta_rule_one_by_one(monkeypatch):
    from gulipel_models import TINY_G
    from xinfer_b200.engine.runner import ModelRunner, StepInput
    from xinfer_b200.parts.base import Workspace
    cfg, seed, ps = TINY_G["G1"]
    ids = np.random.default_rng(1).integers(0, cfg["vocab"], size=200)

    def logits():
        r = ModelRunner.random(cfg, seed, dtype="f32", block_size=ps, num_blocks=400 // ps + 2, max_num_seqs=2, max_model_len=400)
        out = r.step([StepInput(r.open_request(), ids, [9, 198, 199])]).clone()
        r.check_errors()
        return out.double(), "gdelta.prep" in r.workspace._bufs
    got, scratch = logits()
    monkeypatch.setattr(Workspace, "reserve", lambda *a: False)
    want, none = logits()
    assert scratch and not none
    assert (got - want).norm() <= 1e-4 * want.norm()        # float32 sums in another order, through the layers behind them
