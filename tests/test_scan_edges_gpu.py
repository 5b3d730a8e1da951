"""The scans over matrix states where a lane's rows change (64 and 65, 256 and 257, 512 rows), with portions that leave every
remainder of a group of four tokens, against the plain recurrences in float64."""
import pytest
import torch
import torch.nn.functional as F

import plain_gulipel as plain
import test_dalalix_gpu as dalalix
import test_gulipel_gpu as gulipel
import test_napuzen_gpu as napuzen

pytestmark = pytest.mark.gpu

LENS = [23, 4, 1]
PORTIONS = [[7, 5, 1, 2, 3, 4, 1], [3, 1], [1]]


def _tolerance(rows):
    # A sum over rows is rounded at most 16 + 5 times (a lane's own, the shuffles) and a few more where it is formed, the state
    # once per token; the terms of a sum of `rows` random signs are together about sqrt(rows) times the sum.
    return (24 + max(LENS)) * 2.0 ** -24 * rows ** 0.5


@pytest.mark.parametrize("cols", [6, 130])
@pytest.mark.parametrize("rows", [64, 65, 256, 257, 512])
def test_scans_where_a_lanes_rows_change(rows, cols):
    H, slots, cuts = 2, [3, 1, 0], ([[n] for n in LENS], PORTIONS)
    dt_bias, a_log, d_skip = gulipel._rand(H, seed=1), gulipel._rand(H, seed=2), gulipel._rand(H, seed=3)
    f = lambda t: t.float().double()
    ins = gulipel._scan_inputs(LENS, H, cols, rows, 1, seed=rows)
    want = [plain.selective_scan(f(i["x"]), f(i["B"]).repeat_interleave(H, dim=1), f(i["C"]).repeat_interleave(H, dim=1),
                                 F.softplus(f(i["dt"]) + f(dt_bias)), torch.exp(f(a_log)), f(d_skip)).reshape(-1, H * cols)
            for i in ins]
    for c in cuts:
        got = gulipel._run_scan(ins, c, slots, H, cols, rows, 1, dt_bias, a_log, d_skip,
                                torch.zeros(4, H, rows, cols, device="cuda:0"))
        for g, w in zip(got, want):
            gulipel._close(g, w, _tolerance(rows))
    ins, bias = gulipel._delta_inputs(LENS, H, 1, rows, cols, seed=rows), gulipel._rand(H, rows, seed=4)
    want = [gulipel._delta_plain(i, H, 1, rows, cols, bias, a_log) for i in ins]
    for c in cuts:
        got = gulipel._run_delta(ins, c, slots, H, 1, rows, cols, bias, a_log, torch.zeros(4, H, rows, cols, device="cuda:0"))
        for g, w in zip(got, want):
            gulipel._close(g, w, _tolerance(rows))
    steps = [[(r, n) for r, n in enumerate(LENS)]], [[(0, 7), (1, 3)], [(0, 5), (2, 1)], [(1, 1), (0, 1)], [(0, 10)]]
    for c in steps:
        for g, w in zip(*napuzen._scan_steps(H, rows, cols, LENS, c, seed=rows)):
            assert (g - w).abs().max() <= _tolerance(rows) * (1 + w.abs().max())
        for g, w in zip(*dalalix._memory_steps(H, rows, cols, 9.0, LENS, c, seed=rows)):
            assert (g - w).abs().max() <= 1e-4 * (1 + w.abs().max())          # (the divisor may be small: as in its own tests)
