"""The records that carry a batch's sampling options to the device (CPU): field by field what each row asked for."""
import dataclasses

import numpy as np
import pytest

from xinfer_b200 import kernels
from xinfer_b200.sampling import SamplingParams
from xinfer_b200.sampling.sampler import PENALTY_HISTORY, fill_records

SHARED = SamplingParams(temperature=0.6, top_k=20, top_p=0.95)
ROWS = [SamplingParams(), SHARED, SHARED, SamplingParams(temperature=1e-9, top_k=-3), SamplingParams(temperature=1e39, top_p=0.0),
        SamplingParams(temperature=2.0, frequency_penalty=0.5), SamplingParams(temperature=0.3, presence_penalty=-1.5, top_k=2 ** 31 - 1),
        dataclasses.replace(SHARED, presence_penalty=0.25), SHARED]


def _field_by_field(rec, params, seeds, draws, histories, hist):
    off = 0
    for r, p in enumerate(params):
        n = 0
        if p.has_penalties and histories is not None:
            h = list(histories[r])[-PENALTY_HISTORY:]
            n = len(h)
            hist[off:off + n] = h
        s = int(seeds[r]) & (2 ** 64 - 1)
        values = dict(temperature=0.0 if p.greedy else float(p.temperature), top_k=int(p.top_k) if p.top_k and p.top_k > 0 else 0,
                      top_p=1.0 if p.top_p is None else float(p.top_p), seed_lo=s & 0xFFFFFFFF, seed_hi=s >> 32,
                      draw=int(draws[r]) & 0xFFFFFFFF, frequency_penalty=float(p.frequency_penalty or 0.0),
                      presence_penalty=float(p.presence_penalty or 0.0), history_offset=off, history_len=n)
        for name, v in values.items():
            rec[r][name] = v
        off += n
    return off


@pytest.mark.filterwarnings("ignore:overflow encountered")
@pytest.mark.parametrize("rows", [[], [0], [1, 2, 8], list(range(len(ROWS))), [5, 5, 6, 7, 5], [1] * 15, [1] * 16, [4] * 20, [5] * 20,
                                  [1] * 19 + [8, 2]])
@pytest.mark.parametrize("with_histories", [False, True])
def test_records_hold_what_every_row_asked_for(rows, with_histories):
    params = [ROWS[i] for i in rows]
    seeds, draws = ([-1, 0, 2 ** 63, 7, 2 ** 40 + 5, 1, -2 ** 62] * 4)[:len(rows)], ([2 ** 32 + 3, 0, -1, 5, 6] * 5)[:len(rows)]
    histories = [list(range(i, i + (PENALTY_HISTORY + 9 if i % 2 else 3))) for i in range(len(rows))] if with_histories else None
    made = []
    for fill in (fill_records, _field_by_field):
        rec, hist = np.full(24 * 40, 255, dtype=np.uint8).view(kernels.SAMPLE_PARAMS), np.zeros(24 * PENALTY_HISTORY, dtype=np.int32)
        made.append((fill(rec, params, seeds, draws, histories, hist), rec.tobytes(), hist.tobytes()))
    assert made[0] == made[1]


def test_seeds_that_fit_64_signed_bits_and_others_are_filled_alike():
    for seeds in ([2 ** 63] * 16, [2 ** 63 - 1] * 16, [-2 ** 63] * 16, [-2 ** 63 - 1] * 16, [0, 2 ** 64 + 9] * 8):
        rec = np.zeros(16, dtype=kernels.SAMPLE_PARAMS)
        fill_records(rec, [SHARED] * 16, seeds, [1] * 16, None, np.zeros(1, dtype=np.int32))
        assert [int(r["seed_lo"]) | int(r["seed_hi"]) << 32 for r in rec] == [s & (2 ** 64 - 1) for s in seeds]


def test_a_number_that_no_field_holds_is_refused():
    rec = np.zeros(1, dtype=kernels.SAMPLE_PARAMS)
    with pytest.raises(OverflowError):
        fill_records(rec, [SamplingParams(temperature=1.0, top_k=2 ** 40)], [0], [0], None, np.zeros(1, dtype=np.int32))
