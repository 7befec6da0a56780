"""Sampling from a short top-k, which is gathered and sorted: slices of a row that do not fill a block, the
largest row, k at the ends of its range, ties across blocks, and rows that go to the general search."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def kept(row, k):
    """Indices of the k largest, equal logits by rising index."""
    return np.lexsort((np.arange(len(row)), -row.astype(np.float64)))[:k]


def cumulative(row, order, temperature):
    w = np.exp((row[order].astype(np.float64) - float(row[order[0]])) / temperature)
    return np.cumsum(w)


@pytest.mark.parametrize("vocab", [4096, 4099, 32000, 151936, 204800])
def test_short_top_k(vocab):
    from from_scratch_inference_engine_b200.kernels import ops
    rng = np.random.default_rng(vocab)
    cases = [(t, k, p, rng.random()) for t in (0.05, 0.8, 2.0) for k in (1, 2, 40, 103, 104, 105)
             for p in (1.0, 0.95, 0.2)]
    cases += [(1.0, 40, 1.0, 0.0), (1.0, 40, 0.95, 0.99999994), (0.0, 40, 0.9, 0.5), (1.0, vocab, 0.9, 0.5)]
    rows = (rng.standard_normal((len(cases), vocab)) * 3).astype(np.float32)
    rows[1, :] = 0.25                                   # all equal: more candidates than there is room for
    rows[3, vocab // 8 - 3:vocab // 8 + 3] = 30.0       # ties where one block's slice ends
    rows[4, ::2] = -np.inf
    rows[5, 7] = np.nan
    rows[6] = np.round(rows[6])                         # few different logits, many ties at the k-th
    to = lambda v, dtype: torch.tensor(np.array(v), dtype=dtype, device="cuda")
    out = torch.full((len(cases),), -9, dtype=torch.int32, device="cuda")
    ops.sample(torch.from_numpy(rows).cuda(), to([c[0] for c in cases], torch.float32),
               to([c[1] for c in cases], torch.int32), to([c[2] for c in cases], torch.float32),
               to([c[3] for c in cases], torch.float32), out)
    for r, (got, (temperature, k, p, u)) in enumerate(zip(out.tolist(), cases)):
        if temperature <= 0.0:
            assert got == -1
            continue
        row = np.where(np.isnan(rows[r]), -np.inf, rows[r])
        order = kept(row, k)
        run = cumulative(row, order, temperature)
        cut = int(np.argmax(run >= np.float32(p) * run[-1])) if p < 1.0 else len(order) - 1
        want = int(np.argmax(run >= np.float32(u) * run[cut]))
        if got != order[want]:
            # float32 sums of at most 2^18 weights: the boundary lies within their rounding
            assert got in order, (r, cases[r])
            at = int(np.where(order == got)[0][0])
            lo, hi = sorted((at, want))
            assert (run[hi - 1] - run[lo]) / run[-1] < 2e-6 or abs(run[lo] - np.float32(u) * run[cut]) / run[-1] < 2e-6, \
                (r, cases[r], got, order[want])
