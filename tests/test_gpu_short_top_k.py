"""Sampling from a short top-k, which is gathered and sorted: slices of a row that do not fill a block, the
largest row, k at the ends of its range, ties across blocks, and rows that go to the general search."""

import numpy as np
import pytest
import torch

from sampling_ranks import cumulative, kept, ranks

pytestmark = pytest.mark.gpu


def draw(rows, cases, short_lists=True):
    from from_scratch_inference_engine_b200.kernels import ops
    to = lambda i, dtype: torch.tensor(np.array([c[i] for c in cases]), dtype=dtype, device="cuda")
    out = torch.full((len(cases),), -9, dtype=torch.int32, device="cuda")
    ops.sample(torch.from_numpy(rows).cuda(), to(0, torch.float32), to(1, torch.int32), to(2, torch.float32),
               to(3, torch.float32), out, short_lists=short_lists)
    return out.tolist()


@pytest.mark.parametrize("vocab", [4096, 4099, 32000, 151936, 204800])
def test_short_top_k(vocab):
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
    unsettled = 0
    for r, (got, (temperature, k, p, u)) in enumerate(zip(draw(rows, cases), cases)):
        if temperature <= 0.0:
            assert got == -1
            continue
        row = np.where(np.isnan(rows[r]), -np.inf, rows[r])
        order = kept(row, k)
        want, may = ranks(cumulative(row, order, temperature), p, u)
        if got != order[want]:
            assert got in order[sorted(may)], (r, cases[r], got, order[want])
            unsettled += 1
    assert unsettled <= 2


@pytest.mark.parametrize("vocab", [4099, 151936])
def test_order_of_equal_logits(vocab):
    """u in the middle of a token's step: exactly that token, equal logits by rising index across blocks."""
    rng = np.random.default_rng(vocab + 1)
    picks = [(40, r) for r in (0, 1, 7, 20, 38, 39)] + [(104, r) for r in (0, 50, 102, 103)]
    rows, cases, want = [], [], []
    for kind in range(4):
        for k, rank in picks:
            row = (rng.standard_normal(vocab) * 3).astype(np.float32)
            if kind == 1:
                row[vocab // 8 - 60:vocab // 8 + 60] = row.max() + 1       # a run of ties over the end of a slice
            elif kind == 2:
                row = np.round(row)
            elif kind == 3:
                row[:] = 0.25
            order = kept(row, k)
            run = cumulative(row, order, 4.0)
            below = run[rank - 1] if rank else 0.0
            rows.append(row)
            cases.append((4.0, k, 1.0, (below + run[rank]) / 2 / run[-1]))
            want.append(int(order[rank]))
    assert draw(np.stack(rows), cases) == want
    assert draw(np.stack(rows), cases, short_lists=False) == want          # the search alone
