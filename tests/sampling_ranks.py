"""Which tokens a sampler with 32-bit running sums may draw from a sorted short list: for the tests."""

import numpy as np

ROUNDING = 2e-6          # of the mass of the list: running 32-bit sums of its weights


def kept(row, k):
    """Indices of the k largest, equal logits by rising index."""
    return np.lexsort((np.arange(len(row)), -row.astype(np.float64)))[:k]


def cumulative(row, order, temperature):
    w = np.exp((row[order].astype(np.float64) - float(row[order[0]])) / temperature)
    return np.cumsum(w)


def _reaches(run, target):
    """Ranks at which the running mass may be found to reach the target: a boundary within rounding of it counts
    for both of its sides."""
    slack = ROUNDING * run[-1]
    before = np.concatenate(([-np.inf], run[:-1]))
    return np.flatnonzero((run >= target - slack) & (before < target + slack))


def ranks(run, top_p, u):
    """(the rank to draw, the ranks that rounding may turn it into)."""
    cuts = _reaches(run, np.float32(top_p) * run[-1]) if top_p < 1.0 else np.array([len(run) - 1])
    cut = int(np.argmax(run >= np.float32(top_p) * run[-1])) if top_p < 1.0 else len(run) - 1
    want = int(np.argmax(run >= np.float32(u) * run[cut]))
    return want, set(int(r) for c in cuts for r in _reaches(run, np.float32(u) * run[c]))
