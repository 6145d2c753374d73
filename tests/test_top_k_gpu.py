"""The sampler's lists that start with a top-k: which ids survive, with what probability, and which one is drawn."""
import numpy as np
import pytest
import torch

from tests.test_kernels_gpu import DEV, _randn, ops32  # noqa: F401

pytestmark = pytest.mark.gpu


def _rows(vocab):
    """Rows on which a selection can go wrong: random; all equal; two values; the best values all in one thread's share
    (every 1,024th id), more of them than a thread's maximum shows; both zeros among ties; a few finite; none."""
    rows = [_randn((vocab,), 1, scale=3.0), torch.full((vocab,), 2.5, device=DEV), (_randn((vocab,), 2) > 0).float(),
            _randn((vocab,), 3), torch.where(_randn((vocab,), 4) > 0, 0.0, -0.0), torch.full((vocab,), float("nan"), device=DEV),
            torch.full((vocab,), float("-inf"), device=DEV)]
    rows[3][5::1024] += 50.0
    rows[5][[3, vocab // 2, vocab - 1]] = torch.tensor([1.0, -4.0, 1.0], device=DEV)
    rows[0][7] = float("inf")
    return torch.stack(rows)


@pytest.mark.parametrize("vocab", [17, 1025, 2048, 6000, 151936])
@pytest.mark.parametrize("k", [1, 40, 1000, 1024, 1025])        # 1,024: the last that a block collects
def test_top_k_keeps_the_best_ids_and_draws_among_them(ops32, vocab, k):  # noqa: F811
    from leone_b200.sampling.sampler import TRUNCATION_STAGES
    from tests.plain.model import select, uniform
    logits = _rows(vocab)
    n, t = logits.shape[0], 0.9
    stages = [(TRUNCATION_STAGES["top_k"], float(k)), (TRUNCATION_STAGES["top_p"], 0.97)]
    seeds, positions = list(range(50, 50 + n)), [3 * i for i in range(n)]
    args = (logits, [t] * n, seeds, positions, stages)
    out, probs = ops32.sample_truncated(*args, want_probs=True)
    assert torch.equal(out, ops32.sample_truncated(*args))             # the draw without the dense distribution
    for i, row in enumerate(logits.cpu().numpy().astype(np.float64)):
        ids = np.flatnonzero(np.isfinite(row))
        if not len(ids):
            assert out[i].item() == -1
            continue
        best = ids[np.lexsort((ids, -row[ids]))][:k]
        p = np.exp(row[best] / t - row[best[0]] / t)
        p /= p.sum()
        keep = best[:int(np.searchsorted(np.cumsum(p), 0.97) + 1)]
        got = probs[i].cpu().numpy()
        # (a running sum that meets the limit within its rounding may keep one more or one less)
        assert abs(np.count_nonzero(got) - len(keep)) <= 1 and set(np.flatnonzero(got)) <= set(best)
        few = min(np.count_nonzero(got), len(keep))
        assert (got[best[:few]] > 0).all() and abs(got.sum() - 1.0) < 1e-12
        assert out[i].item() == select(got, uniform(seeds[i], positions[i]))


@pytest.mark.parametrize("vocab", [2049, 4096, 4097, 9001, 151936])      # the first radix-sorted size, a tile of 4,096, remainders
def test_rows_sorted_whole_keep_equal_logits_in_id_order(ops32, vocab):  # noqa: F811
    from leone_b200.sampling.sampler import TRUNCATION_STAGES
    logits = _rows(vocab)
    logits[3] = torch.round(logits[3])                                   # many ties
    logits[1, ::7] = -3e38
    n, t = logits.shape[0], 1.3
    # an epsilon of nearly nothing keeps every finite logit: the distribution is the whole row's
    out, probs = ops32.sample_truncated(logits, [t] * n, list(range(n)), [5] * n, [(TRUNCATION_STAGES["epsilon"], 1e-300)],
                                        want_probs=True)
    # a top-k longer than a block collects is cut from the sorted row: ties at the cut keep the lower ids
    k = min(1500, vocab)
    _, cut = ops32.sample_truncated(logits, [t] * n, list(range(n)), [5] * n, [(TRUNCATION_STAGES["top_k"], float(k))], want_probs=True)
    for i, row in enumerate(logits.cpu().numpy().astype(np.float64)):
        ids = np.flatnonzero(np.isfinite(row))
        if not len(ids):
            assert out[i].item() == -1
            continue
        p = np.zeros(vocab)
        p[ids] = np.exp((row[ids] - row[ids].max()) / t)
        assert np.abs(probs[i].cpu().numpy() - p / p.sum()).max() < 1e-13
        best = ids[np.lexsort((ids, -row[ids]))][:k]
        assert set(np.flatnonzero(cut[i].cpu().numpy())) == set(best[p[best] > 0])
