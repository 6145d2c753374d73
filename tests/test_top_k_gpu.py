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
