"""Which form of the latent attention a step's prompt portions take, on the CPU: the estimate against times measured of both forms, and
the short answers against the estimate."""
import random

import pytest

from leone_b200.ops.cuda import latent_short_answer, latent_times

# tokens, cached tokens before them, sequences, heads, window, us on tcgen05, us on mma.sync
MEASURED = [
    (8, 0, 1, 16, 0, 15.2, 8.8), (64, 0, 1, 16, 0, 15.4, 14.2), (96, 0, 1, 16, 0, 17.8, 20.7), (256, 0, 1, 16, 0, 24.8, 36.0),
    (8, 128, 1, 16, 0, 21.1, 17.7), (48, 128, 1, 16, 0, 21.3, 18.8), (64, 128, 1, 16, 0, 21.4, 24.9), (64, 512, 1, 16, 0, 41.0, 48.2),
    (8, 1024, 1, 16, 0, 68.2, 31.3), (64, 1024, 1, 16, 0, 68.2, 82.5), (2, 8192, 1, 16, 1024, 60.3, 21.4), (48, 8192, 1, 16, 1024, 66.6, 57.6),
    (64, 8192, 1, 16, 128, 21.4, 17.3), (96, 8192, 1, 16, 128, 21.5, 27.6), (8, 16384, 1, 16, 0, 824.5, 150.2), (32, 16384, 1, 16, 0, 824.1, 516.7),
    (64, 16384, 1, 16, 0, 823.3, 1012.1), (8, 32768, 1, 16, 0, 1606.9, 275.1), (2048, 0, 1, 16, 0, 233.2, 562.0), (16, 16384, 1, 32, 0, 822.1, 515.9),
    (32, 16384, 1, 32, 0, 823.3, 1012.5), (8, 0, 16, 16, 0, 15.4, 13.3), (128, 0, 16, 16, 0, 63.2, 67.3), (8, 8192, 3, 16, 0, 424.6, 182.0),
    (16, 8192, 3, 16, 0, 423.1, 344.5), (32, 8192, 3, 16, 0, 424.9, 942.3), (4, 4096, 1, 128, 0, 215.6, 140.6), (8, 4096, 1, 128, 0, 222.0, 264.9)]


@pytest.mark.parametrize("q,before,seqs,heads,window,tcgen05,mma", MEASURED)
def test_the_faster_form_is_chosen(q, before, seqs, heads, window, tcgen05, mma):
    a, b = latent_times([q] * seqs, [q + before] * seqs, heads // 16, window, 0)
    assert (a < b) == (tcgen05 < mma)


def test_short_answers_agree_with_the_estimate():
    rng = random.Random(5)
    given = {True: 0, False: 0}
    for _ in range(4000):
        q = [max(1, int(2 ** rng.uniform(0, 11))) for _ in range(rng.choice([1, 1, 2, rng.randint(1, 12)]))]
        ctx = [n + int(2 ** rng.uniform(0, 15)) - 1 for n in q]
        window, groups = rng.choice([0, 0, 100, 1024]), rng.choice([1, 2, 8])
        answer = latent_short_answer(sum(q), len(q), groups, max(ctx), window)
        if answer is not None:
            a, b = latent_times(q, ctx, groups, window, 0)
            assert a < 1.25 * b if answer else b < a, (q, ctx, window, groups, a, b)
            given[answer] += 1
    assert min(given.values()) > 300
