"""State-space scans whose blocks follow the entries' lengths (csrc/ragged.cu): many entries, equal lengths, one long portion among tokens, more blocks than SMs and fewer,
each entry against the oracle by itself."""
import numpy as np
import pytest

from tests.test_fosovik import F32_TOL, FULL, all_rows, make, rel, tokens

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[1] * 12, [3, 3, 3, 90, 90, 1], [1] * 11 + [130], [130] + [1] * 3, [16, 17, 15, 33, 32, 31, 1, 2]])
def test_entries_of_any_order(lens):
    check(lens, 12)


@pytest.mark.parametrize("lens", [[1] * 64, [1] * 40 + [5, 70, 2, 70] + [1] * 20])
def test_every_slot_taken(lens):
    check(lens, 64)


def check(lens, slots):
    m, o = make(FULL, 13, precision="f32", max_tokens=2048 if slots == 12 else 8192, max_batch=slots)
    prompts = [tokens(n + 2, FULL["vocab"], 40 + i) for i, n in enumerate(lens)]
    seqs = [0] + [m.seq_create() for _ in lens[1:]]
    first = m.step_batch([(s, p[:n], all_rows(n)) for s, p, n in zip(seqs, prompts, lens)])
    second = m.step_batch([(s, p[n:], all_rows(2)) for s, p, n in reversed(list(zip(seqs, prompts, lens)))])
    at = 0
    for i, (p, n) in enumerate(zip(prompts, lens)):
        want = o.forward(p, o.new_state()).numpy()
        back = 2 * (len(lens) - 1 - i)
        got = np.concatenate([first[at: at + n], second[back: back + 2]])
        assert rel(got, want) < F32_TOL, (i, n)
        at += n
    m.close()
