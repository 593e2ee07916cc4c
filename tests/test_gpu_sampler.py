"""The sampler's cluster form where its list of values can go wrong: short rows, rows of equal values, rows that are not
finite, against the plain sampler."""
import numpy as np
import pytest
import torch

import plain_sampling as ps
from sonicboom_b200 import ops
from sonicboom_b200.sampling import Sampler, Sampling

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def plain(row, s, position, history=()):
    return ps.sample_token(row.cpu().numpy(), ps.Params(temperature=s.temperature, top_k=s.top_k, top_p=s.top_p, min_p=s.min_p,
                                                        seed=s.seed, repeat_penalty=s.repeat_penalty,
                                                        repeat_last_n=s.repeat_last_n, presence_penalty=s.presence_penalty,
                                                        frequency_penalty=s.frequency_penalty), position, history)


def rows(vocab):
    """Rows of different making: normal, the largest in one block's share, few distinct values (more equal ones than the
    list holds), all equal, both zeros (for the argmax; a draw takes the positive ones first), mostly -inf."""
    g = torch.Generator().manual_seed(vocab)
    x = torch.randn(6, vocab, generator=g) * 2
    at = torch.arange(vocab)
    x[1] += 50.0 * ((at // 32) % 8 == 3)               # the fourth block's values, all of the candidates
    x[2] = torch.round(x[2])
    x[3] = 0.25
    x[4] = torch.where(at % 2 == 0, 0.0, -0.0)
    x[5, : vocab - min(vocab, 5)] = float("-inf")
    return x.to(DEV)


# one value, less than a warp, one more than the candidates, more than the list, up to here in one block; in two blocks; in eight
@pytest.mark.parametrize("vocab", [1, 31, 257, 3000, 9001, 40000])
def test_tokens_of_every_kind_of_row(vocab):
    sampler, x = Sampler(DEV), rows(vocab)
    history = [[3 % vocab, 0, 3 % vocab]] * len(x)
    kinds = [Sampling(), Sampling(temperature=0.7, seed=3), Sampling(temperature=1.3, seed=4, top_p=0.9, min_p=0.01),
             Sampling(temperature=0.9, seed=5, top_k=7), Sampling(temperature=0.8, seed=6, repeat_penalty=1.3, presence_penalty=0.5)]
    for s in (k.checked() for k in kinds):
        if s.temperature > 0:
            x[4] = 0.0
        kept = x.clone()
        got = sampler.sample(x, [s] * len(x), [11 + i for i in range(len(x))], history)
        assert got == [plain(r, s, 11 + i, history[i]) for i, r in enumerate(x)], s
        assert torch.equal(x.view(torch.int32), kept.view(torch.int32))        # the row is as it was


@pytest.mark.parametrize("n", [42, 90, 180])
def test_tokens_of_many_rows(n):
    """Rows whose blocks would not all run at once are shared by four, two or one: the tokens of the same rows with eight."""
    sampler, x = Sampler(DEV), rows(33001)
    x[4] = 0.0
    many = x.repeat(n // 6, 1)
    for s in (Sampling().checked(), Sampling(temperature=0.7, seed=3).checked(), Sampling(temperature=0.9, seed=5, top_p=0.8, repeat_penalty=1.2).checked()):
        few = sampler.sample(x, [s] * 6, [11 + i for i in range(6)], [[7, 3]] * 6)
        assert sampler.sample(many, [s] * n, [11 + i % 6 for i in range(n)], [[7, 3]] * n) == few * (n // 6), s


@pytest.mark.parametrize("vocab", [9, 900, 40000])
@pytest.mark.parametrize("win", [1, 3, 130, 1023, 1024])
def test_penalties_over_windows_of_any_length(vocab, win):
    """Windows that end inside a group of four, with a token in many places, ids outside the vocabulary, up to the longest."""
    sampler, x = Sampler(DEV), rows(vocab)[:2]
    g = torch.Generator().manual_seed(win)
    history = torch.randint(-2, min(vocab, 700) + 2, (2, win), generator=g).tolist()
    for s in (Sampling(repeat_penalty=1.3, presence_penalty=0.5, frequency_penalty=0.2, repeat_last_n=1024).checked(),
              Sampling(temperature=0.8, seed=6, repeat_penalty=1.3, frequency_penalty=0.1, repeat_last_n=1024).checked()):
        kept = x.clone()
        got = sampler.sample(x, [s] * 2, [5, 6], history)
        assert got == [plain(r, s, 5 + i, [t for t in history[i] if 0 <= t < vocab]) for i, r in enumerate(x)], s
        assert torch.equal(x.view(torch.int32), kept.view(torch.int32))


def test_rows_that_are_not_finite():
    x = torch.randn(3, 5000, generator=torch.Generator().manual_seed(1)).to(DEV)
    x[0, 100], x[1, 17], x[2, 4999] = float("nan"), float("inf"), float("nan")
    x[2, 10:20] = float("-inf")
    want = [int(torch.nan_to_num(r, nan=-9.0, posinf=99.0, neginf=-9.0).argmax()) for r in x]
    assert Sampler(DEV).sample(x, [Sampling().checked()] * 3, [0] * 3, [[]] * 3) == want
    ids = torch.empty(3, dtype=torch.int32, device=DEV)
    from sonicboom_b200.sampling.sampler import pack_params
    rec, _ = pack_params([Sampling(temperature=0.7, seed=1).checked()] * 3, [5] * 3, [[]] * 3)
    ops.sample(x, torch.from_numpy(rec).to(DEV), None, ids)
    ids = ids.tolist()
    assert ids[1] == 17 and 0 <= ids[0] < 5000 and ids[0] != 100 and 0 <= ids[2] < 4999
    z = np.where(np.isnan(x[0].cpu().numpy()), -np.inf, x[0].cpu().numpy())
    assert ids[0] == ps.sample_token(z, ps.Params(temperature=0.7, seed=1), 5)
