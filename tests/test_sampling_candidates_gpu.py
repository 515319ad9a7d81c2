"""Candidates of the sampler: the short way to the k largest (csrc/sampling.cu) against the definition, where it can go wrong --
ties at the k-th value, k near the threads' number, zeros of both signs, infinities, short rows."""
import numpy as np
import pytest
import torch

import plain_sampler as PS

pytestmark = pytest.mark.gpu


def rows(kind, n, V, rng):
    x = rng.standard_normal((n, V)).astype(np.float32)
    if kind == "ties":
        x = np.round(x * 2) / 2
    elif kind == "equal":
        x[:] = 1.25
    elif kind == "zeros":
        x = np.where(rng.random((n, V)) < 0.5, np.float32(-0.0), np.float32(0.0))
    elif kind == "masked":
        x[:, V // 3:] = np.finfo(np.float32).min
        x[:, : V // 8] = -np.inf
    elif kind == "few":
        x[:] = -np.inf
        x[:, [0, V // 2, V - 1]] = [1.0, 3.0, 2.0]
    return x


@pytest.mark.parametrize("kind", ["plain", "ties", "equal", "zeros", "masked", "few"])
@pytest.mark.parametrize("V", [7, 331, 1024, 1025, 65536])
def test_top_k_candidates(kind, V):
    from kappai_b200 import SamplingParams
    from kappai_b200.sampling import uniform
    from kappai_b200.sampling.sampler import sample
    n = 6
    x = rows(kind, n, V, np.random.default_rng(V))
    filters = [dict(top_p=1.0, min_p=0.0), dict(top_p=0.9, min_p=0.1), dict(top_p=0.5, min_p=0.0)] * 2
    for k in (2, 3, 40, 200, 1000, 1024):
        if k >= V:
            continue
        got = sample(torch.from_numpy(x).cuda(), [SamplingParams(temperature=0.7, top_k=k, **f) for f in filters],
                     [i + 1 for i in range(n)], [3] * n).cpu().tolist()
        for i, f in enumerate(filters):
            if kind == "zeros":
                # the selection's order puts 0 before -0, the plain sampler's takes them as equal
                assert (np.signbit(x[i]) == 0).sum() < k or not np.signbit(x[i, got[i]])
                continue
            want, slack = PS.sample(x[i], uniform(i + 1, 3), temperature=0.7, top_k=k, **f)
            assert got[i] == want or slack < 1e-5, (kind, V, k, f, got[i], want, slack)


@pytest.mark.parametrize("V", [1024, 1025, 65536])
@pytest.mark.parametrize("k", [512, 600, 601, 0])
def test_rows_on_either_side_of_the_short_way(V, k):
    """k at the line and no k at all (the 1024 largest), of rows that are masked but for fewer than k too."""
    from kappai_b200 import SamplingParams
    from kappai_b200.sampling import uniform
    from kappai_b200.sampling.sampler import sample
    if k >= V:
        return
    rng = np.random.default_rng(V + k)
    x = np.stack([rows(kind, 1, V, rng)[0] for kind in ("plain", "ties", "equal", "masked", "few")])
    f = dict(top_p=0.9, min_p=0.0)
    got = sample(torch.from_numpy(x).cuda(), [SamplingParams(temperature=0.7, top_k=k, **f)] * len(x), [i + 1 for i in range(len(x))],
                 [3] * len(x)).cpu().tolist()
    for i in range(len(x)):
        want, slack = PS.sample(x[i], uniform(i + 1, 3), temperature=0.7, top_k=k, **f)
        assert got[i] == want or slack < 1e-5, (V, k, i, got[i], want, slack)


@pytest.mark.parametrize("V,k", [(65536, 4), (65536, 40), (65536, 601), (65536, 0), (1025, 200), (1000, 0), (500, 3)])
@pytest.mark.parametrize("kind", ["one", "several", "negative", "most"])
def test_a_nan_counts_as_minus_infinity(V, k, kind):
    """... in every row alike: 64 rows of the same values, a uniform number each."""
    from kappai_b200 import SamplingParams
    from kappai_b200.sampling import uniform
    from kappai_b200.sampling.sampler import sample
    x = np.random.default_rng(V).standard_normal(V).astype(np.float32)
    at = {"one": [V // 3], "several": [1, V // 3, int(np.argmax(x)), V - 2], "negative": [V // 3], "most": list(range(2, V))}[kind]
    x[at] = np.array([0xffc00001 if kind == "negative" else 0x7fc00000], np.uint32).view(np.float32)[0]
    plain = np.where(np.isnan(x), np.float32(-np.inf), x)
    for f in (dict(top_p=1.0, min_p=0.01), dict(top_p=0.9, min_p=0.0)):
        got = sample(torch.from_numpy(np.tile(x, (64, 1))).cuda(), [SamplingParams(temperature=0.7, top_k=k, **f)] * 64, list(range(64)), [3] * 64)
        for i, tok in enumerate(got.cpu().tolist()):
            want, slack = PS.sample(plain, uniform(i, 3), temperature=0.7, top_k=k, **f)
            assert tok == want or slack < 1e-5, (i, tok, want, slack)
