"""Results as Python callers hold them: a dataclass whose scales are the norms'
as they were made, and whose arrays are its own."""

import copy
import dataclasses
import pickle

import numpy as np
import pytest

from vqm_b200 import ss2


def _norms(scales=6):
    return np.random.default_rng(scales).random((scales, 18))


@pytest.mark.parametrize("scales", [1, 4, 6])
def test_scales_are_a_field(scales):
    norms = _norms(scales)
    r = ss2.Ssimulacra2Result(norms, 50.0)
    assert [f.name for f in dataclasses.fields(r)] == ["norms", "device_score", "scales"]
    assert "scales=[Ssimulacra2Scale(" in repr(r)
    d = dataclasses.asdict(r)
    assert len(d["scales"]) == scales
    for row, s, e in zip(norms, r.scales, d["scales"]):
        for name, want in (("avg_ssim", row[:6]), ("avg_edgediff", row[6:])):
            assert np.array_equal(getattr(s, name), want) and np.array_equal(e[name], want)
    assert r.scales is r.scales


def test_scales_are_of_the_norms_as_made():
    r = ss2.Ssimulacra2Result(_norms())
    others = [copy.copy(r), copy.deepcopy(r), pickle.loads(pickle.dumps(r))]
    r.norms[:] = -1.0
    for x in [r] + others:
        assert np.array_equal(x.scales[3].avg_edgediff, _norms()[3, 6:])
    r.scales[3].avg_ssim[:] = 2.0
    assert np.all(r.norms == -1.0)
    with pytest.raises(AttributeError):
        r.nothing


@pytest.mark.gpu
def test_a_lists_results_are_each_their_own():
    from tests import synthetic
    pairs = [synthetic.rgb_pair(96, 64, s)[:2] for s in range(3)]
    pairs.append(synthetic.rgb_pair(16, 20, 9)[:2])  # two scales
    with ss2.Ssimulacra2Batch() as b:
        results = b.compute_many(pairs)
        again = b.compute_many(pairs)
    for r, a in zip(results, again):
        assert r.norms.base is None or r.norms.base.size == r.norms.size
        assert np.array_equal(r.norms, a.norms) and r.device_score == a.device_score
    before = results[1].norms.copy()
    results[0].norms[:] = 0.0
    assert np.array_equal(results[1].norms, before)
