"""Thresholds near the smallest numbers there are (the weak lines of a cold gas,
or a threshold that only drops zeros): the default split scheme keeps exactly
the lines at or above them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["I", "S"])
@pytest.mark.parametrize("thresh", [1e-296, 1e-303, 3e-307, 2.3e-308])
def test_threshold_near_the_smallest_number(pkg, synth, which, thresh):
    scale = 1.0 if which == "I" else thresh ** 0.5  # S near the threshold: tiny moments
    prob = synth.make_c2v(66, 150, [1, 2, 3], nvec_max=120, T=25.0 if which == "I" else 500.0)
    prob.mu = np.asarray(prob.mu) * scale
    with pkg.Engine(0) as eng:
        eng.load(prob, precision=pkg.GI_PREC_SPLIT)
        eng.run()
        every = np.sort(eng.lines(), order=["level_i", "level_f"])
        value = every["S"] if which == "S" else every["I"] / 6.0221415e23
        prob.params.thresh_linestrength = thresh if which == "S" else 0.0
        prob.params.thresh_intensity = thresh if which == "I" else 0.0
        eng.set_params(prob.params, precision=pkg.GI_PREC_SPLIT)
        eng.run()
        kept = np.sort(eng.lines(), order=["level_i", "level_f"])
    want = every[value >= thresh]
    assert 0 < len(want) < len(every)
    near = (value >= thresh) & (value < thresh * 1e4)
    assert near.sum() > 0
    assert np.array_equal(kept[["level_i", "level_f"]], want[["level_i", "level_f"]])
