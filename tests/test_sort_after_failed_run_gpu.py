"""gi_sort_lines after a run that failed: the lines of the run before it, whose
level ids the failed run's shorter level table does not cover, are sorted all
the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["host", "device", "compact"])
def test_sort_after_a_failed_run(pkg, synth, mode):
    prob = synth.make_c2v(31, 60, [1, 2], nvec_max=30)
    kw = {"lines_on_device": mode == "device", "compact": mode == "compact"}
    with pkg.Engine(0) as eng:
        eng.load(prob, precision=pkg.GI_PREC_SPLIT)
        eng.run(**kw)
        before, small, nlev = eng.lines(), eng.lines_compact(), len(eng.levels())
        p = prob.params
        p.erange_lower = p.erange_upper = (0.0, 2400.0)  # fewer levels, and at this
        p.q_stat, p.temperature = -1.0, 1e-6             # temperature no partition function
        eng.set_params(p, precision=pkg.GI_PREC_SPLIT)
        with pytest.raises(pkg.GiError):
            eng.run(**kw)
        assert len(eng.levels()) < nlev and before["level_i"].max() >= len(eng.levels())
        eng.sort_lines()
        after, small_after = eng.lines(), eng.lines_compact()
    assert len(before) > 100
    assert np.array_equal(after, np.sort(before, order=["level_i", "level_f"]))
    if mode != "host":
        assert np.array_equal(small_after, np.sort(small, order=["level_i", "level_f"]))
