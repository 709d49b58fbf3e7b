"""gi_sort_lines on the device: the run's lines in (initial level, final level)
order, every record as it was, for full records on the host, on the device and
compact ones; initial levels with few lines (counted places) and with more than
512 (places from a bitmap of the final levels)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["host", "device", "compact"])
@pytest.mark.parametrize("nvec", [1, 30, 400])
def test_sorted_lines_are_the_lines(pkg, synth, mode, nvec):
    prob = synth.make_c2v(21, 1300 if nvec == 400 else 60, [1, 2], nvec_max=nvec)
    kw = {"lines_on_device": mode == "device", "compact": mode == "compact"}
    with pkg.Engine(0) as eng:
        eng.load(prob, precision=pkg.GI_PREC_SPLIT)
        eng.run(**kw)
        before, small = eng.lines(), eng.lines_compact()
        eng.sort_lines()
        after, small_after = eng.lines(), eng.lines_compact()
    want = np.sort(before, order=["level_i", "level_f"])
    per = np.bincount(before["level_i"])
    assert len(before) > 0 and (nvec < 400 or per.max() > 512)
    if mode == "host":
        assert np.array_equal(after, want)
    else:
        assert np.array_equal(after, want)
        assert np.array_equal(small_after, np.sort(small, order=["level_i", "level_f"]))
