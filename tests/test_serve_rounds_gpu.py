"""Serving jobs whose initial vectors take several rounds: jobs of one initial
block to final blocks of unequal sizes share its cached half line strength and
give bit for bit the lines they give without the cache."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,slices", [(0, 0), (1, 0), (1, 9)])
def test_zcache_over_several_rounds(pkg, synth, precision, slices):
    N, jlist, nv = 120, [3, 4, 5, 6], 150
    prob = synth.make_c3v(91, N, jlist, nvec_max=nv)
    for (J, g), b in prob.blocks.items():  # final blocks of unequal sizes
        n = b.nvec - 40 * ((J + g) % 3)
        b.vecs, b.energies, b.quanta = b.vecs[:n], b.energies[:n], b.quanta[:n]
    jobs = [(jI, g, jF, prob.partner(g)) for jI in (4, 5) for g in range(3)
            for jF in (jI - 1, jI, jI + 1)]
    # fewer than 40 of an E block's vectors a round (Z alone takes 24 N bytes for
    # each of a vector's 2 (2J + 1) columns), and by their own final blocks' sizes
    # the three jobs of a block would cut its vectors differently
    slot_ws = 40 * 2 * (2 * 4 + 1) * N * 24
    res, stats = {}, {}
    for cache in (False, True):
        with pkg.Engine(0) as eng:
            eng.load(prob, precision=precision, split_slices=slices)
            eng.serve_start(slots=2, budget=1 << 30, slot_workspace=slot_ws, zcache=cache)
            ids = [(j, eng.submit(*j)) for j in jobs]
            res[cache] = {j: np.sort(eng.job_lines(i), order=["level_i", "level_f"])
                          for j, i in ids}
            stats[cache] = eng.serve_stats()
            eng.serve_stop()
    assert stats[True]["failed"] == stats[False]["failed"] == 0
    assert stats[False]["zcache_hits"] == 0
    # one fill for each initial block, whatever the final block
    assert stats[True]["zcache_misses"] == 6 and stats[True]["zcache_hits"] == len(jobs) - 6
    assert sum(len(v) for v in res[False].values()) > 2000
    for j in jobs:
        assert np.array_equal(res[True][j], res[False][j]), j
