"""gi_half_ls on a context that is serving: single vectors and jobs use the same
tables of the bases, made by whichever comes first."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("loaded", [False, True])
def test_half_ls_between_jobs(pkg, synth, loaded):
    # large enough for the digit path: above 8 million products
    prob = synth.make_c2v(95, 900, [6, 7, 8], nvec_max=40)
    jobs = [(jI, g, jF, prob.partner(g)) for jI in (6, 7) for g in range(4) for jF in (7, 8)
            if abs(jI - jF) <= 1]
    calls = [(J, g, jF) for J in (6, 7) for g in range(4) for jF in (6, 7, 8) if abs(J - jF) <= 1]

    def vec(eng, J, g, jF):
        return eng.half_ls(J, g, 0, jF, prob.blocks[(J, g)].vecs[0], prob.bases[jF].Maxcontracts)

    with pkg.Engine(0) as eng:
        eng.load(prob, precision=pkg.GI_PREC_SPLIT)
        want_v = [vec(eng, *c) for c in calls]
        eng.serve_start(slots=1, zcache=False)
        want = {j: np.sort(eng.job_lines(eng.submit(*j)), order=["level_i", "level_f"])
                for j in jobs}
        eng.serve_stop()
    blocks = dict(prob.blocks)
    for rep in range(3):
        with pkg.Engine(0) as eng:
            prob.blocks = blocks if loaded else {}
            eng.load(prob, precision=pkg.GI_PREC_SPLIT)
            prob.blocks = blocks
            eng.serve_start(slots=3)
            if not loaded:  # blocks that come while serving: no table is there yet
                for (J, g), b in sorted(blocks.items()):
                    eng.set_block(J, g, b.vecs, b.energies, b.quanta)
            ids = [(j, eng.submit(*j)) for j in jobs]
            got_v = [vec(eng, *c) for c in calls]
            got = {j: np.sort(eng.job_lines(i), order=["level_i", "level_f"]) for j, i in ids}
            assert eng.serve_stats()["failed"] == 0
            eng.serve_stop()
        for a, b in zip(got_v, want_v):
            assert np.array_equal(a, b)
        for j in jobs:
            assert np.array_equal(got[j], want[j]), j
