"""A captured run replayed after the dipole was streamed and made resident
again: the order tables of the dipole were remade meanwhile (for panels they are
several times as large), and the graph must not name the old ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_resident_streamed_resident(pkg, synth, precision):
    prob = synth.make_c3v(93, 150, [1, 2, 3], nvec_max=12)
    order = ["level_i", "level_f"]
    with pkg.Engine(0) as eng:
        eng.load(prob, precision=precision)
        eng.run()
        want = np.sort(eng.lines(), order=order)
        got = []
        for _ in range(3):
            for _ in range(2):  # captured, replayed
                eng.run(graph=True)
                got.append(np.sort(eng.lines(), order=order))
            eng.set_dipole_streamed(prob.N, prob.mu, panel_rows=16)
            eng.run(graph=True)
            got.append(np.sort(eng.lines(), order=order))
            # other work in the memory that the tables left
            other = synth.make_c2v(94, 100 + 30 * len(got), [0, 1], nvec_max=4)
            with pkg.Engine(0) as e2:
                e2.load(other, precision=precision)
                e2.run()
                eng.set_dipole(prob.N, prob.mu)
                eng.run(graph=True)
                got.append(np.sort(eng.lines(), order=order))
    assert len(want) > 200
    for g in got:
        assert np.array_equal(g, want)
