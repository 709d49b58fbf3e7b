"""A basis whose vibrational indices no dipole reaches is taken by gi_set_basis
and refused, with a status, by the calls that need the functions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("index", [60, (1 << 20) - 1, 1 << 20, (1 << 31) - 1])
@pytest.mark.parametrize("precision", [0, 1])
def test_index_beyond_the_dipole_is_refused(pkg, synth, index, precision):
    prob = synth.make_c2v(33, 60, [1, 2], nvec_max=5)
    with pkg.Engine(0) as eng:
        eng.load(prob, precision=precision)
        n = eng.run()
        good = prob.bases[2].iroot_correlat_j0.copy()
        prob.bases[2].iroot_correlat_j0[7] = index
        eng.set_basis(prob.bases[2])
        vec = prob.blocks[(1, 0)].vecs[0]
        for call in (eng.run, eng.serve_start,
                     lambda: eng.half_ls(1, 0, 0, 2, vec, prob.bases[2].Maxcontracts)):
            with pytest.raises(pkg.GiError) as e:
                call()
            assert e.value.status == pkg.GI_ERR_ARG
        prob.bases[2].iroot_correlat_j0[:] = good
        eng.set_basis(prob.bases[2])
        assert eng.run() == n > 0
