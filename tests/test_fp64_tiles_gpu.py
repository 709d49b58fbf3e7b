"""FP64 jobs at the edges of the list GEMM's 16 x 16 warp and 32 x 32 block
tiles (vectors per block) and of its 128-row, 32-function classes (functions),
against the oracle."""
import pytest

from paritylib import compare, with_threshold

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group", ["c2v", "c3v"])
@pytest.mark.parametrize("N,nvec", [(2, 1), (33, 15), (64, 16), (65, 17), (130, 33), (270, 9)])
def test_fp64_tile_edges(pkg, synth, oracle, group, N, nvec):
    make = synth.make_c2v if group == "c2v" else synth.make_c3v
    prob = with_threshold(make(N + nvec, N, [0, 1, 2], nvec_max=nvec))
    with pkg.Engine(0) as eng:
        eng.load(prob, precision=pkg.GI_PREC_FP64)
        eng.set_refine(1 << 20)
        eng.run()
        got = pkg.keyed(eng.lines(), eng.levels())
    compare(got, oracle.run_all(prob))
