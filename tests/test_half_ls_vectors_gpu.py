"""The half line strength of single vectors at the sizes where its kernels
change: rows of Y packed to their non-zero values (half full, full, one
element, row strides with and without padding), sizes where the split precision
takes FP64, and the split GEMM's bands and K parts; and the allocation-free call
from several contexts at once."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group,N,jlist,precision", [
    ("c2v", 1, [0, 1], 0), ("c2v", 63, [1, 2], 0), ("c2v", 64, [1, 2], 0), ("c3v", 65, [1, 2], 0),
    ("c3v", 130, [3, 4], 0), ("c2v", 333, [2], 1), ("c2v", 1900, [8, 9], 1), ("c3v", 1250, [6], 1)])
def test_half_ls_sizes(pkg, synth, oracle, group, N, jlist, precision):
    prob = (synth.make_c2v if group == "c2v" else synth.make_c3v)(N, N, jlist, nvec_max=1)
    with pkg.Engine(0) as eng:
        eng.load(prob, precision=precision)
        n = 0
        for (jI, gI), blk in sorted(prob.blocks.items()):
            if blk.nvec == 0:
                continue
            d, jF = prob.degen[gI] - 1, jlist[-1]
            vprim = oracle.correlate(prob.bases[jI], prob.nrep, prob.degen, d, gI, blk.vecs[0])
            want = oracle.half_ls(prob.bases[jI], prob.bases[jF], prob.N, prob.mu, max(jlist), vprim)
            got = [eng.half_ls(jI, gI, d, jF, blk.vecs[0], prob.bases[jF].Maxcontracts)
                   for _ in range(3)]  # eager, captured, replayed
            assert np.abs(got[0] - want).max() <= 1e-13 * np.abs(want).max()
            assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
            n += 1
        assert n > 0


def test_noalloc_calls_of_several_contexts(pkg, synth):
    """Calls on three contexts' own streams, issued without waiting: each gets
    its own vector's result although all share one scratch array."""
    torch = pytest.importorskip("torch")
    probs = [synth.make_c2v(70 + i, 300 + 40 * i, [2, 3], nvec_max=1) for i in range(3)]
    engs = [pkg.Engine(0) for _ in probs]
    for e, p in zip(engs, probs):
        e.load(p)
    vecs = [torch.from_numpy(p.blocks[(2, 0)].vecs[0]).cuda() for p in probs]
    outs = [torch.zeros(p.bases[3].Maxcontracts, dtype=torch.float64, device="cuda") for p in probs]
    want = [e.half_ls(2, 0, 0, 3, p.blocks[(2, 0)].vecs[0], p.bases[3].Maxcontracts)
            for e, p in zip(engs, probs)]
    torch.cuda.synchronize()
    for _ in range(20):
        for e, v, o in zip(engs, vecs, outs):
            st = pkg.lib().gi_half_ls_noalloc(e._h, 2, 0, 0, 3, C.c_void_p(v.data_ptr()),
                                              C.c_void_p(o.data_ptr()), None)
            assert st == pkg.GI_OK
    torch.cuda.synchronize()
    for w, o in zip(want, outs):
        assert np.array_equal(o.cpu().numpy(), w)
    for e in engs:
        e.close()
