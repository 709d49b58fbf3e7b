"""The default split-precision GEMM (e4m3 digits on the fp8 tensor pipe) alone,
at the edges of its 128 x 40 tiles, 32-wide K slices and 5952-wide exact
segments, through gi_probe_split_gemm.

Bound: each operand is rounded to 2^-56 of a power of two at most four times
its row's largest element, and the dropped digit products (diagonals 11 and up,
55 pairs of at most 2^8 with weights from 2^-65) add at most 2^-53 of the two
powers' product per k: together below 2^-48 K max|a| max|b|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (127, 39, 31), (128, 40, 32), (129, 41, 33),
                                   (257, 80, 95), (384, 121, 64), (130, 83, 5952),
                                   (129, 44, 5953), (140, 41, 11969)])
def test_tile_and_segment_edges(pkg, M, N, K):
    rng = np.random.default_rng(M + N + K)
    A = rng.standard_normal((M, K)) * np.exp(rng.uniform(-20.0, 20.0, (M, 1)))
    B = rng.standard_normal((N, K)) * np.exp(rng.uniform(-20.0, 20.0, (N, 1)))
    got = pkg.split_gemm(A, B)
    err = np.abs(got - A @ B.T)
    bound = np.abs(A).max(axis=1)[:, None] * np.abs(B).max(axis=1)[None, :]
    assert (err <= (2.0 ** -48 + 2.0 ** -52) * K * bound).all()


@pytest.mark.parametrize("value", [0.5 - 2.0 ** -54, 16.0 / 31.0, -1.0, 1.0 / 3.0])
@pytest.mark.parametrize("K", [5952, 6000])
def test_constant_rows_stay_exact(pkg, value, K):
    """Every digit of a plane the same sign and size along K: the largest
    diagonal sums a segment can reach, where an inexact one would show at
    2^-24 of the result."""
    A = np.full((130, K), value)
    B = np.full((42, K), value)
    got = pkg.split_gemm(A, B)
    want = K * value * value
    assert np.abs(got - want).max() <= 1e-15 * abs(want)


@pytest.mark.parametrize("value", [15.0 / 31.0, -15.0 / 31.0, 0.5 - 2.0 ** -54])
@pytest.mark.parametrize("K", [1409, 1472, 1473])
def test_short_segments_stay_exact(pkg, value, K):
    """Sums on both sides of the length up to which they are read off the bits
    (46 slices): 15/31 is the digit 15 eleven times, 7/8 of the largest sum
    there is.  Left out of the result are products of 2^-55 of it, about 3e-16;
    its own roundings and those of the value wanted are as much again."""
    A = np.full((130, K), value)
    B = np.full((42, K), 15.0 / 31.0)
    got = pkg.split_gemm(A, B)
    want = K * value * (15.0 / 31.0)
    assert np.abs(got - want).max() <= 1e-15 * abs(want)


@pytest.mark.parametrize("case", ["unused", "few_kinds", "many_kinds", "empty_columns"])
def test_classes_of_functions(pkg, synth, case):
    """The half-line-strength GEMM skips what the symmetries rule out, by
    classes of functions that every basis uses alike: functions no basis uses,
    coefficients missing from some functions (a few classes, or more than the
    32 a launch tells apart), and keys whose columns are empty for a symmetry.
    The same lines as the FP64 path, which contracts everything."""
    rng = np.random.default_rng(3)
    if case == "unused":
        prob = synth.make_c2v(61, 90, [1, 2], nvec_max=12, nsize_scale=0.4)
    else:
        prob = synth.make_c3v(62, 70, [0, 1, 2, 3], nvec_max=12)
        kinds = {"few_kinds": 3, "many_kinds": 64, "empty_columns": 1}[case]
        lost = rng.integers(0, kinds, 70)  # the kind of each function
        for J, b in prob.bases.items():
            D = b.Maxcontracts
            gone = rng.random((kinds, J + 1, 3)) < 0.3
            for g in range(3):
                nt, dg = int(b.Ntotal[g]), prob.degen[g]
                rep = b.repres[g][:nt * dg * b.mat_size].reshape(b.mat_size, dg, nt)
                nsym = b.Nsym.reshape(-1, 3)[:, g]
                s0 = np.cumsum(nsym) - nsym
                for r in range(D):
                    ic, lam = b.icontr2icase[r], b.icontr2icase[r + D]
                    k = b.k[r]
                    if gone[lost[b.iroot_correlat_j0[r]], k, g]:
                        rep[lam, :, s0[ic]:s0[ic] + nsym[ic]] = 0.0
    out = []
    for precision in (pkg.GI_PREC_FP64, pkg.GI_PREC_SPLIT):
        with pkg.Engine(0) as eng:
            eng.load(prob, precision=precision)
            eng.set_refine(1 << 20)
            eng.run()
            out.append(np.sort(eng.lines(), order=["level_i", "level_f"]))
    a, b = out
    assert len(a) > 300 and np.array_equal(a[["level_i", "level_f"]], b[["level_i", "level_f"]])
    scale = np.abs(a["t"]).max()
    assert np.abs(a["t"] - b["t"]).max() <= 1e-12 * scale


@pytest.mark.parametrize("case", ["decay", "blocks", "zero_rows", "tiny"])
def test_zero_planes_of_the_dipole(pkg, synth, case):
    """K slices of the dipole whose leading digit planes are zero skip those
    planes' products, and slices without any digit are not contracted at all: a
    banded dipole, whole zero blocks, rows and components that are zero, and
    blocks 2^-50 of their rows.  Lines and single vectors as the FP64 path's."""
    N = 420
    prob = synth.make_c3v(63, N, [1, 2], nvec_max=20)
    mu = prob.mu.reshape(3, N, N)
    rng = np.random.default_rng(1)
    if case == "blocks":
        mu[:] = rng.standard_normal(mu.shape)
        mu[:, :, 200:330] = 0.0
        mu[:, 100:310, :] = 0.0
    elif case == "zero_rows":
        mu[:] = rng.standard_normal(mu.shape)
        mu[1] = 0.0
        mu[:, rng.random(N) < 0.6] = 0.0
    elif case == "tiny":
        mu[:] = rng.standard_normal(mu.shape)
        mu[:, :, 64:300] *= 2.0 ** -50
        mu[:, :, 300:] *= 2.0 ** -30
    out, vec = [], []
    for precision, streamed in ((0, None), (1, None), (1, 150)):
        with pkg.Engine(0) as eng:
            eng.load(prob, precision=precision, panel_rows=streamed)
            eng.run()
            out.append(np.sort(eng.lines(), order=["level_i", "level_f"]))
            vec.append(eng.half_ls(1, 2, 1, 2, prob.blocks[(1, 2)].vecs[0],
                                   prob.bases[2].Maxcontracts))
    assert len(out[0]) > 300
    scale = np.abs(out[0]["t"]).max()
    for o in out[1:]:
        assert np.array_equal(o[["level_i", "level_f"]], out[0][["level_i", "level_f"]])
        assert np.abs(o["t"] - out[0]["t"]).max() <= 1e-12 * scale
    assert np.array_equal(out[1], out[2])
    for v in vec[1:]:
        assert np.abs(v - vec[0]).max() <= 1e-13 * np.abs(vec[0]).max()


@pytest.mark.parametrize("case", ["c2v", "c3v", "c3v_reduced"])
@pytest.mark.parametrize("which", ["I", "S", "both"])
def test_thresholds_keep_exactly_the_lines_above(pkg, synth, case, which):
    """Lines told to be below a threshold from single-precision logarithms: a
    run with thresholds keeps bit for bit the lines of a run without that are at
    or above them, and counts the same lines through the filters."""
    if case == "c2v":
        prob = synth.make_c2v(64, 150, [1, 2, 3], nvec_max=60)
    else:
        prob = synth.make_c3v(65, 120, [1, 2, 3], nvec_max=50, reduced=case.endswith("reduced"))
    with pkg.Engine(0) as eng:
        eng.load(prob, precision=pkg.GI_PREC_SPLIT)
        eng.run()
        every, n = np.sort(eng.lines(), order=["level_i", "level_f"]), eng.stats()["nlines_filtered"]
        avogno = 6.0221415e23
        tS, tI = np.quantile(every["S"], 0.6), np.quantile(every["I"] / avogno, 0.7)
        prob.params.thresh_linestrength = float(tS) if which in ("S", "both") else 0.0
        prob.params.thresh_intensity = float(tI) if which in ("I", "both") else 0.0
        eng.set_params(prob.params, precision=pkg.GI_PREC_SPLIT)
        eng.run()
        kept, m = np.sort(eng.lines(), order=["level_i", "level_f"]), eng.stats()["nlines_filtered"]
    want = every[(every["S"] >= prob.params.thresh_linestrength) &
                 (every["I"] / avogno >= prob.params.thresh_intensity)]
    assert n == m == len(every) > 2000 and 100 < len(want) < len(every)
    # (a line at the threshold itself is evaluated exactly, its values replaced)
    assert np.array_equal(kept[["level_i", "level_f"]], want[["level_i", "level_f"]])
    assert np.allclose(kept["S"], want["S"], rtol=1e-11, atol=0)
    assert np.count_nonzero(kept["S"] != want["S"]) <= 2
