"""The cut of a serving job's initial vectors into rounds and the layout of its
half line strength (csrc/zlayout.h, compiled here on its own): jobs of one
initial block to different final J share cached columns, so their cuts must
agree, and a layout that differs in anything must not compare equal."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "gpu-intensities_gb300", "csrc")
HARNESS = r"""
#include "zlayout.h"
using namespace gi;
// the cut of nvec vectors (returns the rounds) for a job to final block `mine`
// of the n loaded ones
extern "C" int cut(size_t ws, size_t zbytes, int cols, size_t digit, int n, const int* ld,
                   const int* nvec, int mine, int shared, int nv, int* out) {
  FinalSize f{ld[mine], nvec[mine]};
  if (shared) for (int k = 0; k < n; k++) f = larger(f, FinalSize{ld[k], nvec[k]});
  const int chunk = unit_vectors(ws, zbytes + cols * final_col_bytes(f, digit), nv);
  int r = 0;
  for (int i = 0; i < nv; i += chunk) out[r++] = std::min(chunk, nv - i);
  return r;
}
extern "C" int same(unsigned long long oa, int la, size_t na, int ca, unsigned long long ob, int lb,
                    size_t nb, int cb) {
  return ZLayout{oa, la, na, {ca, 1}} == ZLayout{ob, lb, nb, {cb, 1}};
}
extern "C" size_t elems(int ld, size_t n) { return ZLayout{1, ld, n, {}}.elems(); }
"""


@pytest.fixture(scope="module")
def lay(tmp_path_factory):
    d = tmp_path_factory.mktemp("zlayout")
    (d / "h.cpp").write_text(HARNESS)
    so = str(d / "h.so")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}",
                           str(d / "h.cpp"), "-o", so])
    L = C.CDLL(so)
    L.elems.restype = C.c_size_t
    return L


def cuts(L, ws, zbytes, cols, digit, finals, nv, shared):
    ld = (C.c_int * len(finals))(*[f[0] for f in finals])
    n = (C.c_int * len(finals))(*[f[1] for f in finals])
    out = (C.c_int * nv)()
    res = []
    for k in range(len(finals)):
        r = L.cut(C.c_size_t(ws), C.c_size_t(zbytes), cols, C.c_size_t(digit), len(finals), ld, n,
                  k, shared, nv, out)
        res.append(list(out[:r]))
    return res


@pytest.mark.parametrize("digit", [0, 11, 18])
def test_one_cut_for_every_final_block(lay, digit):
    rng = np.random.default_rng(digit)
    differ = 0
    for _ in range(300):
        J, nvib = int(rng.integers(1, 41)), int(rng.choice([200, 1000, 3000, 5000]))
        ndeg, nv = int(rng.integers(1, 3)), int(np.exp(rng.uniform(np.log(10), np.log(2000))))
        finals = [(-(-(2 * j + 1) * nvib // (3 * 64)) * 64, int(np.exp(rng.uniform(4.6, 7.6))))
                  for j in (J - 1, J, J + 1)]
        zbytes = ndeg * (2 * J + 1) * nvib * (24 + 11)
        ws = int(np.exp(rng.uniform(np.log(1e6), np.log(1.3e10))))
        shared = cuts(lay, ws, zbytes, ndeg * ndeg, digit, finals, nv, 1)
        assert shared[0] == shared[1] == shared[2] and sum(shared[0]) == nv
        own = cuts(lay, ws, zbytes, ndeg * ndeg, digit, finals, nv, 0)
        differ += not (own[0] == own[1] == own[2])
    assert differ > 20  # the cut by a job's own final block is not one cut


def test_layouts_differ_in_every_part(lay):
    U, S = C.c_ulonglong, C.c_size_t
    a = (U(7), 3072, S(284160), 609)
    assert lay.same(*a, *a)
    for b in [(U(8), 3072, S(284160), 609), (U(7), 3008, S(284160), 609),
              (U(7), 3072, S(284040), 609), (U(7), 3072, S(284160), 605)]:
        assert not lay.same(*a, *b)
    assert lay.elems(3072, S(1 << 20)) == 3 * 3072 << 20
