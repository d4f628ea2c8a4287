"""The composed line passes of the fused kernels (csrc/wvlh_lines.cuh), built
for the host: B = magic filter x synthesis, B^T and T = analysis x kinetic x
synthesis on rows and columns, periodic and free lines, against dense matrices
made from the filters.  Lengths run from the shortest lines (shorter than the
windows, which wrap several times) over odd ones to several segments with every
remainder."""
import ctypes as C
import re
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "bigdft-suite_b200" / "csrc"


@pytest.fixture(scope="module")
def line_pass(tmp_path_factory):
    so = tmp_path_factory.mktemp("lines") / "lines.so"
    cuda = Path("/usr/local/cuda/include")
    if not cuda.exists():
        pytest.skip("no CUDA headers")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-w", "-I", str(cuda), "-I",
                    str(CSRC), str(HERE / "native" / "lines_host.cpp"), "-o", str(so)], check=True)
    f = C.CDLL(str(so)).line_pass

    def call(prec, rows, op, n, per, x, nout):
        x = np.ascontiguousarray(x)
        out, e = np.zeros((len(x), nout)), C.c_double()
        p = C.POINTER(C.c_double)
        rc = f(prec, rows, op, n, per, len(x), x.ctypes.data_as(p), out.ctypes.data_as(p), C.byref(e))
        assert rc == 0, "a write outside the buffers"
        return out, e.value
    return call


def table(name):
    t = re.search(r"#define WVL_%s_INIT \{(.*?)\}" % name, (CSRC / "wvl_filters.h").read_text(), re.S).group(1)
    return [float(v) for v in t.replace("\\", "").split(",")]


def matrices(n, per):
    """B (real-space x wavelet) and T (wavelet x wavelet, coarse spacing 1) of one line."""
    ch, cg, mf, kin = table("CH"), table("CG"), table("MF"), table("KIN")
    f, r = (2 * n, 2 * n) if per else (2 * n + 14, 2 * n + 29)
    s, m, k = np.zeros((f, 2 * n)), np.zeros((r, f)), np.zeros((f, f))
    for i in range(n):
        for j in range(16):
            q = 2 * i + j - 7 + (0 if per else 7)
            s[q % f, i] += ch[j]
            s[q % f, n + i] += cg[j]
    for q in range(r):
        for j in range(16):
            p = q - 8 + j if per else q - 15 + j
            if per or 0 <= p < f:
                m[q, p % f] += mf[j]
    for q in range(f):
        for l in range(-14, 15):
            if per or 0 <= q + l < f:
                k[q, (q + l) % f] += kin[abs(l)]
    return m @ s, 4.0 * s.T @ k @ s


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("rows", [1, 0])
@pytest.mark.parametrize("per,n", [(1, v) for v in (8, 9, 11, 12, 13, 17, 24, 30, 35, 48)] +
                         [(0, v) for v in (1, 2, 3, 5, 6, 7, 12, 13, 18, 31)])
def test_line_passes_match_dense(line_pass, prec, rows, per, n):
    B, T = matrices(n, per)
    rng = np.random.default_rng(100 * n + per)
    nl = 5
    w = rng.uniform(-1, 1, (nl, 2 * n))
    r = rng.uniform(-1, 1, (nl, len(B)))
    if prec == 32:
        w, r = w.astype(np.float32).astype(float), r.astype(np.float32).astype(float)
    # a sum of K products of values below 1 with taps c: each product and each
    # partial sum is rounded, so the error is below K eps sum |c|; K <= 62
    eps = 2.0 ** -53 if prec == 64 else 2.0 ** -24
    bound = lambda m: 62 * eps * np.abs(m).sum(axis=1).max()  # noqa: E731
    got, _ = line_pass(prec, rows, 0, n, per, w, len(B))
    assert np.abs(got - w @ B.T).max() <= bound(B)
    got, _ = line_pass(prec, rows, 1, n, per, r, 2 * n)
    assert np.abs(got - r @ B).max() <= bound(B.T)
    got, e = line_pass(prec, rows, 2, n, per, w, 2 * n)
    want = w @ T.T
    ew = (w * want).sum()
    if rows:
        want, ew = 0.25 * w - 0.5 * want, -0.5 * ew
    assert np.abs(got - want).max() <= 2 * bound(T)
    # the energy of a line: the outputs' errors plus a rounding per term (the
    # terms of a segment are summed in T)
    assert abs(e - ew) <= 2 * nl * 2 * n * bound(T)


def test_fp32_energy_is_not_biased_by_tap_rounding(line_pass):
    """<x | T x> in FP32 over many lines: what the taps' rounding leaves stays
    below 5e-9 of the energy (plain FP32 taps: 3e-8)."""
    n, nl = 48, 600
    _, T = matrices(n, 1)
    rng = np.random.default_rng(1)
    w = rng.uniform(-1, 1, (nl, 2 * n)).astype(np.float32).astype(float)
    ew = (w * (w @ T.T)).sum()
    for rows in (1, 0):
        _, e = line_pass(32, rows, 2, n, 1, w, 2 * n)
        assert abs(e / (-0.5 if rows else 1.0) - ew) <= 5e-9 * abs(ew)
