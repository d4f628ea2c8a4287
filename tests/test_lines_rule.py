"""The composed line passes of the fused kernels (csrc/wvlh_lines.cuh), built
for the host: B = magic filter x synthesis, B^T and T = analysis x kinetic x
synthesis on rows and columns, periodic and free lines, against dense matrices
made from the filters, in the segment lengths that the kernels use.  Lengths run from the shortest lines (shorter than the
windows, which wrap several times) over odd ones to several segments with every
remainder."""
import ctypes as C
import re
import subprocess
from fractions import Fraction
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
    dll = C.CDLL(str(so))
    f = dll.line_pass
    dll.b_inv6.restype = C.c_double

    def call(prec, rows, op, n, per, x, nout, seg=8):
        x = np.ascontiguousarray(x)
        out, e = np.zeros((len(x), nout)), C.c_double()
        p = C.POINTER(C.c_double)
        rc = f(prec, rows, op, seg, n, per, len(x), x.ctypes.data_as(p), out.ctypes.data_as(p), C.byref(e))
        assert rc == 0, "a write outside the buffers"
        return (out if op == 2 else out / call.norm[prec]), e.value
    call.norm = {prec: dll.b_inv6(prec) ** (-1 / 6) for prec in (32, 64)}
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
@pytest.mark.parametrize("seg", [6, 8])
@pytest.mark.parametrize("per,n", [(1, v) for v in (8, 9, 11, 12, 13, 17, 24, 30, 35, 48)] +
                         [(0, v) for v in (1, 2, 3, 5, 6, 7, 12, 13, 18, 31)])
def test_line_passes_match_dense(line_pass, prec, rows, seg, per, n):
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
    got, _ = line_pass(prec, rows, 0, n, per, w, len(B), seg)
    assert np.abs(got - w @ B.T).max() <= bound(B)
    got, _ = line_pass(prec, rows, 1, n, per, r, 2 * n, seg)
    assert np.abs(got - r @ B).max() <= bound(B.T)
    got, e = line_pass(prec, rows, 2, n, per, w, 2 * n, seg)
    want = w @ T.T
    ew = (w * want).sum()
    if rows:
        want, ew = 0.25 * w - 0.5 * want, -0.5 * ew
    assert np.abs(got - want).max() <= 2 * bound(T)
    # the energy is x times the outputs: the errors of its up to 62 + 2 seg
    # roundings a term add up like those of independent steps (six deviations);
    # the taps' own rounding goes one way, below 3.3e-8 |x|^2 in FP32
    dev = eps * np.sqrt(62 + 2 * seg) * np.sqrt(((w * (np.abs(w) @ np.abs(T).T)) ** 2).sum())
    assert abs(e - ew) <= 6 * dev + (3.3e-8 if prec == 32 else 1e-16) * (w * w).sum()


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


def b_taps(line_pass, prec):
    """gs(-14..16), gw(-14..16) as the pass holds them: its answers to unit lines"""
    n = 20
    x = np.zeros((2, 2 * n))
    x[0, 3] = x[1, n + 3] = 1.0
    got, _ = line_pass(prec, 1, 0, n, 0, x, 2 * n + 29)
    return [Fraction(v) for v in got[:, 6:37].ravel()]     # j = m + 6 is stored at j + 14


def tap_bias(taps):
    """How far the taps' errors D move |B x|^2: the largest eigenvalue over all
    frequencies of B^T D + D^T B in 2 x 2 symbols (output parity, input half), the
    largest and the zero-frequency scaling-scaling entry of smooth lines, the
    mean (white noise); and the largest |D|"""
    fr = lambda name: [Fraction(v) for v in table(name)]  # noqa: E731
    mf = fr("MF")
    exact = [sum((mf[l + 8] * f[m + l + 7] for l in range(-8, 8) if 0 <= m + l + 7 <= 15), Fraction(0))
             for f in (fr("CH"), fr("CG")) for m in range(-14, 17)]
    th = np.linspace(0, np.pi, 181)
    sym = np.zeros((2, len(th), 2, 2), complex)
    for i, (t, c) in enumerate(zip(taps, exact)):
        m = i % 31 - 14
        ph = np.exp(-1j * th * ((m - (m & 1)) // 2))
        for k, v in enumerate((c, t - c)):
            sym[k, :, m & 1, i // 31] += float(v) * ph
    g, d = sym
    h = np.einsum("toa,tob->tab", g.conj(), d)
    h = h + np.conj(np.swapaxes(h, 1, 2))
    ss = np.abs(h[:, 0, 0])
    return (np.abs(np.linalg.eigvalsh(h)).max(), ss[th < 1].max(), ss[0],
            abs(np.trace(h, axis1=1, axis2=2).real.mean() / 2), np.linalg.norm(d, 2, axis=(1, 2)).max())


def test_fp64_taps_do_not_bias_the_density(line_pass):
    """|B x|^2 per axis stays within 1e-17 of itself (sums of products rounded
    at each step: 4e-16, always the same way), the outputs within 2e-16"""
    worst, smooth, dc, white, dist = tap_bias(b_taps(line_pass, 64))
    assert worst < 1e-17 and white < 3e-18 and dist < 2e-16


def test_fp32_taps_do_not_bias_the_density(line_pass):
    """The FP32 form: within 2.5e-9 at every frequency and 1e-9 on smooth lines
    (nearest taps: 3.1e-8 and 2.4e-8), white noise 3e-10, outputs 1.2e-8"""
    worst, smooth, dc, white, dist = tap_bias(b_taps(line_pass, 32))
    assert worst < 2.5e-9 and smooth < 1e-9 and dc < 4e-10 and white < 3e-10 and dist < 1.2e-8


def test_fp32_norms_of_smooth_and_rough_lines(line_pass):
    """|B x|^2 of Gaussian lines (scaling coefficients of random widths and
    places) and of white noise, in FP32 against the dense matrix: the taps'
    share above plus the roundings of the outputs, which average out"""
    n, nl = 48, 1000
    B, _ = matrices(n, 1)
    rng = np.random.default_rng(2)
    t = (np.arange(n) - rng.uniform(0, n, (nl, 1)) + n / 2) % n - n / 2
    lines = {"smooth": np.hstack([np.exp(-(t / rng.uniform(2, 5, (nl, 1))) ** 2 / 2), np.zeros((nl, n))]),
             "rough": rng.uniform(-1, 1, (nl, 2 * n))}
    for name, w in lines.items():
        w = w.astype(np.float32).astype(float)
        want = ((w @ B.T) ** 2).sum()
        for rows in (1, 0):
            got, _ = line_pass(32, rows, 0, n, 1, w, 2 * n)
            assert abs((got ** 2).sum() / want - 1) < 1.5e-9, name


def t_symbol_errors(line_pass, prec):
    """The errors of T's taps (answers to unit lines) against 4 analysis .
    kinetic . synthesis of the filters' doubles, as 2 x 2 symbols: the scaling-
    scaling entry at frequency 0 and below 0.5, and the largest norm"""
    n, mid = 40, 20
    x = np.zeros((2, 2 * n))
    x[0, mid] = x[1, n + mid] = 1.0
    got, _ = line_pass(prec, 0, 2, n, 0, x, 2 * n)
    kin, fine = [Fraction(v) for v in table("KIN")], [[Fraction(v) for v in table(t)] for t in ("CH", "CG")]
    th = np.linspace(0, np.pi, 181)
    d = np.zeros((len(th), 2, 2), complex)
    for i in range(2):
        y = {}
        for p in range(16):
            for l in range(-14, 15):
                y[p + l] = y.get(p + l, 0) + kin[abs(l)] * fine[i][p]
        for o in range(2):
            for l in range(-14, 15):
                want = 4 * sum((fine[o][p] * y.get(2 * l + p, 0) for p in range(16)), Fraction(0))
                d[:, o, i] += float(Fraction(got[i, o * n + mid + l]) - want) * np.exp(-1j * th * l)
    ss = np.abs(d[:, 0, 0])
    return ss[0], ss[th < 0.5].max(), np.linalg.norm(d, 2, axis=(1, 2)).max()


def test_fp64_taps_do_not_bias_the_kinetic_energy(line_pass):
    """<x | T x> of smooth orbitals is a small difference of large terms: T's
    scaling part is right to 1e-18 at frequency 0 (the published tables of a, c,
    e, taps of the many-digit filters: 1e-15), T's norm is 40"""
    zero, low, worst = t_symbol_errors(line_pass, 64)
    assert zero < 1e-18 and low < 1e-17 and worst < 1.2e-15


def test_fp32_taps_do_not_bias_the_kinetic_energy(line_pass):
    """The FP32 form: 1e-10 at frequency 0, 3e-9 below 0.5 (nearest values of the
    scaled taps: 1.5e-8 throughout)"""
    zero, low, worst = t_symbol_errors(line_pass, 32)
    assert zero < 1e-10 and low < 3e-9 and worst < 4.2e-8
