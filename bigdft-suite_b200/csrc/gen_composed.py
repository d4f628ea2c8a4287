"""Regenerate ``wvl_composed.h``, the taps of the composed operator B = magic
filter . synthesis that the fused kernels use (wvlh_lines.cuh), from the
filters of ``wvl_filters.h``.

The exact taps gs(m), gw(m), m in [-14, 16], are sums of products of the
filters' doubles, taken here as rationals.  Storing a tap moves it by up to half
a rounding, the same way for every output, and so moves |B x|^2, and with it
E_pot and the density, by <x | (B^T D + D^T B) x>, D the taps' errors, whatever
the orbital.  Only 31 of the 62 directions of D do that (to first order the
others turn B x and leave its length).  So the taps are rounded one after the
other, the largest first, each to the neighbour of what the least-squares
solution for the taps still free asks of it: the least norm of
B^T D + D^T B over all frequencies, plus LAMBDA |D|^2, which keeps D small.

FP32 taps are kept times NORM, whose -6th power the kernels multiply back (the
potential's term, E_pot and the density hold six B each): found by a scan of
[2^-1/2, 2^1/2] in steps of 1e-10 among the factors whose taps lie nearest to
FP32 values and whose -6th power lies within 2e-9 of one.  Its four largest taps
take their nearest values, and a local search over the next thirty (steps of a
few roundings, seeded) balances what measure() returns.

Run ``python gen_composed.py`` to rewrite the header; it is committed, so that the
build needs neither this script nor numpy.
"""
import random
import re
from fractions import Fraction
from pathlib import Path

import numpy as np

HERE = Path(__file__).resolve().parent
NORM = {64: 1.0, 32: 0.9752083272817533}
BITS = {64: 53, 32: 24}
LAMBDA = {64: 0.01, 32: 0.1}
KEEP = {64: 0, 32: 4}
TH = np.linspace(0.0, np.pi, 129)


def table(name):
    t = re.search(r"#define WVL_%s_INIT \{(.*?)\}" % name, (HERE / "wvl_filters.h").read_text(), re.S).group(1)
    return [Fraction(float(v)) for v in t.replace("\\", "").split(",")]


def exact_taps():
    """[gs(-14..16) | gw(-14..16)] as rationals"""
    mf = table("MF")
    return [sum((mf[l + 8] * f[m + l + 7] for l in range(-8, 8) if 0 <= m + l + 7 <= 15), Fraction(0))
            for f in (table("CH"), table("CG")) for m in range(-14, 17)]


def symbols():
    """E[i]: the 2 x 2 symbol (output parity, input half) of tap i on TH"""
    E = np.zeros((62, len(TH), 2, 2), complex)
    for i in range(62):
        half, m = i // 31, i % 31 - 14
        E[i, :, m & 1, half] = np.exp(-1j * TH * ((m - (m & 1)) // 2))
    return E


E = symbols()
EXACT = exact_taps()
HERM = np.einsum("toa,itob->itab", np.tensordot(np.array([float(c) for c in EXACT]), E, 1).conj(), E)
HERM = HERM + np.conj(np.swapaxes(HERM, 2, 3))     # tap i's share of B^T D + D^T B


def rounded(x, bits):
    """the rational x to `bits` binary digits"""
    q = Fraction(2) ** (int(np.floor(np.log2(abs(float(x))))) + 1 - bits)
    return round(x / q) * q


def error(tap, i, prec):
    return float(tap / Fraction(NORM[prec]) - EXACT[i])


def measure(d):
    """of B^T D + D^T B: the largest eigenvalue, the largest and the
    zero-frequency scaling-scaling entry (smooth lines), the mean (white noise);
    and the largest |D|"""
    M, D = np.tensordot(d, HERM, 1), np.tensordot(d, E, 1)
    a, b = M[:, 0, 0].real, M[:, 1, 1].real
    return np.array([np.abs(np.linalg.eigvalsh(M)).max(), np.abs(a[TH < 1]).max(), abs(a[0]), abs((a + b).mean() / 2),
                     np.linalg.norm(D, 2, axis=(1, 2)).max()])


ORDER = sorted(range(62), key=lambda i: -abs(EXACT[i]))


def least_squares(prec):
    A = np.stack([HERM[:, :, 0, 0].real, HERM[:, :, 1, 1].real, np.sqrt(2) * HERM[:, :, 0, 1].real,
                  np.sqrt(2) * HERM[:, :, 0, 1].imag], 2).reshape(62, -1).T / np.sqrt(len(TH))
    A = np.vstack([A, np.sqrt(LAMBDA[prec]) * np.eye(62)])
    taps, d = [None] * 62, np.zeros(62)
    for k, i in enumerate(ORDER):
        want = 0.0 if k < KEEP[prec] else np.linalg.lstsq(A[:, ORDER[k:]], -A @ d, rcond=None)[0][0]
        taps[i] = rounded(Fraction(NORM[prec]) * (EXACT[i] + Fraction(want)), BITS[prec])
        d[i] = error(taps[i], i, prec)
    return taps


def refine(taps, prec):
    goal = np.array([2.4e-9, 1.2e-9, 6e-10, 3e-10, 8e-9])
    cost = lambda t: ((measure(np.array([error(v, i, prec) for i, v in enumerate(t)])) / goal) ** 4).sum()  # noqa: E731
    rng, best, idle = random.Random(1), cost(taps), 0
    while idle < 3000:
        t = list(taps)
        for i in rng.sample(ORDER[4:34], rng.choice((1, 1, 2, 2, 3))):
            ulp = Fraction(2) ** (int(np.floor(np.log2(abs(float(t[i]))))) + 1 - BITS[prec])
            t[i] += rng.choice((-1, 1)) * (1 if ulp > 2e-9 else rng.choice((1, 1, 2, 4, 8))) * ulp
        c = cost(t)
        taps, best, idle = (t, c, 0) if c < best else (taps, best, idle + 1)
    return taps


def render():
    out = ["/* Generated by gen_composed.py from wvl_filters.h; do not edit. */", "#pragma once", ""]
    for prec in (64, 32):
        taps = least_squares(prec)
        if prec == 32:
            taps = refine(taps, prec)
        print("FP%d" % prec, *("%.1e" % v for v in measure(np.array([error(t, i, prec) for i, t in enumerate(taps)]))))
        for k, half in enumerate("SW"):
            out += ["/* FP%d taps g%s(-14..16) of magic filter . synthesis%s (index m+14) */"
                    % (prec, half.lower(), ", times %r" % NORM[prec] if NORM[prec] != 1 else ""),
                    "#define WVL_B%d_%s_INIT { \\" % (prec, half),
                    ", \\\n".join("    %s%s" % (float(t).hex(), "f" * (prec == 32)) for t in taps[31 * k:31 * k + 31]) + "}"]
    out += ["/* that factor's -6th power */", "#define WVL_B32_INV6 %s" % float(Fraction(NORM[32]) ** -6).hex()]
    return "\n".join(out) + "\n"


if __name__ == "__main__":
    (HERE / "wvl_composed.h").write_text(render())
