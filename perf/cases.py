"""The framework's work, as a list of cases for measuring it.

Each case is one call (or the few calls that belong together) of a step of a
wavelet DFT calculation through the package's public entry points, on the sizes that the
package's own workloads (``wvlh/workloads.py``), tests and benchmark use:

* ``hpsi``: the local Hamiltonian of ``norb`` orbitals on one box, the call that
  every self-consistency iteration makes once per orbital group;
* ``dropin``: the same operator through the C ABI that the Fortran host drives,
  orbital by orbital with host buffers;
* ``regions``: support functions of the linear-scaling mode, one per free
  localisation region of its own size;
* ``serve``: one launch of the request server: H psi and density of several
  independent clients with boxes of different size and boundary conditions;
* ``density``: the charge density of the occupied orbitals;
* ``precond``: the preconditioner's fixed number of CG iterations;
* ``ortho``: overlap matrix and Cholesky orthonormalisation;
* ``projectors``: the nonlocal pseudopotential part of the Hamiltonian.

``exact`` restates each of them with dense FP64 matrices in plain torch.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bigdft-suite_b200"))
from wvlh import nlpsp, ocl, ortho  # noqa: E402
from wvlh.batch import Batch, Context, OrbitalBatch, Region  # noqa: E402
from wvlh.keys import Locreg  # noqa: E402

H = 0.45          # coarse grid spacing in bohr
DEV = "cuda"

# cells that the largest listed case works on; a drawn case stays below it
MOST_CELLS = 256 * 48 ** 3


def listed():
    return [
        # one orbital of a small molecule: launch latency counts
        dict(name="hpsi_one_f64", kind="hpsi", n1=32, n2=32, n3=32, per=1, norb=1, bits=64),
        # the same orbital as the unchanged Fortran host sends it, from host memory
        dict(name="dropin_f64", kind="dropin", n1=32, n2=32, n3=32, per=1, norb=2),
        # the orbitals of one periodic cell, mixed and full precision
        dict(name="hpsi_batch_f32", kind="hpsi", n1=48, n2=48, n3=48, per=1, norb=256, bits=32),
        dict(name="hpsi_batch_f64", kind="hpsi", n1=48, n2=48, n3=48, per=1, norb=128, bits=64),
        # a large box with uneven sides, full precision
        dict(name="hpsi_large_f64", kind="hpsi", n1=63, n2=61, n3=64, per=1, norb=32, bits=64),
        # support functions of the linear-scaling mode
        dict(name="regions_f32", kind="regions", nlr=192, nmin=20, nmax=40, shapes=2, bits=32),
        # a launch of the server: clients of different boxes and boundary conditions
        dict(name="serve_f32", kind="serve", clients=8, nmin=16, nmax=48, omin=4, omax=32, shapes=4, bits=32),
        # density of one cell's orbitals
        dict(name="density_f32", kind="density", n1=48, n2=48, n3=48, per=1, norb=128, bits=32),
        # preconditioner of one cell's residuals, mixed and full precision
        dict(name="precond_f32", kind="precond", n1=40, n2=40, n3=40, per=1, norb=128, ncong=5, bits=32),
        dict(name="precond_f64", kind="precond", n1=40, n2=40, n3=40, per=1, norb=64, ncong=5, bits=64),
        # orthonormalisation of one cell's orbitals (always full precision)
        dict(name="ortho_f64", kind="ortho", norb=256, ncoeff=8 * 40 ** 3),
        # projectors of the atoms of one cell on its orbitals (always full precision)
        dict(name="projectors_f64", kind="projectors", n1=40, n2=40, n3=40, norb=128, atoms=32, m=4, shapes=6),
    ]


def draw(rng):
    def logu(a, b):
        return max(a, min(b, int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))))

    kind = rng.choice(["hpsi", "hpsi", "hpsi", "regions", "serve", "density", "precond", "precond", "ortho",
                       "projectors", "dropin"])
    bits = rng.choice([32, 64])
    if kind in ("hpsi", "density", "precond"):
        n = [rng.randint(12, 64) for _ in range(3)]
        per = rng.choice([1, 1, 0])
        if not per:
            n = [min(v, 44) for v in n]
        cells = n[0] * n[1] * n[2]
        top = MOST_CELLS // (cells * (4 if bits == 64 else 2) * (4 if kind == "precond" else 1))
        c = dict(kind=kind, n1=n[0], n2=n[1], n3=n[2], per=per, norb=logu(1, max(1, min(256, top))), bits=bits)
        if kind == "precond":
            c["ncong"] = rng.randint(3, 6)
        return c
    if kind == "regions":
        return dict(kind=kind, nlr=logu(4, 128), nmin=rng.randint(12, 24), nmax=rng.randint(25, 40),
                    shapes=rng.randrange(1 << 20), bits=bits)
    if kind == "serve":
        return dict(kind=kind, clients=rng.randint(2, 10), nmin=16, nmax=rng.randint(24, 44), omin=2,
                    omax=rng.randint(4, 24), shapes=rng.randrange(1 << 20), bits=bits)
    if kind == "ortho":
        return dict(kind=kind, norb=logu(3, 256), ncoeff=logu(4000, 500000))
    if kind == "projectors":
        n = [rng.randint(16, 44) for _ in range(3)]
        return dict(kind=kind, n1=n[0], n2=n[1], n3=n[2], norb=logu(1, 128), atoms=logu(1, 40), m=rng.choice([1, 4, 9]),
                    shapes=rng.randrange(1 << 20))
    n = [rng.randint(12, 40) for _ in range(3)]
    return dict(kind=kind, n1=n[0], n2=n[1], n3=n[2], per=rng.choice([1, 0]), norb=rng.randint(1, 3))


# ---------------------------------------------------------------------------
# geometry

def box_masks(n, per):
    """Coarse and fine masks [i3, i2, i1]: all cells; the fine ones fill a
    periodic box and an ellipsoid of 0.4 times a free one."""
    full = np.ones(n[::-1], bool)
    if per:
        return full, full
    r2 = np.zeros(n[::-1])
    for ax, (m, axis) in enumerate(zip(n[::-1], range(3))):
        shape = [1, 1, 1]
        shape[axis] = m
        r2 = r2 + (((np.arange(m) - (m - 1) / 2.0) / (0.4 * m)) ** 2).reshape(shape)
    return full, r2 <= 1.0


def box(n, per):
    c, f = box_masks(n, per)
    return Locreg.from_masks(c, f, (per,) * 3, (H,) * 3)


def dims(case):
    return (case["n1"], case["n2"], case["n3"])


def region_sizes(case):
    r = random.Random(case["shapes"])
    return [tuple(r.randint(case["nmin"], case["nmax"]) for _ in range(3)) for _ in range(case["nlr"])]


def client_boxes(case):
    """(n, per, norb) of each client."""
    r = random.Random(case["shapes"])
    return [(tuple(r.randint(case["nmin"], case["nmax"]) for _ in range(3)), int(r.random() < 0.5),
             r.randint(case["omin"], case["omax"])) for _ in range(case["clients"])]


def isf(n, per):
    return tuple(2 * v if per else 2 * v + 29 for v in n)


def sphere(n, cen, rad):
    z, y, x = np.ogrid[:n[2], :n[1], :n[0]]
    return (x - cen[0]) ** 2 + (y - cen[1]) ** 2 + (z - cen[2]) ** 2 <= rad * rad


# ---------------------------------------------------------------------------
# inputs

def generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 11)
    return g


def coefficients(norb, ncoeff, g):
    """Rows of uniform(-1, 1) coefficients, each normalised."""
    psi = torch.rand(norb, ncoeff, generator=g, device=DEV, dtype=torch.float64)
    psi.mul_(2).sub_(1)
    psi /= psi.norm(dim=1, keepdim=True)
    return psi


def potential(n, per, seed):
    """Sum of four Gaussians on the real-space grid (z, y, x): random centres,
    widths 1-3 bohr, depths -2..-0.5 Ha, minimum image where periodic."""
    r = random.Random(int(seed) * 31 + 5)
    out = 0.0
    for _ in range(4):
        w, dep, f = r.uniform(1.0, 3.0), r.uniform(-2.0, -0.5), []
        for m, pts in zip(n, isf(n, per)):
            length = m * H
            d = (torch.arange(pts, dtype=torch.float64, device=DEV) - (0 if per else 14)) * (0.5 * H) - r.uniform(0, length)
            if per:
                d = d - length * torch.round(d / length)
            f.append(torch.exp(-d * d / (2 * w * w)))
        out = out + dep * f[2][:, None, None] * f[1][None, :, None] * f[0][None, None, :]
    return out.reshape(-1)


def dtype_of(case):
    return torch.float32 if case.get("bits", 64) == 32 else torch.float64


def shifts(case, seed):
    """c = 0.5 - eps of each orbital, eps uniform(-1, -0.1) Ha."""
    r = random.Random(int(seed) + 77)
    return [0.5 + r.uniform(0.1, 1.0) for _ in range(case["norb"])]


def atom_list(case):
    """(masks, m) of each atom: projectors on balls of 8 coarse / 4 fine cells."""
    r, n = random.Random(case["shapes"]), dims(case)
    out = []
    for _ in range(case["atoms"]):
        cen = [r.uniform(0, v - 1) for v in n]
        out.append((sphere(n, cen, 8.0), sphere(n, cen, 4.0)))
    return out


def raw(case, seed):
    """The inputs in FP64 as plain tensors, the same ones for prepare and exact."""
    g, k = generator(seed), case["kind"]
    if k in ("hpsi", "dropin", "density", "precond"):
        n = dims(case)
        c, f = box_masks(n, case["per"])
        psi = coefficients(case["norb"], int(c.sum()) + 7 * int(f.sum()), g)
        if k in ("hpsi", "dropin"):
            return dict(psi=psi, pot=potential(n, case["per"], seed))
        if k == "density":
            return dict(psi=psi, hfac=[2.0 / (0.5 * H) ** 3] * case["norb"])
        return dict(b=psi, c=shifts(case, seed))
    if k == "regions":
        out = []
        for i, n in enumerate(region_sizes(case)):
            c, f = box_masks(n, 0)
            out.append((n, coefficients(1, int(c.sum()) + 7 * int(f.sum()), g)[0], potential(n, 0, seed * 1000 + i)))
        return out
    if k == "serve":
        out = []
        for i, (n, per, norb) in enumerate(client_boxes(case)):
            c, f = box_masks(n, per)
            out.append((n, per, coefficients(norb, int(c.sum()) + 7 * int(f.sum()), g), potential(n, per, seed * 1000 + i)))
        return out
    if k == "ortho":
        return dict(psi=coefficients(case["norb"], case["ncoeff"], g))
    n, out = dims(case), []
    c, f = box_masks(n, 0)
    nc = int(c.sum()) + 7 * int(f.sum())
    for mc, mf in atom_list(case):
        mf = mf & f                          # projectors live inside the orbitals' region
        p = coefficients(case["m"], int(mc.sum()) + 7 * int(mf.sum()), g)
        h = torch.rand(case["m"], case["m"], generator=g, device=DEV, dtype=torch.float64)
        out.append((mc, mf, p, h + h.T))
    return dict(atoms=out, psi=coefficients(case["norb"], nc, g), hpsi=coefficients(case["norb"], nc, g))


# ---------------------------------------------------------------------------
# what a user's program holds, and one pass

def prepare(case, seed):
    k, dt, x = case["kind"], dtype_of(case), raw(case, seed)
    if k == "dropin":
        q = ocl.OclQueue()
        gp = ocl.GpuPointers(q, box(dims(case), case["per"]))
        return dict(kind=k, q=q, gp=gp, psi=x["psi"].cpu().numpy(), pot=x["pot"].cpu().numpy())
    ctx = Context(0)
    s = dict(kind=k, ctx=ctx)
    if k in ("hpsi", "density", "precond"):
        lr = box(dims(case), case["per"])
        s["batch"] = Batch(ctx, [lr], [0] * case["norb"])
    if k == "hpsi":
        s.update(psi=x["psi"].to(dt).reshape(-1), pot=x["pot"].to(dt), hpsi=torch.empty(x["psi"].numel(), dtype=dt, device=DEV),
                 ekin=torch.empty(case["norb"], dtype=torch.float64, device=DEV),
                 epot=torch.empty(case["norb"], dtype=torch.float64, device=DEV))
    elif k == "density":
        s.update(psi=x["psi"].to(dt).reshape(-1), hfac=torch.tensor(x["hfac"], dtype=torch.float64, device=DEV),
                 rho=torch.empty(lr.nisf, dtype=torch.float64, device=DEV))
    elif k == "precond":
        b = x["b"].to(dt).reshape(-1)
        s.update(b=b, x=torch.empty_like(b), c=torch.tensor(x["c"], dtype=torch.float64, device=DEV), ncong=case["ncong"])
    elif k == "regions":
        offs = np.cumsum([0] + [p.numel() for _, _, p in x])
        s["batch"] = Batch(ctx, [box(n, 0) for n, _, _ in x], list(range(len(x))), pot_offset=offs[:-1])
        s.update(psi=torch.cat([p for _, p, _ in x]).to(dt), pot=torch.cat([p for _, _, p in x]).to(dt),
                 ekin=torch.empty(len(x), dtype=torch.float64, device=DEV), epot=torch.empty(len(x), dtype=torch.float64, device=DEV))
        s["hpsi"] = torch.empty_like(s["psi"])
    elif k == "serve":
        cl = []
        for n, per, psi, pot in x:
            lr = box(n, per)
            psi = psi.to(dt)
            cl.append(dict(reg=Region(ctx, lr), psi=psi, hpsi=torch.empty_like(psi), pot=pot.to(dt),
                           rho=torch.empty(lr.nisf, dtype=torch.float64, device=DEV)))
        norb = sum(c["psi"].shape[0] for c in cl)
        s.update(clients=cl, ekin=torch.empty(norb, dtype=torch.float64, device=DEV),
                 epot=torch.empty(norb, dtype=torch.float64, device=DEV),
                 hfac=torch.full((norb,), 2.0 / (0.5 * H) ** 3, dtype=torch.float64, device=DEV))
    elif k == "ortho":
        s.update(psi=x["psi"], out=torch.empty_like(x["psi"]), work=torch.empty_like(x["psi"]))
    elif k == "projectors":
        n = dims(case)
        reg = Region(ctx, box(n, 0))
        s["region"] = reg
        s["proj"] = nlpsp.Projectors(ctx, reg, [(Locreg.from_masks(mc, mf, (0, 0, 0), (H,) * 3), p, h.cpu().numpy())
                                                for mc, mf, p, h in x["atoms"]])
        s.update(psi=x["psi"], hpsi0=x["hpsi"], hpsi=torch.empty_like(x["hpsi"]))
    return s


def run(s):
    k = s["kind"]
    if k in ("hpsi", "regions"):
        return s["batch"].locham(s["psi"], s["pot"], hpsi=s["hpsi"], ekin=s["ekin"], epot=s["epot"])
    if k == "dropin":
        hpsi, ekin, epot, _, _ = ocl.local_hamiltonian_ocl(s["q"], s["gp"], s["psi"], s["pot"])
        return hpsi, ekin, epot
    if k == "density":
        s["rho"].zero_()
        return s["batch"].locden(s["psi"], s["hfac"], s["rho"])
    if k == "precond":
        s["x"].zero_()                       # the CG starts from zero
        return s["batch"].precond(s["x"], s["b"], s["c"], s["ncong"])
    if k == "serve":
        cl = s["clients"]
        b = OrbitalBatch(s["ctx"], [(c["reg"], c["psi"][o], c["hpsi"][o], c["pot"], None)
                                    for c in cl for o in range(c["psi"].shape[0])])
        b.locham(s["ekin"], s["epot"])
        torch._foreach_zero_([c["rho"] for c in cl])
        b = OrbitalBatch(s["ctx"], [(c["reg"], c["psi"][o], None, None, c["rho"])
                                    for c in cl for o in range(c["psi"].shape[0])])
        b.locden(s["hfac"])
        return s["ekin"], s["epot"], [c["hpsi"] for c in cl], [c["rho"] for c in cl]
    if k == "ortho":
        s["out"].copy_(s["psi"])
        return ortho.orthonormalize(s["ctx"], s["out"], "cholesky", work=s["work"])
    s["hpsi"].copy_(s["hpsi0"])
    return s["hpsi"], s["proj"].apply(s["psi"], s["hpsi"])


# ---------------------------------------------------------------------------
# what a pass cannot do without

def grids(n, per):
    """(wavelet, fine, real-space) points of a box."""
    w = 8 * n[0] * n[1] * n[2]
    f = math.prod(2 * v if per else 2 * v + 14 for v in n)
    return w, f, math.prod(isf(n, per))


def hpsi_flops(n, per):
    """16-tap synthesis, magic filter and their transposes and the 29-tap
    kinetic filter, each once per axis, on the grids that they produce."""
    w, f, r = grids(n, per)
    return 2.0 * 3 * (16 * f + 16 * r + 16 * f + 16 * w + 29 * f) + 3 * r


def box_coeffs(n, per):
    c, f = box_masks(n, per)
    return int(c.sum()) + 7 * int(f.sum())


def work(case):
    k, e = case["kind"], case.get("bits", 64) // 8
    if k in ("hpsi", "dropin"):
        n, o, per = dims(case), case["norb"], case["per"]
        return dict(bytes=2.0 * e * o * box_coeffs(n, per) + e * math.prod(isf(n, per)), flops=o * hpsi_flops(n, per))
    if k == "regions":
        ns = region_sizes(case)
        return dict(bytes=sum(e * (2.0 * box_coeffs(n, 0) + math.prod(isf(n, 0))) for n in ns),
                    flops=sum(hpsi_flops(n, 0) for n in ns))
    if k == "serve":
        by = fl = 0.0
        for n, per, o in client_boxes(case):
            r = math.prod(isf(n, per))
            by += o * 3.0 * e * box_coeffs(n, per) + r * (e + 8)
            fl += o * (hpsi_flops(n, per) + 2.0 * 3 * (16 * grids(n, per)[1] + 16 * r) + 3 * r)
        return dict(bytes=by, flops=fl)
    if k == "density":
        n, o, per = dims(case), case["norb"], case["per"]
        _, f, r = grids(n, per)
        return dict(bytes=1.0 * e * o * box_coeffs(n, per) + 8 * r, flops=o * (2.0 * 3 * (16 * f + 16 * r) + 3 * r))
    if k == "precond":
        n, o, per = dims(case), case["norb"], case["per"]
        w, f, _ = grids(n, per)
        nc, it = box_coeffs(n, per), case["ncong"]
        # an iteration reads and writes d, r and x and forms A d; synthesis,
        # kinetic filter and analysis once per axis
        return dict(bytes=1.0 * e * o * nc * 6 * it, flops=o * it * (2.0 * 3 * (16 * f + 29 * f + 16 * w) + 10.0 * nc))
    if k == "ortho":
        m, c = case["norb"], case["ncoeff"]
        return dict(bytes=16.0 * m * c, flops=2.0 * m * (m + 1) * c)
    n, o = dims(case), case["norb"]
    pts = sum(int(mc.sum()) + 7 * int((mf & box_masks(n, 0)[1]).sum()) for mc, mf in atom_list(case))
    return dict(bytes=24.0 * o * box_coeffs(n, 0) + 8.0 * pts * case["m"], flops=4.0 * pts * case["m"] * o)


def tolerance(case):
    # against exact(): 32 bits 1.7e-7 (H psi), 5e-8 (density), about 8e-7 (the
    # preconditioner, whose CG iterations add up); 64 bits below 5e-16, where
    # another order of the sums shows up to a few 1e-15 (CG: a few 1e-14)
    cg = case["kind"] == "precond"
    if case.get("bits", 64) == 32:
        return {"rel": 4e-6 if cg else 8e-7, "max": 4e-4 if cg else 4e-5}
    return {"rel": 1e-12 if cg else 2e-14, "max": 1e-10 if cg else 2e-12}


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits

CH = [-0.0033824159510050025955, -0.00054213233180001068935, 0.031695087811525991431, 0.0076074873249766081919,
      -0.14329423835127266284, -0.061273359067811077843, 0.48135965125905339159, 0.77718575169962802862,
      0.36444189483617893676, -0.051945838107881800736, -0.027219029917103486322, 0.049137179673730286787,
      0.0038087520138944894631, -0.014952258337062199118, -0.00030292051472413308126, 0.0018899503327676891843]
CG = [-CH[15 - k] if k % 2 == 0 else CH[15 - k] for k in range(16)]
MF = [8.4334247333529341094733325815816e-7, -0.1290557201342060969516786758559028e-4, 0.8762984476210559564689161894116397e-4,
      -0.30158038132690463167163703826169879e-3, 0.174723713672993903449447812749852942e-2,
      -0.942047030201080385922711540948195075e-2, 0.2373821463724942397566389712597274535e-1, 0.612625895831207982195380597e-1,
      0.9940415697834003993178616713, -0.604895289196983516002834636e-1, -0.2103025160930381434955489412839065067e-1,
      0.1337263414854794752733423467013220997e-1, -0.344128144493493857280881509686821861e-2,
      0.49443227688689919192282259476750972e-3, -0.5185986881673432922848639136911487e-4, 2.72734492911979659657715313017228e-6]
KIN = [-3.5536922899131901941296809374, 2.2191465938911163898794546405, -0.6156141465570069496314853949,
       0.2371780582153805636239247476, -0.0822663999742123340987663521, 0.02207029188482255523789911295638968409,
       -0.409765689342633823899327051188315485e-2, 0.45167920287502235349480037639758496e-3,
       -0.2398228524507599670405555359023135e-4, 2.0904234952920365957922889447361e-6, -3.7230763047369275848791496973044e-7,
       -1.05857055496741470373494132287e-8, -5.813879830282540547959250667e-11, 2.70800493626319438269856689037647576e-13,
       -6.924474940639200152025730585882e-18]
A2, B2 = 3.55369228991319019, 24.8758460293923314


def matrices(n, per):
    """Synthesis (fine x wavelet), magic filter (real-space x fine) and kinetic
    matrix (fine x fine, times -1/(2 (h/2)^2)) of one axis."""
    f, r = (2 * n, 2 * n) if per else (2 * n + 14, 2 * n + 29)
    s, m, t = np.zeros((f, 2 * n)), np.zeros((r, f)), np.zeros((f, f))

    def put(a, row, col, v):
        if per:
            a[row % a.shape[0], col % a.shape[1]] += v
        elif 0 <= row < a.shape[0] and 0 <= col < a.shape[1]:
            a[row, col] += v

    for i in range(n):
        for k in range(16):
            q = 2 * i + k - 7 + (0 if per else 7)
            put(s, q, i, CH[k])
            s[q % f if per else q, n + i] += CG[k]
    for q in range(r):
        for k in range(16):
            put(m, q, q - 8 + k if per else q - 15 + k, MF[k])
    for q in range(f):
        for l in range(-14, 15):
            put(t, q, q + l, KIN[abs(l)] * (-0.5 / (0.5 * H) ** 2))
    return [torch.tensor(a, device=DEV) for a in (s, m, t)]


class Box:
    """One box's dense operators: B = magic filter x synthesis and the kinetic
    matrix in the wavelet basis, per axis, and the maps between compressed
    vectors and the dense wavelet grid [z][y][x], each axis [scaling | wavelet]."""

    def __init__(self, n, per):
        self.n, self.per = n, per
        self.B, self.T = [], []
        for v in n:
            s, m, t = matrices(v, per)
            self.B.append(m @ s)
            self.T.append(s.T @ t @ s)
        c, f = box_masks(n, per)
        g1, g2 = 2 * n[0], 2 * n[1]
        zc, yc, xc = np.nonzero(c)
        zf, yf, xf = np.nonzero(f)
        idx = [(zc * g2 + yc) * g1 + xc]
        fine = [((zf + n[2] * (q >> 2 & 1)) * g2 + yf + n[1] * (q >> 1 & 1)) * g1 + xf + n[0] * (q & 1) for q in range(1, 8)]
        idx.append(np.stack(fine, axis=1).reshape(-1))
        comp = [np.zeros(len(zc), np.int64), np.tile(np.arange(1, 8), len(zf))]
        self.idx = torch.tensor(np.concatenate(idx), device=DEV)
        self.comp = torch.tensor(np.concatenate(comp), device=DEV)

    def dense(self, v):
        d = torch.zeros(v.shape[0], 8 * self.n[0] * self.n[1] * self.n[2], dtype=torch.float64, device=DEV)
        d[:, self.idx] = v
        return d.reshape(-1, 2 * self.n[2], 2 * self.n[1], 2 * self.n[0])

    def packed(self, d):
        return d.reshape(d.shape[0], -1)[:, self.idx]

    @staticmethod
    def along(a, axis, d):
        if axis == 0:
            return d @ a.T
        if axis == 1:
            return torch.matmul(a, d)
        o, z, y, x = d.shape
        return torch.matmul(a, d.reshape(o, z, y * x)).reshape(o, a.shape[0], y, x)

    def real(self, d):
        for ax in range(3):
            d = self.along(self.B[ax], ax, d)
        return d

    def kinetic(self, d):
        return sum(self.along(self.T[ax], ax, d) for ax in range(3))

    def hpsi(self, psi, pot):
        hp, ek, ep = [], [], []
        v = pot.reshape(isf(self.n, self.per)[::-1])
        for p in psi.split(16):
            d = self.dense(p)
            r = self.real(d)
            w = r * v
            ep.append((w * r).sum(dim=(1, 2, 3)))
            for ax in range(3):
                w = self.along(self.B[ax].T, ax, w)
            t = self.kinetic(d)
            ek.append((d * t).sum(dim=(1, 2, 3)))
            hp.append(self.packed(w + t))
        return torch.cat(hp), torch.cat(ek), torch.cat(ep)

    def density(self, psi, hfac):
        rho = 0.0
        for p, h in zip(psi.split(16), hfac.split(16)):
            rho = rho + (self.real(self.dense(p)) ** 2 * h[:, None, None, None]).sum(dim=0)
        return rho.reshape(-1)

    def precond(self, b, c, ncong):
        """CG on D^-1/2 (c + T) D^-1/2 from zero, the result scaled by D^-1/2."""
        xs, hist = [], []
        hf = 0.5 * H
        for bb, cc in zip(b.split(16), c.split(16)):
            k = self.comp
            diag = sum(A2 + (B2 - A2) * (k >> d & 1).to(torch.float64) for d in range(3)) * (0.125 / hf ** 2)
            sc = 1.0 / torch.sqrt(cc[:, None] + diag[None, :])

            def op(v):
                u = sc * v
                return sc * (cc[:, None] * u + self.packed(self.kinetic(self.dense(u))))

            x, r = torch.zeros_like(bb), bb.clone()
            d, rr = r.clone(), (r * r).sum(dim=1)
            hh = [rr]
            for _ in range(ncong):
                ad = op(d)
                al = rr / (d * ad).sum(dim=1)
                x, r = x + al[:, None] * d, r - al[:, None] * ad
                new = (r * r).sum(dim=1)
                d, rr = r + (new / rr)[:, None] * d, new
                hh.append(rr)
            xs.append(sc * x)
            hist.append(torch.stack(hh))
        return torch.cat(xs), torch.cat(hist, dim=1)


def rounded(t, case):
    """Inputs as the call receives them."""
    return t.to(dtype_of(case)).to(torch.float64)


def exact(case, seed):
    k, x = case["kind"], raw(case, seed)
    if k in ("hpsi", "dropin"):
        hp, ek, ep = Box(dims(case), case["per"]).hpsi(rounded(x["psi"], case), rounded(x["pot"], case))
        if k == "hpsi":
            return hp.reshape(-1), ek, ep
        return tuple(t.cpu().numpy() for t in (hp, ek, ep))
    if k == "density":
        return Box(dims(case), case["per"]).density(rounded(x["psi"], case), torch.tensor(x["hfac"], dtype=torch.float64, device=DEV))
    if k == "precond":
        xx, hist = Box(dims(case), case["per"]).precond(rounded(x["b"], case), torch.tensor(x["c"], dtype=torch.float64, device=DEV), case["ncong"])
        return xx.reshape(-1), hist
    if k == "regions":
        got = [Box(n, 0).hpsi(rounded(p[None], case), rounded(v, case)) for n, p, v in x]
        return tuple(torch.cat([g[i].reshape(-1) for g in got]) for i in range(3))
    if k == "serve":
        hp, ek, ep, rho = [], [], [], []
        for n, per, psi, pot in x:
            b, p = Box(n, per), rounded(psi, case)
            a, e1, e2 = b.hpsi(p, rounded(pot, case))
            hp.append(a), ek.append(e1), ep.append(e2)
            rho.append(b.density(p, torch.full((p.shape[0],), 2.0 / (0.5 * H) ** 3, dtype=torch.float64, device=DEV)))
        return torch.cat(ek), torch.cat(ep), hp, rho
    if k == "ortho":
        p = x["psi"]
        s = p @ p.T
        return torch.linalg.solve_triangular(torch.linalg.cholesky(s), p, upper=False), s
    n = dims(case)
    w = Box(n, 0)
    size = 8 * n[0] * n[1] * n[2]
    hp, ep = x["hpsi"].clone(), 0.0
    where = torch.full((size,), -1, dtype=torch.int64, device=DEV)
    where[w.idx] = torch.arange(len(w.idx), device=DEV)
    g1, g2 = 2 * n[0], 2 * n[1]
    for mc, mf, p, h in x["atoms"]:
        zc, yc, xc = np.nonzero(mc)
        zf, yf, xf = np.nonzero(mf)
        fine = [((zf + n[2] * (q >> 2 & 1)) * g2 + yf + n[1] * (q >> 1 & 1)) * g1 + xf + n[0] * (q & 1) for q in range(1, 8)]
        at = np.concatenate([(zc * g2 + yc) * g1 + xc, np.stack(fine, axis=1).reshape(-1)])
        at = where[torch.tensor(at, device=DEV)]
        c = x["psi"][:, at] @ p.T
        hc = c @ h.T
        ep = ep + (c * hc).sum(dim=1)
        hp[:, at] += hc @ p
    return hp, ep
