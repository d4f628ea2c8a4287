"""What an earlier call left in the scratch does not reach a later call: every
entry point of the fused kernels gives the same bits after a call whose
orbitals and potential were all NaN as after one whose were all zero, on the
same context (for the allocation-free entry point: in the same static array).
The earlier call fills its scratch without gaps (a periodic box) and more of it
than the later one uses.  Free boxes of odd and even sizes: their real-space
rows have odd lengths and pad columns."""
import numpy as np
import pytest

from test_zz_no_alloc import call_noalloc
from wvlh.batch import Batch, OrbitalBatch, Region
from wvlh.keys import Locreg
from wvlh.workloads import full_periodic

pytestmark = pytest.mark.gpu
DTYPES = ["float64", "float32"]


def region(N, per, seed):
    rng = np.random.default_rng(seed)
    return Locreg.from_masks(np.ones(N[::-1], bool), rng.random(N[::-1]) < 0.5, per, (0.45, 0.4, 0.5))


def filler(ctx, dt, torch):
    """fill(v): calls of psi = pot = v over buffers larger than the tests'."""
    lr = full_periodic(24)
    b = Batch(ctx, [lr], [0] * 4)

    def fill(v):
        psi = torch.full((b.psi_size,), v, dtype=dt, device="cuda")
        b.precond(psi.clone(), psi, np.full(4, 0.7), 2)
        b.locden(psi, np.ones(4), torch.zeros(lr.nisf, dtype=torch.float64, device="cuda"))
        b.locham(psi, torch.full((lr.nisf,), v, dtype=dt, device="cuda"))
    return fill


def same_after(fill, call, torch):
    fill(0.0)
    want = [t.clone() for t in call()]
    fill(float("nan"))
    got = call()
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.isfinite(b).all()
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype_name", DTYPES)
def test_several_regions(torch_cuda, wctx, dtype_name):
    torch, dt = torch_cuda, getattr(torch_cuda, dtype_name)
    lrs = [region((9, 8, 11), (0, 0, 0), 1), region((12, 11, 8), (0, 1, 0), 2), region((6, 7, 5), (0, 0, 0), 3)]
    orb = [0, 1, 2, 1, 0]
    off = np.cumsum([0] + [lr.nisf for lr in lrs])
    b = Batch(wctx, lrs, orb, off[orb])
    g = torch.Generator(device="cuda").manual_seed(1)
    psi = torch.rand(b.psi_size, dtype=dt, device="cuda", generator=g) - 0.5
    pot = -torch.rand(int(off[-1]), dtype=dt, device="cuda", generator=g)
    hfac = torch.ones(len(orb), dtype=torch.float64, device="cuda")
    cprec = np.full(len(orb), 0.7)

    def precond():
        x = torch.zeros_like(psi)
        b.precond(x, psi, cprec, 3)
        return [x]
    fill = filler(wctx, dt, torch)
    same_after(fill, lambda: list(b.locham(psi, pot)), torch)
    same_after(fill, lambda: [b.locden(psi, hfac, torch.zeros(int(off[-1]), dtype=torch.float64, device="cuda"))], torch)
    same_after(fill, precond, torch)


@pytest.mark.parametrize("dtype_name", DTYPES)
def test_orbital_batch_of_two_boxes(torch_cuda, wctx, dtype_name):
    torch, dt = torch_cuda, getattr(torch_cuda, dtype_name)
    regs = [Region(wctx, region((11, 9, 8), (0, 0, 0), 4)), Region(wctx, region((8, 10, 9), (0, 0, 1), 5))]
    g = torch.Generator(device="cuda").manual_seed(2)
    psi = [torch.rand(r.psi_size, dtype=dt, device="cuda", generator=g) - 0.5 for r in regs]
    pot = [-torch.rand(r.grid_size, dtype=dt, device="cuda", generator=g) for r in regs]
    hpsi = [torch.zeros_like(p) for p in psi]

    def call():
        b = OrbitalBatch(wctx, [(regs[i], psi[i], hpsi[i], pot[i], None) for i in range(2)])
        e = torch.empty(2, 2, dtype=torch.float64, device="cuda")
        b.locham(e[0], e[1])
        return [*hpsi, e]
    same_after(filler(wctx, dt, torch), call, torch)


@pytest.mark.parametrize("prec", [64, 32])
def test_noalloc(torch_cuda, prec):
    torch, dt = torch_cuda, torch_cuda.float64 if prec == 64 else torch_cuda.float32
    lr, big = region((11, 9, 8), (0, 0, 0), 6), full_periodic(24)
    g = torch.Generator(device="cuda").manual_seed(3)
    psi = torch.rand(lr.ncoeff, dtype=dt, device="cuda", generator=g) - 0.5
    pot = -torch.rand(lr.nisf, dtype=dt, device="cuda", generator=g)
    st = torch.cuda.current_stream()

    def fill(v):
        call_noalloc(torch, big, torch.full((big.ncoeff,), v, dtype=dt, device="cuda"),
                     torch.full((big.nisf,), v, dtype=dt, device="cuda"), prec, st)

    def call():
        h, ek, ep = call_noalloc(torch, lr, psi, pot, prec, st)
        return [h, torch.tensor([ek, ep])]
    same_after(fill, call, torch)
