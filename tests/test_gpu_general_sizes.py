"""Sizes off the presets: every kind of two-pass grid length (even and odd,
with and without the band-pruned first DFT, the row-split FP64 density pass),
odd state counts, state counts at the edges of the product tiles and of
several tiles, and the three Newton-Schulz forms, against the oracle."""
import dataclasses
import math

import numpy as np
import pytest

from openatom_b200.system import make_system
from oracle import cp_oracle as O

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.max(np.abs(np.asarray(a) - b)) / max(float(np.max(np.abs(b))), 1e-300))


def grid_system(n, nstate, box=7.0, frac=1.0):
    """A 2-water cell whose state sphere reaches kmax = (n - 1) / 4 (times frac).
    The radius lies 0.3 above it: no squared radius of the states or of the
    density is then a whole number, so that no point lies on the cutoff, where
    the last bit of |g|^2 would decide which sphere it is in."""
    kmax = max(2.5, frac * ((n - 1) // 4)) + 0.3
    return make_system("w2", seed=3, nfft=(n, n, n), nstate=nstate, box=box,
                       ecut_ry=(kmax * 2.0 * math.pi / box) ** 2)


# FP64: rounding; mixed: FP32 transforms, about 3 log2(n) roundings of 6e-8
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("mixed", 1e-5)])
@pytest.mark.parametrize("n,nstate", [(12, 3), (15, 2), (18, 3), (20, 5), (30, 3), (32, 2), (36, 3), (40, 3), (48, 5),
                                      (54, 3), (60, 2), (75, 3), (81, 2), (90, 3), (96, 3), (108, 5), (150, 3),
                                      (24, 16), (64, 15), (64, 17), (96, 64),
                                      (16, 4), (25, 5), (27, 3), (45, 3), (50, 2), (72, 5), (80, 3), (100, 3),
                                      (120, 3), (125, 2), (128, 3), (135, 2), (144, 3), (160, 2)])
def test_grid_lengths(n, nstate, precision, tol):
    import torch
    from openatom_b200.gpu import CPContext
    s = grid_system(n, nstate)
    ctx = CPContext(s, precision)
    psi = torch.from_numpy(s.psi).cuda()
    rho = torch.zeros(n, n, n, dtype=torch.float64, device="cuda")
    f = torch.zeros_like(psi)
    f2 = torch.zeros_like(psi)
    v = np.random.default_rng(4).standard_normal((n, n, n)) * 0.3
    ctx.state_fft_fwd(psi, rho)
    ctx.set_vks(torch.from_numpy(v).cuda())
    ctx.vks_apply_fft_bwd(psi, f)
    ctx.vks_apply_fft_bwd(psi, f2, recompute_fwd=True)
    torch.cuda.synchronize()
    psir = O.state_g_to_r(s.psi, s)
    fr, _ = O.eke(s.psi, O.add_forces(O.vks_forces(psir, v, s), None, s), s)
    assert rel(rho.cpu().numpy(), O.density(psir, s)) < tol
    assert rel(f.cpu().numpy(), fr) < tol
    assert rel(f2.cpu().numpy(), fr) < tol


def with_lines(s, order):
    """The same system with its z-lines (and their coefficients) in another
    order; returns it and the map new -> old of the coefficients."""
    ln = s.line_nneg + s.line_npos
    src = np.concatenate([np.arange(s.line_off[l], s.line_off[l] + ln[l]) for l in order])
    lines = {k: getattr(s, k)[order] for k in ("line_kx", "line_ky", "line_nneg", "line_npos")}
    off = np.concatenate([[0], np.cumsum(ln[order])[:-1]]).astype(np.int32)
    pts = {k: getattr(s, k)[src] for k in ("kx", "ky", "kz", "cmass")}
    return dataclasses.replace(s, psi=np.ascontiguousarray(s.psi[:, src]), line_off=off, **lines, **pts), src


# planes with per-state two-pass kernels, with the runtime plan only, and (FP64) without pair kernels
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("mixed", 1e-5)])
@pytest.mark.parametrize("n", [40, 45, 125])
@pytest.mark.parametrize("order", ["columns", "shuffled", "rows"])
def test_line_orders(n, order, precision, tol):
    """Whole kx columns in another order (the state-pair kernels take them),
    lines shuffled or sorted by ky (they do not): the same density, forces
    and nonlocal forces as the oracle's."""
    import torch
    from openatom_b200.gpu import CPContext
    s0 = grid_system(n, 3)
    first = int((s0.line_kx == 0).sum())      # kx = 0 stays first, in the reference's order
    rest = np.arange(first, s0.nlines)
    if order == "columns":
        rest = np.concatenate([rest[s0.line_kx[rest] == k] for k in sorted(set(s0.line_kx[rest]), reverse=True)])
    elif order == "shuffled":
        rest = np.random.default_rng(5).permutation(rest)
    else:
        rest = rest[np.argsort(s0.line_ky[rest], kind="stable")]
    s, src = with_lines(s0, np.concatenate([np.arange(first), rest]))
    ctx = CPContext(s, precision)
    pairs = order == "columns" and not (n == 125 and precision == "fp64")
    assert ctx.sizes()["pair_planes"] == int(pairs)
    psi = torch.from_numpy(s.psi).cuda()
    rho = torch.zeros(n, n, n, dtype=torch.float64, device="cuda")
    f, f2, fnl, fees = (torch.zeros_like(psi) for _ in range(4))
    v = np.random.default_rng(4).standard_normal((n, n, n)) * 0.3
    ctx.state_fft_fwd(psi, rho)
    ctx.set_vks(torch.from_numpy(v).cuda())
    ctx.vks_apply_fft_bwd(psi, f)
    ctx.vks_apply_fft_bwd(psi, f2, recompute_fwd=True)
    ctx.nl_sf(psi, fnl)
    ctx.ees_init(1.2, 4)
    ctx.nl_ees(psi, fees)
    torch.cuda.synchronize()
    psir = O.state_g_to_r(s0.psi, s0)
    fr, _ = O.eke(s0.psi, O.add_forces(O.vks_forces(psir, v, s0), None, s0), s0)
    assert rel(rho.cpu().numpy(), O.density(psir, s0)) < tol
    assert rel(f.cpu().numpy(), fr[:, src]) < tol
    assert rel(f2.cpu().numpy(), fr[:, src]) < tol
    assert rel(fnl.cpu().numpy(), O.nl_energy_forces(s0.psi, s0)[0][:, src]) < 1e-9
    fe = O.nl_ees_energy_forces(s0.psi, s0, O.ees_setup(s0, 1.2, 4))[0]
    assert rel(fees.cpu().numpy(), fe[:, src]) < (1e-9 if precision == "fp64" else 1e-5)


@pytest.mark.parametrize("n", [15, 25, 27, 45, 60, 81, 90, 100, 120, 125, 128, 135, 144, 150, 160])
def test_density_path_lengths(n):
    """The density transforms and the Hartree / XC path off the preset lengths."""
    import torch
    from openatom_b200.gpu import CPContext
    s = grid_system(n, 2, frac=0.5)
    ctx = CPContext(s, "fp64")
    vks = torch.zeros(n, n, n, dtype=torch.float64, device="cuda")
    ctx.state_fft_fwd(torch.from_numpy(s.psi).cuda())
    ctx.vks_build(vks)
    en = ctx.energies()
    _, vref, eref = O.vks_build(O.state_g_to_r(s.psi, s), s)
    assert rel(vks.cpu().numpy(), vref) < 1e-10
    for k in ("EHART", "EEXT", "EEXC", "MUXC"):
        assert abs(en[k] - eref[k]) <= 1e-10 * max(1.0, abs(eref[k])), k


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-9), ("mixed", 1e-5)])
@pytest.mark.parametrize("n,nstate,order,scale", [(40, 5, 4, 1.2), (45, 3, 6, 1.3), (64, 4, 8, 1.0), (96, 3, 4, 1.2),
                                                (24, 15, 4, 1.2), (24, 33, 6, 1.2), (40, 16, 4, 1.2), (64, 9, 8, 1.0),
                                                (96, 8, 4, 1.2)])
def test_ees_pairs(n, nstate, order, scale, precision, tol):
    import torch
    from openatom_b200.gpu import CPContext
    s = grid_system(n, nstate)
    ctx = CPContext(s, precision)
    ctx.ees_init(scale, order)
    f = torch.zeros(s.psi.shape, dtype=torch.complex128, device="cuda")
    enl = torch.zeros(nstate, dtype=torch.float64, device="cuda")
    ctx.nl_ees(torch.from_numpy(s.psi).cuda(), f, enl_out=enl)
    torch.cuda.synchronize()
    fr, er, _ = O.nl_ees_energy_forces(s.psi, s, O.ees_setup(s, scale, order))
    assert rel(enl.cpu().numpy(), er) < tol
    assert rel(f.cpu().numpy(), fr) < tol


@pytest.mark.parametrize("nstate", [5, 31, 33, 64, 65, 100, 129, 150, 199, 256, 300])
def test_products_of_several_tiles(nstate):
    """S (symmetric tiles), Lambda, the two-term backward product and the
    rotation: FP64 to rounding; split-BF16 to the rounding of FP32 sums of six
    products (three per term) over the longest inner dimension, a random walk
    of sqrt(6 nstate) steps of 2^-24 with a factor 4."""
    import torch
    from openatom_b200.gpu import CPContext
    s = make_system("w4", seed=9, nstate=nstate, pseudo="analytic")
    rng = np.random.default_rng(2)
    F = (rng.standard_normal(s.psi.shape) + 1j * rng.standard_normal(s.psi.shape)) * 0.1
    T = np.eye(nstate) + 1e-3 * rng.standard_normal((nstate, nstate))
    fref, lref = O.lambda_step(s.psi, F, T, s)
    ps = O.kx0_scale(s.psi, s, 1.0 / math.sqrt(2.0))
    sref = O.pc_forward(ps, ps, s, 2.0)
    psi, Fg, Tg = (torch.from_numpy(a).cuda() for a in (s.psi, F, T))
    for precision, tol in (("fp64", 1e-12), ("mixed", 4 * math.sqrt(6 * nstate) * 2.0**-24)):
        c = CPContext(s, precision)
        S = torch.zeros(nstate, nstate, dtype=torch.float64, device="cuda")
        lam, gam, out, rot = torch.zeros_like(S), torch.zeros_like(S), torch.zeros_like(psi), torch.zeros_like(psi)
        fwd, bwd = (c.pc_forward, c.pc_backward) if precision == "fp64" else (c.pc_forward_mixed, c.pc_backward_mixed)
        c.pc_forward(psi, psi, 2.0, 0.5, S)
        fwd(psi, Fg, 1.0, 1.0, lam)
        c.small_gemm(Tg, torch.from_numpy(lref).cuda(), 1.0, gam)
        bwd(gam, psi, -0.5, -1.0, out, M2=Tg, X2=Fg, a2=1.0)
        c.pc_backward(Tg, psi, 1.0, 1.0, rot)
        c.check()
        assert rel(S.cpu().numpy(), sref) < 1e-12 and torch.equal(S, S.T)
        assert rel(lam.cpu().numpy(), lref) < tol
        assert rel(out.cpu().numpy(), fref) < tol
        assert rel(rot.cpu().numpy(), T.T @ s.psi) < 1e-12


@pytest.mark.parametrize("nstate", [1, 2, 7, 8, 31, 32, 48, 50, 51, 130, 161, 199, 288])
def test_newton_schulz_sizes(nstate):
    import torch
    from openatom_b200.gpu import CPContext
    s = make_system("w2", seed=9, nstate=nstate, pseudo="analytic")
    e = np.random.default_rng(nstate).standard_normal((nstate, nstate)) * 5e-3
    S = 2.0 * np.eye(nstate) + e + e.T
    T = torch.zeros(nstate, nstate, dtype=torch.float64, device="cuda")
    it, err, ok, smax = CPContext(s, "fp64").ortho_invsqrt(torch.from_numpy(S).cuda(), T, 1e-15, 100, with_smax=True)
    tref, iref, _ = O.newton_schulz(S, 1e-15, 100)
    assert ok and abs(it - iref) <= 1
    assert rel(T.cpu().numpy(), tref) < 1e-13
    assert abs(smax - np.max(np.abs(S - 2.0 * np.eye(nstate)))) < 1e-15
