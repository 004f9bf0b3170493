"""Failure detection without a GPU fault (the reference ends such runs with
CkAbort / EXIT: ortho.C:129-133, cp_lowdin.C:246-252):

* a pipeline wait of a tcgen05 product runs out of time because a host-set
  hook made one block skip the loads of one stage: the block takes its
  error path (loads landed, TMEM freed), oa_gpu_check reports it once, and
  the context gives the right product on the next call;
* a non-finite coefficient and a singular overlap matrix injected from the
  host: the native run returns OA_ERR_NONFINITE / OA_ERR_NOT_CONVERGED and
  names the first failing step;
* a step capture reported as failed by a host hook: the stage calls that
  follow sum their energies, and the next native run captures again;
* a device allocation reported as failed by a host hook: psi(r) gives its
  memory back and the per-state kernels take the system."""
import time

import numpy as np
import pytest

from openatom_b200.system import make_system

pytestmark = pytest.mark.gpu


def test_bounded_wait_runs_out_and_is_reported():
    import torch
    from openatom_b200.gpu import CPContext, OaError, OA_ERR_CUDA
    s = make_system("w8", nstate=16, seed=31)
    ctx = CPContext(s, "mixed")
    rng = np.random.default_rng(3)
    psi = torch.from_numpy(s.psi).cuda()
    F = torch.from_numpy((rng.standard_normal(s.psi.shape) + 1j * rng.standard_normal(s.psi.shape)) * 0.1).cuda()
    lam0 = torch.zeros(s.nstate, s.nstate, dtype=torch.float64, device="cuda")
    ctx.pc_forward_mixed(psi, F, 1.0, 1.0, lam0)
    ctx.check()
    ctx.fault_inject(1)
    lam1 = torch.zeros_like(lam0)
    t0 = time.perf_counter()
    ctx.pc_forward_mixed(psi, F, 1.0, 1.0, lam1)
    with pytest.raises(OaError) as ei:
        ctx.check()
    dt = time.perf_counter() - t0
    assert ei.value.status == OA_ERR_CUDA and "ran out of time" in str(ei.value)
    # one 200 ms wait (plus the bounded clean-up waits), not an iteration count
    assert 0.15 < dt < 10.0, dt
    # the failed block's partial was zeroed: the product differs, is finite
    got = lam1.cpu().numpy()
    assert np.all(np.isfinite(got)) and not np.array_equal(got, lam0.cpu().numpy())
    # reported once; the context is usable and the hook was consumed
    ctx.check()
    lam2 = torch.zeros_like(lam0)
    ctx.pc_forward_mixed(psi, F, 1.0, 1.0, lam2)
    ctx.check()
    assert np.array_equal(lam2.cpu().numpy(), lam0.cpu().numpy())
    ctx.close()


def test_nonfinite_coefficient_names_the_step():
    from openatom_b200.gpu import CPDriver, OaError, OA_ERR_NONFINITE
    s = make_system("w2", seed=32, dt=0.5)
    d = CPDriver(s, "fp64")
    d.psi[1, 7] = float("nan")
    d.psi_t[1, 7] = float("nan")
    st = d.native_state(use_graph=True)
    with pytest.raises(OaError) as ei:
        d.run_native(st, 3)
    assert ei.value.status == OA_ERR_NONFINITE
    assert "step 1 of 3" in str(ei.value)


def test_singular_overlap_names_the_step():
    """Two equal states make S singular: the Schulz iteration cannot reach
    its tolerance (it overflows), the run reports the first step."""
    from openatom_b200.gpu import CPDriver, OaError, OA_ERR_NONFINITE, OA_ERR_NOT_CONVERGED
    s = make_system("w2", seed=33, dt=0.5)
    p0 = s.psi.copy()
    p0[1] = p0[0]
    d = CPDriver(s, "fp64", psi0=p0)
    st = d.native_state(use_graph=True)
    with pytest.raises(OaError) as ei:
        d.run_native(st, 2)
    assert ei.value.status in (OA_ERR_NONFINITE, OA_ERR_NOT_CONVERGED)
    assert "step 1 of 2" in str(ei.value)


@pytest.mark.parametrize("nstate", [8, 49])
def test_failed_capture_leaves_the_context_usable(nstate):
    """One graph per step (8 states) and two around the cooperative
    Newton-Schulz launch (49 states: the first one's capture fails)."""
    import torch
    from openatom_b200.gpu import CPDriver, OaError, OA_ERR_CUDA
    s = make_system("w2", seed=34, nstate=nstate, dt=0.5, pseudo="analytic")
    d, ref = CPDriver(s, "fp64"), CPDriver(s, "fp64")
    st, sr = d.native_state(use_graph=True), ref.native_state(use_graph=True)
    d.run_native(st, 1)
    ref.run_native(sr, 1)
    it = st.iteration
    d.ctx.fault_inject(2)
    with pytest.raises(OaError) as ei:
        d.run_native(st, 2)
    assert ei.value.status == OA_ERR_CUDA
    # stage calls of other coefficients: their own energies
    d.psi.mul_(0.9)
    ref.psi.mul_(0.9)
    d.forces()
    ref.forces()
    got, want = d.ctx.energies(), ref.ctx.energies()
    for k in ("EKE", "EHART", "EEXT", "EEXC", "ENL"):
        assert got[k] == want[k], k
    # and the run goes on
    d.psi.div_(0.9)
    ref.psi.copy_(d.psi)
    torch.cuda.synchronize()
    st.iteration = it
    for g, r in zip(d.run_native(st, 2), ref.run_native(sr, 2)):
        for k in ("EKE", "EHART", "EEXT", "EEXC", "ENL", "FICT_KE"):
            assert g[k] == r[k], k


KEYS = ("EKE", "EHART", "EEXT", "EEXC", "ENL", "FICT_KE")


def agree(got, ref, s, precision):
    """Two transform paths: FP64 to rounding; mixed, FP32 transforms with and
    without the renormalised density, as for the tuning choices."""
    tol = 1e-11 if precision == "fp64" else 2e-6
    for g, r in zip(got, ref):
        for k in KEYS:
            assert abs(g[k] - r[k]) <= tol * max(1.0, abs(r[k])), (k, g[k], r[k])
        assert abs(sum(g[k] - r[k] for k in KEYS[:5])) / s.natm <= (1e-11 if precision == "fp64" else 1e-6)


# lengths whose per-state kernels are the runtime plan (45) and the two-pass kernels (64)
@pytest.mark.parametrize("n,nstate", [(45, 5), (64, 8)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_no_memory_for_psir(n, nstate, precision):
    from openatom_b200.gpu import CPContext, CPDriver
    s = make_system("w2", seed=35, nfft=(n, n, n), nstate=nstate, box=7.0, ecut_ry=60.0, dt=0.5)
    def driver():
        return CPDriver(s, precision, tuning="default")
    ref = driver()
    assert ref.ctx.sizes()["pair_planes"] == 1
    want = ref.run_native(ref.native_state(), 3)
    # at init
    other = CPContext(make_system("w2", seed=3), "fp64")
    other.fault_inject(3)
    d = driver()
    assert d.ctx.sizes()["pair_planes"] == 0
    agree(d.run_native(d.native_state(), 3), want, s, precision)
    # at the first native call, between two passes of the force half
    d = driver()
    d.ctx.state_fft_fwd(d.psi)
    d.ctx.fault_inject(3)
    agree(d.run_native(d.native_state(), 3), want, s, precision)
    assert d.ctx.sizes()["pair_planes"] == 0
    # with a captured step in hand
    d = driver()
    st, sr = d.native_state(), ref.native_state()
    d.run_native(st, 3)
    assert d.ctx.sizes()["pair_planes"] == 1
    d.ctx.fault_inject(3)
    d.ctx.set_xc("blyp")
    ref.ctx.set_xc("blyp")
    assert d.ctx.sizes()["pair_planes"] == 0
    agree(d.run_native(st, 3), ref.run_native(sr, 3), s, precision)
