"""Batching form (oa_gpu_cp_run_batch): several independent systems of
different sizes advanced together, one CUDA graph per step with the systems
on concurrent streams.  Each system's energies and coefficients match its
own single-system run (oa_gpu_cp_run) bit for bit."""
import numpy as np
import pytest

from openatom_b200.system import make_system

pytestmark = pytest.mark.gpu

# (preset, states, seed): uneven sizes and grids (the whole step is one graph
# per system: up to 48 states, or an even number up to 128)
SYSTEMS = [("w2", None, 21), ("w2", 6, 22), ("w4", 12, 23), ("w8", 16, 24)]
ODD = [("w2", 1, 26), ("w2", 5, 27), ("w4", 31, 28), ("w4", 47, 29), ("w4", 50, 30)]


@pytest.mark.parametrize("systems", [SYSTEMS, ODD])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_batch_matches_single_runs(precision, systems):
    from openatom_b200.gpu import CPDriver, run_batch
    nsteps = 4
    syss = [make_system(p, nstate=n, seed=sd, dt=0.5) for p, n, sd in systems]
    single = [CPDriver(s, precision) for s in syss]
    ref = []
    for d in single:
        st = d.native_state(use_graph=True)
        ref.append(d.run_native(st, nsteps))
    batch = [CPDriver(s, precision) for s in syss]
    states = [d.native_state(use_graph=True) for d in batch]
    got = run_batch(batch, states, nsteps)
    for i in range(len(syss)):
        for k in range(nsteps):
            for key in ("EKE", "EHART", "EEXT", "EEXC", "ENL", "FICT_KE", "SMAX"):
                assert got[i][k][key] == ref[i][k][key], (i, k, key, got[i][k][key], ref[i][k][key])
        assert np.array_equal(batch[i].psi.cpu().numpy(), single[i].psi.cpu().numpy())
        assert np.array_equal(batch[i].v.cpu().numpy(), single[i].v.cpu().numpy())
    # one graph per steady step holds the kernels of every system
    assert states[0].last_kernels > 4 * 20


def test_batch_rejects_bad_input():
    """A context that appears twice is refused before anything runs."""
    import torch
    from openatom_b200.gpu import CPDriver, run_batch, OaError
    s = make_system("w2", seed=25, dt=0.5)
    d = CPDriver(s, "fp64")
    st = d.native_state()
    with pytest.raises(OaError):
        run_batch([d, d], [st, d.native_state()], 2)


def test_batch_refuses_counts_it_cannot_capture():
    from openatom_b200.gpu import CPDriver, run_batch, OaError, OA_ERR_UNSUPPORTED
    d = CPDriver(make_system("w2", nstate=49, seed=25, dt=0.5), "fp64")
    with pytest.raises(OaError) as ei:
        run_batch([d], [d.native_state()], 2)
    assert ei.value.status == OA_ERR_UNSUPPORTED


@pytest.mark.parametrize("nstate", [5, 8, 47, 49])
def test_graphed_step_follows_the_newton_schulz_limits(nstate):
    """A captured step is made again when the tolerance or the iteration
    limit of the next call differs: the same bits as steps run eagerly."""
    from openatom_b200.gpu import CPDriver, OaError, OA_ERR_NOT_CONVERGED
    s = make_system("w2", nstate=nstate, seed=31, dt=0.5)
    out = []
    for graph in (True, False):
        d = CPDriver(s, "fp64")
        st = d.native_state(use_graph=graph)
        recs = d.run_native(st, 3)
        st.ns_tol = 1e-3
        recs += d.run_native(st, 2)
        assert recs[-1]["ORTHO_ITERS"] < recs[2]["ORTHO_ITERS"]
        st.ns_tol, st.ns_max_iter = 1e-15, 1
        with pytest.raises(OaError) as ei:
            d.run_native(st, 1)
        assert ei.value.status == OA_ERR_NOT_CONVERGED
        out.append((recs, d.psi.cpu().numpy()))
    for g, r in zip(out[0][0], out[1][0]):
        assert g == r
    assert np.array_equal(out[0][1], out[1][1])
