"""The step-by-step sign-parity kernel's launch shapes on the sets that stay with it (several basis sites, five-member clusters):
over thread-block clusters and in batches, in both precisions.  (Sets that have window tables ignore these shapes.)"""
import ctypes as C

import numpy as np
import pytest

from tests.test_chunk_kernel_gpu import _fcc, _job, _state

pytestmark = pytest.mark.gpu


def _equal(torch, a, b):
    for f in ("sigma", "E", "n_acc", "n_near", "rep_of_slot", "E_min_rep", "cv"):
        assert torch.equal(getattr(a, f), getattr(b, f)), f


@pytest.mark.parametrize("kind,L", [("b2", 4), ("b2", 7), ("rocksalt", 5), ("five members", 4)])
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("cluster", [2, 4, 8, 16])
def test_step_kernel_cluster_equals_single_cta(cuda, kind, L, precision, cluster):
    torch = cuda
    from neuralce_gb300.pt import chunk_kernel, run_chunk
    from oracle.ce_oracle import OracleCE, new_state
    gce, sig = _job(kind, L, 3, 11)
    a, b = _state(cuda, gce, sig), _state(cuda, gce, sig)
    assert chunk_kernel([gce], [a], precision)[0] == "sign parity"
    E0 = a.E.cpu().numpy()
    ref, orc = new_state(sig, E0, a.beta_slot.cpu().numpy()), OracleCE(gce.info)
    T = 400
    for c in range(2):
        Ea = torch.zeros((T // 10, 3), dtype=torch.float64, device="cuda"); Eb = torch.zeros_like(Ea)
        run_chunk(gce, a, T, c * T, 31, precision, 8, None, 10, Ea, True)
        run_chunk(gce, b, T, c * T, 31, precision, 8, None, 10, Eb, True, cluster=cluster)
        orc.run(ref, T, c * T, 31, None, 10, None, True, near_eV=1e-9 if precision == 64 else 1e-6)
        torch.cuda.synchronize()
        _equal(torch, a, b)
        assert torch.equal(Ea, Eb)
    assert np.array_equal(b.sigma.cpu().numpy(), ref["sigma"]) and np.array_equal(b.n_acc.cpu().numpy(), ref["n_acc"])
    assert np.abs(b.E.cpu().numpy() - ref["E"]).max() < (1e-9 if precision == 64 else 1e-6 * int(ref["n_acc"].max()))
    assert torch.equal(b.cv, gce.cluster_counts(b.sigma)) and int(ref["n_acc"].sum()) > 0


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("warps,cluster", [(4, 1), (8, 2), (8, 8)])
@pytest.mark.parametrize("kind,cutoffs", [("b2", (6.0, 4.2)), ("rocksalt", (6.0,))])
def test_step_kernel_batch_equals_alone(cuda, precision, warps, cluster, kind, cutoffs):
    """two-sublattice jobs and a one-sublattice job (of the same cluster order) that alone would run in windows, all step by
    step in one launch"""
    torch = cuda
    from neuralce_gb300 import _lib
    from neuralce_gb300.pt import chunk_kernel, make_chunk, run_chunk
    jobs = [_job(kind, 4, 3, 5), _job(kind, 6, 2, 6), _fcc(cutoffs, (4, 5, 6), 4, 7)]
    T = 300
    alone, sts = [_state(cuda, g, s) for g, s in jobs], [_state(cuda, g, s) for g, s in jobs]
    for k, (g, _) in enumerate(jobs):
        run_chunk(g, alone[k], T, 0, 7 + k, precision, warps, None, 1, None, True)
    assert chunk_kernel([jobs[2][0]], alone[2:], precision)[0] == "windowed"
    assert chunk_kernel([g for g, _ in jobs], sts, precision)[0] == "sign parity"
    hs = (C.c_void_p * 3)(*[g.handle.value for g, _ in jobs])
    ss = (_lib.NcePtState * 3)(*[s.struct() for s in sts])
    cks = (_lib.NcePtChunk * 3)(*[make_chunk(T, 0, 7 + k, precision, warps, None, 1, None, True, cluster=cluster) for k in range(3)])
    _lib.check(_lib.lib().nce_ce_run_batch(3, hs, ss, cks, _lib.stream_ptr()), "batch")
    torch.cuda.synchronize()
    for a, b in zip(alone, sts):
        _equal(torch, a, b)


@pytest.mark.parametrize("cluster", [1, 4])
def test_step_kernel_fp32_per_swap_error(cuda, cluster):
    """float32 dE of single accepted swaps within 1e-6 eV of the oracle's, in the five-member set"""
    torch = cuda
    from neuralce_gb300.pt import PTState, chunk_kernel, run_chunk
    from oracle.ce_oracle import OracleCE
    gce, sig = _job("five members", 4, 1, 13)
    orc, rng = OracleCE(gce.info), np.random.default_rng(4)
    worst = n = 0
    while n < 40:
        ia, ib = (int(x) for x in rng.integers(0, sig.shape[1], 2))
        if sig[0, ia] == sig[0, ib]:
            continue
        st = PTState(sig, np.zeros(1), np.zeros(1, np.float32), np.zeros(1, np.int32))   # beta 0: accepted
        assert chunk_kernel([gce], [st], 32)[0] == "sign parity"
        p = tuple(torch.as_tensor(x).cuda() for x in (np.array([[ia]], np.int32), np.array([[ib]], np.int32), np.array([[0.5]])))
        run_chunk(gce, st, 1, 0, 1, 32, 8, p, cluster=cluster)
        worst = max(worst, abs(float(st.E.item()) - orc.delta(sig[0], ia, ib, sig[0, ib], sig[0, ia])))
        n += 1
    assert worst < 1e-6
