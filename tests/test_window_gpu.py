"""The windowed sign-parity kernel against the step-by-step oracle: window and warp edges, tiny cells whose neighbourhood
entries alias, skewed cells, compositions with few or many evaluated swaps, ladders at which nearly every or nearly no
swap is accepted (predictions right and wrong), host streams that propose the same few sites again and again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cell(L, x, R, seed):
    from neuralce_gb300.ce import GPUClusterExpansion
    from neuralce_gb300.ce_tables import synthetic_eci
    from neuralce_gb300.io import Z_OF, fcc_conventional
    from neuralce_gb300.workloads import A_FCC, cluster_space, random_occupancy
    from oracle.ce_oracle import OracleCE
    s = fcc_conventional(A_FCC, L)
    s.numbers = np.full(len(s), Z_OF["Ni"], np.int64)
    cs = cluster_space()
    gce = GPUClusterExpansion((cs, synthetic_eci(cs, 3)), s, energy_scale=len(s))
    return gce, OracleCE(gce.info), random_occupancy(len(s), x, R, seed)


def _run(cuda, gce, orc, sig, beta, chunks, T, si, precision=64, props=None, near_eV=0.0, track=True):
    torch = cuda
    from neuralce_gb300.pt import PTState, run_chunk
    from oracle.ce_oracle import new_state
    R = len(sig)
    E0 = np.array([orc.energy(x) for x in sig])
    st = PTState(sig, E0, beta, np.zeros(R, np.int32))
    if track:
        st.track_counts(gce)
    ref = new_state(sig, E0, beta)
    for c in range(chunks):
        Es = torch.zeros((max(T // si, 1), R), dtype=torch.float64, device="cuda")
        Er = np.zeros((max(T // si, 1), R))
        p = None if props is None else tuple(x[c * T:(c + 1) * T] for x in props)
        pd = None if p is None else tuple(torch.as_tensor(np.ascontiguousarray(x)).cuda() for x in p)
        run_chunk(gce, st, T, c * T, 99, precision, 0, pd, si, Es if T >= si else None, True, near_eV=near_eV)
        orc.run(ref, T, c * T, 99, p, si, Er if T >= si else None, True, near_eV=near_eV or (1e-9 if precision == 64 else 1e-6))
        torch.cuda.synchronize()
        assert np.array_equal(st.n_near.cpu().numpy(), ref["n_near"])
        assert np.array_equal(st.sigma.cpu().numpy(), ref["sigma"])
        assert np.array_equal(st.n_acc.cpu().numpy(), ref["n_acc"])
        assert np.array_equal(st.rep_of_slot.cpu().numpy(), ref["rep_of_slot"])
        # carried energies: float64 rounding of sums below 1e4 eV, or 1e-6 eV a float32 swap
        tol = 1e-9 if precision == 64 else 1e-6 * max(1, int(ref["n_acc"].max()))
        assert np.abs(st.E.cpu().numpy() - ref["E"]).max() < tol
        if T >= si:
            assert np.abs(Es.cpu().numpy() - Er).max() < tol
        if track:
            assert torch.equal(st.cv, gce.cluster_counts(st.sigma))
    gce.check_errors()
    return st, ref


@pytest.mark.parametrize("L", [(3, 3, 3), (4, 4, 4), (5, 6, 7), (10, 4, 9), (8, 8, 8)])
@pytest.mark.parametrize("T,si", [(1, 1), (31, 1), (33, 3), (400, 7)])
def test_windows_match_oracle(cuda, L, T, si):
    from neuralce_gb300.workloads import ladder
    R = 5
    gce, orc, sig = _cell(L, 0.5, R, 11)
    _run(cuda, gce, orc, sig, ladder(R, 300.0, 1400.0)[1], 3, T, si)


@pytest.mark.parametrize("x", [0.01, 0.1, 0.9])
@pytest.mark.parametrize("precision", [64, 32])
def test_compositions(cuda, x, precision):
    from neuralce_gb300.workloads import ladder
    gce, orc, sig = _cell((5, 5, 6), x, 4, 5)
    _run(cuda, gce, orc, sig, ladder(4, 400.0, 1200.0)[1], 2, 700, 50, precision)


@pytest.mark.parametrize("precision", [64, 32])
def test_hot_and_cold(cuda, precision):
    """beta 0 (every swap accepted), nearly free, and frozen replicas side by side"""
    gce, orc, sig = _cell((5, 5, 5), 0.5, 4, 8)
    _run(cuda, gce, orc, sig, np.array([0.0, 1e-3, 5.0, 400.0], np.float32), 2, 600, 100, precision)


def test_repeated_sites(cuda):
    """A host stream over 40 sites of the cell: most windows hold steps that share a site with an earlier swap."""
    gce, orc, sig = _cell((5, 5, 5), 0.5, 3, 9)
    rng = np.random.default_rng(4)
    T, pool = 600, rng.permutation(sig.shape[1])[:40]
    a, b = (rng.choice(pool, (2 * T, 3)).astype(np.int32) for _ in range(2))
    _run(cuda, gce, orc, sig, np.array([2.0, 10.0, 30.0], np.float32), 2, T, 60, props=(a, b, 1.0 - rng.random((2 * T, 3))))


def test_wide_near_band(cuda):
    """A near-threshold band far above float32's error counts the same steps as the oracle's definition."""
    from neuralce_gb300.workloads import ladder
    gce, orc, sig = _cell((5, 5, 5), 0.5, 3, 13)
    st, ref = _run(cuda, gce, orc, sig, ladder(3, 500.0, 1400.0)[1], 2, 500, 100, near_eV=0.02)
    assert int(ref["n_near"].sum()) > 20
