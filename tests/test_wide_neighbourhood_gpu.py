"""Cluster sets whose neighbourhoods exceed what the full-energy kernel keeps on chip (more than about 1,400 sites): counts, energies,
tracked sums and the sign-parity and local-field chunks run as for any other set."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cutoffs,L,n_nbr", [((17.5, 4.2), (10, 10, 10), 1481), ((18.0, 4.2), (9, 10, 11), 1601)])
def test_wide_neighbourhood(cuda, cutoffs, L, n_nbr):
    torch = cuda
    from test_energy_bits_gpu import _counts
    from neuralce_gb300.ce import GPUClusterExpansion
    from neuralce_gb300.ce_tables import synthetic_eci
    from neuralce_gb300.io import Z_OF, fcc_conventional
    from neuralce_gb300.pt import PTState, run_chunk
    from neuralce_gb300.workloads import A_FCC, cluster_space, ladder, random_occupancy
    from oracle.ce_oracle import OracleCE, new_state
    cs = cluster_space(cutoffs)
    s = fcc_conventional(A_FCC, L)
    s.numbers = np.full(len(s), Z_OF["Ni"], np.int64)
    gce = GPUClusterExpansion((cs, synthetic_eci(cs, 1)), s, energy_scale=len(s))
    assert gce.info["n_nbr"] == n_nbr
    R, T = 3, 120
    sig = random_occupancy(len(s), 0.4, R, 2)
    dev = torch.as_tensor(sig).cuda()
    tb = dict(gce.info, counts=[len(o.clusters) for o in cs.orbits])
    want = _counts(torch, tb, dev)
    assert torch.equal(gce.cluster_counts(dev)[:, :-1], want[:, :-1])
    orc = OracleCE(gce.info)
    E0 = np.array([orc.energy(x) for x in sig])
    E = gce.batched_energy(dev).cpu().numpy()
    assert np.abs(E - E0).max() < 1e-10 * max(1.0, np.abs(E0).max())
    assert torch.equal(gce.energy_from_counts(gce.cluster_counts(dev)).cpu(), torch.as_tensor(E))
    _, beta = ladder(R)
    for path in (0, 2) + ((3,) if gce.has_local_field else ()):
        st, ref = PTState(sig, E0, beta, np.zeros(R, np.int32)), new_state(sig, E0, beta)
        st.track_counts(gce)
        if path == 3:
            st.enable_field(gce)
        run_chunk(gce, st, T, 0, 5, do_exchange=True, path=path)
        orc.run(ref, T, 0, 5, None, 1, None, True, near_eV=1e-9)
        torch.cuda.synchronize()
        assert np.array_equal(st.sigma.cpu().numpy(), ref["sigma"]) and np.array_equal(st.n_acc.cpu().numpy(), ref["n_acc"])
        assert np.abs(st.E.cpu().numpy() - ref["E"]).max() < 1e-9
        assert torch.equal(st.cv, gce.cluster_counts(st.sigma))
    gce.check_errors()
