"""Bit-sliced kernels on cluster sets beyond the usual one: five-member clusters (more members a row) and a column of 384
rows a site (counts past one byte).  Cluster-vector sums and layer 0 against the template rows and the float64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _space(kind):
    from neuralce_gb300.ce_tables import ClusterSpace
    from neuralce_gb300.io import fcc_primitive
    from neuralce_gb300.workloads import A_FCC, cluster_space
    if kind == "five members":
        return ClusterSpace.build(fcc_primitive(A_FCC), [4.2, 4.2, 4.2, 4.2])
    import copy
    cs = copy.deepcopy(cluster_space())
    big = [k for k, o in enumerate(cs.orbits) if len(o.clusters) == 48 and o.order == 4]
    cs.orbits[big[0]].clusters = cs.orbits[big[0]].clusters + cs.orbits[big[1]].clusters
    del cs.orbits[big[1]]
    return cs


@pytest.mark.parametrize("kind", ["five members", "wide column"])
@pytest.mark.parametrize("L,R", [((4, 4, 4), 3), ((16, 16, 16), 2)])
def test_counts_and_layer0(cuda, kind, L, R):
    torch = cuda
    from test_energy_bits_gpu import _counts
    from neuralce_gb300.ce import GPUClusterExpansion
    from neuralce_gb300.ce_tables import synthetic_eci
    from neuralce_gb300.io import Z_OF, fcc_conventional
    from neuralce_gb300.nce import NCEModel, NCEState, synthetic_model
    from neuralce_gb300.workloads import A_FCC, random_occupancy
    from oracle.nce_oracle import NCEOracle
    cs = _space(kind)
    assert max(len(o.clusters[0]) for o in cs.orbits) == (5 if kind == "five members" else 4)
    s = fcc_conventional(A_FCC, L)
    s.numbers = np.full(len(s), Z_OF["Ni"], np.int64)
    gce = GPUClusterExpansion((cs, synthetic_eci(cs, 1)), s, energy_scale=len(s))
    sig = random_occupancy(len(s), 0.45, R, 2)
    dev = torch.as_tensor(sig).cuda()
    tb = dict(gce.info, counts=[len(o.clusters) for o in cs.orbits])
    assert torch.equal(gce.cluster_counts(dev)[:, :-1], _counts(torch, tb, dev)[:, :-1])
    P = synthetic_model(len(cs.orbits) + 1, 1, 16, 1, 0)
    m = NCEModel(cs, s, P, shell_edges=(0.0, 3.3), act="silu", pool="sum")
    st = NCEState(m, sig, np.ones(R)).full_cache()
    h0 = NCEOracle(m.geo, P, act="silu", pool="sum").h0s(sig[0].astype(np.int64))
    assert np.abs(st.h0[0].cpu().numpy() - h0).max() < 2e-5         # float32 of sums of at most a few units


@pytest.mark.parametrize("kind", ["five members", "wide column"])
def test_trajectory(cuda, kind):
    """the first set runs step by step, the second in windows"""
    torch = cuda
    from neuralce_gb300.ce import GPUClusterExpansion
    from neuralce_gb300.ce_tables import synthetic_eci
    from neuralce_gb300.io import Z_OF, fcc_conventional
    from neuralce_gb300.pt import PTState, run_chunk
    from neuralce_gb300.workloads import A_FCC, ladder, random_occupancy
    from oracle.ce_oracle import OracleCE, new_state
    cs = _space(kind)
    s = fcc_conventional(A_FCC, (5, 5, 5))
    s.numbers = np.full(len(s), Z_OF["Ni"], np.int64)
    gce = GPUClusterExpansion((cs, synthetic_eci(cs, 1)), s, energy_scale=len(s))
    orc = OracleCE(gce.info)
    sig = random_occupancy(len(s), 0.5, 3, 4)
    _, beta = ladder(3)
    E0 = np.array([orc.energy(x) for x in sig])
    st, ref = PTState(sig, E0, beta, np.zeros(3, np.int32)), new_state(sig, E0, beta)
    run_chunk(gce, st, 300, 0, 5, do_exchange=True)
    orc.run(ref, 300, 0, 5, None, 1, None, True, near_eV=1e-9)
    torch.cuda.synchronize()
    assert np.array_equal(st.sigma.cpu().numpy(), ref["sigma"]) and np.array_equal(st.n_acc.cpu().numpy(), ref["n_acc"])
    assert np.abs(st.E.cpu().numpy() - ref["E"]).max() < 1e-9
