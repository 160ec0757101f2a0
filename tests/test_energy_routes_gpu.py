"""The full energy's two kernels on the sets and cells at either side of their rule: pairs only (every member fetched), the same
with triplets and quadruplets (words shared on chip), several and few blocks an SM.  Cluster-vector sums against the template rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cutoffs", [(8.0,), (12.0,), (12.0, 6.0), (12.0, 6.0, 5.0), (13.0, 6.0, 5.0), (14.5,), (14.5, 6.0, 5.0)])
@pytest.mark.parametrize("L,R", [((4, 4, 4), 3), ((8, 8, 8), 9), ((16, 16, 16), 4), ((32, 32, 32), 5)])
def test_counts(cuda, cutoffs, L, R):
    torch = cuda
    from test_energy_bits_gpu import _counts
    from neuralce_gb300.ce import GPUClusterExpansion
    from neuralce_gb300.ce_tables import synthetic_eci
    from neuralce_gb300.io import Z_OF, fcc_conventional
    from neuralce_gb300.workloads import A_FCC, cluster_space, random_occupancy
    cs = cluster_space(cutoffs)
    s = fcc_conventional(A_FCC, L)
    s.numbers = np.full(len(s), Z_OF["Ni"], np.int64)
    gce = GPUClusterExpansion((cs, synthetic_eci(cs, 2)), s, energy_scale=len(s))
    dev = torch.as_tensor(random_occupancy(len(s), 0.4, R, 6)).cuda()
    tb = dict(gce.info, counts=[len(o.clusters) for o in cs.orbits])
    cv = gce.cluster_counts(dev)
    assert torch.equal(cv[:, :-1], _counts(torch, tb, dev)[:, :-1]) and not cv[:, -1].any()
