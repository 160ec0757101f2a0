"""Layer 0 of the full caches by its two bit-sliced kernels: sets at either side of their rule (few and many rows a word, narrow and
wide neighbourhoods) and one of more than 700 distinct member words, against the float64 oracle."""
import copy

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _space(kind):
    from neuralce_gb300.workloads import cluster_space
    if kind != "merged":
        return cluster_space(kind)
    cs = copy.deepcopy(cluster_space((14.5,)))                # pairs to 14.5 A in three columns: few channels, 887 words
    pairs = [o for o in cs.orbits if o.order == 2]
    for k, o in enumerate(pairs):
        if k >= 3:
            pairs[k % 3].clusters = pairs[k % 3].clusters + o.clusters
            cs.orbits.remove(o)
    return cs


@pytest.mark.parametrize("kind", [(10.0,), (11.0,), (11.0, 6.0, 5.0), (12.0, 6.0), (13.0,), "merged"])
@pytest.mark.parametrize("L,R", [((4, 4, 4), 3), ((9, 10, 11), 2), ((16, 16, 16), 2)])
def test_layer0(cuda, kind, L, R):
    from neuralce_gb300.io import Z_OF, fcc_conventional
    from neuralce_gb300.nce import NCEModel, NCEState, synthetic_model
    from neuralce_gb300.workloads import A_FCC, random_occupancy
    from oracle.nce_oracle import NCEOracle
    cs = _space(kind)
    s = fcc_conventional(A_FCC, L)
    s.numbers = np.full(len(s), Z_OF["Ni"], np.int64)
    P = synthetic_model(len(cs.orbits) + 1, 0, 16, 1, 0)
    m = NCEModel(cs, s, P, shell_edges=(0.0, 3.3), act="silu", pool="sum")
    if kind == "merged":
        assert m.geo["J"] == 887 and m.C0 == 5
    sig = random_occupancy(len(s), 0.45, R, 2)
    st = NCEState(m, sig, np.ones(R)).full_cache()
    orc = NCEOracle(m.geo, P, act="silu", pool="sum")
    for r in range(R):
        h0 = orc.h0s(sig[r].astype(np.int64))
        # a float32 rounding of sums of at most a few units
        assert np.abs(st.h0[r].cpu().numpy() - h0).max() < 2e-5
