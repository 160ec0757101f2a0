"""The bit-sliced full energy over its launch forms: one and two words a thread, rows split into slices, planes packed four
sites a lane (rows of whole words) or bit by bit, an unaligned occupancy buffer.  Cluster-vector sums against a float64 sum
over the template rows (exact integers) and energies against the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _counts(torch, tb, sig):
    """(R, n_cols) from the template rows: products of point-function signs, site by site, on the device"""
    d, nB = [int(x) for x in tb["d"]], int(tb["nB"])
    assert nB == 1
    R, N = sig.shape
    k = torch.arange(N, device="cuda")
    k = torch.stack([k // (d[1] * d[2]), k // d[2] % d[1], k % d[2]], 1)
    dd = torch.tensor(d, device="cuda")
    spin = (2 * sig.to(torch.int8) - 1)                       # theta(2, 0, s) = -cos(pi s)
    out = torch.zeros((R, tb["n_cols"]), dtype=torch.int64, device="cuda")
    cols = np.repeat(np.arange(len(tb["counts"])), tb["counts"])
    cache = {}
    for row in range(tb["Rt"]):
        p = None
        for m in range(tb["mo"]):
            if not tb["T_msk"][row, m]:
                continue
            key = tuple(int(v) for v in tb["T_uo"][row, m])
            if key not in cache:
                q = (k + torch.tensor(key, device="cuda")) % dd
                cache[key] = spin[:, (q[:, 0] * d[1] + q[:, 1]) * d[2] + q[:, 2]]
            p = cache[key] if p is None else p * cache[key]
        out[:, cols[row]] += p.sum(1, dtype=torch.int64)
    return out


@pytest.mark.parametrize("L,R", [((2, 2, 2), 3), ((3, 3, 3), 2), ((5, 6, 7), 5), ((8, 8, 8), 33), ((16, 16, 16), 1), ((16, 16, 16), 40),
                                 ((10, 4, 9), 65), ((20, 20, 20), 12), ((32, 32, 32), 6)])
@pytest.mark.parametrize("shift", [0, 1])
def test_counts_and_energies(cuda, L, R, shift):
    torch = cuda
    from neuralce_gb300.ce import GPUClusterExpansion
    from neuralce_gb300.ce_tables import synthetic_eci
    from neuralce_gb300.io import Z_OF, fcc_conventional
    from neuralce_gb300.workloads import A_FCC, cluster_space, random_occupancy
    from oracle.ce_oracle import OracleCE
    s = fcc_conventional(A_FCC, L)
    s.numbers = np.full(len(s), Z_OF["Ni"], np.int64)
    cs = cluster_space()
    gce = GPUClusterExpansion((cs, synthetic_eci(cs, 2)), s, energy_scale=len(s))
    sig = random_occupancy(len(s), 0.4, R, 6)
    buf = torch.zeros(sig.size + 8, dtype=torch.int8, device="cuda")
    dev = buf[shift:shift + sig.size].view(R, -1)             # shift 1: not aligned to four bytes
    dev.copy_(torch.as_tensor(sig))
    tb = dict(gce.info, counts=[len(o.clusters) for o in cs.orbits])
    cv = gce.cluster_counts(dev)
    assert torch.equal(cv[:, :-1], _counts(torch, tb, dev)[:, :-1]) and not cv[:, -1].any()
    E = gce.batched_energy(dev).cpu().numpy()
    orc = OracleCE(gce.info)
    for r in range(min(R, 2)):
        e = orc.energy(sig[r])
        assert abs(E[r] - e) < 1e-10 * max(1.0, abs(e))
