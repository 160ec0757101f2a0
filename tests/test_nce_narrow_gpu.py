"""Layer-0 inputs of 21 to 32 channels over several shells (a gather of its own), in the float32 and mma.sync forms: full caches
and a forced-move chain against the oracle, on tiles that a cell's sites fill unevenly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edges", [(0.0, 3.3, 4.2), (0.0, 3.3, 4.2, 5.0)])
@pytest.mark.parametrize("width,mma", [(16, 0), (64, 0), (128, 0), (64, 1), (64, 3)])
def test_narrow_inputs(cuda, edges, width, mma):
    torch = cuda
    from neuralce_gb300.io import Z_OF, fcc_conventional
    from neuralce_gb300.nce import NCEModel, NCEState, synthetic_model
    from neuralce_gb300.workloads import A_FCC, cluster_space, random_occupancy
    from oracle.nce_oracle import NCEOracle, run_chain
    cs = cluster_space((7.5, 6.0, 4.2))
    assert len(cs.orbits) + 1 == 24
    s = fcc_conventional(A_FCC, (3, 4, 5))
    s.numbers = np.full(len(s), Z_OF["Ni"], np.int64)
    P = synthetic_model(24, 2, width, len(edges) - 1, 1)
    m = NCEModel(cs, s, P, shell_edges=edges, act="silu", pool="sum", mma=mma)
    orc = NCEOracle(m.geo, P, act="silu", pool="sum")
    sig = random_occupancy(len(s), 0.4, 2, 3)
    st = NCEState(m, sig, np.ones(2)).full_cache()
    c = orc.full_cache(sig[0].astype(np.int64))
    # 1e-4 eV for the float32 and split forms, 2e-2 for plain bf16 operands: the bounds of the other cache tests
    assert np.abs(st.e[0].cpu().numpy() - np.asarray(c["e"])).max() < (2e-2 if mma == 1 else 1e-4)
    T = 6
    rng = np.random.default_rng(8)
    pi, pj = rng.integers(0, m.N, T).astype(np.int32), rng.integers(0, m.N, T).astype(np.int32)
    one = NCEState(m, sig[:1], np.ones(1)).full_cache()
    dE = torch.zeros((T, 1), dtype=torch.float64, device="cuda")
    one.run_chunk(T, 0, proposals=tuple(torch.as_tensor(x.reshape(T, 1)).cuda() for x in (pi, pj, np.full(T, 0.5))), dE_out=dE, force=1)
    torch.cuda.synchronize()
    m.check_errors()
    _, sig_ref, _, _, dEs, _ = run_chain(orc, c, sig[0].astype(np.int64), pi, pj, np.full(T, 0.5), 0.0, m.scale_eV)
    assert np.abs((dE.cpu().numpy()[:, 0] - dEs) * m.scale_eV).max() < (1e-2 if mma == 1 else 1e-4)
    assert np.array_equal(one.sigma[0].cpu().numpy(), sig_ref.astype(np.int8))
