"""Full NeuralCE caches of many replicas: tiles run across replica boundaries, so a batch equals its replicas one by one
(bit for bit), on cells whose sites do not fill a tile, in every contraction form, and the first replica the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [(3, 3, 3), (3, 4, 5), (2, 2, 17)])
@pytest.mark.parametrize("width,mma", [(16, 0), (64, 0), (128, 0), (32, 2), (64, 4), (128, 4)])
def test_batch_of_caches_equals_single(cuda, L, width, mma):
    torch = cuda
    from neuralce_gb300.io import Z_OF, fcc_conventional
    from neuralce_gb300.nce import NCEModel, NCEState, synthetic_model
    from neuralce_gb300.workloads import A_FCC, cluster_space, random_occupancy
    from oracle.nce_oracle import NCEOracle
    s = fcc_conventional(A_FCC, L)
    s.numbers = np.full(len(s), Z_OF["Ni"], np.int64)
    cs = cluster_space()
    P = synthetic_model(len(cs.orbits) + 1, 2, width, 1, 1)
    m = NCEModel(cs, s, P, shell_edges=(0.0, 3.3), act="silu", pool="sum", mma=mma)
    R = 5
    sig = random_occupancy(len(s), 0.4, R, 3)
    a = NCEState(m, sig, np.ones(R)).full_cache()
    for r in range(R):
        b = NCEState(m, sig[r:r + 1], np.ones(1)).full_cache()
        assert torch.equal(a.h0[r], b.h0[0]) and torch.equal(a.e[r], b.e[0]) and torch.equal(a.E[r], b.E[0])
        assert torch.equal(a.hmid[:, r], b.hmid[:, 0])
    c = NCEOracle(m.geo, P, act="silu", pool="sum").full_cache(sig[0].astype(np.int64))
    # per-site energies: 1e-4 eV, the bound of the float32 and split forms; 2e-2 for plain bf16 operands
    assert np.abs(a.e[0].cpu().numpy() - np.asarray(c["e"])).max() < (2e-2 if mma == 2 else 1e-4)
    m.check_errors()


@pytest.mark.parametrize("mma", [2, 4])
def test_layer0_buffer_aligned_to_eight_bytes(cuda, mma):
    """24 layer-0 channels (rows a multiple of four floats) in a buffer that starts between two 16-byte boundaries: caches and
    steps equal those of an aligned buffer."""
    torch = cuda
    from neuralce_gb300.io import Z_OF, fcc_conventional
    from neuralce_gb300.nce import NCEModel, NCEState, synthetic_model
    from neuralce_gb300.workloads import A_FCC, cluster_space, random_occupancy
    cs = cluster_space((7.5, 6.0, 4.2))
    assert (len(cs.orbits) + 1) % 4 == 0
    s = fcc_conventional(A_FCC, (4, 4, 4))
    s.numbers = np.full(len(s), Z_OF["Ni"], np.int64)
    P = synthetic_model(len(cs.orbits) + 1, 2, 32, 1, 1)
    m = NCEModel(cs, s, P, shell_edges=(0.0, 3.3), act="silu", pool="sum", mma=mma)
    sig = random_occupancy(len(s), 0.5, 2, 3)
    a, b = NCEState(m, sig, np.full(2, 5.0)), NCEState(m, sig, np.full(2, 5.0))
    buf = torch.zeros(b.h0.numel() + 2, dtype=torch.float32, device="cuda")
    b.h0 = buf[2:].view(b.h0.shape)
    assert b.h0.data_ptr() % 16 == 8
    for st in (a, b):
        st.full_cache()
        st.run_chunk(12, 0, seed=4)
    torch.cuda.synchronize()
    for f in ("sigma", "h0", "hmid", "e", "E", "n_acc"):
        assert torch.equal(getattr(a, f), getattr(b, f)), f
