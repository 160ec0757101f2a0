"""Layer-0 buffers at any float alignment on the tensor-core forms: a view that starts between two 8-byte boundaries (two
shells, an even channel count) gives the caches and the steps of an aligned buffer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mma", [2, 4])
@pytest.mark.parametrize("cutoffs,C0", [((8.0, 6.0, 5.0), 38), ((7.5, 6.0, 4.2), 24)])
@pytest.mark.parametrize("off", [1, 2, 3])
def test_layer0_buffer_at_float_alignment(cuda, mma, cutoffs, C0, off):
    torch = cuda
    from neuralce_gb300.io import Z_OF, fcc_conventional
    from neuralce_gb300.nce import NCEModel, NCEState, synthetic_model
    from neuralce_gb300.workloads import A_FCC, cluster_space, random_occupancy
    cs = cluster_space(cutoffs)
    assert len(cs.orbits) + 1 == C0
    s = fcc_conventional(A_FCC, (4, 4, 4))
    s.numbers = np.full(len(s), Z_OF["Ni"], np.int64)
    P = synthetic_model(C0, 2, 32, 2, 1)
    m = NCEModel(cs, s, P, shell_edges=(0.0, 3.3, 4.2), act="silu", pool="sum", mma=mma)
    sig = random_occupancy(len(s), 0.5, 2, 3)
    a, b = NCEState(m, sig, np.full(2, 5.0)), NCEState(m, sig, np.full(2, 5.0))
    buf = torch.zeros(b.h0.numel() + 4, dtype=torch.float32, device="cuda")
    assert buf.data_ptr() % 16 == 0
    b.h0 = buf[off:off + b.h0.numel()].view(b.h0.shape)
    assert b.h0.data_ptr() % 16 == 4 * off and b.h0.is_contiguous()
    for st in (a, b):
        st.full_cache()
        st.run_chunk(12, 0, seed=4)
    torch.cuda.synchronize()
    m.check_errors()
    for f in ("sigma", "h0", "hmid", "e", "E", "n_acc"):
        assert torch.equal(getattr(a, f), getattr(b, f)), f
