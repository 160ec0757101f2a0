"""The chunk-end exchange takes a lane per pair of slots: ladders around the edges of a warp of pairs, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("R", [2, 3, 64, 65, 66, 131])
def test_exchange_matches_oracle(cuda, R, fused):
    torch = cuda
    from neuralce_gb300.pt import PTState, run_chunk
    from neuralce_gb300.workloads import ce_config, ladder, replica_configs
    from oracle.ce_oracle import OracleCE, new_state
    gce, sig = ce_config(3, seed=1)
    orc = OracleCE(gce.info)
    sig_r = replica_configs(sig, R, 7)
    _, beta = ladder(R, 900.0, 1400.0)                       # close temperatures: many accepted exchanges
    lid = (np.arange(R) * 2 // (R + 1)).astype(np.int32)     # two ladders: the pair across them never exchanges
    E0 = np.array([orc.energy(x) for x in sig_r])
    st = PTState(sig_r, E0, beta, lid)
    if not fused:
        st.ex_sync = None
    ref = new_state(sig_r, E0, beta, lid)
    for c in range(3):
        Es = torch.zeros((2, R), dtype=torch.float64, device="cuda")
        run_chunk(gce, st, 20, c * 20, 31, 64, 4, None, 10, Es, True)
        Er = np.zeros((2, R))
        orc.run(ref, 20, c * 20, 31, None, 10, Er, True)
        torch.cuda.synchronize()
        assert np.array_equal(st.rep_of_slot.cpu().numpy(), ref["rep_of_slot"])
        assert np.array_equal(st.slot_of_rep.cpu().numpy()[ref["rep_of_slot"]], np.arange(R))
        assert np.array_equal(st.sigma.cpu().numpy(), ref["sigma"])
        assert np.abs(Es.cpu().numpy() - Er).max() < 1e-9
    assert int(st.n_ex.item()) == int(np.asarray(ref["n_ex"]).reshape(-1)[0])
    assert R < 64 or int(st.n_ex.item()) > 0
