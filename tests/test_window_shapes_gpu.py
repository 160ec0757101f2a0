"""Launch shapes of the windowed kernel: a job in a launch of more replicas than SMs (two CTAs an SM) and of more than two an SM
(256 threads) equals the job alone, bit for bit, in both precisions; the ladder that fills such a launch equals the oracle."""
import ctypes as C

import numpy as np
import pytest

from tests.test_chunk_kernel_gpu import _fcc, _state
from tests.test_step_kernel_gpu import _equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cutoffs", [(8.0, 6.0, 5.0), (6.0,)])
@pytest.mark.parametrize("per_sm", [1, 2, 3])
@pytest.mark.parametrize("precision", [64, 32])
def test_shared_launch_equals_alone(cuda, cutoffs, per_sm, precision):
    torch = cuda
    from neuralce_gb300 import _lib
    from neuralce_gb300.pt import chunk_kernel, make_chunk, run_chunk
    from oracle.ce_oracle import OracleCE, new_state
    n_sm = torch.cuda.get_device_properties(0).multi_processor_count
    jobs = [_fcc(cutoffs, (5, 5, 6), 20, 2), _fcc(cutoffs, (3, 3, 3), per_sm * n_sm + 5, 3), _fcc(cutoffs, (9, 8, 7), 7, 4)]
    alone, sts = [_state(cuda, g, s) for g, s in jobs], [_state(cuda, g, s) for g, s in jobs]
    T, si = 90, 7
    for j in (0, 2):
        assert chunk_kernel([jobs[j][0]], [alone[j]], precision) == ("windowed", 512)
    assert chunk_kernel([g for g, _ in jobs], sts, precision) == ("windowed", 512 if per_sm == 1 else 256)
    hs = (C.c_void_p * 3)(*[g.handle.value for g, _ in jobs])
    for c in range(2):
        Es = [[torch.zeros((T // si, len(s)), dtype=torch.float64, device="cuda") for _, s in jobs] for _ in range(2)]
        for j in (0, 2):
            run_chunk(jobs[j][0], alone[j], T, c * T, 7 + j, precision, 0, None, si, Es[0][j], True)
        ss = (_lib.NcePtState * 3)(*[s.struct() for s in sts])
        cks = (_lib.NcePtChunk * 3)(*[make_chunk(T, c * T, 7 + j, precision, 0, None, si, Es[1][j], True) for j in range(3)])
        _lib.check(_lib.lib().nce_ce_run_batch(3, hs, ss, cks, _lib.stream_ptr()), "batch")
        torch.cuda.synchronize()
        for j in (0, 2):
            _equal(torch, alone[j], sts[j])
            assert torch.equal(Es[0][j], Es[1][j])
    if precision == 64:                                       # (float32 decisions may differ from float64's near a threshold)
        gce, sig = jobs[1]
        ref = new_state(sig, alone[1].E.cpu().numpy(), alone[1].beta_slot.cpu().numpy())
        orc = OracleCE(gce.info)
        for c in range(2):
            orc.run(ref, T, c * T, 8, None, si, None, True, n_threads=8, near_eV=1e-9)
        assert np.array_equal(sts[1].sigma.cpu().numpy(), ref["sigma"]) and np.array_equal(sts[1].n_acc.cpu().numpy(), ref["n_acc"])
        assert np.array_equal(sts[1].rep_of_slot.cpu().numpy(), ref["rep_of_slot"])
        assert np.abs(sts[1].E.cpu().numpy() - ref["E"]).max() < 1e-9
    for (g, _), st in zip(jobs, sts):
        assert torch.equal(st.cv, g.cluster_counts(st.sigma))
