"""Which kernel a chunk takes (nce_ce_chunk_kernel), and what the tuners and split batches make of it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fcc(cutoffs, L, R, seed):
    from neuralce_gb300.ce import GPUClusterExpansion
    from neuralce_gb300.ce_tables import synthetic_eci
    from neuralce_gb300.io import Z_OF, fcc_conventional
    from neuralce_gb300.workloads import A_FCC, cluster_space, random_occupancy
    s = fcc_conventional(A_FCC, L)
    s.numbers = np.full(len(s), Z_OF["Ni"], np.int64)
    cs = cluster_space(cutoffs)
    return GPUClusterExpansion((cs, synthetic_eci(cs, 3)), s, energy_scale=len(s)), random_occupancy(len(s), 0.5, R, seed)


def _job(kind, L, R, seed):
    """(gce, occupancies) of a set without window tables"""
    if kind == "five members":
        return _fcc((4.2, 4.2, 4.2, 4.2), (L, L, L), R, seed)
    from neuralce_gb300.ce import GPUClusterExpansion
    from tests.test_multisublattice import _system
    cs, params, s = _system(kind, L, seed)
    gce = GPUClusterExpansion((cs, params), s)
    sig, sl, rng = gce.encode(s), gce.info["site_to_sl"], np.random.default_rng(seed)
    out = np.stack([sig] * R).astype(np.int8)
    for r in range(R):
        for k in np.unique(sl):
            i = np.where(sl == k)[0]
            out[r, i] = out[r, i[rng.permutation(len(i))]]
    return gce, out


def _state(cuda, gce, sig, track=True):
    from neuralce_gb300.pt import PTState
    from neuralce_gb300.workloads import ladder
    E = gce.batched_energy(cuda.as_tensor(sig).cuda()).cpu().numpy()
    st = PTState(sig, E, ladder(len(sig))[1], np.zeros(len(sig), np.int32))
    if track:
        st.track_counts(gce)
    return st


def test_which_kernel(cuda):
    from neuralce_gb300 import _lib
    from neuralce_gb300.pt import chunk_kernel
    n_sm = cuda.cuda.get_device_properties(0).multi_processor_count
    fcc, sig = _fcc((6.0, 4.2), (5, 5, 5), 4, 1)
    st = _state(cuda, fcc, sig)
    for prec in (64, 32):
        for path in (0, 2):
            assert chunk_kernel([fcc], [st], prec, path) == ("windowed", 512)
    assert chunk_kernel([fcc]) == ("windowed", 0)
    many = _state(cuda, fcc, np.repeat(sig[:1], 2 * n_sm, 0))
    assert chunk_kernel([fcc], [many]) == ("windowed", 512)
    assert chunk_kernel([fcc, fcc], [many, st]) == ("windowed", 256)
    st.cv = None
    assert chunk_kernel([fcc], [st], 64, 1) == ("general", 0)
    for kind in ("b2", "rocksalt", "five members"):
        g, s = _job(kind, 4, 2, 2)
        assert chunk_kernel([g], [_state(cuda, g, s)]) == ("sign parity", 0)
    b2, s = _job("b2", 4, 2, 2)
    assert chunk_kernel([fcc, b2], [st, _state(cuda, b2, s)])[0] == "sign parity"
    st.enable_field(fcc)
    assert chunk_kernel([fcc], [st]) == ("local field", 0)
    assert chunk_kernel([fcc], [st], 32) == ("windowed", 512)
    with pytest.raises(_lib.NceError, match="path must be"):
        chunk_kernel([fcc], [st], 64, 4)
    with pytest.raises(_lib.NceError, match="precision"):
        chunk_kernel([fcc], [st], 16)


@pytest.mark.parametrize("L", [(3, 3, 3), (4, 4, 4), (5, 5, 5), (5, 5, 6), (5, 6, 7), (10, 4, 9), (8, 8, 8)])
def test_cells_of_the_window_tests_run_in_windows(cuda, L):
    from neuralce_gb300.pt import chunk_kernel
    from tests.test_window_gpu import _cell
    gce, _, _ = _cell(L, 0.5, 1, 1)
    assert chunk_kernel([gce])[0] == "windowed" and chunk_kernel([gce], None, 32)[0] == "windowed"


def test_tuners_time_the_windowed_kernel_once(cuda):
    from neuralce_gb300.autotune import best_launch
    from neuralce_gb300.batch import CEBatch, tune_launch
    from neuralce_gb300.workloads import ladder
    fcc, sig = _fcc((6.0, 4.2), (4, 4, 4), 4, 1)
    best, t = best_launch(fcc, _state(cuda, fcc, sig), 64, 2, (4, 8), (1, 2), steps=50)
    assert best == (4, 1) and set(t) == {(4, 1)}
    b2, s = _job("b2", 4, 4, 2)
    _, t = best_launch(b2, _state(cuda, b2, s), 64, 2, (4, 8), (1, 2), steps=50)
    assert set(t) == {(4, 1), (8, 1), (4, 2), (8, 2)}
    job = lambda g, x: {"gce": g, "sigma": x, "beta": ladder(len(x))[1], "R": len(x), "N": g.n_atoms}
    big, x = _fcc((6.0, 4.2), (24, 24, 24), 2, 3)
    jobs = [job(fcc, sig), job(big, x)]
    best, t = tune_launch(jobs, 32, (8, 16), (1, 2), steps=20)
    assert best == (8, 1) and set(t) == {(8, 1)}
    assert len(tune_launch([job(b2, s)], 32, (8, 16), (1, 2), steps=20)[1]) == 4
    a = CEBatch(jobs, 32, cluster=2)
    assert len(a.launch_groups()) == 2 and a._launches() == [([0, 1], 1)]
    c = CEBatch([job(b2, s), job(big, x)], 32, cluster=2)
    assert c._launches() == c.launch_groups()
