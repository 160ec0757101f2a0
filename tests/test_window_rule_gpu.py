"""The windowed kernel's float32 filter settles no step that the float64 rule decides otherwise: negative beta (in float64 every
swap between different species is accepted, as by the step-by-step kernel's threshold; in float32 ln u < -beta dE, also with
a wide near band) and host uniforms without a logarithm (rejected)."""
import numpy as np
import pytest

from tests.test_window_gpu import _cell, _run

pytestmark = pytest.mark.gpu


def test_negative_beta_float64(cuda):
    torch = cuda
    from neuralce_gb300.pt import PTState, run_chunk
    R, T = 3, 500
    gce, orc, sig = _cell((5, 5, 5), 0.5, R, 21)
    rng = np.random.default_rng(5)
    a, b = (rng.integers(0, sig.shape[1], (T, R)).astype(np.int32) for _ in range(2))
    u = 1.0 - rng.random((T, R))
    st = PTState(sig, np.array([orc.energy(x) for x in sig]), np.array([-0.5, -5.0, -40.0], np.float32), np.zeros(R, np.int32))
    run_chunk(gce, st, T, 0, 1, 64, 0, tuple(torch.as_tensor(x).cuda() for x in (a, b, u)), do_exchange=False)
    want, n = sig.copy(), np.zeros(R, np.int64)
    for s in range(T):
        for r in range(R):
            x, y = want[r, a[s, r]], want[r, b[s, r]]
            if x != y:
                want[r, a[s, r]], want[r, b[s, r]] = y, x
                n[r] += 1
    torch.cuda.synchronize()
    assert np.array_equal(st.n_acc.cpu().numpy(), n) and np.array_equal(st.sigma.cpu().numpy(), want)
    assert not st.n_near.any()


@pytest.mark.parametrize("near_eV", [0.0, 0.05])
def test_negative_beta_float32(cuda, near_eV):
    gce, orc, sig = _cell((5, 5, 5), 0.5, 3, 22)
    _run(cuda, gce, orc, sig, np.array([-0.5, -5.0, -40.0], np.float32), 2, 300, 50, 32, near_eV=near_eV)


@pytest.mark.parametrize("precision", [64, 32])
def test_uniforms_without_a_logarithm(cuda, precision):
    gce, orc, sig = _cell((5, 5, 5), 0.5, 3, 23)
    rng = np.random.default_rng(6)
    T = 300
    a, b = (rng.integers(0, sig.shape[1], (2 * T, 3)).astype(np.int32) for _ in range(2))
    u = 1.0 - rng.random((2 * T, 3))
    u[::7] = np.nan
    u[3::7] = -0.25
    u[5::7] = -1.0
    _run(cuda, gce, orc, sig, np.array([2.0, 10.0, 30.0], np.float32), 2, T, 60, precision, props=(a, b, u))
