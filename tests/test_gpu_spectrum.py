"""The spectrum's half of the frequencies and their conjugates, at lengths around
the blocks of its sums, and what non-finite samples do to it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 2, 3, 63, 64, 65, 255, 256, 257, 1021, 4096])
def test_lengths(N):
    import torch

    from python_code_to_check_c_gb300.spectrum import spectrum
    rng = np.random.default_rng(N)
    mu = rng.standard_normal(N) + 1e-9j * rng.standard_normal(N)
    n = np.arange(N)
    ang = 2 * np.pi * ((n[:, None] * n[None, :]) % N).astype(np.longdouble) / N
    w = np.cos(ang) - 1j * np.sin(ang)
    _, Yr, Yi = spectrum(mu, 0.01)
    for Y, x in ((Yr, mu.real), (Yi, mu.imag)):
        ref = np.fft.fftshift((x.astype(np.longdouble)[:, None] * w).sum(0))
        # N terms, each off by 2^-53 of the twiddle and of the sum so far, which log2 N + 8 additions round
        tol = (np.log2(N) + 10) * 2.0**-53 * np.sqrt(N) * np.abs(x).max() * 4
        assert np.abs(Y - ref).max() <= tol
    # under capture the same
    d = torch.as_tensor(mu, device="cuda")
    lib, Y = _call(d, N)
    assert np.array_equal(Y[0], Yr) and np.array_equal(Y[1], Yi)


def _call(d, N):
    import torch

    from python_code_to_check_c_gb300 import _lib
    from python_code_to_check_c_gb300.engine import _ptr, _stream
    lib = _lib.load()
    Y = torch.zeros((2, N), dtype=torch.complex128, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        assert lib.tdcc_spectrum(_ptr(d), N, 1, 0.01, _ptr(Y[0]), _ptr(Y[1]), None, _stream()) == 0
    g.replay()
    return lib, Y.cpu().numpy()


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_non_finite_samples_stay_in_their_part(bad):
    from python_code_to_check_c_gb300.spectrum import spectrum
    mu = np.random.default_rng(3).standard_normal(130) * (1 + 0.1j)
    mu.imag[7] = bad
    _, Yr, Yi = spectrum(mu, 0.01)
    assert np.isfinite(Yr).all() and not np.isfinite(Yi).any()
