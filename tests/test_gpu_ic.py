"""Device initial conditions against the float64 numpy oracle over lattices that do and do not
divide the mesh, with and without noise, and the stream-ordered form against the synchronous one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("noise_frac", [0.0, 0.01])
@pytest.mark.parametrize("N,Np", [(8, 8), (16, 5), (16, 16), (16, 48), (32, 27), (32, 64), (64, 32)])
def test_recipe_particles_match_the_oracle(N, Np, noise_frac):
    import torch
    from oracle.pm3d_oracle import Mesh
    from oracle.recipe_oracle import recipe_ic
    from pbh_b200.ic import KIND_GAUSS, make_particles
    R, delta0, L = (0.10, 0.09, 0.08), 0.03, 2.0
    ref = recipe_ic(Mesh(N, L, Np), R, delta0, noise_frac, 7)
    noise = np.random.default_rng(7).standard_normal((N, N, N)) if noise_frac else None
    x, p, dl, rms = make_particles(N, Np, L, KIND_GAUSS, delta0, R, noise=noise, noise_frac=noise_frac, delta_lin=True)
    d = (x.cpu().numpy() - ref["x"] + L / 2) % L - L / 2
    assert np.abs(d).max() < 1e-12 * L
    scale = np.abs(ref["p"]).max()
    assert np.abs(p.cpu().numpy() - ref["p"]).max() < 1e-12 * scale
    assert np.abs(dl.cpu().numpy() - ref["delta_lin"]).max() < 1e-12 * np.abs(ref["delta_lin"]).max()
    # without delta_lin one transform fewer, the same particles
    x3, p3, _, rms3 = make_particles(N, Np, L, KIND_GAUSS, delta0, R, noise=noise, noise_frac=noise_frac)
    assert float((x3 - x).abs().max()) < 1e-13 * L and float((p3 - p).abs().max()) < 1e-13 * scale and rms3 == rms
    if noise_frac:
        k = 2 * np.pi * np.fft.fftfreq(N, d=L / N)
        kk = np.sqrt(k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2)
        kk[0, 0, 0] = np.inf
        assert rms == pytest.approx(float(np.std(np.fft.ifftn(np.fft.fftn(noise) / kk).real)), rel=1e-12)
