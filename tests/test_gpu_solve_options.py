"""Gradient and smoothing options of the native solve on the sizes of five passes, whose row and z
passes take their factors from the table of the finite differences, against the cuFFT path; and
smoothed forces of every native size against float64."""
import pytest

pytestmark = pytest.mark.gpu


def _particles(Np, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand((Np ** 3, 3), generator=g, device="cuda", dtype=torch.float64)
    return x, torch.zeros_like(x)


def _rel(a, b):
    return float((a - b).norm() / b.norm())


def _forces(N, Np, native, x, p, **kw):
    from pbh_b200.engine import Engine, PeakConfig
    eng = Engine([PeakConfig(N=N, Np=Np, L=1.0, **kw)], native_fft=native)
    eng.set_particles(0, x, p, 1.0)
    eng.run(1)
    out = eng.acc(0, 1.0)
    assert eng.stats(0).status == 0
    eng.close()
    return out


@pytest.mark.parametrize("gradient,smooth", [("fd2", 0.0), ("fd4", 0.0), ("fd4", 1.0), ("spectral", 1.5)])
@pytest.mark.parametrize("N,Np", [(256, 96), (512, 64)])
def test_options_match_the_cufft_path(N, Np, gradient, smooth):
    # Two FP32 transforms of a few 1e-7 relative L2 each (the same bound as on the slab sizes).
    x, p = _particles(Np, N)
    kw = dict(gradient=gradient, smooth=smooth)
    assert _rel(_forces(N, Np, True, x, p, **kw), _forces(N, Np, False, x, p, **kw)) < 2e-6


@pytest.mark.parametrize("N,smooth", [(32, 1.5), (128, 1.0), (256, 2.0)])
def test_smoothed_forces_match_float64(N, smooth):
    from oracle.pm3d_torch64 import TorchMesh
    Np = min(N, 96)
    x, p = _particles(Np, N + 1)
    mesh = TorchMesh(N, 1.0, Np, smooth=smooth, device="cuda")
    ref, _ = mesh.forces(x, 1.0)
    assert _rel(_forces(N, Np, True, x, p, smooth=smooth), ref) < 2e-6
