"""The native Poisson solve (density to force grids, native_fft.cu) of every mesh size it serves
against the float64 torch restatement of pm3d on the same positions, its gradient and smoothing
options against the cuFFT path, and a batch with idle slots."""
import pytest

pytestmark = pytest.mark.gpu


def _particles(N, seed):
    import torch
    from pbh_b200 import recipe
    from pbh_b200.ic import recipe_particles
    x, p = recipe_particles(recipe.single_peak(N=N, steps=20, seed=seed), device=0, device_noise=True)
    # Off the lattice by up to half a cell, so that every mode of the mesh is excited, the Nyquist
    # planes included.
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (x + (torch.rand(x.shape, device="cuda", generator=g, dtype=torch.float64) - 0.5) / N) % 1.0, p


def _rel(a, b):
    return float((a - b).norm() / b.norm())


def _engine(N, native=True, **kw):
    from pbh_b200.engine import Engine, PeakConfig
    return Engine([PeakConfig(N=N, Np=N, L=1.0, **kw)], native_fft=native)


@pytest.mark.parametrize("N,smooth", [(32, 0.0), (64, 0.0), (64, 2.0), (128, 0.0), (256, 0.0)])
def test_forces_match_float64(N, smooth):
    # FP32 transforms agree with float64 to a few 1e-7 relative L2 (N = 512: test_gpu_large).
    import torch
    from oracle.pm3d_torch64 import TorchMesh
    x, p = _particles(N, 3)
    eng = _engine(N, smooth=smooth)
    eng.set_particles(0, x, p, 1.0)
    eng.step_explicit(0, 1.0, 0.01)
    a = 1.01
    xe, pe = eng.particles(0)
    mesh = TorchMesh(N, 1.0, N, smooth=smooth, device="cuda")
    ref, delta = mesh.forces(xe, a)
    assert _rel(eng.acc(0, a), ref) < 2e-6
    # the potential energy of the solve is sampled at the next push
    phi = torch.fft.irfftn(mesh.potential_k(delta, a), s=(N, N, N))
    pot = 0.5 * 3.0 * 25.0 / (8.0 * torch.pi) * (1.0 / N) ** 3 * float((delta * phi).sum())
    eng.step_explicit(0, a, 0.01)
    s = eng.stats(0)
    assert s.a_energy == pytest.approx(a) and s.potential == pytest.approx(pot, rel=2e-6)
    assert s.status == 0
    eng.close()


@pytest.mark.parametrize("gradient,smooth", [("fd2", 0.0), ("fd4", 1.0)])
@pytest.mark.parametrize("N", [32, 64, 128])
def test_finite_difference_gradients_match_the_cufft_path(N, gradient, smooth):
    x, p = _particles(N, 4)
    acc = []
    for native in (False, True):
        eng = _engine(N, native, gradient=gradient, smooth=smooth)
        eng.set_particles(0, x, p, 1.0)
        eng.step_explicit(0, 1.0, 0.01)
        acc.append(eng.acc(0, 1.01))
        eng.close()
    assert _rel(acc[1], acc[0]) < 2e-6


def test_idle_slots_keep_their_forces_and_do_not_disturb_the_others():
    """Slots of one mesh size: one never loaded, one loaded once and held, one that keeps
    stepping.  The held one's forces stay what they were, the stepping one's equal its run alone."""
    import torch
    from pbh_b200.engine import Engine, PeakConfig
    x, p = _particles(64, 5)
    eng = Engine([PeakConfig(N=64, Np=64, L=1.0)] * 3)
    eng.set_particles(1, x, p, 1.0)
    eng.run(1)
    held = eng.acc(1, 1.0)
    eng.set_particles(2, x, p, 1.0, mode=0, param=0.02, max_steps=50)
    eng.run(6)
    alone = _engine(64)
    alone.set_particles(0, x, p, 1.0, mode=0, param=0.02, max_steps=50)
    alone.run(6)
    a = alone.clock(0).a
    assert torch.equal(eng.acc(1, 1.0), held)
    assert torch.equal(eng.acc(2, a), alone.acc(0, a))
    assert eng.stats(1).status == 0 and eng.stats(2).status == 0
    eng.close()
    alone.close()
