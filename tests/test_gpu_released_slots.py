"""A slot of a served (dynamic) engine that is stepped explicitly after its release: the solve covers
it, and nothing of the step is left behind for the next run loaded there."""
import pytest

pytestmark = pytest.mark.gpu


def _particles(N, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand((N ** 3, 3), generator=g, device="cuda", dtype=torch.float64)
    return x, 0.05 * torch.randn(x.shape, generator=g, device="cuda", dtype=torch.float64)


@pytest.mark.parametrize("N", [16, 32, 64, 128])     # cuFFT; node sums; node sums; face partials
def test_explicit_step_of_a_released_slot(N):
    import torch
    from pbh_b200.engine import Engine, PeakConfig
    x, p = _particles(N, 1)
    y, q = _particles(N, 2)
    out = []
    for dynamic in (False, True):
        eng = Engine([PeakConfig(N=N, Np=N, L=1.0)] * 2, dynamic=dynamic)
        for i in range(2):
            eng.set_particles(i, x, p, 1.0, mode=0, param=0.02, max_steps=3)
        eng.run(5)
        eng.release(1)
        eng.step_explicit(1, 1.1, 0.02)
        got = [eng.delta(1), eng.acc(1, 1.12), *eng.particles(1)]
        eng.release(1)
        eng.set_particles(1, y, q, 1.0, mode=0, param=0.02, max_steps=3)
        eng.run(1)
        got += [eng.delta(1), eng.acc(1, 1.0)]
        assert abs(eng.stats(1).mass_defect) <= N ** 3 * 2.0 ** -39 and eng.stats(1).status == 0
        out.append(got)
        eng.close()
    for k, (a, b) in enumerate(zip(*out)):
        assert torch.equal(a, b), k
