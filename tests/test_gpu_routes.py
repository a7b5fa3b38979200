"""Choices the engine makes by itself give the results of the choices a caller can force: the
super-tile side, the way a load is grouped into bins, and explicit steps that start where the
last one ended."""
import pytest

pytestmark = pytest.mark.gpu


def _particles(N, Np, seed, jitter=0.0):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    q = (torch.arange(Np, device="cuda", dtype=torch.float64) + 0.5) / Np
    x = torch.stack(torch.meshgrid(q, q, q, indexing="ij"), dim=-1).reshape(-1, 3)
    p = 0.5 * torch.randn(x.shape, generator=g, device="cuda", dtype=torch.float64)
    return (x + jitter * torch.randn(x.shape, generator=g, device="cuda", dtype=torch.float64)) % 1.0, p


def _run(cfg, x, p, steps=6, **kw):
    from pbh_b200.engine import Engine, PeakConfig
    eng = Engine([PeakConfig(**cfg)], **kw)
    eng.set_particles(0, x, p, 1.0, mode=0, param=0.03, max_steps=steps)
    eng.run(steps + 2)
    out = (*eng.particles(0), eng.delta(0), eng.stats(0))
    eng.close()
    return out


def _same(a, b):
    import torch
    assert all(torch.equal(u, v) for u, v in zip(a[:3], b[:3]))
    assert a[3].status == 0 and b[3].status == 0
    assert a[3].kinetic == pytest.approx(b[3].kinetic, rel=1e-12)
    assert a[3].potential == pytest.approx(b[3].potential, rel=1e-12)


@pytest.mark.parametrize("N,Np", [(8, 8), (16, 20), (32, 32), (64, 50), (64, 64), (128, 64)])
def test_automatic_super_tile_side(N, Np):
    x, p = _particles(N, Np, N + Np, jitter=0.02)
    auto = _run(dict(N=N, Np=Np, L=1.0), x, p)
    for tile in (4, 8, 16):
        if tile <= N:
            _same(auto, _run(dict(N=N, Np=Np, L=1.0, tile=tile), x, p))


@pytest.mark.parametrize("N,Np,n", [(32, 32, 0), (32, 31, 0), (64, 36, 0), (16, 16, 4000), (32, 32, 7)])
def test_placing_a_load_equals_sorting_it(N, Np, n):
    """An engine with a refresh period primes by the radix sort, one without by counting and placing
    (lattices with and without whole 4^3 blocks, explicit particle counts)."""
    x, p = _particles(N, Np, 3, jitter=0.05)
    if n:
        x, p = x[:n].contiguous(), p[:n].contiguous()
    cfg = dict(N=N, Np=Np, L=1.0, n=n)
    _same(_run(cfg, x, p), _run(cfg, x, p, full_every=200))


def test_reloading_twice_before_a_step_and_a_shrunk_cloud():
    """A load replaced before it was placed, and one whose particles all sit in one super-tile."""
    import torch
    from pbh_b200.engine import Engine, PeakConfig
    x, p = _particles(32, 32, 5, jitter=0.05)
    small = 0.4 + 0.05 * x
    eng = Engine([PeakConfig(N=32, Np=32, L=1.0)])
    eng.set_particles(0, x, p, 1.0)
    eng.set_particles(0, small, p, 1.0, mode=0, param=0.03, max_steps=4)
    eng.run(6)
    ref = _run(dict(N=32, Np=32, L=1.0), small, p, steps=4)
    assert torch.equal(eng.delta(0), ref[2]) and torch.equal(eng.particles(0)[0], ref[0])
    assert eng.stats(0).status == 0
    eng.close()


def test_explicit_steps_with_and_without_reading_the_clock_back():
    import torch
    from pbh_b200 import _lib
    from pbh_b200.engine import Engine, PeakConfig
    x, p = _particles(32, 32, 9, jitter=0.02)
    out = []
    for disturb in (False, True):
        eng = Engine([PeakConfig(N=32, Np=32, L=1.0)] * 2)
        for i in range(2):
            eng.set_particles(i, x, p, 1.0)
        a = 1.0
        for k in range(6):
            if k == 4:
                a = a * 1.01          # a step that does not start where the last one ended
            eng.step_explicit(0, a, 0.02 * a)
            a += 0.02 * a
            if disturb:               # each of these makes the engine read the clock back
                if k % 2:
                    eng.run(1)
                else:
                    _lib.check(_lib.load().pm_set_collapse_threshold(eng._h, 0, 0.0, 0), "threshold")
        eng.set_particles(0, x, p, 1.0)
        eng.step_explicit(0, 1.0, 0.02)   # reloaded: not held any more
        out.append((eng.delta(0), *eng.particles(0), eng.clock(0).a))
        eng.step_explicit(0, 1.02, 0.02)
        out[-1] += (eng.delta(0), *eng.particles(0))
        eng.close()
    for u, v in zip(*out):
        assert torch.equal(u, v) if hasattr(u, "shape") else u == v
