"""The widths of the push and the ways of reading particles back, by the number and density of an
engine's super-tiles, give the same bits: few dense bins, many sparse ones, one bin far denser than
the mean, and a load that was not placed yet."""
import pytest

pytestmark = pytest.mark.gpu


def _particles(Np, seed, size=1.0):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand((Np ** 3, 3), generator=g, device="cuda", dtype=torch.float64)
    return 0.37 + size * x if size < 1 else x, 0.05 * torch.randn(x.shape, generator=g, device="cuda", dtype=torch.float64)


def _outputs(N, Np, tile, x, p, peaks=1):
    from pbh_b200.engine import Engine, PeakConfig
    eng = Engine([PeakConfig(N=N, Np=Np, L=1.0, tile=tile)] * peaks)
    eng.set_particles(peaks - 1, x, p, 1.0, mode=0, param=0.02, max_steps=4)
    out = [*eng.particles(peaks - 1)]                    # from the loading area
    eng.run(3)
    a = eng.clock(peaks - 1).a
    out += [*eng.particles(peaks - 1), eng.acc(peaks - 1, a), eng.delta(peaks - 1)]
    assert eng.stats(peaks - 1).status == 0
    eng.close()
    return out


@pytest.mark.parametrize("N,Np,size,forms", [
    (8, 40, 1.0, [(4, 1), (8, 1)]),                      # eight bins of 8000, one of 64000
    (32, 32, 1.0, [(4, 1), (8, 1), (16, 1)]),            # 512 bins of 64, 64 of 512, 8 of 4096
    (32, 16, 1.0, [(4, 1), (8, 1), (8, 10), (16, 1)]),   # sparser than the widest push; 640 super-tiles
    (64, 64, 0.08, [(4, 1), (8, 1), (8, 2), (16, 1)]),   # one place far denser than the mean
    (64, 33, 1.0, [(4, 1), (8, 1), (16, 1)]),
    (64, 104, 1.0, [(8, 1), (8, 2), (16, 1)]),           # 512 super-tiles of 2197, 1024
])
def test_density_and_number_of_bins_change_no_bit(N, Np, size, forms):
    import torch
    x, p = _particles(Np, N + Np, size)
    ref = None
    for tile, peaks in forms:
        out = _outputs(N, Np, tile, x, p, peaks)
        d = (out[0] - x + 0.5) % 1.0 - 0.5
        assert float(d.abs().max()) <= 2.0 ** -24 / N * 1.01 and float((out[1] - p).abs().max()) <= 2.0 ** -24 * float(p.abs().max())
        if ref is not None:
            assert all(torch.equal(u, v) for u, v in zip(out, ref)), (tile, peaks)
        ref = out
