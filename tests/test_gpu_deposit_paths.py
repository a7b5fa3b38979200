"""The deposit's two ways of finishing its node sums: 64-bit integers (folded chunks, float64
counts, large mean counts) and exact FP64 arithmetic (a single chunk), on the same positions."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,Np,tile,spread", [
    (16, 16, 8, 1.0),     # one chunk per super-tile
    (32, 45, 16, 1.0),    # about 11 000 particles a super-tile: two chunks
    (64, 32, 16, 1.0),    # sparse: most nodes empty
    (8, 60, 8, 1.0),      # n_mean = 422, many chunks
    (8, 96, 8, 1.0),      # n_mean = 1728: integers throughout
    (32, 32, 16, 0.02),   # all particles in a few cells (one node takes thousands)
    (32, 19, 4, 1.0),
])
def test_delta_is_the_same_from_both_paths(N, Np, tile, spread):
    import torch
    from pbh_b200.engine import Engine, PeakConfig
    n = Np ** 3
    g = torch.Generator(device="cuda").manual_seed(N + Np)
    x = (0.37 + spread * torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64)) % 1.0
    eng = Engine([PeakConfig(N=N, Np=Np, L=1.0, tile=tile)])
    eng.set_particles(0, x, torch.zeros_like(x), 1.0)
    eng.run(1)
    delta = eng.delta(0)
    s = eng.stats(0)
    counts = eng.counts(0)                       # the same kernels with the integer path
    assert torch.equal(eng.delta(0), delta)      # rewritten with identical bits
    t = eng.stats(0)
    assert (s.mass_defect, s.rho_max_over_mean, s.status) == (t.mass_defect, t.rho_max_over_mean, t.status)
    assert s.status == 0
    # Counts are exact multiples of 2^-38 and n_mean is not always: the defect is its rounding.
    assert abs(s.mass_defect) <= N ** 3 * 2.0 ** -39
    assert float(counts.sum()) == pytest.approx(n, rel=1e-14)
    assert s.rho_max_over_mean == pytest.approx(float(counts.max()) / (n / N ** 3), rel=1e-14)
    ref = (counts / (n / N ** 3) - 1.0).to(torch.float32)
    # float32 rounding of the same FP64 value, whose subtraction of 1 here loses up to 2^-53 of it
    assert float((delta - ref).abs().max()) <= 2.0 ** -23 * float(ref.abs().max())
    eng.close()


@pytest.mark.parametrize("sizes", [
    [(32, 32, 4)], [(32, 19, 16), (32, 45, 16)], [(32, 32, 0), (64, 32, 0)],
    [(64, 64, 8), (64, 75, 8)],                  # 2^19 cells: the last size that adds node sums
    [(64, 64, 16)], [(64, 64, 0), (64, 64, 0), (32, 32, 0)],
])
def test_node_sums_of_small_meshes_start_from_zero_every_step(sizes):
    """Engines of a few small meshes add their node sums to grids that the solve reads and clears:
    after several steps delta and its statistics have the bits of the face partials' path, and
    the delta of a peak that went idle stays."""
    import torch
    from pbh_b200 import _lib
    from pbh_b200.engine import Engine, PeakConfig
    eng = Engine([PeakConfig(N=N, Np=Np, L=1.0, tile=tile) for N, Np, tile in sizes])
    g = torch.Generator(device="cuda").manual_seed(len(sizes))
    for i, (N, Np, tile) in enumerate(sizes):
        x = torch.rand((Np ** 3, 3), generator=g, device="cuda", dtype=torch.float64)
        p = 0.05 * torch.randn((Np ** 3, 3), generator=g, device="cuda", dtype=torch.float64)
        eng.set_particles(i, x, p, 10.0, mode=_lib.SCHED_RATIO, param=0.02, max_steps=6 - 4 * (i % 2))
    eng.run(4)
    held = [eng.delta(i) for i in range(len(sizes))]
    eng.run(2)
    for i in range(len(sizes)):
        delta, s = eng.delta(i), eng.stats(i)
        assert torch.equal(delta, held[i]) == (i % 2 == 1)
        eng.counts(i)
        t = eng.stats(i)
        assert torch.equal(eng.delta(i), delta)
        assert (s.mass_defect, s.rho_max_over_mean, s.status) == (t.mass_defect, t.rho_max_over_mean, 0)
    eng.close()
