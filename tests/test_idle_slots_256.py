"""Every pass of the solve leaves the slots alone whose peak did not deposit, on the sizes of five
passes too (test_gpu_solve has 64^3, whose solve has no row pass)."""
import re
from pathlib import Path

import pytest

SRC = Path(__file__).resolve().parent.parent / "pbh_b200" / "csrc" / "native_fft.cu"


def test_every_launch_of_the_solve_knows_the_slots_and_returns_on_idle_ones():
    text = re.sub(r"//[^\n]*", "", SRC.read_text())
    solve = text[text.index("int solve_n("):text.index("int c2r_n(")]
    launches = re.findall(r"pdl_launch\((\w+)<[^;]*?\);", solve)
    assert len(launches) >= 8
    for call in re.findall(r"pdl_launch\([^;]*\);", solve):
        assert call.rstrip(");").endswith("slot_peak"), call
    for kernel in set(launches):
        code = text[re.search(rf"\b{kernel}\(", text).start():]
        code = code[:code.index("\n}\n")]
        assert re.search(r"if \((slot_peak && )?!(slot_active\(A, slot_peak, [^)]+\)|\(A\.plan\[pk\]\.flags & PLAN_DEP\))\) return;",
                         code), kernel


@pytest.mark.gpu
def test_idle_slots_of_256():
    """One slot never loaded, one loaded once and held, one that keeps stepping."""
    import torch
    from pbh_b200.engine import Engine, PeakConfig
    N, Np = 256, 64
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.rand((Np ** 3, 3), generator=g, device="cuda", dtype=torch.float64)
    p = 0.05 * torch.randn(x.shape, generator=g, device="cuda", dtype=torch.float64)
    eng = Engine([PeakConfig(N=N, Np=Np, L=1.0)] * 3)
    eng.set_particles(1, x, p, 1.0)
    eng.run(1)
    held = eng.acc(1, 1.0)
    eng.set_particles(2, x, p, 1.0, mode=0, param=0.02, max_steps=50)
    eng.run(30)
    alone = Engine([PeakConfig(N=N, Np=Np, L=1.0)])
    alone.set_particles(0, x, p, 1.0, mode=0, param=0.02, max_steps=50)
    alone.run(30)
    a = alone.clock(0).a
    assert torch.equal(eng.acc(1, 1.0), held)
    assert torch.equal(eng.acc(2, a), alone.acc(0, a))
    # the held slot steps again: its spectra are made anew
    eng.step_explicit(1, 1.0, 0.02)
    one = Engine([PeakConfig(N=N, Np=Np, L=1.0)])
    one.set_particles(0, x, p, 1.0)
    one.step_explicit(0, 1.0, 0.02)
    assert torch.equal(eng.acc(1, 1.02), one.acc(0, 1.02))
    assert eng.stats(1).status == 0 and eng.stats(2).status == 0
    for e in (eng, alone, one):
        e.close()
