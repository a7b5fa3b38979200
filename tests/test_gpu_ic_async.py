"""Stream-ordered initial conditions: the bits of the synchronous call, and host threads that share a
work area on one stream, while it is made, grows or is released."""
import ctypes as C
import threading

import pytest

pytestmark = pytest.mark.gpu

R, AMP, L = (0.10, 0.09, 0.08), 0.03, 2.0


def _params(N, Np, seed=0, noise=None):
    from pbh_b200 import _lib
    from pbh_b200.ic import KIND_GAUSS
    prm = _lib.ICParams()
    prm.N, prm.Np, prm.L, prm.kind, prm.amp = N, Np, L, KIND_GAUSS, AMP
    prm.axes = (C.c_double * 3)(*R)
    prm.noise_frac = 0.01 if seed or noise is not None else 0.0
    prm.noise_seed = seed
    if noise is not None:
        prm.noise = noise.data_ptr()
    return prm


def _buffers(Np):
    import torch
    x = torch.empty((Np ** 3, 3), dtype=torch.float64, device="cuda")
    return x, torch.empty_like(x)


def _sync(N, Np, seed=0, noise=None, delta_lin=False):
    from pbh_b200.ic import KIND_GAUSS, make_particles
    frac = 0.01 if seed or noise is not None else 0.0
    return make_particles(N, Np, L, KIND_GAUSS, AMP, R, noise=noise, noise_frac=frac, noise_seed=seed, delta_lin=delta_lin)


@pytest.mark.parametrize("N,Np", [(4, 4), (8, 40), (16, 5), (32, 32), (64, 64), (128, 128), (256, 64)])
def test_the_same_bits_from_both_calls(N, Np):
    import torch
    from pbh_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(N)
    noise = torch.randn((N, N, N), generator=g, device="cuda", dtype=torch.float64)
    s = torch.cuda.Stream()
    for kw in (dict(), dict(seed=5), dict(noise=noise)):
        x, p = _buffers(Np)
        torch.cuda.synchronize()
        prm = _params(N, Np, **kw)
        _lib.check(_lib.load().pm_make_ic_async(C.byref(prm), x.data_ptr(), p.data_ptr(), s.cuda_stream), "async")
        s.synchronize()
        for delta_lin in (False, True):
            a, b, _, _ = _sync(N, Np, delta_lin=delta_lin, **kw)
            assert torch.equal(x, a) and torch.equal(p, b), (kw.keys(), delta_lin)


@pytest.mark.parametrize("release", [False, True])
def test_host_threads_that_share_a_work_area(release):
    import torch
    from pbh_b200 import _lib
    lib = _lib.load()
    lib.pm_ic_release_cache()                       # the first calls make the work area
    s = torch.cuda.Stream()
    jobs = [(N, Np, 1 + k) for k, (N, Np) in enumerate([(16, 16), (16, 70), (32, 32), (16, 90), (32, 140), (16, 8)] * 4)]
    out = [_buffers(Np) for _, Np, _ in jobs]
    torch.cuda.synchronize()
    codes = [0] * len(jobs)
    start = threading.Barrier(5 if release else 4)

    def work(t):
        start.wait()
        for k in range(t, len(jobs), 4):
            N, Np, seed = jobs[k]
            prm = _params(N, Np, seed)
            codes[k] = lib.pm_make_ic_async(C.byref(prm), out[k][0].data_ptr(), out[k][1].data_ptr(), s.cuda_stream)

    def drop():
        start.wait()
        for _ in range(5):
            assert lib.pm_ic_release_cache() == 0

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)] + ([threading.Thread(target=drop)] if release else [])
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    s.synchronize()
    assert not any(codes)
    for (N, Np, seed), (x, p) in zip(jobs, out):
        a, b, _, _ = _sync(N, Np, seed)
        assert torch.equal(x, a) and torch.equal(p, b), (N, Np, seed)


def test_later_calls_of_a_mesh_size_allocate_nothing():
    import torch
    from pbh_b200 import _lib
    lib = _lib.load()
    lib.pm_ic_release_cache()
    s = torch.cuda.Stream()
    bufs = {Np: _buffers(Np) for Np in (8, 33, 96, 200)}
    torch.cuda.synchronize()
    for k, (Np, (x, p)) in enumerate(bufs.items()):
        prm = _params(8, Np, seed=k + 1)
        if k == 0:
            _lib.check(lib.pm_make_ic_async(C.byref(prm), x.data_ptr(), p.data_ptr(), s.cuda_stream), "async")
            s.synchronize()
            continue
        g = torch.cuda.CUDAGraph()      # a capture refuses the calls that an allocation needs
        with torch.cuda.graph(g, stream=s):
            rc = lib.pm_make_ic_async(C.byref(prm), x.data_ptr(), p.data_ptr(), s.cuda_stream)
        assert rc == 0
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(x, _sync(8, Np, k + 1)[0])
