"""Batch rules: the band batch that follows the call (growth, even split, frozen
by a capture or by the caller) and the k-point projector products batched over
whole k-points.  The same kernels run on every batch shape, so results agree to
the bit where only the batch changes; FP32 k-points against one k at a time
differ by the split-K partition of the projector sums (1e-5, the FP32 bar)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
A = 10.26


def _ctx(prec, n=(16, 16, 16), **kw):
    from oracle import pw
    from pwdft_develop_b200 import Context
    L, z, pos = pw.make_crystal("Si", (1, 1, 1), A, 0.02, 77)
    c = Context(L, n, tuple(2 * x for x in n), precision=prec)
    c.set_atoms([z] * len(pos), pos)
    rng = np.random.default_rng(3)
    c.set_vtot(rng.uniform(-1, 0.5, c.ntotFine))
    return c


def _rand(c, nb, seed=5):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((nb, c.ntot), generator=g, device="cuda", dtype=torch.float64).to(c.torch_dtype)


@pytest.mark.parametrize("nb", [1, 64, 65, 150, 307])
def test_batch_follows_the_call(nb):
    import torch
    c, d = _ctx("f64"), _ctx("f64")
    d.set_band_batch(14)
    x = _rand(c, nb)
    ref = torch.cat([c.teter(x[i:i + 2]) for i in range(0, nb, 2)])
    assert torch.equal(c.teter(x), ref)
    assert torch.equal(d.teter(x), ref)
    # the projector products take all bands of a call, however they are batched
    assert torch.equal(c.hpsi(x), d.hpsi(x))


def test_a_captured_call_outlives_larger_ones():
    import torch
    c = _ctx("f32")
    x = _rand(c, 7)
    out = torch.empty_like(x)
    g = c.capture_hpsi(x, out)
    g.replay()
    torch.cuda.synchronize()
    ref = out.clone()
    big = _rand(c, 200, seed=9)
    y = c.hpsi(big)
    assert torch.isfinite(y).all()
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, ref)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("batch", [None, 2, 10, 22, 30])
def test_kpoint_batches(prec, batch):
    """nk = 5 of nb = 7: all together, whole k-points per batch (22, 30 fields)
    and k-points cut by the batch (1, 5 fields); the projector products take
    whole k-points in all of them, so the bits are those of one batch."""
    import torch
    c = _ctx(prec)
    if batch:
        c.set_band_batch(2 * batch)
    rng = np.random.default_rng(1)
    ks = rng.uniform(-0.3, 0.3, (5, 3))
    c.set_kpoints(ks)
    g = torch.Generator(device="cuda").manual_seed(2)
    ct = torch.complex128 if prec == "f64" else torch.complex64
    x = torch.randn((5, 7, c.ntot, 2), generator=g, device="cuda", dtype=torch.float64)
    x = torch.view_as_complex(x).to(ct)
    got = c.hpsi_kbatch(x)
    if batch:
        c.set_band_batch(2 * 5 * 7)
        assert torch.equal(got, c.hpsi_kbatch(x))
    for i, k in enumerate(ks):
        c.set_kpoint(k)
        ref = c.hpsi_k(x[i].contiguous())
        err = (got[i] - ref).abs().max() / ref.abs().max()
        assert err <= (1e-5 if prec == "f32" else 1e-13), (i, float(err))


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_a_refused_growth_leaves_the_batch(prec):
    """No room for a larger batch: the call runs in the batch that is there."""
    import torch
    from pwdft_develop_b200._lib import PwError
    c = _ctx(prec)
    x = _rand(c, 900)
    out = torch.empty_like(x)
    ref = torch.cat([c.hpsi(x[i:i + 30]) for i in range(0, 900, 30)])
    with pytest.raises(PwError):
        c.set_band_batch(2000000000)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (40 << 20), dtype=torch.uint8, device="cuda")
    for _ in range(3):
        out.zero_()
        c.hpsi(x, out=out)
        torch.cuda.synchronize()
    del fill
    torch.cuda.empty_cache()
    # other widths of the projector products: equal to rounding
    assert (out - ref).abs().max() <= (1e-5 if prec == "f32" else 1e-13) * ref.abs().max()
    assert (c.hpsi(x) - ref).abs().max() <= (1e-5 if prec == "f32" else 1e-13) * ref.abs().max()


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_capture_of_a_call_wider_than_any_before(prec):
    """Recorded on a capturing stream, a block wider than the scratch runs in the
    batch that is there and its projector products still find their operands."""
    import torch
    c = _ctx(prec)
    c.hpsi(_rand(c, 6))
    x = _rand(c, 203, seed=8)
    out = torch.zeros_like(x)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        c.hpsi(x, out=out)
    x.copy_(_rand(c, 203, seed=9))
    g.replay()
    torch.cuda.synchronize()
    ref = c.hpsi(x)
    assert (out - ref).abs().max() <= (1e-5 if prec == "f32" else 1e-13) * ref.abs().max()


def test_projector_products_of_more_than_one_group():
    """363 bands of 72^3 are two groups of split bands and seven batches; against
    narrow calls, whose products have other tiles and partitions (FP32 bar)."""
    import torch
    c = _ctx("f32", n=(72, 72, 72))
    nb = 363
    assert nb * 4 * c.ntot > 512 << 20
    x = _rand(c, nb)
    ref = torch.cat([c.hpsi(x[i:i + 33]) for i in range(0, nb, 33)])
    top = ref.abs().max()
    assert (c.hpsi(x) - ref).abs().max() <= 1e-5 * top
    base = torch.randn_like(x[:1]).expand(nb, -1).contiguous()
    got = c.hpsi(x, out=base.clone(), accumulate=True)
    assert (got - (base + ref)).abs().max() <= 1e-5 * top


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("mode", ["planes", "sphere"])
def test_a_captured_exchange_outlives_larger_ones(mode, prec):
    """H*psi with the full exchange, recorded; then a wider exchange and another
    scratch limit: the recorded workspaces are still the graph's."""
    import torch
    if mode == "planes":
        c = _ctx(prec)
    else:
        from oracle import pw
        from pwdft_develop_b200 import Context
        L, z, pos = pw.make_crystal("Si", (1, 1, 1), A, 0.02, 77)
        c = Context.gspace(L, (32, 32, 32), 6.0, precision=prec)
        c.set_atoms([z] * len(pos), pos)
        c.set_vtot(np.random.default_rng(3).uniform(-1, 0.5, c.ntotFine))
    phi = _rand(c, 5, seed=4) / np.sqrt(c.ntot)
    c.exx_setup(0.25, 0.0, 1, 6.0)
    c.exx_set_phi(phi, np.ones(5))
    c.exx_set_mode("full")
    x = _rand(c, 3)
    out = torch.empty_like(x)
    g = c.capture_hpsi(x, out)
    g.replay()
    torch.cuda.synchronize()
    ref = out.clone()
    c.exx_apply(_rand(c, 64, seed=9))
    from pwdft_develop_b200._lib import check, lib
    check(lib.pw_exx_set_scratch(c.handle, 1 << 24))
    y = torch.full((1 << 22,), 3.0, dtype=c.torch_dtype, device="cuda")
    c.exx_apply(_rand(c, 70, seed=10))
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, ref) and bool((y == 3.0).all())


def _count(c, f):
    for _ in range(3):       # past any growth
        f()
    n = c.launches()
    f()
    return c.launches() - n


@pytest.mark.parametrize("solver", ["eigsolve", "scf", "twin"])
def test_a_solver_leaves_the_batch_to_the_calls(solver):
    """After a narrow solve on the same context the wide calls and the k-point
    batches take as many launches as on a fresh one."""
    import torch
    prec = "f32" if solver == "eigsolve" else "f64"
    c, d = _ctx(prec), _ctx(prec)
    if solver == "eigsolve":
        c.eigsolve(_rand(c, 4) / np.sqrt(c.ntot), solver="lobpcg", maxit=2)
    elif solver == "scf":
        c.scf(nocc=16, nextra=4, ecut=5.0, solver="chebfsi", mixed=True, max_iter=2)
    else:
        c.build_twin()
    x = _rand(c, 200)
    ks = np.random.default_rng(1).uniform(-0.3, 0.3, (4, 3))
    g = torch.Generator(device="cuda").manual_seed(2)
    y = torch.view_as_complex(torch.randn((4, 24, c.ntot, 2), generator=g, device="cuda", dtype=x.dtype))
    for e in (c, d):
        e.set_vtot(np.linspace(-1, 0.5, c.ntotFine))
        e.set_wfn_filter(None)
        e.set_kpoints(ks)
    for f in (lambda e: e.hpsi(x), lambda e: e.teter(x), lambda e: e.hpsi_kbatch(y)):
        assert _count(c, lambda: f(c)) == _count(d, lambda: f(d))


@pytest.mark.parametrize("mode", ["sphere", "serial", "full", "full filter", "ace"])
@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_no_result_depends_on_the_batch(mode, prec):
    """Serial and sphere-cut projector products and the exchange after them: the
    bits of one batch in batches of 3 pairs, accumulated or not."""
    import torch
    if mode == "sphere":
        from oracle import pw
        from pwdft_develop_b200 import Context
        L, z, pos = pw.make_crystal("Si", (1, 1, 1), A, 0.02, 77)
        c = Context.gspace(L, (32, 32, 32), 6.0, precision=prec)
        c.set_atoms([z] * len(pos), pos)
        c.set_vtot(np.random.default_rng(3).uniform(-1, 0.5, c.ntotFine))
    else:
        c = _ctx(prec)
    if mode == "serial":
        from pwdft_develop_b200._lib import check, lib
        check(lib.pw_set_nl_overlap(c.handle, 0))
    x = _rand(c, 25) / np.sqrt(c.ntot)
    if mode != "serial":
        phi = _rand(c, 30, seed=4) / np.sqrt(c.ntot)
        c.exx_setup(0.25, 0.0, 1, 6.0)
        c.exx_set_phi(phi, np.ones(30))
        c.exx_set_mode("full")
    if mode == "ace":
        c.ace_build(phi)
    if mode == "full filter":
        c.set_wfn_filter(5.0)
    c.set_band_batch(26)
    base = torch.randn_like(x)
    ref, refa = c.hpsi(x), c.hpsi(x, out=base.clone(), accumulate=True)
    c.set_band_batch(6)
    assert torch.equal(c.hpsi(x), ref)
    assert torch.equal(c.hpsi(x, out=base.clone(), accumulate=True), refa)


def _grown(f):
    """Device memory that a call takes and keeps."""
    import torch
    torch.cuda.synchronize()
    a = torch.cuda.mem_get_info()[0]
    f()
    torch.cuda.synchronize()
    return a - torch.cuda.mem_get_info()[0]


def test_one_wide_call_takes_no_new_scratch():
    """The first call wider than the scratch runs in the batches that are there,
    with the bits of the later ones; the second takes what it needs, Teter its
    one block of coarse fields; a narrower call takes nothing."""
    import torch
    c, w = _ctx("f64", n=(24, 24, 24)), _ctx("f64", n=(24, 24, 24))
    c.set_band_batch(64)         # w's: the kernels and library handles of both calls are there
    x = _rand(c, 200)
    out, wout = torch.empty_like(x), torch.empty_like(x)
    c.hpsi(x, out=out), c.teter(x, out=out)
    pair = 16 * (2 * 24 ** 3 + 48 * 25 * 25)
    assert _grown(lambda: w.teter(x, out=wout)) < 4 << 20
    first = wout.clone()
    coarse = 100 * 16 * 24 ** 3
    assert coarse <= _grown(lambda: w.teter(x, out=wout)) < coarse + (4 << 20)
    assert torch.equal(wout, first)
    assert _grown(lambda: w.hpsi(x, out=wout)) < 4 << 20
    first = wout.clone()
    rest = 100 * pair - coarse
    assert rest <= _grown(lambda: w.hpsi(x, out=wout)) < rest + (6 << 20)
    assert torch.equal(wout, first)
    assert _grown(lambda: (w.hpsi(x, out=wout), w.teter(x[:150], out=wout[:150]))) == 0


def test_the_scratch_stays_within_its_limit():
    """Ever wider calls: the blocks in use hold at most 640 MiB, all of them less
    than three times that, and the batch no longer grows there."""
    import torch
    c = _ctx("f64", n=(24, 24, 24))
    c.set_atoms([14], [(0.0, 0.0, 0.0)])
    x = _rand(c, 3000)
    out = torch.empty_like(x)
    pair = 16 * (2 * 24 ** 3 + 48 * 25 * 25)
    lim = (640 << 20) // pair
    c.hpsi(x[:66], out=out[:66])

    def grow():
        for nb in range(80, 3000, 40):
            c.hpsi(x[:nb], out=out[:nb])
    assert _grown(grow) < 3 * (640 << 20)
    n = c.launches()
    c.hpsi(x, out=out)
    batches = -(-1500 // lim)
    assert c.launches() - n == 5 * batches + 1


def test_sphere_cut_scratch():
    """Sphere-cut calls take slot fields alone, and Teter nothing."""
    import torch
    from oracle import pw
    from pwdft_develop_b200 import Context
    L, z, pos = pw.make_crystal("Si", (1, 1, 1), A, 0.02, 77)
    c = Context.gspace(L, (48, 48, 48), 10.0, precision="f64")
    c.set_vtot(np.random.default_rng(3).uniform(-1, 0.5, c.ntotFine))
    x = _rand(c, 200)
    out = torch.empty_like(x)
    c.hpsi(x[:8], out=out[:8])
    c.teter(x[:8], out=out[:8])
    assert _grown(lambda: (c.teter(x, out=out), c.teter(x, out=out))) == 0
    assert _grown(lambda: c.hpsi(x, out=out)) == 0
    first = out.clone()
    slots = 100 * 16 * 48 * 25 * 25
    assert slots <= _grown(lambda: c.hpsi(x, out=out)) < slots + (4 << 20)
    assert torch.equal(out, first)


def test_projector_builds_take_fields_for_their_projectors():
    """After a wide k-point batch the temporary fields of a build still go with
    the projectors: there is room for them on a nearly full device."""
    import torch
    c, d = _ctx("f32", n=(24, 24, 24)), _ctx("f32", n=(24, 24, 24))
    ks = np.random.default_rng(1).uniform(-0.3, 0.3, (4, 3))
    c.set_kpoints(ks)
    g = torch.Generator(device="cuda").manual_seed(2)
    y = torch.view_as_complex(torch.randn((4, 300, c.ntot, 2), generator=g, device="cuda"))
    for _ in range(3):
        c.hpsi_kbatch(y)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (200 << 20), dtype=torch.uint8, device="cuda")
    c.set_kpoint(ks[1] / 2)
    from oracle import pw
    _, z, pos = pw.make_crystal("Si", (1, 1, 1), A, 0.02, 77)
    c.set_atoms([z] * len(pos), pos)
    del fill
    torch.cuda.empty_cache()
    d.set_kpoint(ks[1] / 2)
    x = y[0, :5].contiguous()
    assert torch.equal(c.hpsi_k(x), d.hpsi_k(x))


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("by", ["hpsi", "teter", "kbatch"])
def test_a_captured_call_outlives_a_growth(by, prec):
    """A graph recorded before wide H*psi, Teter or k-point calls grew the scratch
    still reads and writes its own blocks."""
    import torch
    c = _ctx(prec)
    x = _rand(c, 7)
    out = torch.empty_like(x)
    g = c.capture_hpsi(x, out)
    g.replay()
    torch.cuda.synchronize()
    ref = out.clone()
    if by == "kbatch":
        c.set_kpoints(np.random.default_rng(1).uniform(-0.3, 0.3, (5, 3)))
        r = torch.Generator(device="cuda").manual_seed(2)
        big = torch.view_as_complex(torch.randn((5, 40, c.ntot, 2), generator=r, device="cuda", dtype=x.dtype))
        f = c.hpsi_kbatch
    else:
        big = _rand(c, 200, seed=9)
        f = c.hpsi if by == "hpsi" else c.teter
    y = [f(big) for _ in range(3)]
    assert all(torch.equal(v, y[0]) for v in y)
    for _ in range(2):
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, ref)
    assert torch.equal(f(big), y[0])


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_the_exchange_of_a_wide_call_takes_64_bands_at_a_time(prec):
    """The pair fields' chunks, and with them the sums over the orbitals, do not
    follow the width of an H*psi call: the bits of calls of 64 bands."""
    import torch
    from pwdft_develop_b200 import Context
    from pwdft_develop_b200._lib import check, lib
    c = Context((A,) * 3, (16, 16, 16), (32, 32, 32), precision=prec)
    c.set_vtot(np.random.default_rng(3).uniform(-1, 0.5, c.ntotFine))
    c.exx_setup(0.25, 0.0, 1, 6.0)
    c.exx_set_phi(_rand(c, 30, seed=4) / np.sqrt(c.ntot), np.ones(30))
    c.exx_set_mode("full")
    x = _rand(c, 150) / np.sqrt(c.ntot)
    # room for 256 pair fields: 4 orbital pairs of 64 bands, 1 of 150
    check(lib.pw_exx_set_scratch(c.handle, 256 * c.ntot * (16 if prec == "f64" else 8)))
    ref = torch.cat([c.hpsi(x[i:i + 64]) for i in range(0, 150, 64)])
    assert torch.equal(c.hpsi(x), ref)
