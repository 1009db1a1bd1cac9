"""Register-resident transforms at the sizes where they can go wrong: one- and
two-lane lengths, planes that leave lanes or planes of a CTA idle, band counts
with an unpaired last band, Nyquist rows of unequal axes, the cut-off mask and
the exchange over an odd number of orbitals, against the FP64 oracle.
Tolerances: FP64 1e-12 and FP32 1e-5 of the largest value, the bars of every
H*psi test of this repository."""
import numpy as np
import pytest

from oracle import exx, pw

pytestmark = pytest.mark.gpu
TOL = {"f64": 1e-12, "f32": 1e-5}
GRIDS = [(12, 12, 12), (24, 16, 20), (20, 20, 20), (30, 30, 30), (36, 36, 36), (40, 20, 20), (48, 24, 24),
         (48, 48, 48), (60, 60, 60), (72, 72, 72)]


def _case(n, prec):
    from pwdft_develop_b200 import Context
    L = [0.35 * x for x in n]
    nf = tuple(2 * x for x in n)
    dm = pw.Domain(tuple(L), tuple(n), nf)
    ekin, teter = pw.ekin_teter(dm)
    rng = np.random.default_rng(sum(n))
    T = pw.HamTables(dm, ekin, teter, rng.uniform(-1, 0.5, dm.ntotFine), [])
    return Context(L, n, nf, precision=prec), T, rng


def _close(got, ref, prec):
    err = np.abs(got.double().cpu().numpy() - ref).max() / np.abs(ref).max()
    assert err <= TOL[prec], err


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n", GRIDS)
def test_transforms_of_every_length(n, prec):
    import torch
    c, T, rng = _case(n, prec)
    c.set_vtot(T.vtot)
    # white noise: every Nyquist row, column and corner carries weight
    nb = 1 if n[0] >= 60 else 3
    psi = rng.standard_normal((nb, T.dm.ntot)) / np.sqrt(T.dm.ntot)
    x = torch.tensor(psi, dtype=c.torch_dtype, device="cuda")
    ref = pw.mult_spinor(T, psi)
    _close(c.hpsi(x), ref, prec)
    _close(c.hpsi(x, out=x.clone(), accumulate=True), ref + x.double().cpu().numpy(), prec)
    _close(c.teter(x), pw.add_teter_precond(T, psi), prec)
    ecut = 0.6 * float(T.ekin.max())
    c.set_wfn_filter(ecut)
    _close(c.hpsi(x), pw.mult_spinor(T, psi, wfn_ecut=ecut), prec)


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n", [(12, 12, 12), (24, 16, 20), (36, 36, 36), (40, 20, 20), (60, 60, 60)])
def test_exchange_of_an_odd_number_of_orbitals(n, prec):
    import torch
    c, T, rng = _case(n, prec)
    psi = rng.standard_normal((2, T.dm.ntot)) / np.sqrt(T.dm.ntot)
    phi = rng.standard_normal((3, T.dm.ntot)) / np.sqrt(T.dm.ntot)
    occ = np.array([1.0, 0.5, 1.0])
    c.exx_setup(fraction=0.25, screen_mu=0.0, divergence_type=1, ecut=10.0)
    c.exx_set_phi(torch.tensor(phi, dtype=c.torch_dtype, device="cuda"), occ)
    # the device's own kernel table: its G = 0 entry is a small difference of two
    # sums over the grid (here 1e-12 from the oracle's at 60^3), which is not a
    # matter of the transforms
    kern = c.exx_kernel()[1][:, :, : n[0] // 2 + 1]
    ref = exx.add_mult_spinor_exx(T.dm, psi, exx.set_phi(T.dm, phi), kern, 0.25, occ)
    _close(c.exx_apply(torch.tensor(psi, dtype=c.torch_dtype, device="cuda")), ref, prec)


@pytest.mark.parametrize("n", [(12, 12, 12), (16, 16, 16), (20, 20, 20), (24, 16, 20), (24, 24, 24), (30, 30, 30),
                               (32, 32, 32), (36, 36, 36), (40, 40, 40), (48, 48, 48), (60, 60, 60), (72, 72, 72)])
def test_rounding_of_the_transforms(n):
    """FP32 Teter (a 3-D transform there and back) on damped bands: the rms error of
    an FFT of N points grows as u sqrt(log2 N) (Gentleman and Sande 1966), here
    with a factor of 0.36-0.49 over the lengths.  The bound of 0.52 leaves 5 % and is
    passed by one more rounded twiddle product per point: with twiddles between all
    radix steps 40 points are at 0.63, 36 at 0.56 and 72 at 0.521."""
    import torch
    c, T, _ = _case(n, "f32")
    g = torch.Generator(device="cuda").manual_seed(5)
    f = [2 * np.pi / (0.35 * m) * torch.fft.fftfreq(m, 1.0 / m, dtype=torch.float64, device="cuda") for m in n]
    a = f[2][:, None, None] ** 2 + f[1][None, :, None] ** 2 + f[0][None, None, :] ** 2
    b = 27.0 + a * (18.0 + a * (12.0 + a * 8.0))
    x = torch.randn((16,) + n[::-1], generator=g, device="cuda", dtype=torch.float64)
    x = torch.fft.ifftn(torch.fft.fftn(x, dim=(1, 2, 3)) / (1.0 + a / 6.0) ** 2, dim=(1, 2, 3)).real
    x = x.reshape(16, -1).float()
    ref = torch.fft.ifftn(torch.fft.fftn(x.double().reshape((16,) + n[::-1]), dim=(1, 2, 3)) * (b / (b + 16.0 * a ** 4)),
                          dim=(1, 2, 3))
    ref = ref.real.reshape(16, -1)
    err = float((c.teter(x).double() - ref).norm() / ref.norm())
    assert err <= 0.52 * 2.0 ** -24 * np.sqrt(2 * np.log2(c.ntot)), err
