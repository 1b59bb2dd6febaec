"""The in-place row and column passes (inplace.cuh): every retained mode against
a plain FP64 evaluation, the members of a batch, and the closure's forcing."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [64, 128, 256, 512, 1024, 2048, 4096, 8192, 9216]


def P():
    import optimizec_b200 as mod
    return mod


def _white(N, seed):
    """A field whose velocity has the same amplitude in every mode, so that the products and the
    nonlinear term have no mode below rounding: a wrong position of any stage shows."""
    r = np.random.default_rng(seed)
    H = N // 2
    kz = np.where(np.arange(N) < H, np.arange(N), np.arange(N) - N)[:, None]
    k = np.sqrt(kz.astype(np.float64) ** 2 + np.arange(H)[None, :] ** 2)
    om = (k / N) * np.exp(2j * np.pi * r.random((N, H)))
    om[H] = 0.0
    om[0, 0] = 0.0
    om[H + 1:, 0] = np.conj(om[1:H, 0][::-1])
    return om.astype(np.complex64)


def _nonlinear64(om):
    """FN of a compact spectrum with torch's FP64 transforms."""
    N, H = om.shape
    L = 3 * N // 2
    o = torch.from_numpy(om).cuda().to(torch.complex128)
    iz = torch.arange(N, device="cuda", dtype=torch.float64)
    kz = torch.where(iz < H, iz, iz - N)[:, None]
    kx = torch.arange(H, device="cuda", dtype=torch.float64)[None, :]
    inv = torch.where((kx ** 2 + kz ** 2) > 0, 1.0 / (kx ** 2 + kz ** 2).clamp(min=1.0), 0.0)

    def phys(f):
        pad = torch.zeros((L, L // 2 + 1), dtype=torch.complex128, device="cuda")
        pad[:H, :H], pad[L - H:, :H] = f[:H], f[H:]
        return torch.fft.irfft2(pad, s=(L, L), norm="forward")

    def spec(p):
        f = torch.fft.rfft2(p, norm="forward")
        return torch.cat([f[:H, :H], f[L - H:, :H]])

    u, w = phys(-1j * kz * inv * o), phys(1j * kx * inv * o)
    fn = kx * kz * spec(u * u - w * w) + (kz ** 2 - kx ** 2) * spec(u * w)
    fn[H] = 0.0
    return fn.cpu().numpy()


@pytest.mark.parametrize("N", SIZES)
def test_nonlinear_term_of_every_mode(N):
    """FP32 transforms of at most 14 butterfly levels, four in a row, leave a relative L2 error of about
    6e-8 sqrt(4 x 13) = 4e-7 on white data; ten times that is allowed.  One wrong mode among N^2 / 2 would
    be 1e-3 or more."""
    om = _white(N, N)
    s = P().Solver(N, 1e6, 4.0, 0.1)
    s.init_vorticity(om)
    s.next_dt()
    s.step(1)
    fn = s.fnm1().astype(np.complex128)
    s.close()
    ref = _nonlinear64(om)
    assert np.linalg.norm(fn - ref) <= 4e-6 * np.linalg.norm(ref)
    assert np.all(fn[N // 2] == 0)


@pytest.mark.parametrize("N", [1024, 2048, 4096])
def test_energies_of_a_step_are_those_of_its_field(N):
    """E and Z of a step are FP64 sums over the FP32 field with 1 / K^2 to FP64 rounding: sums of N^2 / 2
    positive terms, each within a few 2^-52, differ from any other order's by less than 1e-12."""
    s = P().Solver(N, 1e4, 4.0, 0.1)
    s.init_vorticity(_white(N, N + 1))
    s.next_dt()
    E, Z = s.step(2, history=True)
    om = s.om2().astype(np.complex128)
    s.close()
    kz = np.where(np.arange(N) < N // 2, np.arange(N), np.arange(N) - N)[:, None].astype(np.float64)
    kx = np.arange(N // 2, dtype=np.float64)[None, :]
    k2 = kx ** 2 + kz ** 2
    p = np.abs(om.real) ** 2 + np.abs(om.imag) ** 2
    p *= np.where(kx == 0, 0.5, 1.0)
    e = np.sum(np.where(k2 > 0, p / np.maximum(k2, 1.0), 0.0))
    assert abs(E[-1] - e) <= 1e-12 * e
    assert abs(Z[-1] - p.sum()) <= 1e-12 * p.sum()


def test_members_of_a_batch_equal_single_runs():
    members = [(1024, 1e4, 4.0, 0.1, 3), (2048, 1e5, 5.0, 0.1, 4), (1024, 1e3, 3.0, 0.1, 5)]
    b = P().Batch(members)
    b.init_k4()
    b.next_dt()
    b.step(3)
    for m, (N, Re, K0, cfl, seed) in enumerate(members):
        s = P().Solver(N, Re, K0, cfl)
        s.init_k4(seed)
        s.next_dt()
        s.step(3)
        np.testing.assert_array_equal(b.om2(m), s.om2())
        s.close()
    b.close()


def test_closure_forcing_enters_the_nonlinear_term():
    """FNM1 of a closed step = FNM1 of the plain step + the forcing, within FP32 rounding."""
    N = 1024
    om = _white(N, 7)
    runs = []
    net = P().CNN(3, 8, seed=11)
    for closed in (False, True):
        s = P().Solver(N, 1e4, 4.0, 0.1)
        s.init_vorticity(om)
        s.next_dt()
        if closed:
            s.attach_closure(net, (1.0, 1.0, 1.0, 50.0), energy_check=0)
            F = s.closure_forcing().astype(np.complex128)
        s.step(1)
        runs.append(s.fnm1().astype(np.complex128))
        s.close()
    net.close()
    scale = np.abs(runs[0]).max() + np.abs(F).max()
    assert np.abs(runs[1] - runs[0] - F).max() <= 1e-6 * scale
