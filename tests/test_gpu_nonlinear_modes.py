"""The nonlinear term of every compiled size up to N = 9216 against a plain FP64 evaluation, mode by mode: each
mode's error is measured against what one mode of the products' spectra contributes there, so that a wrong mode
of any wavenumber shows, the lowest and the kx = 0 column too."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def white_velocity(N, seed):
    """A field whose velocity has the same amplitude in every mode."""
    r = np.random.default_rng(seed)
    H = N // 2
    kz = np.where(np.arange(N) < H, np.arange(N), np.arange(N) - N)[:, None]
    k = np.sqrt(kz.astype(np.float64) ** 2 + np.arange(H)[None, :] ** 2)
    om = (k / N) * np.exp(2j * np.pi * r.random((N, H)))
    om[H] = 0.0
    om[H + 1:, 0] = np.conj(om[1:H, 0][::-1])
    return om.astype(np.complex64)


@pytest.mark.parametrize("N", [16, 32, 64, 128, 256, 512, 840, 1024, 2048, 4096, 8192, 9216])
def test_every_mode_of_the_nonlinear_term(N):
    """FN = kx kz D + (kz^2 - kx^2) E, D = F[u^2 - w^2], E = F[u w]; |kx kz| <= k^2 / 2 and |kz^2 - kx^2| <= k^2,
    so FN / k^2 has the products' scale and a wrong mode an error of their RMS amplitude.  FP32 transforms of at
    most 14 butterfly levels, four in a row, leave 6e-8 sqrt(52) = 4e-7 of that RMS per mode, the largest of
    4e7 Gaussian modes sqrt(ln 4e7) = 4.2 times as much: 2e-6.  Ten times that is allowed."""
    import optimizec_b200 as P

    H, L = N // 2, 3 * N // 2
    om = white_velocity(N, N)
    s = P.Solver(N, 1e6, 4.0, 0.1)
    s.init_vorticity(om)
    s.next_dt()
    s.step(1)
    fn = torch.from_numpy(s.fnm1()).cuda().to(torch.complex128)
    s.close()
    o = torch.from_numpy(om).cuda().to(torch.complex128)
    iz = torch.arange(N, device="cuda", dtype=torch.float64)
    kz = torch.where(iz < H, iz, iz - N)[:, None]
    kx = torch.arange(H, device="cuda", dtype=torch.float64)[None, :]
    k2 = (kx ** 2 + kz ** 2).clamp(min=1.0)

    def phys(f):
        pad = torch.zeros((L, L // 2 + 1), dtype=torch.complex128, device="cuda")
        pad[:H, :H], pad[L - H:, :H] = f[:H], f[H:]
        return torch.fft.irfft2(pad, s=(L, L), norm="forward")

    def spec(p):
        f = torch.fft.rfft2(p, norm="forward")
        return torch.cat([f[:H, :H], f[L - H:, :H]])

    u, w = phys(-1j * kz / k2 * o), phys(1j * kx / k2 * o)
    d, e = spec(u * u - w * w), spec(u * w)
    ref = kx * kz * d + (kz ** 2 - kx ** 2) * e
    ref[H] = 0.0
    rms = max(float(d.abs().square().mean().sqrt()), float(e.abs().square().mean().sqrt()))
    err = (fn - ref).abs() / (k2 * rms)
    assert float(err.max()) <= 2e-5
    assert float(fn[H].abs().max()) == 0.0
    # two low modes exchanged would be found
    wrong = ref.clone()
    wrong[1, 1], wrong[2, 1] = ref[2, 1], ref[1, 1]
    assert float(((wrong - ref).abs() / (k2 * rms)).max()) > 2e-3
