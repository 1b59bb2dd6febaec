"""The work that users of this framework run, as cases that can be timed and checked.

Kinds of case
  run       an initial-value problem through Solver, the way the command line and the benchmark
            drive it: the vorticity from pinned host memory, NEXTDT, time steps with the
            diagnostics of every `update` steps, the final vorticity back to pinned memory.
  ensemble  independent runs of uneven sizes advanced together through Batch.
  closure   a coarse run with the learned closure attached (its CNN evaluated every step).
  train     Adam iterations of the closure network on a resident data set.
  grad      loss and gradient of the closure network on one batch from host memory.

Grid sizes are the compiled ones that the tests, the benchmark and the reference's recorded runs
use (64 ... 16384; a transform has 3N/2 points, so 96, 192 ... 24576, with the odd factors 3 and,
at 9216, 27).  Flow parameters are the ranges of the benchmark and the ensemble configuration.
"""
import math

import numpy as np
import torch

import optimizec_b200 as P


def listed():
    return [
        # one step of a small run between two host reads: a program that couples the solver to its
        # own loop; launches and copies are all of its time
        dict(name="run_64_one_step", kind="run", N=64, Re=1e3, K0=4.0, cfl=0.1, steps=1, update=100, history=False, spectrum="k4"),
        # the smallest grids in earnest (parameter studies), energies read back every step
        dict(name="run_256_history", kind="run", N=256, Re=1e4, K0=4.0, cfl=0.1, steps=150, update=100, history=True, spectrum="k4"),
        # the reference's N = 512 configuration, a part of its 1000 steps
        dict(name="run_512", kind="run", N=512, Re=1e4, K0=4.0, cfl=0.1, steps=200, update=100, history=False, spectrum="k4"),
        # a medium grid from a developed (k^-3) field, an odd number of steps
        dict(name="run_1024_developed", kind="run", N=1024, Re=3e4, K0=6.0, cfl=0.1, steps=77, update=25, history=False, spectrum="k-3"),
        # the DNS that training data of the closure comes from
        dict(name="run_2048", kind="run", N=2048, Re=1e5, K0=4.0, cfl=0.1, steps=50, update=100, history=False, spectrum="k-3"),
        # the headline configuration of the benchmark, end to end with energies per step
        dict(name="run_4096_headline", kind="run", N=4096, Re=1e5, K0=4.0, cfl=0.1, steps=20, update=100, history=True, spectrum="k4"),
        # the large grids (rows spread over several CTAs): 8192, and 16384 as in the reference's
        # recorded runs (UPDATE = 10 there)
        dict(name="run_8192", kind="run", N=8192, Re=1e5, K0=4.0, cfl=0.1, steps=11, update=10, history=False, spectrum="k-3"),
        dict(name="run_16384", kind="run", N=16384, Re=1e6, K0=4.0, cfl=0.1, steps=5, update=10, history=False, spectrum="k-3"),
        # the 64-member ensemble of the benchmark
        dict(name="ensemble_64", kind="ensemble", n128=32, n256=24, n512=8, cfl=0.1, steps=300),
        # the closed N = 256 run (6 x 32 network, BF16 inference, device-side energy gate)
        dict(name="closure_256", kind="closure", N=256, Re=1e5, K0=4.0, cfl=0.1, steps=100, layers=6),
        # training at the closure's grid (384^2), tensor-core convolutions as the experiment uses them
        dict(name="train_384_b4", kind="train", size=384, batch=4, samples=12, iters=4, layers=6, tensor_cores=True),
        # a gradient of the small network grid in the default FP32 arithmetic, batch from the host
        dict(name="grad_48_b32_fp32", kind="grad", size=48, batch=32, layers=6, tensor_cores=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["run", "ensemble", "closure", "train", "grad"], [10, 2, 2, 2, 2])[0]
    Re = round(10.0 ** rng.uniform(3.0, 6.0), 1)
    K0 = float(rng.randint(2, 8))
    cfl = round(rng.uniform(0.05, 0.2), 3)
    if kind == "run":
        N = rng.choice([16, 32, 64, 128, 256, 512, 1024, 2048, 4096, 8192, 9216, 16384])
        # the number of steps falls with the grid, so that no drawn case costs more than the largest listed one
        most = 5 if N == 16384 else max(8, min(300, 20 * 4096 // N))
        steps = _log_int(rng, 1, most)
        return dict(kind="run", N=N, Re=Re, K0=K0, cfl=cfl, steps=steps, update=rng.choice([10, 25, 100]),
                    history=rng.random() < 0.3, spectrum=rng.choice(["k4", "k-3"]))
    if kind == "ensemble":
        return dict(kind="ensemble", n128=rng.randint(1, 40), n256=rng.randint(0, 16), n512=rng.randint(0, 8), cfl=cfl,
                    steps=_log_int(rng, 8, 300))
    if kind == "closure":
        return dict(kind="closure", N=rng.choice([128, 256, 512]), Re=round(10.0 ** rng.uniform(4.0, 5.0), 1), K0=K0,
                    cfl=cfl, steps=_log_int(rng, 2, 120), layers=rng.randint(4, 7))
    if kind == "train":
        size = rng.choice([48, 96, 192, 384])
        batch = rng.randint(1, 4 if size >= 192 else 32)
        return dict(kind="train", size=size, batch=batch, samples=batch + rng.randint(1, 8), iters=rng.randint(1, 6),
                    layers=rng.randint(4, 7), tensor_cores=True)
    size = rng.choice([48, 64, 96, 192])
    return dict(kind="grad", size=size, batch=rng.randint(1, 32 if size <= 96 else 4), layers=rng.randint(3, 7),
                tensor_cores=rng.random() < 0.5)


# ---- inputs ----------------------------------------------------------------------------------

def _vorticity(N, K0, spectrum, rng, out):
    """A random-phase vorticity field of energy 1/2 in the solver's compact layout [iz][ix], in
    place: E(k) ~ k^4 exp(-2 (k/K0)^2), or k^4 at low k and k^-3 with a viscous cut-off above K0.
    Modes beyond the band have amplitudes below single precision and stay zero."""
    H = N // 2
    kb = min(H - 1, 64 if spectrum == "k4" else 256)
    kx = np.arange(kb + 1, dtype=np.float64)[None, :]
    kz = np.arange(-kb, kb + 1, dtype=np.float64)[:, None]
    k = np.sqrt(kx * kx + kz * kz)
    q = k / K0
    e = q ** 4 * np.exp(-2.0 * q * q) if spectrum == "k4" else q ** 4 / (1.0 + q ** 7) * np.exp(-((3.0 * k / (kb + 1)) ** 2))
    om = np.sqrt(k * e) * np.exp(2j * np.pi * rng.random((2 * kb + 1, kb + 1)))
    om[kb, 0] = 0.0
    om[:kb, 0] = np.conj(om[:kb:-1, 0])  # a real field: Hermitian on kx = 0
    w = np.where(kx == 0, 0.5, 1.0)
    E = np.sum(np.where(k > 0, w * np.abs(om) ** 2 / np.maximum(k * k, 1.0), 0.0))
    om *= math.sqrt(0.5 / E)
    out[:kb + 1, :kb + 1] = om[kb:]
    out[N - kb:, :kb + 1] = om[:kb]
    return out


def _pinned(shape, dtype):
    pin = torch.cuda.is_available()
    return torch.zeros(shape, dtype=dtype, pin_memory=pin).numpy()


def _field(case, seed):
    om = _pinned((case["N"], case["N"] // 2), torch.complex64)
    return _vorticity(case["N"], case["K0"], case.get("spectrum", "k4"), np.random.default_rng(seed), om)


def _members(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for N in (128, 256, 512):
        for _ in range(case["n%d" % N]):
            out.append((N, float(np.float32(10.0 ** rng.uniform(3.0, 5.0))), float(rng.integers(2, 9)), case["cfl"],
                        int(rng.integers(1, 1 << 40))))
    return out


def _smooth(rng, n, channels, size):
    """Unit-variance periodic fields with a falling spectrum, like normalised vorticity planes."""
    k = np.fft.fftfreq(size, 1.0 / size)
    k2 = k[:, None] ** 2 + np.arange(size // 2 + 1)[None, :] ** 2
    f = np.fft.irfft2(np.fft.rfft2(rng.standard_normal((n, channels, size, size), dtype=np.float32)) / (1.0 + k2 / 16.0),
                      s=(size, size))
    return (f / f.std(axis=(-2, -1), keepdims=True)).astype(np.float32)


def _net_params(layers, channels, rng):
    parts = []
    for l in range(layers):
        ci, co = (3 if l == 0 else channels), (1 if l == layers - 1 else channels)
        parts += [rng.standard_normal(co * ci * 9) * math.sqrt(2.0 / (9 * ci)), 0.05 * rng.standard_normal(co)]
    return np.concatenate(parts).astype(np.float32)


def _net_data(case, seed):
    rng = np.random.default_rng(seed)
    n = case.get("samples", case["batch"])
    x = _smooth(rng, n, 3, case["size"])
    t = _smooth(rng, n, 1, case["size"])
    return x, t, _net_params(case["layers"], 32, rng)


_TRAIN_SEED = 7   # of the minibatch draws
_LR = 1e-5        # the end of a schedule


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("run", "closure"):
        s = P.Solver(case["N"], case["Re"], case["K0"], case["cfl"])
        state = dict(case=case, solver=s, om0=_field(case, seed),
                     out=_pinned((case["N"], case["N"] // 2), torch.complex64))
        if kind == "closure":
            net = P.CNN(case["layers"], 32)
            net.set_params(_net_params(case["layers"], 32, np.random.default_rng(seed + 1)))
            s.attach_closure(net, (5.0, 1.0, 1.0, 0.01), energy_check=1)
            state["net"] = net
        return state
    if kind == "ensemble":
        b = P.Batch(_members(case, seed))
        b.init_k4()
        return dict(case=case, batch=b)
    x, t, params = _net_data(case, seed)
    net = P.CNN(case["layers"], 32)
    net.set_params(params)
    net.set_train_tc(case["tensor_cores"])
    if kind == "train":
        net.set_dataset(x, t)
        return dict(case=case, net=net)
    px, pt = _pinned(x.shape, torch.float32), _pinned(t.shape, torch.float32)
    px[...], pt[...] = x, t
    return dict(case=case, net=net, x=px, t=pt)


# ---- one pass --------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "run":
        s, sigma, E, Z = state["solver"], [], [], []
        s.init_vorticity(state["om0"])
        s.next_dt()
        left = case["steps"]
        while left:
            n = min(left, case["update"])
            h = s.step(n, history=case["history"])
            if h is not None:
                E.append(h[0])
                Z.append(h[1])
            left -= n
            # the diagnostics of a printed line, as the command line makes them
            s.next_dt()
            s.om2phys()
            sigma.append(s.display_sigma(2))
        out = dict(om2=s.om2(out=state["out"]), sigma=np.array(sigma, dtype=np.float32))
        if E:  # the field that they are sums over is 32-bit, so the histories are kept at that precision
            out.update(E=np.concatenate(E).astype(np.float32), Z=np.concatenate(Z).astype(np.float32))
        return out
    if kind == "closure":
        s = state["solver"]
        s.init_vorticity(state["om0"])
        s.next_dt()
        s.step(case["steps"])
        return dict(om2=s.om2(out=state["out"]))
    if kind == "ensemble":  # goes on from where the last pass ended
        b = state["batch"]
        b.next_dt()
        b.step(case["steps"])
        return [b.om2(m) for m in range(len(b.members))]
    if kind == "train":  # likewise
        state["net"].train(case["iters"], case["batch"], _LR, seed=_TRAIN_SEED)
        return dict(params=state["net"].params())
    loss, g = state["net"].loss_grad(state["x"], state["t"])
    return dict(loss=np.float32(loss), grad=g)  # the loss is a mean over 32-bit activations


# ---- what a pass cannot do without -------------------------------------------------------------

def _step_work(N):
    """One time step.  Bytes: om2 and fnm1 read and written (4 x 4 N^2), and the two half-spectra
    of 3N/2 rows (12 N^2) handed over twice between the row and the column transforms, written and
    read each time.  Operations: complex transforms of length L = 3N/2, one inverse and one forward
    per row, two of each per retained column, at 5 L log2 L."""
    L = 3 * N // 2
    return 64.0 * N * N, 5.0 * L * math.log2(L) * (2 * L + 4 * (N // 2))


def _net_work(layers, size, batch, passes):
    """Convolutions of one evaluation (passes = 1) or of forward, data and weight gradients (3).
    Bytes: the 32-bit input planes and output, and every hidden activation written once and read
    once per pass that needs it."""
    px = batch * size * size
    macs = px * 9 * (3 * 32 + (layers - 2) * 32 * 32 + 32)
    return px * 4.0 * (4 + 32 * (layers - 1) * 2 * passes), 2.0 * passes * macs


def work(case):
    kind = case["kind"]
    if kind in ("run", "closure"):
        b, f = _step_work(case["N"])
        if kind == "closure":
            L = 3 * case["N"] // 2
            nb, nf = _net_work(case["layers"], L, 1, 1)
            px = float(L * L)
            # the hidden activations are bf16 here; the fields' inverse and the forcing's forward transforms
            b, f = b + nb / 2 + 4 * 4 * px, f + nf + 5.0 * L * math.log2(L) * 3 * L
        return dict(bytes=case["steps"] * b + 8.0 * case["N"] ** 2, flops=case["steps"] * f)
    if kind == "ensemble":
        w = [(case["n%d" % N],) + _step_work(N) + (4.0 * N * N,) for N in (128, 256, 512)]
        return dict(bytes=sum(n * (case["steps"] * b + o) for n, b, _, o in w), flops=sum(n * case["steps"] * f for n, _, f, _ in w))
    b, f = _net_work(case["layers"], case["size"], case["batch"], 3)
    it = case.get("iters", 1)
    return dict(bytes=it * b, flops=it * f)


# ---- 64-bit values -----------------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Flow:
    """The scheme in 64 bits with torch's transforms, for a batch of fields of one size."""

    def __init__(self, om, Re, cfl):
        dev = _device()
        self.m, self.N, self.H = om.shape
        self.L = 3 * self.N // 2
        col = lambda v: torch.as_tensor(v, dtype=torch.float64, device=dev).reshape(-1, 1, 1)  # noqa: E731
        self.om = torch.from_numpy(om).to(dev, torch.complex128)
        self.fo = torch.zeros_like(self.om)
        self.visc, self.cfl = 1.0 / col(Re), col(cfl)
        iz = torch.arange(self.N, device=dev, dtype=torch.float64)
        self.kz = torch.where(iz < self.H, iz, iz - self.N).reshape(1, -1, 1)
        self.kx = torch.arange(self.H, device=dev, dtype=torch.float64).reshape(1, 1, -1)
        self.k2 = self.kx ** 2 + self.kz ** 2
        self.inv = torch.where(self.k2 > 0, 1.0 / self.k2.clamp(min=1.0), 0.0)
        self.dt = self.cn = self.cnm1 = None
        self.E, self.Z = [], []

    def _physical(self, f):
        L, H, N = self.L, self.H, self.N
        pad = torch.zeros((self.m, L, L // 2 + 1), dtype=torch.complex128, device=f.device)
        pad[:, :H, :H] = f[:, :H]
        pad[:, L - H:, :H] = f[:, H:]
        return torch.fft.irfft2(pad, s=(L, L), norm="forward")

    def _velocity(self):
        return (self._physical(-1j * self.kz * self.inv * self.om), self._physical(1j * self.kx * self.inv * self.om))

    def next_dt(self):
        u, w = self._velocity()
        cflm = ((u.abs() + w.abs()) * (self.N / (2.0 * math.pi))).amax(dim=(1, 2), keepdim=True)
        if self.dt is None:
            self.dt, self.cn, self.cnm1 = self.cfl / cflm / math.pi, torch.ones_like(cflm), torch.zeros_like(cflm)
        else:
            self.cn = 0.8 + 0.2 * self.cfl / (cflm * self.dt * math.pi)
            self.dt = self.dt * self.cn

    def _spectrum(self, p):
        f = torch.fft.rfft2(p, norm="forward")
        return torch.cat([f[:, :self.H, :self.H], f[:, self.L - self.H:, :self.H]], dim=1)

    def step(self):
        u, w = self._velocity()
        d, e = self._spectrum(u * u - w * w), self._spectrum(u * w)
        del u, w
        fn = self.kx * self.kz * d + (self.kz ** 2 - self.kx ** 2) * e
        del d, e
        fn[:, self.H] = 0.0
        a = 0.5 * self.visc * self.dt * self.k2
        self.om = ((1.0 - a) * self.om + 0.5 * self.dt * ((2.0 + self.cnm1) * fn - self.cnm1 * self.fo)) / (1.0 + a)
        self.fo, self.cnm1 = fn, self.cn

    def sums(self):
        p = self.om.abs() ** 2 * torch.where(self.kx == 0, 0.5, 1.0)
        self.E.append(float((p * self.inv).sum()))
        self.Z.append(float(p.sum()))


def _exact_run(case, seed):
    om = _vorticity(case["N"], case["K0"], case["spectrum"], np.random.default_rng(seed),
                    np.zeros((case["N"], case["N"] // 2), dtype=np.complex64))
    f = _Flow(om[None], [np.float32(case["Re"])], [np.float32(case["cfl"])])
    f.next_dt()
    for i in range(1, case["steps"] + 1):
        f.step()
        if case["history"]:
            f.sums()
        if i % case["update"] == 0:
            f.next_dt()
    out = dict(om2=f.om[0].cpu(), sigma=None)  # sigma is over quantised pixels
    if case["history"]:
        out.update(E=torch.tensor(f.E, dtype=torch.float64), Z=torch.tensor(f.Z, dtype=torch.float64))
    return out


def _splitmix(z):
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _k4_field(N, K0, seed):
    """The seeded k^4 field that Batch.init_k4 starts its members from (splitmix64 phases)."""
    H = N // 2
    i = np.arange(N * H, dtype=np.uint64).reshape(N, H)
    with np.errstate(over="ignore"):
        u = (_splitmix(np.uint64(seed) + (i + np.uint64(1)) * np.uint64(0x9E3779B97F4A7C15)) >> np.uint64(11)) * 2.0 ** -53
    kz = np.where(np.arange(N) < H, np.arange(N), np.arange(N) - N)[:, None].astype(np.float64)
    kx = np.arange(H, dtype=np.float64)[None, :]
    k = np.sqrt(kx * kx + kz * kz)
    q = k / K0
    om = np.sqrt(k * q ** 4 * np.exp(-2.0 * q * q)) * np.exp(2j * np.pi * u)
    om[H] = 0.0
    om[H + 1:, 0] = np.conj(om[1:H, 0][::-1])
    E = np.sum(np.where(k > 0, np.where(kx == 0, 0.5, 1.0) * np.abs(om) ** 2 / np.maximum(k * k, 1.0), 0.0))
    return (om * math.sqrt(0.5 / E)).astype(np.complex64)


def _exact_ensemble(case, seed):
    members, out = _members(case, seed), []
    for N in (128, 256, 512):
        of = [m for m in members if m[0] == N]
        if not of:
            continue
        f = _Flow(np.stack([_k4_field(N, m[2], m[4]) for m in of]), [np.float32(m[1]) for m in of], [np.float32(m[3]) for m in of])
        f.next_dt()
        for _ in range(case["steps"]):
            f.step()
        out += list(f.om.cpu())
    return out


def _conv3x3(x, w, b):
    """A periodic 3x3 convolution in 64 bits as nine matrix products."""
    x = torch.nn.functional.pad(x, (1, 1, 1, 1), mode="circular")
    h, v = x.shape[2] - 2, x.shape[3] - 2
    y = b.reshape(1, -1, 1, 1)
    for i in range(3):
        for j in range(3):
            y = y + torch.einsum("oc,bchw->bohw", w[:, :, i, j], x[:, :, i:i + h, j:j + v])
    return y


def _loss(p, layers, x, t):
    off, a = 0, x
    for l in range(layers):
        ci, co = (3 if l == 0 else 32), (1 if l == layers - 1 else 32)
        w = p[off:off + co * ci * 9].reshape(co, ci, 3, 3)
        off += co * ci * 9
        a = _conv3x3(a, w, p[off:off + co])
        off += co
        if l + 1 < layers:
            a = torch.nn.functional.gelu(a)
    return torch.mean((a - t) ** 2)


def _exact_net(case, seed):
    dev = _device()
    x, t, params = _net_data(case, seed)
    x, t = (torch.from_numpy(v).to(dev, torch.float64) for v in (x, t))
    p = torch.from_numpy(params).to(dev, torch.float64).requires_grad_()
    if case["kind"] == "grad":
        loss = _loss(p, case["layers"], x, t)
        return dict(loss=loss.detach().cpu(), grad=torch.autograd.grad(loss, p)[0].cpu())
    m, v, state, n = torch.zeros_like(p), torch.zeros_like(p), np.uint64(_TRAIN_SEED), x.shape[0]
    for it in range(1, case["iters"] + 1):
        idx = list(range(n))  # a minibatch without replacement, by splitmix64
        for i in range(min(case["batch"], n)):
            with np.errstate(over="ignore"):
                state = state + np.uint64(0x9E3779B97F4A7C15)
                j = i + int(_splitmix(state)) % (n - i)
            idx[i], idx[j] = idx[j], idx[i]
        idx = [idx[i % n] for i in range(case["batch"])]
        g = torch.autograd.grad(_loss(p, case["layers"], x[idx], t[idx]), p)[0]
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        step = _LR * (m / (1 - 0.9 ** it)) / (torch.sqrt(v / (1 - 0.999 ** it)) + 1e-8)
        p = (p.detach() - step.detach()).requires_grad_()
    return dict(params=p.detach().cpu())


def exact(case, seed):
    if case["kind"] == "run":
        return _exact_run(case, seed)
    if case["kind"] == "ensemble":
        return _exact_ensemble(case, seed)
    if case["kind"] in ("train", "grad"):
        return _exact_net(case, seed)
    return None  # the closure evaluates its network in bf16 with hardware tanh
