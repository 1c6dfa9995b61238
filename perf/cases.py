"""The framework's work as its users have it done, case by case, for measuring it.

A case is one pass of a program's main loop through the public entry points: a
stretch of imaginary- or real-time iterations with the energy and the state that
are read at its end (the cadence of ``solve()``), a parameter sweep, the
interface's single steps, the dipolar field on a caller's device buffers, the
warm-start network forward and its training gradients.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare(case, seed)`` is what a program has in hand before the pass,
``run(state)`` is the pass, ``work(case)`` is what a pass cannot do without, and
``exact(case, seed)`` is what ``run`` returns, computed in 64 bits by plain torch.
"""
import ctypes
import math

import numpy as np
import torch

# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # the smallest call: a short look at a small box with a ramped dipolar
        # strength; launches and host work count
        dict(name="rt_small", kind="real", nx=32, ny=32, nz=16, precision="c64", trap="HARMONIC", droplets=1,
             edd=0.75, ramp=True, before=0, iters=10),
        # plain imaginary-time ground state at 64 x 64 x 16: the stretch between two
        # checkpoints (every 100 iterations)
        dict(name="it_64", kind="imag", nx=64, ny=64, nz=16, precision="c64", trap="HARMONIC", droplets=1,
             edd=1.5, ramp=False, before=0, iters=100),
        # real time at the size of the full simulation, from an imaginary-time
        # state in the double well that is let go
        dict(name="rt_128", kind="real", nx=128, ny=128, nz=32, precision="c64", trap="DOUBLE", droplets=2,
             edd=1.5, ramp=False, before=100, iters=200),
        # the largest grid: droplets in a trap that binds along z only, dipolar strength ramped
        dict(name="rt_256_ramp", kind="real", nx=256, ny=256, nz=64, precision="c64", trap="FREE", droplets=9,
             edd=1.4, ramp=True, before=0, iters=100),
        # a box that is no power of two (odd factors on every axis), real time
        dict(name="rt_odd", kind="real", nx=100, ny=90, nz=30, precision="c64", trap="CYLINDRICAL", droplets=1,
             edd=1.2, ramp=False, before=20, iters=50),
        # complex128: the reference's own precision, imaginary and real time
        dict(name="it_c128", kind="imag", nx=64, ny=64, nz=16, precision="c128", trap="CYLINDRICAL", droplets=1,
             edd=1.5, ramp=False, before=0, iters=50),
        dict(name="rt_c128", kind="real", nx=128, ny=128, nz=32, precision="c128", trap="DOUBLE", droplets=2,
             edd=1.5, ramp=False, before=20, iters=20),
        # a parameter sweep of uneven grids, run as one batch
        dict(name="sweep", kind="sweep", members=24, iters=100),
        # the interface's steps one by one, as a host program's own loop calls them
        dict(name="virtuals", kind="virtuals", nx=64, ny=64, nz=16, precision="c64", trap="HARMONIC", droplets=1,
             edd=1.2, ramp=False, before=0, iters=10),
        # the dipolar field on a framework's own device buffers
        dict(name="field", kind="field", nx=128, ny=128, nz=32),
        # warm start: one prediction (a solve is about to start), and the gradients of one training batch
        dict(name="predict", kind="predict", nx=128, ny=128, nz=32, levels=4, batch=1),
        dict(name="train", kind="train", nx=128, ny=128, nz=32, levels=4, batch=8),
    ]


# the grids a sweep draws its members from, and the boxes programs use most
SWEEP_GRIDS = ((64, 64, 16), (96, 96, 24), (128, 128, 32))
POW2_XY, POW2_Z = (32, 64, 96, 128, 256), (8, 16, 24, 32, 64)


def _smooth(lo, hi):
    """Lengths in [lo, hi] with no prime factor above 7, as the transforms take them."""
    out = []
    for n in range(lo, hi + 1):
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m == 1:
            out.append(n)
    return out


def _pick(rng, lo, hi, values):
    """One of `values`, spread over the logarithm of [lo, hi]."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(values, key=lambda v: abs(v - x))


def draw(rng):
    kind = rng.choice(("imag", "imag", "real", "real", "real", "sweep", "virtuals", "field", "predict", "train"))
    if kind == "sweep":
        return dict(kind=kind, members=rng.randint(4, 24), iters=rng.randint(20, 100))
    if kind in ("predict", "train"):
        levels = rng.choice((3, 4))
        f = 1 << levels
        return dict(kind=kind, nx=f * rng.randint(2, 128 // f), ny=f * rng.randint(2, 128 // f),
                    nz=f * rng.randint(1, 32 // f), levels=levels, batch=rng.randint(1, 8))
    precision = "c64" if kind in ("virtuals", "field") or rng.random() < 0.7 else "c128"
    if rng.random() < 0.4:
        top = 256 if precision == "c64" and kind in ("imag", "real") else 128
        nx, ny = (rng.choice([v for v in POW2_XY if v <= top]) for _ in range(2))
        nz = rng.choice([v for v in POW2_Z if v <= (64 if top == 256 else 32)])
    else:
        xy, zz = _smooth(12, 144), _smooth(6, 40)
        nx, ny = (_pick(rng, 12, 144, xy) for _ in range(2))
        nz = _pick(rng, 6, 40, zz)
    if kind == "field":
        return dict(kind=kind, nx=min(nx, 128), ny=min(ny, 128), nz=min(nz, 32))
    n = nx * ny * nz
    most = 10 if kind == "virtuals" else max(5, min(100, int((1.2e8 if precision == "c64" else 1e7) / n)))
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=precision,
                trap=rng.choice(("HARMONIC", "CYLINDRICAL", "DOUBLE", "FREE")), droplets=rng.choice((1, 1, 2, 9)),
                edd=round(rng.uniform(0.7, 1.3), 3), ramp=kind == "real" and rng.random() < 0.4, before=0,
                iters=rng.randint(max(2, most // 4), most))


# ---------------------------------------------------------------------------
# physics of a case (atomic units)
# ---------------------------------------------------------------------------
NM, HZ, DA = 18.897261260649092, 4.1356e-12 / 27211.6, 1 / 0.000548579909


def _physics(case, seed):
    """The solve's parameters: those of the configurations, spread a little by the seed."""
    u = np.random.RandomState(seed % (1 << 31)).uniform(0.95, 1.05, 8)
    p = dict(nx=case["nx"], ny=case["ny"], nz=case["nz"], m=163.929 * DA, n_atoms=2e4 * u[0])
    # the box is at least 7.7 x 7.7 x 9.6 um, the spacing at least 120 x 120 x 600 nm
    p["dx"], p["dy"] = (max(120.0, 7680.0 / n) * NM for n in (p["nx"], p["ny"]))
    p["dz"] = max(600.0, 9600.0 / p["nz"]) * NM
    p["wx"], p["wy"], p["wz"] = 60 * HZ * u[1], 60 * HZ * u[1], 120 * HZ * u[2]
    if case["trap"] == "HARMONIC":
        p["wy"] *= u[3]
    p["edd0"] = case["edd"] * u[4]
    p["edd1"] = p["edd0"] * 1.1
    p["iter_real"] = 2000
    p["dt"], p["dtau"] = 1.00e10, 1.25e11
    p["cdd"] = 12.0 * math.pi * 131.0 / p["m"]
    p["shift"], p["width"] = 0.2 * (u[5] - 1.0), u[6]
    return p


def _contact(p, edd):
    a = 131.0 / edd
    return (4 * math.pi * a / p["m"],
            128.0 * math.sqrt(math.pi) * a ** 2.5 / 3.0 / p["m"] * (1.0 + 1.5 * edd ** 2))


def _axes(p, device):
    return [(torch.arange(p["n" + c], dtype=torch.float64, device=device) - p["n" + c] // 2) * p["d" + c] for c in "xyz"]


def _grid(p, device):
    x, y, z = _axes(p, device)
    return x[:, None, None], y[None, :, None], z[None, None, :]


def _trap(p, trap, device):
    x, y, z = _grid(p, device)
    m, dd = p["m"], 1500.0 * NM
    v = 0.5 * m * p["wz"] ** 2 * z ** 2 + 0 * x + 0 * y
    if trap in ("HARMONIC", "CYLINDRICAL"):
        v = v + 0.5 * m * (p["wx"] ** 2 * x ** 2 + p["wy"] ** 2 * y ** 2)
    elif trap == "DOUBLE":
        v = v + 0.5 * m * p["wy"] ** 2 * y ** 2 - 0.5 * m * p["wx"] ** 2 * x ** 2 + \
            0.25 * m * p["wx"] ** 2 / dd ** 2 * x ** 4
    elif trap == "DOUBLE_FREE":
        v = v + 0.5 * m * p["wy"] ** 2 * y ** 2 + 0.25 * m * p["wx"] ** 2 / dd ** 2 * x ** 4
    return v.contiguous()


def _start(p, droplets, device):
    """psi_0: Gaussian droplets on the interior, zero on the boundary, real."""
    x, y, z = _grid(p, device)
    lx, ly, lz = p["nx"] * p["dx"], p["ny"] * p["dy"], p["nz"] * p["dz"]
    w = (10.0 if droplets == 1 else 16.0) / p["width"]
    rows = int(round(math.sqrt(droplets))) if droplets > 2 else 1
    cols = droplets // rows
    out = torch.zeros(p["nx"], p["ny"], p["nz"], dtype=torch.float64, device=device)
    for i in range(cols):
        for j in range(rows):
            cx = lx * ((i + 1) / (cols + 1) - 0.5 + p["shift"])
            cy = ly * ((j + 1) / (rows + 1) - 0.5 - p["shift"])
            out += torch.exp(-0.5 * ((x - cx) * w / lx) ** 2) * torch.exp(-0.5 * ((y - cy) * w / ly) ** 2) * \
                torch.exp(-0.5 * (z * w / lz) ** 2)
    inside = torch.zeros_like(out)
    inside[1:-1, 1:-1, 1:-1] = 1.0
    return out * inside


def _json(p, case):
    """The solve as a gpe_params.json (file units)."""
    j = dict(nx=p["nx"], ny=p["ny"], nz=p["nz"], dx=p["dx"] / NM, dy=p["dy"] / NM, dz=p["dz"] / NM, m=163.929,
             n_atoms=p["n_atoms"], omega_x=p["wx"] / HZ, omega_y=p["wy"] / HZ, omega_z=p["wz"] / HZ, dd=1500.0,
             calc_strategy="IT" if case["kind"] in ("imag", "sweep") else "RT", init_strategy="GAUSS",
             pote_strategy="HARMONIC", iter_imag=1000, iter_real=p["iter_real"])
    if case.get("ramp"):
        j.update(edd_start=p["edd0"], edd_stop=p["edd1"])
    else:
        j.update(edd=p["edd0"])
    return j


def _member_cases(case, seed):
    """A sweep's members: the three grids in turn, dipolar strength and trap drawn from the sweep's ranges."""
    r = np.random.RandomState(seed % (1 << 31))
    out = []
    for m in range(case["members"]):
        g = SWEEP_GRIDS[m % 3]
        out.append((dict(kind="sweep", nx=g[0], ny=g[1], nz=g[2], trap="CYLINDRICAL", droplets=1,
                         edd=float(r.uniform(1.2, 1.8)), ramp=False), int(r.randint(1 << 30))))
    return out


def _features(case, seed):
    r = np.random.RandomState(seed % (1 << 31))
    return r.uniform(-1.0, 1.0, (case["batch"], 4)).astype(np.float32)


CHANNELS = {3: (16, 16, 8, 4), 4: (32, 32, 16, 8, 8)}
HIDDEN = {3: 64, 4: 256}


def _net_layout(case):
    """Sizes of the flat weight vector's pieces: dense, dense, then the convolutions."""
    ch, lv, hidden = CHANNELS[case["levels"]], case["levels"], HIDDEN[case["levels"]]
    g0 = [case[a] >> lv for a in ("nx", "ny", "nz")]
    latent = ch[0] * g0[0] * g0[1] * g0[2]
    layers = [(ch[s], ch[s + 1] if s < lv else 1) for s in range(lv + 1)]
    return ch, hidden, g0, latent, layers


def _net_weights(case, seed):
    """Fan-in scaled weights, small biases (a network at the start of its training)."""
    ch, hidden, g0, latent, layers = _net_layout(case)
    r = np.random.RandomState((seed + 7) % (1 << 31))
    parts = []
    for out, fan in [(hidden, 4), (latent, hidden)] + [(o, i * 27) for i, o in layers]:
        parts += [r.uniform(-1, 1, out * fan) * math.sqrt(3.0 / fan), r.uniform(-0.05, 0.05, out)]
    return np.concatenate(parts).astype(np.float32)


def _net_targets(case, seed, device):
    """Amplitudes of mean square 1: one Gaussian droplet a sample, its place and width from the seed."""
    r = np.random.RandomState((seed + 3) % (1 << 31))
    out = []
    for _ in range(case["batch"]):
        t = 1.0
        for n, shape in ((case["nx"], (-1, 1, 1)), (case["ny"], (1, -1, 1)), (case["nz"], (1, 1, -1))):
            x = (torch.arange(n, dtype=torch.float64, device=device) - n / 2 - r.uniform(-0.1, 0.1) * n) / n
            t = t * torch.exp(-0.5 * (x * r.uniform(6, 12)) ** 2).reshape(shape)
        out.append((t / t.square().mean().sqrt()).reshape(-1))
    return torch.stack(out).to(torch.float32)


def _field_psi(case, seed, device):
    p = _physics(dict(case, trap="HARMONIC", edd=1.0), seed)
    psi = _start(p, 2, device)
    x, y, z = _grid(p, device)
    psi = psi / torch.sqrt(psi.square().sum() * p["dx"] * p["dy"] * p["dz"])
    turn = 2.0 * math.pi * (x / (p["nx"] * p["dx"]) + 2 * y / (p["ny"] * p["dy"]))
    return p, torch.polar(psi, turn + 0 * z).to(torch.complex64).contiguous()


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def _solver_state(case, seed):
    import gpesolver_b200 as G

    p = _physics(case, seed)
    s = G.B200GrossPitaevskiSolver(G.params_from_json(_json(p, case)), precision=case["precision"])
    s.load_pote(_trap(p, case["trap"], "cuda").cpu().numpy())
    s.load_buffer(_start(p, case["droplets"], "cuda").cpu().numpy().astype(np.complex128))
    if case["before"]:
        s.imag_steps(case["before"])
        if case["trap"] == "DOUBLE":
            s.load_pote(_trap(p, "DOUBLE_FREE", "cuda").cpu().numpy())
    s.calc_fi3d()
    # pinned, as a program that writes checkpoints keeps it
    buf = torch.empty(2 * s.n, dtype=torch.float64, pin_memory=True)
    # a complex64 solver's state is handed on in its own precision
    out = torch.empty(2 * s.n, dtype=torch.float32) if case["precision"] == "c64" else None
    return dict(case=case, solver=s, buf=buf, out=out, done=0)


def prepare(case, seed):
    if case["kind"] in ("imag", "real", "virtuals"):
        return _solver_state(case, seed)
    if case["kind"] == "sweep":
        import gpesolver_b200 as G

        members = [(c, _physics(c, s)) for c, s in _member_cases(case, seed)]
        b = G.B200Batch([G.params_from_json(_json(p, c)) for c, p in members])
        amps = []
        for (c, p), s in zip(members, b.members):
            s.load_pote(_trap(p, c["trap"], "cuda").cpu().numpy())
            s.load_buffer(_start(p, c["droplets"], "cuda").cpu().numpy().astype(np.complex128))
            amps.append(torch.empty(s.n, dtype=torch.float32, device="cuda"))
        return dict(case=case, batch=b, amps=amps)
    if case["kind"] == "field":
        p, psi = _field_psi(case, seed, "cuda")
        phi = torch.zeros(psi.numel(), dtype=torch.float32, device="cuda")
        return dict(case=case, p=p, psi=psi, phi=phi)
    from gpesolver_b200 import warmstart as W

    cfg = W.WarmConfig(nx=case["nx"], ny=case["ny"], nz=case["nz"], levels=case["levels"],
                       channels=CHANNELS[case["levels"]], hidden=HIDDEN[case["levels"]], max_batch=case["batch"])
    net = W.WarmStartNet(cfg)
    net.set_weights(_net_weights(case, seed))
    st = dict(case=case, net=net, x=_features(case, seed))
    if case["kind"] == "predict":
        st["amp"] = torch.empty(case["batch"], net.n_voxels, dtype=torch.float32, device="cuda")
    else:
        st["target"] = _net_targets(case, seed, "cuda")
    return st


def _state_out(st):
    """Energies and the state on the host, as at a checkpoint."""
    s, buf = st["solver"], st["buf"]
    s.export_async(buf.numpy())
    e = s.calc_energy()
    s.export_wait()
    if st["out"] is None:
        return dict(energy=np.array(e), psi=buf)
    return dict(energy=np.array(e, dtype=np.float32), psi=st["out"].copy_(buf))


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "imag":
        st["solver"].imag_steps(case["iters"])
        return _state_out(st)
    if kind == "real":
        st["solver"].real_steps(case["iters"], st["done"] % 2000)
        st["done"] += case["iters"]
        return _state_out(st)
    if kind == "virtuals":
        s = st["solver"]
        for _ in range(case["iters"]):
            s.imag_time_iter()
        for _ in range(case["iters"]):
            s.real_time_iter()
        return _state_out(st)
    if kind == "sweep":
        from gpesolver_b200 import capi

        st["batch"].imag_steps(case["iters"])
        energy = []
        for s, a in zip(st["batch"].members, st["amps"]):
            energy.append(s.calc_energy().e_total)
            capi.check(capi.lib().gpe_export_amplitude_device(s.handle, ctypes.c_void_p(a.data_ptr()), s.n))
        return dict(energy=np.array(energy, dtype=np.float32), amps=st["amps"])
    if kind == "field":
        from gpesolver_b200 import capi

        p = st["p"]
        capi.check(capi.lib().gpe_calc_fi3d_noalloc(
            ctypes.c_void_p(st["psi"].data_ptr()), ctypes.c_void_p(st["phi"].data_ptr()), p["nx"], p["ny"], p["nz"],
            p["dx"], p["dy"], p["dz"], p["n_atoms"], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return st["phi"]
    if kind == "predict":
        st["net"].forward(st["x"], st["amp"].data_ptr())
        return st["amp"]
    loss, grad = st["net"].gradients(st["x"], st["target"].data_ptr())
    return dict(loss=loss, grad=grad)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _field_flops(nx, ny, nz):
    """The dipolar convolution: pruned real transforms of the doubled box, there and back."""
    def line(n):
        return 5.0 * n * math.log2(n)

    one = nx * ny * 0.5 * line(2 * nz) + nx * (nz + 1) * line(2 * ny) + 2 * ny * (nz + 1) * line(2 * nx)
    return 2 * one + 6.0 * 4 * nx * ny * (nz + 1)


def _iter_work(nx, ny, nz, precision, real):
    """One iteration: psi read and written, the trap read; its transforms and its pointwise arithmetic."""
    n, w = nx * ny * nz, 4 if precision == "c64" else 8
    flops = _field_flops(nx, ny, nz) + 45.0 * n
    if real:
        flops += 2 * 5.0 * n * math.log2(n) + 8.0 * n
    return 5.0 * w * n, flops


def work(case):
    kind = case["kind"]
    if kind == "sweep":
        b = f = 0.0
        for c, _ in _member_cases(case, 0):
            x, y = _iter_work(c["nx"], c["ny"], c["nz"], "c64", False)
            n = c["nx"] * c["ny"] * c["nz"]
            b, f = b + case["iters"] * x + 16.0 * n + 12.0 * n, f + case["iters"] * y + 60.0 * n
        return {"bytes": b, "flops": f}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    if kind == "field":
        return {"bytes": 12.0 * n, "flops": _field_flops(nx, ny, nz)}
    if kind in ("predict", "train"):
        ch, hidden, g0, latent, layers = _net_layout(case)
        flops, acts, weights = 2.0 * hidden * (4 + latent), 0.0, hidden * 4 + latent * hidden
        for s, (i, o) in enumerate(layers):
            vox = g0[0] * g0[1] * g0[2] * 8 ** min(s + 1, case["levels"])
            flops += 2.0 * 27 * i * o * vox
            acts += 4.0 * o * vox
            weights += 27 * i * o
        b = case["batch"]
        if kind == "predict":
            return {"bytes": 2.0 * weights + 4.0 * n * b, "flops": flops * b}
        # the activations are written by the forward pass and read by the backward one
        return {"bytes": 6.0 * weights + (4.0 * n + 2 * acts) * b, "flops": 3 * flops * b}
    w = 4 if case["precision"] == "c64" else 8
    bi, fi = _iter_work(nx, ny, nz, case["precision"], False)
    br, fr = _iter_work(nx, ny, nz, case["precision"], True)
    k = case["iters"]
    b, f = {"imag": (bi, fi), "real": (br, fr), "virtuals": (bi + br, fi + fr)}[kind]
    # at the end psi, the trap and the field are read for the energy, psi is handed over as complex128
    return {"bytes": k * b + 4.0 * w * n + 16.0 * n, "flops": k * f + 60.0 * n}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
class _Exact:
    """The reference's iterations in FP64: Euler steps with a 7-point Laplacian
    in imaginary time, Strang splitting in real time, the dipolar field by a
    zero-padded convolution."""

    def __init__(self, p, case, device):
        self.p, self.ramp = p, case.get("ramp", False)
        self.V = _trap(p, case["trap"], device)
        self.dV = p["dx"] * p["dy"] * p["dz"]
        self.psi = _start(p, case["droplets"], device).to(torch.complex128)
        self.normalise()
        self.g, self.gamma = _contact(p, p["edd0"])
        k = []
        for c in "xyz":
            n = 2 * p["n" + c]
            k.append(2 * math.pi * torch.fft.fftfreq(n, p["d" + c], dtype=torch.float64, device=device))
        kz = k[2][: p["nz"] + 1].abs()
        k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + kz[None, None, :] ** 2
        k2[0, 0, 0] = 1.0
        self.vk = (kz ** 2)[None, None, :] / k2
        q = [2 * math.pi * torch.fft.fftfreq(p["n" + c], p["d" + c], dtype=torch.float64, device=device) for c in "xyz"]
        q2 = q[0][:, None, None] ** 2 + q[1][None, :, None] ** 2 + q[2][None, None, :] ** 2
        self.kin = torch.polar(torch.ones_like(q2), -p["dt"] / (2 * p["m"]) * q2)
        self.inside = torch.zeros_like(self.V, dtype=torch.bool)
        self.inside[1:-1, 1:-1, 1:-1] = True
        self.field()

    def normalise(self):
        self.psi = self.psi / torch.sqrt(self.psi.abs().square().sum() * self.dV)

    def field(self):
        p = self.p
        rho = p["n_atoms"] * self.psi.abs().square()
        s = (2 * p["nx"], 2 * p["ny"], 2 * p["nz"])
        r = torch.fft.irfftn(torch.fft.rfftn(rho, s=s) * self.vk, s=s)
        self.phi = r[: p["nx"], : p["ny"], : p["nz"]].contiguous()

    def nonlinear(self):
        p = self.p
        d = self.psi.abs().square()
        return self.V + p["cdd"] * self.phi + (self.g - p["cdd"] / 3) * p["n_atoms"] * d + \
            self.gamma * p["n_atoms"] ** 1.5 * d * torch.sqrt(d)

    def laplacian(self):
        p, f = self.p, self.psi
        c = f[1:-1, 1:-1, 1:-1]
        return (f[2:, 1:-1, 1:-1] + f[:-2, 1:-1, 1:-1] - 2 * c) / p["dx"] ** 2 + \
            (f[1:-1, 2:, 1:-1] + f[1:-1, :-2, 1:-1] - 2 * c) / p["dy"] ** 2 + \
            (f[1:-1, 1:-1, 2:] + f[1:-1, 1:-1, :-2] - 2 * c) / p["dz"] ** 2

    def imag(self, k):
        for _ in range(k):
            self.field()
            h = (self.nonlinear() * self.psi)[1:-1, 1:-1, 1:-1] - 0.5 / self.p["m"] * self.laplacian()
            new = torch.zeros_like(self.psi)
            new[1:-1, 1:-1, 1:-1] = self.psi[1:-1, 1:-1, 1:-1] - self.p["dtau"] * h
            self.psi = new
            self.normalise()

    def half(self):
        t = torch.where(self.inside, -0.5 * self.p["dt"] * self.nonlinear(), torch.zeros_like(self.V))
        self.psi = self.psi * torch.polar(torch.ones_like(t), t)

    def real(self, k):
        p = self.p
        for it in range(k):
            if self.ramp:
                self.g, self.gamma = _contact(p, p["edd0"] + (p["edd1"] - p["edd0"]) * it / p["iter_real"])
            self.half()
            self.field()
            self.psi = torch.fft.ifftn(torch.fft.fftn(self.psi) * self.kin)
            self.half()

    def energy(self):
        p = self.p
        f, w, i = self.psi[1:-1, 1:-1, 1:-1], p["n_atoms"], (slice(1, -1),) * 3
        d = f.abs().square()
        e = [-(self.laplacian() * f.conj()).real.sum() * self.dV / (2 * p["m"]) * w,
             (self.V[i] * d).sum() * self.dV * w,
             0.5 * self.g * d.square().sum() * self.dV * w ** 2,
             (0.5 * p["cdd"] * self.phi[i] * d * w - p["cdd"] / 6.0 * d.square() * w ** 2).sum() * self.dV,
             0.4 * self.gamma * (d.square() * d.sqrt()).sum() * self.dV * w ** 2.5]
        e = [float(v) for v in e]
        return e + [sum(e)]


def _bf16(w):
    return torch.from_numpy(w).to(torch.bfloat16).to(torch.float64)


def _net_exact(case, seed, device):
    ch, hidden, g0, latent, layers = _net_layout(case)
    w = _bf16(_net_weights(case, seed)).to(device).requires_grad_(case["kind"] == "train")
    x = torch.from_numpy(_features(case, seed)).to(torch.float64).to(device)
    at = 0

    def take(*shape):
        nonlocal at
        n = math.prod(shape)
        at += n
        return w[at - n:at].reshape(shape)

    f = torch.nn.functional
    h = f.silu(f.linear(x, take(hidden, 4), take(hidden)))
    h = f.silu(f.linear(h, take(latent, hidden), take(latent))).reshape(-1, ch[0], *g0)
    for s, (i, o) in enumerate(layers):
        last = s == case["levels"]
        if not last:
            h = h.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)
        k, b = take(o, i, 3, 3, 3), take(o)
        q = f.pad(h, (1, 1, 1, 1, 1, 1))
        y = b.reshape(1, o, 1, 1, 1)
        for a in range(3):
            for c in range(3):
                for e in range(3):
                    part = q[:, :, a:a + h.shape[2], c:c + h.shape[3], e:e + h.shape[4]]
                    y = y + torch.einsum("oi,bixyz->boxyz", k[:, :, a, c, e], part)
        h = y if last else f.silu(y)
    out = h.reshape(x.shape[0], -1)
    if case["kind"] == "predict":
        return out
    loss = (out - _net_targets(case, seed, device).to(torch.float64)).square().mean()
    loss.backward()
    return dict(loss=float(loss.detach()), grad=w.grad)


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind in ("predict", "train"):
        return _net_exact(case, seed, device)
    if kind == "field":
        p, psi = _field_psi(case, seed, device)
        e = _Exact(p, dict(case, trap="FREE", droplets=1, edd=1.0), device)
        e.psi = psi.to(torch.complex128)
        e.field()
        return e.phi.reshape(-1)
    if kind == "sweep":
        energy, amps = [], []
        for c, s in _member_cases(case, seed):
            e = _Exact(_physics(c, s), c, device)
            e.imag(case["iters"])
            energy.append(e.energy()[5])
            amps.append(e.psi.abs().reshape(-1))
        return dict(energy=np.array(energy), amps=amps)
    e = _Exact(_physics(case, seed), case, device)
    if kind in ("imag", "virtuals"):
        e.imag(case["iters"])
    if kind == "real":
        if case["before"]:
            e.imag(case["before"])
            if case["trap"] == "DOUBLE":
                e.V = _trap(e.p, "DOUBLE_FREE", device)
        e.field()
    if kind in ("real", "virtuals"):
        e.real(case["iters"])
    return dict(energy=np.array(e.energy()), psi=torch.view_as_real(e.psi).reshape(-1))
