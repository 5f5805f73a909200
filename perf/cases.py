"""The work that is timed when a kernel changes: what a user's program asks
of the propagator, the batched sweep and the learned guess, through their
public entry points.

A propagator case is one monitoring interval of the reference's time loop
(fortress_b200.driver.run): `steps` split steps, then NORMC, ENERGY/RAD, in
imaginary time CONV, and the state read back in device memory.  The state
goes on from pass to pass as in that loop.  Sizes, spacings, time steps and
couplings are those of the benchmark workloads, the published 1D input, the
parity tests' configurations and the kernel tour; draw() spreads them.

The FP32 bulk path promises single precision, so its results are returned
in single precision; CONV is left to the FP64 path there, since the FP32
path's one-step difference is at its rounding floor.
"""
import math

import numpy as np
import torch

from fortress_b200 import Propagator, RunConfig
from fortress_b200.batch import Batch
from fortress_b200.fno import FNO, init_params, input_channels, normalise_params

DEV = "cuda"


# ------------------------------------------------------------------- cases
def _propagation(name, cfg, steps, precision="fp64"):
    p = cfg.params(precision)
    n, d, g = list(p["n"]) + [1] * 3, list(p["d"]) + [1.0] * 3, list(p["gamma"]) + [0.0] * 3
    return dict(name=name, kind="propagate", dim=p["dim"], spin=p["spin"], nx=n[0], ny=n[1], nz=n[2], dx=d[0],
                dy=d[1], dz=d[2], dt=p["dt"], imag=bool(p["imag_time"]), tau0=p["tau"][0], tau1=p["tau"][1],
                tau2=p["tau"][2], gx=g[0], gy=g[1], gz=g[2], ay=p["alpha"][1], az=p["alpha"][2], mag=p["mag"],
                precision=precision, steps=steps)


def listed():
    box = dict(dim=3, spin=1, n=(256, 256, 256), d=(0.1, 0.1, 0.1), dt=1e-3, mass=87.0, a=(101.8, 100.4, 0.0),
               natoms=100000, nu=(50.0, 50.0, 50.0), gamma=(0.5, 0.5, 0.5), switch_im=1)
    line = dict(dim=1, spin=2, mass=23.0, a=(34.9, 45.8, 64.5), natoms=10000, nu=(20.0, 400.0, 400.0),
                gamma=(0.5, 0.0, 0.0))
    plane = dict(dim=2, spin=2, mass=87.0, a=(87.93, 91.28, 99.18), natoms=50000, nu=(20.0, 20.0, 500.0))
    return [
        # the smallest call: a short q1D line watched every 10 steps
        _propagation("q1d_256_spin1", RunConfig(dim=1, spin=1, n=(256, 1, 1), d=(0.1, 1.0, 1.0), dt=5e-4, mass=23.0,
                                                a=(50.0, 55.01, 0.0), natoms=10000, nu=(20.0, 400.0, 400.0),
                                                switch_im=1, gamma=(0.5, 0.0, 0.0)), 10),
        # the reference's published run: one of its STP = 400 intervals
        _propagation("q1d_2048_spin2", RunConfig(n=(2048, 1, 1), d=(0.05, 1.0, 1.0), dt=1.25e-4, switch_im=1, **line), 400),
        # a long q1D line in real time
        _propagation("q1d_8192_spin2_real", RunConfig(n=(8192, 1, 1), d=(0.02, 1.0, 1.0), dt=1e-4, switch_im=0, **line), 100),
        # the q2D spin-2 quench in real time
        _propagation("q2d_512_spin2_real", RunConfig(n=(512, 512, 1), d=(0.05, 0.05, 1.0), dt=1e-4, switch_im=0,
                                                     gamma=(1.2, 1.0, 0.0), **plane), 40),
        # a q2D ground state without SO coupling at an imposed magnetisation,
        # on a grid of no size-specialised length
        _propagation("q2d_320x240_spin1_mag", RunConfig(dim=2, spin=1, n=(320, 240, 1), d=(0.08, 0.1, 1.0), dt=5e-4,
                                                        mass=87.0, a=(101.8, 100.4, 0.0), natoms=50000,
                                                        nu=(20.0, 24.0, 500.0), switch_im=1, mag=0.3), 40),
        # 3D SO-coupled ground state, the benchmark's grid, both precisions
        _propagation("box_256_spin1", RunConfig(**box), 10),
        _propagation("box_256_spin1_fp32", RunConfig(**box), 10, "fp32"),
        # a ragged 3D spin-2 grid in real time
        _propagation("box_96x80x120_spin2_real", RunConfig(dim=3, spin=2, n=(96, 80, 120), d=(0.25, 0.3, 0.2), dt=5e-4,
                                                           mass=87.0, a=(87.93, 91.28, 99.18), natoms=50000,
                                                           nu=(50.0, 60.0, 50.0), switch_im=0, gamma=(0.5, 0.3, 0.4)), 8),
        # the phase-diagram sweep, in the two launch modes its autotuner picks from
        dict(name="sweep_64_grouped_fp32", kind="sweep", count=64, mode="grouped", precision="fp32", steps=32),
        dict(name="sweep_64_persistent_fp32", kind="sweep", count=64, mode="persistent", precision="fp32", steps=32),
        # learned guess: one training step, and guesses for a block of points
        dict(name="guess_train_64_b64", kind="train", n=64, batch=64),
        dict(name="guess_infer_256_b8", kind="infer", n=256, batch=8),
    ]


_SIZES = sorted(n for a in range(1, 14) for b in range(5) for c in range(4)
                if 16 <= (n := 2 ** a * 3 ** b * 5 ** c) <= 8192)
_FAST = (128, 192, 256, 384, 512)


def draw(rng):
    kind = rng.choice(("line", "plane", "plane", "box", "box", "sweep", "train", "infer"))

    def size(lo, hi):
        x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        return min((n for n in _SIZES if lo <= n <= hi), key=lambda n: abs(math.log(n / x)))

    precision = rng.choice(("fp64", "fp64", "fp32"))
    if kind == "sweep":
        return dict(kind="sweep", count=rng.randint(4, 64), mode=rng.choice(("branches", "grouped", "persistent")),
                    precision=precision, steps=rng.choice((8, 16, 32)))
    if kind == "train":
        n = size(32, 128)
        return dict(kind="train", n=n, batch=rng.randint(1, max(1, 262144 // (n * n))))
    if kind == "infer":
        n = size(32, 256)
        return dict(kind="infer", n=n, batch=rng.randint(1, max(1, min(64, 524288 // (n * n)))))
    dim = {"line": 1, "plane": 2, "box": 3}[kind]
    lo, hi = {1: (64, 8192), 2: (32, 512), 3: (16, 256)}[dim]
    # half of the 2D and 3D axes at the lengths of the compiled kernels
    n = [rng.choice([f for f in _FAST if f <= hi]) if dim > 1 and rng.random() < 0.5 else size(lo, hi)
         for _ in range(dim)] + [1] * (3 - dim)
    d = [min(25.6 / m, 0.4) if dim > 1 else rng.choice((0.05, 0.1)) for m in n[:dim]] + [1.0] * (3 - dim)
    spin = rng.choice((1, 2))
    imag = rng.random() < 0.6
    soc = rng.random() < 0.8
    g = [round(rng.uniform(0.1, 1.5), 3) if soc and a < dim else 0.0 for a in range(3)]
    c0 = rng.uniform(100.0, 2000.0)
    # a drawn case costs no more than ten steps of the largest box
    most = 10 * 3 * 256 ** 3 // (n[0] * n[1] * n[2] * (2 * spin + 1))
    steps = min(rng.choice({1: (1, 10, 100, 400), 2: (1, 10, 40, 100), 3: (1, 2, 5, 10)}[dim]), max(1, most))
    return dict(kind="propagate", dim=dim, spin=spin, nx=n[0], ny=n[1], nz=n[2], dx=d[0], dy=d[1], dz=d[2],
                dt=5e-4 if imag else 1e-4, imag=imag, tau0=2.0 * c0, tau1=2.0 * c0 * rng.uniform(-0.05, 0.05),
                tau2=2.0 * c0 * rng.uniform(-0.05, 0.05) if spin == 2 else 0.0, gx=g[0], gy=g[1], gz=g[2],
                ay=round(rng.uniform(1.0, 2.0), 3), az=round(rng.uniform(1.0, 2.0), 3),
                mag=0.0 if soc or not imag else round(rng.uniform(-0.5, 0.5), 3), precision=precision, steps=steps)


# ------------------------------------------------------------------ inputs
def _params(c):
    dim = c["dim"]
    return dict(dim=dim, spin=c["spin"], n=(c["nx"], c["ny"], c["nz"])[:dim], d=(c["dx"], c["dy"], c["dz"])[:dim],
                dt=c["dt"], imag_time=c["imag"], tau=(c["tau0"], c["tau1"], c["tau2"]),
                gamma=(c["gx"], c["gy"], c["gz"])[:dim], alpha=(1.0, c["ay"], c["az"]), mag=c["mag"],
                precision=c["precision"])


def _axis(n, d, a):
    """Grid points of one axis, shaped to broadcast over [z][y][x]."""
    x = (-1.0 + 2.0 * torch.arange(n, dtype=torch.float64, device=DEV) / n) * n * d / 2.0 if n > 1 else torch.zeros(1, dtype=torch.float64, device=DEV)
    return x.reshape([-1 if q == a else 1 for q in (2, 1, 0)])


def _start(p, seed):
    """A Gaussian of the trap's widths in every component, with 5 % of
    amplitude noise and a smooth phase of its own per component: [m][z][y][x]."""
    n, d = list(p["n"]) + [1] * (3 - p["dim"]), list(p["d"]) + [1.0] * (3 - p["dim"])
    r = torch.Generator(DEV).manual_seed(int(seed))
    x, y, z = (_axis(n[a], d[a], a) for a in range(3))
    al = p["alpha"]
    # as wide as the repulsion makes the cloud, within the box
    w = min(1.0 + 0.15 * p["tau"][0] ** (1.0 / (2 + p["dim"])), 0.15 * min(m * e for m, e in zip(p["n"], p["d"])))
    gauss = torch.exp(-(al[0] * x * x + al[1] * y * y + al[2] * z * z) / (2.0 * w * w))
    ms = 2 * p["spin"] + 1
    phi = torch.empty((ms, n[2], n[1], n[0]), dtype=torch.complex128, device=DEV)
    for m in range(ms):
        u = torch.rand(5, generator=r, dtype=torch.float64, device=DEV) - 0.5
        amp = gauss * (1.0 + 0.05 * torch.rand(gauss.shape, generator=r, dtype=torch.float64, device=DEV)) * (1.0 + u[4])
        phi[m] = torch.polar(amp, u[0] * x + u[1] * y + u[2] * z + 3.0 * u[3] + 0.0 * amp)
    return phi


def _sweep(c, seed):
    """Instances of the phase-diagram box: q2D spin-1 on sizes from
    {128, 192, 256, 384, 512}^2, in equal shares."""
    r = np.random.default_rng(seed)
    out = []
    for k in range(c["count"]):
        g = r.uniform(0, 2, 2)
        c0 = r.uniform(100, 2000)
        n = _FAST[k % 5]
        out.append(dict(dim=2, spin=1, n=(n, n), d=(0.1, 0.1), dt=5e-4, imag_time=True,
                        tau=(2 * c0, 2 * c0 * r.uniform(-0.05, 0.05), 0.0), gamma=(float(g[0]), float(g[1])),
                        alpha=(1.0, r.uniform(1, 2), 1.0), precision=c["precision"]))
    return out


def _points(c, seed):
    """Network inputs [7][B][n][n] (host) of seeded points of the sweep box."""
    r = np.random.default_rng(seed)
    pts = [normalise_params(*r.uniform(0, 2, 2), r.uniform(100, 2000), r.uniform(-0.05, 0.05), r.uniform(1, 2))
           for _ in range(c["batch"])]
    return input_channels(np.array(pts), c["n"])


def _weights(seed):
    """Initial weights, with biases that are not zero."""
    r = np.random.default_rng(seed + 2)
    w = init_params(seed=seed)
    for k in ("bP", "c1", "c2", "b0", "b1", "b2", "b3"):
        w[k] = 0.1 * r.standard_normal(w[k].shape)
    return w


def _training(c, seed):
    """Inputs and targets on the device, weights, and Adam moments of a run
    that is under way."""
    r = np.random.default_rng(seed + 1)
    a = torch.from_numpy(_points(c, seed)).to(DEV).reshape(7, -1)
    x = torch.linspace(-1, 1, c["n"], device=DEV)
    w = torch.tensor(r.uniform(2, 6, (6, c["batch"], 1, 1)), dtype=torch.float32, device=DEV)
    tgt = torch.exp(-w * (x[:, None] ** 2 + x[None, :] ** 2)) * torch.tensor(
        r.uniform(-1, 1, (6, c["batch"], 1, 1)), dtype=torch.float32, device=DEV)
    weights = _weights(seed)
    m = {k: 1e-3 * r.standard_normal(v.shape) for k, v in weights.items()}
    v = {k: 1e-4 * r.uniform(0.5, 2, v.shape) for k, v in weights.items()}
    return a, tgt.reshape(6, -1).contiguous(), weights, m, v


_T, _LR = 100, 1e-3


def _device_layout(v):
    return torch.tensor(np.ascontiguousarray(np.transpose(v, (2, 3, 0, 1)) if v.ndim == 4 else v), dtype=torch.float64,
                        device=DEV)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "propagate":
        p = _params(case)
        phi = _start(p, seed)
        prop = Propagator(**p)
        torch.cuda.synchronize()
        prop.set_state_device(phi.data_ptr())
        prop.normt()
        return dict(case=case, prop=prop, out=torch.empty_like(phi))
    if kind == "sweep":
        insts = _sweep(case, seed)
        phis = [_start(p, seed + 1000 * k) for k, p in enumerate(insts)]
        b = Batch(insts)
        torch.cuda.synchronize()
        for q, phi in zip(b.props, phis):
            q.set_state_device(phi.data_ptr())
            q.normt()
        b.mode(grouped=case["mode"] == "grouped", persistent=case["mode"] == "persistent")
        if case["mode"] == "persistent":
            b.variant(2)
        b.config(min(case["count"], 64), 8)
        flat = torch.empty(sum(x.numel() for x in phis), dtype=torch.complex128, device=DEV)
        at = np.cumsum([0] + [x.numel() for x in phis])
        return dict(case=case, batch=b, out=flat, at=at)
    if kind == "train":
        a, tgt, weights, m, v = _training(case, seed)
        net = FNO(case["n"], case["batch"], params=weights)
        net.a.copy_(a)
        for k in net.p:
            net.m[k].copy_(_device_layout(m[k]))
            net.v[k].copy_(_device_layout(v[k]))
        net.t = _T
        return dict(case=case, net=net, tgt=tgt)
    net = FNO(case["n"], case["batch"], params=_weights(seed))
    return dict(case=case, net=net, a=_points(case, seed))


# -------------------------------------------------------------------- pass
def run(s):
    c = s["case"]
    if c["kind"] == "propagate":
        prop = s["prop"]
        prop.step(c["steps"])
        res = {"norms": prop.normc()}
        en, mu, mz, rms = prop.observables()
        res["observables"] = np.concatenate([[en, mz], mu, rms])
        fp64 = c["precision"] == "fp64"
        if c["imag"] and fp64:
            res["conv"] = prop.conv()
        prop.get_state_device(s["out"].data_ptr())
        res["state"] = s["out"]
        return res if fp64 else _single(res)
    if c["kind"] == "sweep":
        b = s["batch"]
        b.step(c["steps"])
        obs = b.observables(with_conv=False)
        for i in range(len(b)):
            b[i].get_state_device(s["out"].data_ptr() + 16 * int(s["at"][i]))
        res = {"observables": np.concatenate([np.concatenate([[o["en"], o["mz"]], o["mu"], o["rms"], o["norm"]]) for o in obs]),
               "state": s["out"]}
        return res if c["precision"] == "fp64" else _single(res)
    net = s["net"]
    if c["kind"] == "infer":
        return {"out": net.forward(s["a"])}
    out = net.forward()
    loss = net.loss(s["tgt"])
    net.backward()
    net.adam(lr=_LR)
    return {"out": out, "loss": loss.float(), "grads": dict(net.g), "weights": dict(net.p)}


def _single(res):
    return {k: v.to(torch.complex64) if isinstance(v, torch.Tensor) else v.astype(np.float32) for k, v in res.items()}


# -------------------------------------------------------------------- work
def _spinor_work(npts, ms, steps, size):
    """A step depends on all of the one before (transforms, norm), so a
    spinor larger than the 126 MB L2 is read and written once per step; a
    smaller one once per pass.  flops: two transforms, KE and SO coupling,
    spin exchange (closed form for spin 1; two coupling sets and about
    eight products with a 5 x 5 matrix for spin 2), SP, norms."""
    state = npts * ms * size
    point = 10.0 * math.log2(npts) * ms + 8.0 * ms * ms + 10.0 * ms + (90.0 if ms == 3 else 1500.0) + 20.0 * ms
    return 2.0 * state * (steps if state > 126e6 else 1), point * npts * steps


def work(case):
    kind = case["kind"]
    if kind in ("propagate", "sweep"):
        size = 16 if case["precision"] == "fp64" else 8
        if kind == "propagate":
            b, f = _spinor_work(case["nx"] * case["ny"] * case["nz"], 2 * case["spin"] + 1, case["steps"], size)
            return {"bytes": b, "flops": f}
        each = [_spinor_work(_FAST[k % 5] ** 2, 3, case["steps"], size) for k in range(case["count"])]
        total = sum(b for b, _ in each)
        return {"bytes": total * (case["steps"] if total / 2 > 126e6 else 1), "flops": sum(f for _, f in each)}
    # width 32, 16 modes, 4 layers, 7 -> 32 -> ... -> 128 -> 6 channels
    n, pts = case["n"], case["n"] ** 2 * case["batch"]
    dense = 2.0 * pts * (7 * 32 + 4 * 32 * 32 + 32 * 128 + 128 * 6)
    spec = 4 * case["batch"] * 32 * 2.0 * (4 * n * n * 16 + 8 * n * 32 * 16) + 4 * 512 * 2.0 * 64 * 64 * case["batch"]
    weights = 4.0 * (4 * 2 * 32 * 32 * 32 * 16 + 4 * 32 * 32 + 7 * 32 + 32 * 128 + 128 * 6)
    if kind == "infer":
        return {"bytes": weights + 4.0 * pts * (7 + 6), "flops": dense + spec}
    # backward: input and weight gradients; weights, moments and gradients
    return {"bytes": 7 * weights + 4.0 * pts * (7 + 6 + 6), "flops": 3 * (dense + spec)}


# ------------------------------------------------- the same in 64-bit torch
def _simpson(n, d):
    """Node weights of the composite rule: Simpson 1/3 on the first n-3
    nodes, 3/8 on the last four."""
    if n == 1:
        return torch.ones(1, dtype=torch.float64, device=DEV)
    w = np.zeros(n)
    w[0] = 1 / 3
    w[1:n - 4:2] = 4 / 3
    w[2:n - 5:2] = 2 / 3
    w[n - 4] = 1 / 3 + 3 / 8
    w[n - 3] = w[n - 2] = 9 / 8
    w[n - 1] = 3 / 8
    return torch.tensor(w * d, dtype=torch.float64, device=DEV)


def _couplings(v, t1, t2):
    s = math.sqrt(1.5)
    z = [v[m].conj() * v[m + 1] for m in range(4)]
    f = 2 * (z[0] + s * z[1] + s * z[2] + z[3]).conj()
    a, b = 0.4 * t2, 0.2 * t2
    return {(0, 1): t1 * f - a * v[3] * v[4].conj(), (0, 2): b * v[2] * v[4].conj(),
            (1, 2): s * t1 * f - b * v[2] * v[3].conj(), (2, 3): s * t1 * f - b * v[1] * v[2].conj(),
            (2, 4): b * v[0] * v[2].conj(), (3, 4): t1 * f - a * v[0] * v[1].conj()}


def _apply(h, v):
    out = [torch.zeros_like(x) for x in v]
    for (i, j), c in h.items():
        out[i] += c * v[j]
        out[j] += c.conj() * v[i]
    return out


class _Exact:
    """The split step and the observables in complex128 torch."""

    def __init__(self, p, phi):
        self.p, self.ms, self.S = p, 2 * p["spin"] + 1, p["spin"]
        dim = p["dim"]
        self.n = list(p["n"]) + [1] * (3 - dim)
        self.d = list(p["d"]) + [1.0] * (3 - dim)
        self.g = list(p["gamma"]) + [0.0] * (3 - dim)
        shape = lambda t, a: t.reshape([-1 if q == a else 1 for q in (2, 1, 0)])  # noqa: E731
        self.w = [shape(_simpson(self.n[a], self.d[a]), a) for a in range(3)]
        self.x = [_axis(self.n[a], self.d[a], a) for a in range(3)]
        self.k = [shape(2 * math.pi * torch.fft.fftfreq(self.n[a], self.d[a], dtype=torch.float64, device=DEV).abs()
                        * torch.where(torch.arange(self.n[a], device=DEV) <= self.n[a] // 2, 1.0, -1.0), a)
                  if self.n[a] > 1 else torch.zeros(1, 1, 1, dtype=torch.float64, device=DEV) for a in range(3)]
        self.V = sum((p["alpha"][a] * self.x[a]) ** 2 for a in range(dim))
        self.cdt = -1j * p["dt"] if p["imag_time"] else p["dt"] + 0j
        self.project = p["imag_time"] and not any(abs(v) > 1e-40 for v in p["gamma"])
        self.sig = (20.0, 20.0)
        self.v = [phi[m] for m in range(self.ms)]
        self._scale([1.0 / math.sqrt(sum(self.norms()))] * self.ms)

    def _sum(self, f):
        return float((f * self.w[0] * self.w[1] * self.w[2]).sum())

    def _scale(self, s):
        for m in range(self.ms):
            self.v[m] = self.v[m] * s[m]

    def norms(self):
        return [self._sum(x.abs() ** 2) for x in self.v]

    def phase(self, e):
        return torch.exp(-1j * self.cdt * e)

    def _fourier(self):
        kx, ky, kz = self.k
        ms, S, (gx, gy, gz) = self.ms, self.S, self.g
        v = [torch.fft.fftn(x) for x in self.v]
        for m in range(ms):
            v[m] = v[m] * self.phase(kx ** 2 + ky ** 2 + kz ** 2 - 2 * (m - S) * gz * kz)
        h, q = math.sqrt(0.5), math.sqrt(0.375)
        a0 = ([[0.5, -h, 0.5], [-h, 0, h], [0.5, h, 0.5]] if ms == 3 else
              [[0.25, -0.5, q, -0.5, 0.25], [-0.5, 0.5, 0, -0.5, 0.5], [q, 0, -0.5, 0, q], [-0.5, -0.5, 0, 0.5, 0.5],
               [0.25, 0.5, q, 0.5, 0.25]])
        if self.p["dim"] == 1:
            al, beta = 2 * gx * kx, torch.zeros_like(kx)
        else:
            al, beta = 2 * torch.sqrt((gx * kx) ** 2 + (gy * ky) ** 2), torch.atan2(gy * ky, gx * kx)
        e = [torch.exp(-1j * (S - m) * beta) for m in range(ms)]
        w = [e[m].conj() * v[m] for m in range(ms)]
        u = [self.phase((r - S) * al) * sum(a0[j][r] * w[j] for j in range(ms)) for r in range(ms)]
        self.v = [torch.fft.ifftn(e[r] * sum(a0[r][j] * u[j] for j in range(ms))) for r in range(ms)]

    def _exchange(self):
        v, dt, imag = self.v, self.p["dt"], self.p["imag_time"]
        t1, t2 = self.p["tau"][1:]
        if self.ms == 3:
            A, B = t1 * v[1] * v[2].conj(), t1 * v[1] * v[0].conj()
            r2 = A.abs() ** 2 + B.abs() ** 2
            x = dt * torch.sqrt(r2)
            y = torch.where(x > 1e-6, x, torch.ones_like(x))
            if imag:
                f = torch.where(x > 1e-6, torch.sinh(y) / y, 1 + x * x / 6)
                g = torch.where(x > 1e-6, 2 * (torch.sinh(y / 2) / y) ** 2, 0.5 + x * x / 24)
                kf, dc = -dt * f, dt * dt * g
            else:
                f = torch.where(x > 1e-6, torch.sin(y) / y, 1 - x * x / 6)
                g = torch.where(x > 1e-6, 2 * (torch.sin(y / 2) / y) ** 2, 0.5 - x * x / 24)
                kf, dc = -1j * dt * f, -dt * dt * g
            h = {(0, 1): A, (1, 2): B.conj()}
            hv = _apply(h, v)
            hhv = _apply(h, hv)
            self.v = [v[m] + kf * hv[m] + dc * hhv[m] for m in range(3)]
            return
        c = _couplings(v, t1, t2)
        half = 0.5 if self.p["dim"] == 1 else 1.0
        hv = _apply(c, v)
        c1 = _couplings([v[m] - 1j * self.cdt * half * hv[m] for m in range(5)], t1, t2)
        mean = {q: (0.5 * (c[q] + c1[q])).reshape(-1) for q in c}
        flat = torch.stack([x.reshape(-1) for x in v], 1)
        for at in range(0, len(flat), 1 << 20):
            part = slice(at, at + (1 << 20))
            H = torch.zeros(len(flat[part]), 5, 5, dtype=torch.complex128, device=DEV)
            for (i, j), z in mean.items():
                H[:, i, j], H[:, j, i] = z[part], z[part].conj()
            flat[part] = (torch.matrix_exp(-1j * self.cdt * H) @ flat[part][:, :, None])[:, :, 0]
        self.v = [flat[:, m].reshape(v[0].shape) for m in range(5)]

    def _spin_density(self, a):
        return sum((self.S - m) * a[m] for m in range(self.ms))

    def _density(self):
        t0, t1, t2 = self.p["tau"]
        a = [x.abs() ** 2 for x in self.v]
        rho = sum(a)
        if self.ms == 3:
            b = [t1 * (a[0] + a[1] - a[2]), t1 * (a[0] + a[2]), t1 * (a[2] + a[1] - a[0])]
        else:
            fz = self._spin_density(a)
            b = [(2 - m) * t1 * fz + (0.2 if m == 2 else 0.4) * t2 * a[4 - m] for m in range(5)]
        return a, rho, [self.V + t0 * rho + b[m] for m in range(self.ms)]

    def step(self):
        self._fourier()
        self._exchange()
        for m, t in enumerate(self._density()[2]):
            self.v[m] = self.v[m] * self.phase(t)
        n = self.norms()
        if self.p["imag_time"]:
            s = self._projection(n) if self.project else [1.0] * self.ms
            tot = math.sqrt(sum(s[m] ** 2 * n[m] for m in range(self.ms)))
            self._scale([x / tot for x in s])
        return n

    def _projection(self, n):
        mag, dt = self.p["mag"], self.p["dt"]
        if self.ms == 3:
            s0 = math.sqrt(1 - mag ** 2) / math.sqrt(n[1] + math.sqrt(4 * (1 - mag ** 2) * n[0] * n[2] + (mag * n[1]) ** 2))
            return [math.sqrt(1 + mag - s0 ** 2 * n[1]) / math.sqrt(2 * n[0]), s0,
                    math.sqrt(1 - mag - s0 ** 2 * n[1]) / math.sqrt(2 * n[2])]
        x1, x2 = self.sig
        for _ in range(1000):
            e = [n[m] * math.exp(2 * (x1 + (2 - m) * x2) * dt) for m in range(5)]
            f1, f2 = sum(e) - 1.0, sum((2 - m) * e[m] for m in range(5)) - mag
            j11, j12 = 2 * dt * sum(e), 2 * dt * sum((2 - m) * e[m] for m in range(5))
            j22 = 2 * dt * sum((2 - m) ** 2 * e[m] for m in range(5))
            p2 = (f2 * j11 - f1 * j12) / (j12 * j12 - j11 * j22)
            p1 = (-f1 - j12 * p2) / j11
            x1, x2 = x1 + p1, x2 + p2
            if max(abs(p1), abs(p2)) <= 1e-6:
                break
        self.sig = (x1, x2)
        return [math.exp((x1 + (2 - m) * x2) * dt) for m in range(5)]

    def _gradient(self, u, a):
        """DIFF along axis a: nine points inside, five at the four nodes of each end."""
        if self.n[a] == 1:
            return torch.zeros_like(u)
        at, n, h = 2 - a, self.n[a], self.d[a]
        r = lambda q: torch.roll(u, -q, at)  # noqa: E731
        inner = (3 * (r(-4) - r(4)) - 32 * (r(-3) - r(3)) + 168 * (r(-2) - r(2)) - 672 * (r(-1) - r(1))) / (840 * h)
        i = torch.arange(n, device=DEV).reshape([-1 if q == a else 1 for q in (2, 1, 0)])
        return torch.where((i >= 4) & (i <= n - 5), inner, (r(-2) - 8 * r(-1) + 8 * r(1) - r(2)) / (12 * h))

    def observables(self):
        ms, S, v = self.ms, self.S, self.v
        t0, t1, t2 = self.p["tau"]
        a, rho, t = self._density()
        c = [0.5 * math.sqrt(S * (S + 1) - (S - m) * (S - m - 1)) for m in range(ms - 1)]
        G = [[self._gradient(x, q) for q in range(3)] for x in v]
        e = self.V * rho + t0 * rho ** 2 / 2
        f = 2 * sum(c[m] * v[m].conj() * v[m + 1] for m in range(ms - 1))
        e = e + t1 * (f.abs() ** 2 + self._spin_density(a) ** 2) / 2
        mu = [t[m] * a[m] for m in range(ms)]
        if ms == 3:
            x = t1 * (v[1] ** 2 * (v[0] * v[2]).conj()).real
            mu = [mu[0] + x, mu[1] + 2 * x, mu[2] + x]
        else:
            th = (2 * v[0] * v[4] - 2 * v[1] * v[3] + v[2] ** 2) / math.sqrt(5.0)
            e = e + t2 * th.abs() ** 2 / 2
            hv = _apply(_couplings(v, t1, t2), v)
            mu = [mu[m] + (hv[m] * v[m].conj()).real for m in range(ms)]
        for m in range(ms):
            so = (S - m) * self.g[2] * G[m][2]
            if m > 0:
                so = so + c[m - 1] * (self.g[0] * G[m - 1][0] + 1j * self.g[1] * G[m - 1][1])
            if m < ms - 1:
                so = so + c[m] * (self.g[0] * G[m + 1][0] - 1j * self.g[1] * G[m + 1][1])
            k = sum(x.abs() ** 2 for x in G[m]) + (v[m].conj() * (-2j) * so).real
            e, mu[m] = e + k, mu[m] + k
        n = self.norms()
        r2 = self.x[0] ** 2 + self.x[1] ** 2 + self.x[2] ** 2
        return np.array([self._sum(e) / sum(n), self._sum(self._spin_density(a))] + [self._sum(mu[m]) / n[m] for m in range(ms)]
                        + [math.sqrt(self._sum(r2 * x)) for x in a])


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _network(w, a, n, modes=16, layers=4):
    """The operator network in float64 torch on [c][B][n][n]; w in the device's layout (R [kx][ky][o][c])."""
    pick = torch.cat([torch.arange(modes, device=DEV), torch.arange(n - modes, n, device=DEV)])
    mix = lambda m, x, b: torch.einsum("oc,cbij->obij", m, x) + b[:, None, None, None]  # noqa: E731
    h = mix(w["P"], a, w["bP"])
    for q in range(layers):
        H = torch.fft.rfft2(h)[:, :, pick, :modes]
        full = torch.zeros(h.shape[0], h.shape[1], n, n // 2 + 1, dtype=torch.complex128, device=DEV)
        G = torch.einsum("akoc,cbak->obak", torch.complex(w[f"Rr{q}"], w[f"Ri{q}"]), H)
        full[:, :, pick, :modes] = G
        # Re of the sum over the kept modes, ky > 0 doubled (the kept ky stay below n/2)
        full[..., 0] = 0
        zero = torch.zeros(h.shape[0], h.shape[1], n, dtype=torch.complex128, device=DEV)
        zero[:, :, pick] = G[..., 0]
        col = torch.fft.ifft(zero, dim=2).real[..., None] / n
        z = mix(w[f"W{q}"], h, w[f"b{q}"]) + torch.fft.irfft2(full, s=(n, n)) + col
        h = _gelu(z) if q < layers - 1 else z
    return mix(w["Q2"], _gelu(mix(w["Q1"], h, w["c1"])), w["c2"])


def exact(case, seed):
    kind = case["kind"]
    if kind == "propagate" and case["spin"] == 2 and case["nx"] * case["ny"] * case["nz"] * case["steps"] > 3e7:
        return None  # its matrix exponentials take longer than is worth waiting for
    if kind in ("propagate", "sweep"):
        insts = [_params(case)] if kind == "propagate" else _sweep(case, seed)
        got = []
        for k, p in enumerate(insts):
            x = _Exact(p, _start(p, seed + 1000 * k))
            for i in range(case["steps"]):
                before = x.v if i == case["steps"] - 1 else None
                norms = x.step()
            got.append((x, norms, before))
        x, norms, before = got[0]
        if kind == "sweep":
            return {"observables": np.concatenate([np.concatenate([x.observables(), n]) for x, n, _ in got]),
                    "state": torch.cat([torch.stack(x.v).reshape(-1) for x, _, _ in got])}
        res = {"norms": np.array(norms), "observables": x.observables(), "state": torch.stack(x.v)}
        if case["imag"] and case["precision"] == "fp64":
            res["conv"] = max(float((u - v).abs().max()) for u, v in zip(x.v, before))
        return res
    n, B = case["n"], case["batch"]
    if kind == "infer":
        w = {k: _device_layout(v) for k, v in _weights(seed).items()}
        a = torch.from_numpy(_points(case, seed)).to(DEV, torch.float64)
        return {"out": torch.cat([_network(w, a[:, b:b + 1], n) for b in range(B)], 1).reshape(6, -1)}
    a, tgt, weights, m, v = _training(case, seed)
    w = {k: _device_layout(x).requires_grad_() for k, x in weights.items()}
    out = _network(w, a.double().reshape(7, B, n, n), n).reshape(6, -1)
    loss = ((out - tgt.double()) ** 2).mean()
    loss.backward()
    new, t = {}, _T + 1
    for k, x in w.items():
        mm = 0.9 * _device_layout(m[k]) + 0.1 * x.grad
        vv = 0.999 * _device_layout(v[k]) + 0.001 * x.grad ** 2
        new[k] = x.detach() - _LR * (mm / (1 - 0.9 ** t)) / (torch.sqrt(vv / (1 - 0.999 ** t)) + 1e-8)
    return {"out": out.detach(), "loss": loss.detach(), "grads": {k: x.grad for k, x in w.items()}, "weights": new}
