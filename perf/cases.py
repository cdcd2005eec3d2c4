"""The work a user of this framework has it do, as measurable cases.

  step      time steps of one channel (``Channel.step``): plain DNS in FP64 and
            on the mixed path, fixed or CFL-limited dt, and LES with the AMD or
            the learned closure; a pass advances the state ``steps`` steps and
            brings the five step fields to the program's own host arrays
  ensemble  steps of a batched ensemble of independent small channels
            (``Ensemble.step``), the closure's data-generation runs
  fft       a device-resident field to Fourier space and back
            (``fft_xz_to_fourier_dev``, ``fft_xz_to_physical_dev``)
  train     Adam steps of the closure network (``SgsNet.train_step``)

``exact`` restates the same work in plain torch in 64 bits.
"""
import ctypes
import math
import os

import numpy as np
import torch

STEP_FIELDS = 5   # cu1, cu2, cu3, cp, cth: what a time step reads and leaves


def _step(name, nx, ny, nz, **kw):
    c = dict(name=name, kind="step", nx=nx, ny=ny, nz=nz, precision=0, les=0, front=0, variable_dt=1, re=5000.0,
             steps=4)
    c.update(kw)
    return c


def listed():
    return [
        # the parity/latency grid: a small DNS at a fixed dt, launches and serial chains count
        _step("dns_64x65x64_f64", 64, 65, 64, variable_dt=0, re=1000.0, steps=20),
        # a thin ragged box on the mixed path
        _step("dns_32x41x128_mixed", 32, 41, 128, precision=1, re=1000.0, steps=20),
        # an ordinary DNS, twice the learned closure's LES grid
        _step("dns_256x129x256_f64", 256, 129, 256, steps=6),
        # the headline DNS, FP64 throughout, CFL-limited
        _step("dns_512x257x512_f64", 512, 257, 512),
        # the same on the mixed path
        _step("dns_512x257x512_mixed", 512, 257, 512, precision=1),
        # finite-front LES, AMD closure, mixed precision
        _step("les_amd_256x129x256_mixed", 256, 129, 256, precision=1, les=5, front=1, re=1e5),
        # finite-front LES, AMD closure, FP64
        _step("les_amd_128x65x128_f64", 128, 65, 128, les=5, front=1, re=1e4, steps=10),
        # the same with the trained network in place of AMD
        _step("les_net_128x65x128_mixed", 128, 65, 128, precision=1, les=6, front=1, re=1e4, steps=10),
        # closure-data generation: small channels with their own seeds and Ri, stepped together
        dict(name="ensemble_32x128x65x128_mixed", kind="ensemble", nx=128, ny=65, nz=128, precision=1, members=32,
             re=2000.0, steps=12),
        # one field through the transforms: a large one in FP64, a small odd one in FP32 arithmetic
        dict(name="fft_512x129x512_f64", kind="fft", nx=512, ny=129, nz=512, precision=0),
        dict(name="fft_64x33x256_f32", kind="fft", nx=64, ny=33, nz=256, precision=1),
        # training of the closure network at its batch size
        dict(name="train_65536", kind="train", points=65536, steps=8),
    ]


def _pow2(rng, lo, hi):
    return 1 << rng.randint(lo, hi)


def _odd_ny(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "les", "ensemble", "fft", "fft", "train"])
    if kind == "train":
        return dict(kind="train", points=int(round(math.exp(rng.uniform(math.log(1000), math.log(400000))))),
                    steps=rng.randint(4, 8))
    nx, nz, ny = _pow2(rng, 5, 9), _pow2(rng, 5, 9), _odd_ny(rng, 17, 257)
    precision = rng.randint(0, 1)
    if kind == "fft":
        return dict(kind="fft", nx=nx, ny=_odd_ny(rng, 17, 129), nz=nz, precision=precision)
    if kind == "ensemble":
        nx, nz, ny = _pow2(rng, 5, 7), _pow2(rng, 5, 7), _odd_ny(rng, 17, 65)
        return dict(kind="ensemble", nx=nx, ny=ny, nz=nz, precision=precision, members=rng.randint(2, 32),
                    re=2000.0, steps=rng.randint(6, 12))
    c = _step("", nx, ny, nz, precision=precision, variable_dt=rng.randint(0, 1), steps=rng.randint(3, 6),
              re=rng.choice([1000.0, 2000.0, 5000.0]))
    del c["name"]
    if kind == "les":
        nx, nz, ny = _pow2(rng, 5, 8), _pow2(rng, 5, 8), _odd_ny(rng, 33, 129)
        c.update(nx=nx, ny=ny, nz=nz, les=rng.choice([5, 5, 6]), front=1, variable_dt=1, re=rng.choice([1e4, 1e5]))
    return c


# ---------------------------------------------------------------------------
# inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _grid(ny):
    """GY(1..ny+1): tanh-stretched to both walls of [-1, 1] (create_grid type 1, strength 1.5)."""
    s = np.tanh(1.5 * (2.0 * np.arange(ny + 1) / ny - 1.0)) / np.tanh(1.5)
    f = 0.5 * (s[:-1] + s[1:])
    scale = (s[-1] - s[0]) / (f[-1] - f[0])
    return np.ascontiguousarray(s * scale + (s[0] - f[0] * scale))


def _metrics(gy):
    n = len(gy) - 1
    y, yf, dy, dyf = (np.zeros(n + 2) for _ in range(4))
    y[1:] = gy
    yf[1:n + 1] = 0.5 * (y[1:n + 1] + y[2:])
    yf[0], yf[n + 1] = 2 * yf[1] - yf[2], 2 * yf[n] - yf[n - 1]
    dy[1:] = yf[1:] - yf[:-1]
    dyf[1:n + 1] = y[2:] - y[1:n + 1]
    dyf[0], dyf[n + 1] = dyf[1], dyf[n]
    return y, yf, dy, dyf


def _noise(case, g, lead=()):
    """Band-limited noise (|k| below a third of the largest wavenumber) of unit deviation."""
    nx, nz, npl = case["nx"], case["nz"], case["ny"] + 2
    w = torch.fft.rfft2(torch.randn((npl,) + lead + (nz, nx), generator=g, device="cuda", dtype=torch.float64))
    kx = torch.arange(nx // 2 + 1, device="cuda")
    kz = (torch.fft.fftfreq(nz, device="cuda") * nz).abs()
    w *= (kx[None, :] < nx / 6.0) & (kz[:, None] < nz / 6.0)
    f = torch.fft.irfft2(w, s=(nz, nx))
    return f / f.std()


def _ri(case, seed):
    """Ri of an ensemble's members, U[0.5, 2]."""
    return np.random.Generator(np.random.PCG64(int(seed) + 1000)).uniform(0.5, 2.0, case["members"])


def _pack(case, f):
    """Physical [j, ..., z, x] -> retained modes [j, ..., 2 nkz + 1, nkx + 1], normalised."""
    nx, nz = case["nx"], case["nz"]
    h = torch.fft.rfft2(f, norm="forward")
    kz = nz // 3
    return torch.cat([h[..., :kz + 1, :nx // 3 + 1], h[..., nz - kz:, :nx // 3 + 1]], dim=-2)


def _to_ref(case, s):
    """Retained modes -> the reference layout [j, ..., nz + 2, nx / 2 + 1], zero elsewhere."""
    out = torch.zeros(s.shape[:-2] + (case["nz"] + 2, case["nx"] // 2 + 1), dtype=torch.complex128, device=s.device)
    out[..., :s.shape[-2], :s.shape[-1]] = s
    return out


def _initial(case, seed):
    """Spectral u1, u2, u3, th of the infinite front (IC 4) or the finite front (IC 6), with seeded noise."""
    g = _gen(seed)
    lead = (case["members"],) if case["kind"] == "ensemble" else ()
    _, yf, _, _ = _metrics(_grid(case["ny"]))
    ny, nx, nz = case["ny"], case["nx"], case["nz"]
    kick = 0.02 if case.get("front") else 1e-3
    u1, u2, u3 = (kick * _noise(case, g, lead) for _ in range(3))
    th = torch.zeros((ny + 2,) + lead + (nz, nx), dtype=torch.float64, device="cuda")
    y = torch.tensor(yf - 1.0, device="cuda").view(-1, 1, 1)          # gyf - ly / 2
    if case.get("front"):
        lx, d = 2 * math.pi, 0.5
        x = torch.arange(nx, device="cuda", dtype=torch.float64) * (lx / nx) - 0.5 * lx
        s = math.sqrt(2.0)
        t = torch.tanh((x + y[:ny + 1]) / (d * s))
        u3[:ny + 1] += d * s * t - 2.0 * d / lx * y[:ny + 1]
        th[1:ny + 1] = s * t[1:] + (1.0 - 2.0 / lx * (x + 0.5 * lx))
    else:
        th[1:ny + 1] = y[1:ny + 1].view((-1,) + (1,) * (th.dim() - 1))
    return [_pack(case, f) for f in (u1, u2, u3, th)]


def _params(case, m2=float("nan")):
    from diablo3_b200.params import make_params
    front = case.get("front", 0)
    return make_params(
        nx=case["nx"], ny=case["ny"], nz=case["nz"], re=case["re"], precision=case["precision"], ic_type=6 if front else 4,
        delta=0.5 if front else 1.0, delta_t=1e-3, variable_dt=case.get("variable_dt", 0), cfl=0.5, time_limit=1e9,
        use_les=1 if case.get("les") else 0, les_model_type=case.get("les") or 5,
        create_new_flow=0 if case.get("les") else 1, dthdx_override=m2)


def _net_file():
    import diablo3_b200
    return np.load(os.path.join(os.path.dirname(diablo3_b200.__file__), "data", "closure_config3.npz"))


def _move(ch, call, fid, host):
    ch._ck(call(ch.h, fid, ctypes.cast(ctypes.c_void_p(host.data_ptr()), ctypes.POINTER(ctypes.c_double))))


_UP = (0, 1, 2, 4)        # cu1, cu2, cu3, cth
_DOWN = (0, 1, 2, 3, 4)   # cu1, cu2, cu3, cp, cth


def _train_data(case, seed):
    g = _gen(seed)
    n = case["points"]
    d = _net_file()
    mean, std, scale = (torch.tensor(d[k], device="cuda") for k in ("mean", "std", "scale"))
    feat = mean + std * torch.randn((n, 16), generator=g, device="cuda")
    feat[:, 15] = feat[:, 10]
    strain = feat[:, :9].square().sum(1).sqrt() / std[:9].square().sum().sqrt()
    tgt = scale * torch.stack([strain, strain * torch.rand((n,), generator=g, device="cuda") * 2], 1)
    w = torch.randn((9538,), generator=g, device="cuda") * 0.05
    params = torch.tensor(d["params"], device="cuda") + w * (torch.rand((9538,), generator=g, device="cuda") < 0.5)
    return feat.contiguous(), tgt.contiguous(), params.cpu().numpy(), d


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        from diablo3_b200.sgs_net import SgsNet
        feat, tgt, params, d = _train_data(case, seed)
        net = SgsNet()
        net.set(params, d["mean"], d["std"], d["scale"])
        return dict(case=case, net=net, feat=feat, tgt=tgt)
    from diablo3_b200 import Channel
    shape = (case["ny"] + 2, case["nz"] + 2, case["nx"] // 2 + 1)
    if kind == "fft":
        t = torch.zeros((case["ny"] + 2, case["nz"] + 2, case["nx"] + 2), dtype=torch.float64, device="cuda")
        t[:, :case["nz"], :case["nx"]] = torch.randn((case["ny"] + 2, case["nz"], case["nx"]), generator=_gen(seed),
                                                     device="cuda", dtype=torch.float64)
        ch = Channel(_params(dict(case, re=1000.0)), _grid(case["ny"]))
        return dict(case=case, ch=ch, t=t)
    spec = _initial(case, seed)
    if kind == "ensemble":
        from diablo3_b200.ensemble import Ensemble
        n = case["members"]
        ens = Ensemble([_params(case, math.sqrt(1.0 / r)) for r in _ri(case, seed)], _grid(case["ny"]), init=False)
        host = [torch.zeros((n,) + shape, dtype=torch.complex128, pin_memory=True) for _ in _DOWN]
        for fid, s in zip(_UP, spec):
            host[fid].copy_(_to_ref(case, s).transpose(0, 1))
        for i, ch in enumerate(ens.members):
            for fid in _UP:
                _move(ch, ch.L.db_upload_field, fid, host[fid][i])
            ch.apply_bc_vel_post()
            ch.rem_div_chan()
        return dict(case=case, ens=ens, host=host)
    ch = Channel(_params(case), _grid(case["ny"]))
    state = dict(case=case, ch=ch)
    if case["les"] == 6:
        from diablo3_b200.sgs_net import SgsNet
        d = _net_file()
        net = SgsNet()
        net.set(d["params"], d["mean"], d["std"], d["scale"])
        net.set_range(d["lo"], d["hi"])
        ch.set_sgs_net(net)
    host = [torch.zeros(shape, dtype=torch.complex128, pin_memory=True) for _ in _DOWN]
    for fid, s in zip(_UP, spec):
        host[fid].copy_(_to_ref(case, s))
        _move(ch, ch.L.db_upload_field, fid, host[fid])
    ch.apply_bc_vel_post()
    ch.rem_div_chan()
    state["host"] = host
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        net = state["net"]
        loss = [net.train_step(state["feat"], state["tgt"], 1e-3) for _ in range(case["steps"])]
        return dict(loss=np.array(loss), params=net.get())
    if kind == "fft":
        ch, t = state["ch"], state["t"]
        ch.fft_xz_to_fourier_dev(t)
        ch.fft_xz_to_physical_dev(t)
        return t[:, :case["nz"], :case["nx"]]
    host = state["host"]
    if kind == "ensemble":
        state["ens"].step(case["steps"])
        for i, ch in enumerate(state["ens"].members):
            for fid in _DOWN:
                _move(ch, ch.L.db_download_field, fid, host[fid][i])
        return host
    ch = state["ch"]
    ch.step(case["steps"])
    for fid in _DOWN:
        _move(ch, ch.L.db_download_field, fid, host[fid])
    return host


# ---------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    if case["kind"] == "train":
        n, s = case["points"], case["steps"]
        # forward and backward of 16-64-64-64-2
        return {"bytes": s * (n * 18 * 4 + 9538 * 4 * 6.0), "flops": s * n * 6.0 * (16 * 64 + 2 * 64 * 64 + 64 * 2)}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    pts = float(nx * nz * (ny + 2))
    spec = 16.0 * (nx // 3 + 1) * (2 * (nz // 3) + 1) * (ny + 2)
    fft2 = 2.5 * pts * math.log2(nx * nz)
    if case["kind"] == "fft":
        full = 16.0 * (nx // 2 + 1) * (nz + 2) * (ny + 2)
        return {"bytes": 2 * 8.0 * pts + full + spec, "flops": 2 * fft2}
    m = case.get("members", 1)
    # a substep reads and writes the state and the history of the explicit
    # terms (9 fields), transforms 4 fields to physical space (12 with the
    # closure's gradients) and 11 products back; the last step's fields go out
    subs = 3 * case["steps"] * m
    nfft = 15 + (8 if case.get("les") else 0)
    flops = subs * (nfft * fft2 + 60.0 * pts)
    if case.get("les") == 6:
        flops += subs * pts * 2.0 * (16 * 64 + 2 * 64 * 64 + 64 * 2)
    return {"bytes": subs * 18 * spec + m * STEP_FIELDS * spec, "flops": flops}


def tolerance(case):
    # about four times the distance to the same work in 64 bits, worst field (cp) and worst listed case
    if case["kind"] == "fft":
        return {"rel": 1.2e-6, "max": 1e-5} if case["precision"] else {"rel": 3e-15, "max": 3e-14}
    if case["kind"] == "train":
        return {"rel": 1.5e-3, "max": 5e-3}
    if case.get("les") == 6:
        return {"rel": 3e-4, "max": 1e-2}   # BF16 activations
    if case["precision"]:
        return {"rel": 1.5e-5, "max": 2e-3}
    return {"rel": 1e-11, "max": 2e-9}


# ---------------------------------------------------------------------------
# the same work in plain torch, 64 bits

class _Exact:
    """RKW3 + Crank-Nicolson steps of the channel in plain torch (FP64).  Axis 0 is the wall-normal row, the last two
    are z and x (physical) or kz and kx (retained modes), members of an ensemble lie between."""

    def __init__(self, case, m2=None):
        T = lambda a: torch.tensor(np.asarray(a, dtype=np.float64), device="cuda")   # noqa: E731
        self.case, self.ny, self.nx, self.nz = case, case["ny"], case["nx"], case["nz"]
        self.lead = (case["members"],) if case["kind"] == "ensemble" else ()
        self.y, self.yf, self.dy, self.dyf = _metrics(_grid(self.ny))
        nkx, nkz = self.nx // 3, self.nz // 3
        pi = float(np.float32(4.0) * np.arctan(np.float32(1.0)))
        self.pi, self.lx = pi, 2 * math.pi
        kz = np.concatenate([np.arange(nkz + 1), -np.arange(nkz, 0, -1)])
        self.kx = T(np.arange(nkx + 1) * (2.0 * pi) / self.lx)[None, :]
        self.kz = T(kz * (2.0 * pi) / self.lx)[:, None]
        self.k2 = self.kx ** 2 + self.kz ** 2
        self.nu = 1.0 / case["re"]
        front = case.get("front", 0)
        if front:
            self.f = 1.0 / 0.5            # ro_inv / delta
            self.m2, self.w_max = 2.0 / self.lx, -2.0 * 0.5 / self.lx
        else:
            self.f = 1.0
            self.m2 = 1.0 if m2 is None else T(m2).view(-1, 1, 1)
            self.w_max = -1.0 if m2 is None else -T(m2)
        self.dt = 1e-3
        self.jst, self.jth = 2, 1         # first rows of u1, u3 (no slip) and of th (flux)
        self.les = case.get("les", 0)
        if self.les == 6:
            d = _net_file()
            self.net = {k: T(d[k]) for k in ("params", "mean", "std", "scale", "lo", "hi")}
        shp = (self.ny + 2,) + self.lead + (2 * nkz + 1, nkx + 1)
        self.cp = torch.zeros(shp, dtype=torch.complex128, device="cuda")
        self.cf = [torch.zeros(shp, dtype=torch.complex128, device="cuda") for _ in range(4)]

    def col(self, a):
        """A row table as a column that broadcasts over a field."""
        return torch.tensor(np.asarray(a), device="cuda").view((-1,) + (1,) * (2 + len(self.lead)))

    def phys(self, s):
        full = torch.zeros(s.shape[:-2] + (self.nz, self.nx // 2 + 1), dtype=torch.complex128, device="cuda")
        nkz = self.nz // 3
        full[..., :nkz + 1, :s.shape[-1]] = s[..., :nkz + 1, :]
        full[..., self.nz - nkz:, :s.shape[-1]] = s[..., nkz + 1:, :]
        return torch.fft.irfft2(full, s=(self.nz, self.nx), norm="forward")

    def spec(self, f):
        return _pack(self.case, f)

    def bc_vel_post(self, u1, u2, u3):
        n, m0 = self.ny, (Ellipsis, 0, 0)
        for u in (u1, u3):
            u[0], u[1] = 0, 0
            u[n] = u[n - 1]
            u[n + 1] = u[n]
        u3[n][m0] = u3[n - 1][m0] + self.dy[n] * self.w_max
        u3[n + 1][m0] = u3[n][m0] + self.dy[n] * self.w_max
        u2[1] = -u2[2]
        u2[0] = u2[1]
        u2[n + 1][m0] = -u2[n][m0]

    def rem_div(self, u1, u2, u3, h):
        n, dy, dyf = self.ny, self.dy, self.dyf
        zero = self.k2 == 0
        rhs = [None] * (n + 1)
        b = [None] * (n + 1)
        up = [None] * (n + 1)
        for j in range(1, n + 1):
            if j == 1:
                l, d, u, r = 0.0, torch.ones_like(self.k2), torch.where(zero, 0.0, -1.0), torch.zeros_like(u1[1])
            elif j == n:
                l, d, u, r = 1.0, -torch.ones_like(self.k2), torch.zeros_like(self.k2), torch.zeros_like(u1[1])
            else:
                l, u = 1.0 / (dy[j] * dyf[j]), torch.full_like(self.k2, 1.0 / (dy[j + 1] * dyf[j]))
                d = -self.k2 - 1.0 / (dy[j + 1] * dyf[j]) - l
                r = 1j * self.kx * u1[j] + (u2[j + 1] - u2[j]) / dyf[j] + 1j * self.kz * u3[j]
            if j > 1:
                a = -l / b[j - 1]
                d = d + a * up[j - 1]
                r = r + a * rhs[j - 1]
            b[j], up[j], rhs[j] = d, u, r
        phi = [None] * (n + 1)
        for j in range(n, 0, -1):
            phi[j] = rhs[j] / b[j] if j == n else (rhs[j] - up[j] * phi[j + 1]) / b[j]
        for j in range(1, n + 1):
            u1[j] -= 1j * self.kx * phi[j]
            u3[j] -= 1j * self.kz * phi[j]
            if j >= 2:
                u2[j] -= (phi[j] - phi[j - 1]) / dy[j]
            if h is not None and self.jst <= j <= n:
                self.cp[j] += phi[j] / h

    def start(self, spec):
        u1, u2, u3, th = spec
        self.bc_vel_post(u1, u2, u3)
        self.rem_div(u1, u2, u3, None)
        self.u = [u1, u2, u3, th]

    # the implicit rows of one equation: (l, d, u, cn_lo, cn_hi, ef_lo, ef_hi) of the interior, BC rows by number
    def rows(self, eq, h):
        n, dy, dyf = self.ny, self.dy, self.dyf
        t = 0.5 * self.nu * h
        R = {}
        lo, hi = (self.jth if eq == "th" else 2 if eq == "u2" else self.jst), n
        for j in range(lo, hi + 1):
            if eq == "u2":
                lo_, hi_ = 1.0 / (dyf[j - 1] * dy[j]), 1.0 / (dyf[j] * dy[j])
                ef = 0.5
            else:
                lo_, hi_ = 1.0 / (dy[j] * dyf[j]), 1.0 / (dy[j + 1] * dyf[j])
                ef = 1.0
            R[j] = dict(l=-t * lo_, d=1.0 + t * hi_ + t * lo_, u=-t * hi_, lo=t * lo_, hi=t * hi_, elo=ef * lo_,
                        ehi=ef * hi_, bc=None)
        def put(j, l, d, u, v):
            R[j] = dict(l=l, d=d, u=u, bc=v)
        for j in range(0, n + 2):
            if j not in R:
                put(j, 0.0, 1.0, 0.0, 0.0)
        if eq == "u2":
            for j in (0, 1, 2, n, n + 1):
                put(j, 0.0, 1.0, 0.0, 0.0)
        else:
            put(0, 0.0, 1.0, 0.0, 0.0)
            put(n + 1, 0.0, 1.0, 0.0, 0.0)
            if eq == "th":
                put(1, 0.0, -1.0, 1.0, dy[2] * 1.0)
                put(n, -1.0, 1.0, 0.0, dy[n] * 1.0)
            else:
                put(1, 0.0, 1.0, 0.0, 0.0)
                put(n, -1.0, 1.0, 0.0, dy[n] * (self.w_max if eq == "u3" else 0.0))
        return R

    def solve(self, eq, u, r, h, nut=None, spectral=True):
        """u of the new time level (rows the solve stores) from the explicit right-hand side r."""
        n = self.ny
        R = self.rows(eq, h)
        t2 = 0.5 * h
        bs, gs, us = [None] * (n + 2), [None] * (n + 2), [None] * (n + 2)
        for j in range(n + 2):
            q = R[j]
            l, d, up = q["l"], q["d"], q["u"]
            if q["bc"] is not None:
                v = torch.zeros_like(u[0])
                if spectral:
                    v[..., 0, 0] = q["bc"]
                else:
                    v += q["bc"]
            else:
                v = r[j] + (q["hi"] * (u[j + 1] - u[j]) - q["lo"] * (u[j] - u[j - 1]))
                if nut is not None:
                    a, b = ((nut[j] + nut[j - 1], nut[j] + nut[j + 1]) if eq == "u2" else (nut[j], nut[j + 1]))
                    a, b = a * q["elo"], b * q["ehi"]
                    v = v + t2 * (b * (u[j + 1] - u[j]) - a * (u[j] - u[j - 1]))
                    l, d, up = l - t2 * a, d + t2 * b + t2 * a, up - t2 * b
            if j > 0:
                a = -l / bs[j - 1]
                d = d + a * us[j - 1]
                v = v + a * gs[j - 1]
            bs[j], gs[j], us[j] = d, v, up
        new = u.clone()
        lo, hi = (0, n + 1) if eq == "th" else (1, n + 1)
        x = None
        for j in range(n + 1, -1, -1):
            x = gs[j] / bs[j] if x is None else (gs[j] - us[j] * x) / bs[j]
            if lo <= j <= hi:
                new[j] = x
        return new

    @staticmethod
    def up(a):
        """Rows j + 1 in place of j (the last row repeated)."""
        return torch.cat([a[1:], a[-1:]])

    @staticmethod
    def dn(a):
        return torch.cat([a[:1], a[:-1]])

    def amd(self, s1, s2, s3, s4, s5, s6, o4, o5, o6):
        i3 = (s1 ** 3 + s2 ** 3 + s3 ** 3 + 3 * (s1 * s4 * s4 + s1 * s5 * s5 + s2 * s4 * s4 + s2 * s6 * s6 + s3 * s5 * s5 +
              s3 * s6 * s6) + 6 * s4 * s5 * s6)
        v = (-i3 - s1 * o4 * o4 - s1 * o5 * o5 - s2 * o4 * o4 - s2 * o6 * o6 - s3 * o5 * o5 - s3 * o6 * o6 -
             2 * s4 * o5 * o6 + 2 * s5 * o4 * o6 - 2 * s6 * o4 * o5)
        den = s1 ** 2 + s2 ** 2 + s3 ** 2 + 2 * (s4 ** 2 + o4 ** 2 + s5 ** 2 + o5 ** 2 + s6 ** 2 + o6 ** 2)
        return torch.where(v > 0, v / torch.where(v > 0, den, 1.0), 0.0)

    def amd_th(self, dx, dy, dz, u1x, u2y, u3z, u1y, u2x, u1z, u3x, u2z, u3y, tx, ty, tz):
        v = -(dx * dx * u1x * tx * tx + dy * dy * u2y * ty * ty + dz * dz * u3z * tz * tz +
              (dy * dy * u1y + dx * dx * u2x) * tx * ty + (dz * dz * u1z + dx * dx * u3x) * tx * tz +
              (dz * dz * u2z + dy * dy * u3y) * ty * tz)
        den = (dx * tx) ** 2 + (dy * ty) ** 2 + (dz * tz) ** 2
        return torch.where(v > 0, v / torch.where(v > 0, den, 1.0), 0.0)

    def mlp(self, feat):
        p, n = self.net["params"], self.net
        sh = [(0, (64, 16)), (1024, (64,)), (1088, (64, 64)), (5184, (64,)), (5248, (64, 64)), (9344, (64,)),
              (9408, (2, 64)), (9536, (2,))]
        w = [p[o:o + int(np.prod(s))].view(s) for o, s in sh]
        h = (feat - n["mean"]) / n["std"]
        for i in range(3):
            h = torch.nn.functional.gelu(h @ w[2 * i].T + w[2 * i + 1], approximate="tanh")
        return torch.nn.functional.softplus(h @ w[6].T + w[7]) * n["scale"]

    def closure(self, ghosted):
        """nu_t, kappa_t at GY rows and the nine forcing terms of the SGS stress and flux."""
        n = self.ny
        up, dn, col = self.up, self.dn, self.col
        u1, u2, u3, th = self.pu
        gx = [self.phys(1j * self.kx * s) for s in ghosted]
        gz = [self.phys(1j * self.kz * s) for s in ghosted]
        a1x, a2x, a3x, atx = gx
        a1z, a2z, a3z, atz = gz
        dxs, dzs = 3.0 * self.lx / self.nx, 3.0 * self.lx / self.nz
        idy = np.where(self.dy != 0, 1.0 / np.where(self.dy != 0, self.dy, 1.0), 0.0)
        dly = 2.0 * self.dy
        rxy, rzy = dxs * idy / 2, dzs * idy / 2
        coef = lambda h: np.where(h != 0, -2.0 * 0.2887 ** 2 * 3.0 / (1 / dxs ** 2 + 1 / np.where(h != 0, 2 * h, 1) ** 2 + 1 / dzs ** 2), 0.0)   # noqa: E731
        delt, dlf = col(coef(self.dy)), col(coef(self.dyf))
        wa, wb = np.zeros(n + 2), np.zeros(n + 2)
        wa[1:], wb[1:] = self.dyf[:-1] * idy[1:] / 2, self.dyf[1:] * idy[1:] / 2
        wa, wb = col(wa), col(wb)
        gyi = lambda a: a * wa + dn(a) * wb   # noqa: E731
        cidy = col(idy)
        d1y, d3y, dty = ((q - dn(q)) * cidy for q in (u1, u3, th))
        c2y = (up(u2) - u2) / col(self.dyf)
        c2y[n + 1] = 0
        ryx, ryz = col(dly / dxs), col(dly / dzs)
        rxy, rzy = col(rxy), col(rzy)
        rzx, rxz = dzs / dxs, dxs / dzs
        SI4, O4 = 0.5 * (d1y * ryx + a2x * rxy), 0.5 * (d1y * ryx - a2x * rxy)
        SI6, O6 = 0.5 * (a2z * rzy + d3y * ryz), 0.5 * (a2z * rzy - d3y * ryz)
        SI5, O5 = 0.5 * (a1z * rzx + a3x * rxz), 0.5 * (a1z * rzx - a3x * rxz)
        temp = self.amd(gyi(a1x), gyi(c2y), gyi(a3z), SI4, gyi(SI5), SI6, O4, gyi(O5), O6)
        temp_th = self.amd_th(dxs, col(dly), dzs, gyi(a1x), gyi(c2y), gyi(a3z), d1y, a2x, gyi(a1z), gyi(a3x), a2z, d3y,
                              gyi(atx), dty, gyi(atz))
        mid = lambda a: 0.5 * (a + up(a))   # noqa: E731
        s1 = self.amd(a1x, c2y, a3z, mid(SI4), SI5, mid(SI6), mid(O4), O5, mid(O6))
        s1t = self.amd_th(dxs, col(2.0 * self.dyf), dzs, a1x, c2y, a3z, mid(d1y), mid(a2x), a1z, a3x, mid(a2z), mid(d3y),
                          atx, mid(dty), atz)
        if self.les == 6:
            one = torch.ones_like(u1)
            feat = torch.stack([gyi(a1x), d1y, gyi(a1z), a2x, gyi(c2y), a2z, gyi(a3x), d3y, gyi(a3z), gyi(atx), dty,
                                gyi(atz), dxs * one, col(dly) * one, dzs * one, dty], -1)
            ok = ((feat >= self.net["lo"]) & (feat <= self.net["hi"])).all(-1)
            f32 = feat[..., 12:15].float().double()
            ok = ok | (((feat[..., :12] >= self.net["lo"][:12]) & (feat[..., :12] <= self.net["hi"][:12])).all(-1) &
                       ((f32 >= self.net["lo"][12:15]) & (f32 <= self.net["hi"][12:15])).all(-1))
            ok[0] = False
            out = self.mlp(feat)
            nu_m, ka_m = out[..., 0], out[..., 1]
            sd = torch.where(delt != 0, delt, 1.0)
            temp = torch.where(ok, -2.0 * nu_m / sd, temp)
            temp_th = torch.where(ok, -2.0 * ka_m / sd, temp_th)
            both = ok & up(ok)
            s1 = torch.where(both, -(nu_m + up(nu_m)) / dlf, s1)
            s1t = torch.where(both, -(ka_m + up(ka_m)) / dlf, s1t)
        for t in (temp, temp_th):
            t[:2] = 0
            t[n + 1] = 0
        nut, kat = -0.5 * delt * temp, -0.5 * delt * temp_th
        for t in (nut, kat):
            t[:3] = 0
            t[n:] = 0
        S4, S6 = 0.5 * (d1y + a2x), 0.5 * (a2z + d3y)
        P4, P6 = temp * (S4 - 0.5 * d1y), temp * (S6 - 0.5 * d3y)
        P4[1], P6[1] = S4[1], S6[1]
        L5, L6 = delt * P4 - nut * d1y, delt * P6 - nut * d3y
        cidyf = col(1.0 / self.dyf)
        L1, L3 = (up(delt * P4) - delt * P4) * cidyf, (up(delt * P6) - delt * P6) * cidyf
        L0, L2, L4 = dlf * s1 * a1x, dlf * s1 * 0.5 * (a1z + a3x), dlf * s1 * a3z
        L7, L8 = 0.5 * dlf * s1t * atx, 0.5 * dlf * s1t * atz
        L = [L0, L1, L2, L3, L4, L5, L6, L7, L8]
        for i, t in enumerate(L):
            lo, hi = (self.jst, n - 1) if i < 5 else (2, n) if i < 7 else (self.jth, n)
            t[:lo] = 0
            t[hi + 1:] = 0
        return nut, kat, L

    def nonlinear(self, L):
        """NL of u1, u2, u3, th (retained modes), the SGS forcing added to the products."""
        n, col, up, dn = self.ny, self.col, self.up, self.dn
        u1, u2, u3, th = self.pu
        Lt = (lambda i: L[i]) if L else (lambda i: 0.0)
        i2dyf = col(0.5 / self.dyf)
        idy = np.where(self.dy != 0, 1.0 / np.where(self.dy != 0, self.dy, 1.0), 0.0)
        wj = col(self.dyf * idy / 2)
        wm = col(np.concatenate([[0.0], self.dyf[:-1]]) * idy / 2)
        u2p = up(u2)
        Dy = lambda q: (up(q) * u2p + q * u2p - q * u2 - dn(q) * u2) * i2dyf   # noqa: E731
        gy = lambda q: wj * q + wm * dn(q)   # noqa: E731
        ikx, ikz = 1j * self.kx, 1j * self.kz
        sp = self.spec
        x13 = sp(u1 * u3 + Lt(2))
        n1 = ikx * sp(u1 * u1 + Lt(0)) + sp(Dy(u1) + Lt(1)) + ikz * x13
        n3 = ikx * x13 + sp(Dy(u3) + Lt(3)) + ikz * sp(u3 * u3 + Lt(4))
        q = 0.25 * (u2 + u2p) ** 2
        n2 = ikx * sp(gy(u1) * u2 + Lt(5)) + sp((q - dn(q)) * col(idy)) + ikz * sp(gy(u3) * u2 + Lt(6))
        nt = ikx * sp(th * u1 + Lt(7)) + sp(Dy(th)) + ikz * sp(th * u3 + Lt(8))
        return n1, n2, n3, nt

    def substep(self, rk):
        case, n, col = self.case, self.ny, self.col
        h = self.dt * (8.0 / 15.0, 2.0 / 15.0, 5.0 / 15.0)[rk]
        beta, zeta = (1.0, 25.0 / 8.0, 9.0 / 4.0)[rk], (0.0, -17.0 / 8.0, -5.0 / 4.0)[rk]
        cu1, cu2, cu3, cth = self.u
        L = nut = kat = None
        if self.les:
            g = [s.clone() for s in self.u]
            self.bc_vel_post(g[0], g[1], g[2])
            for s in (g[0], g[2], g[3]):
                s[n] = s[n - 1]
                s[n + 1] = s[n]
            g[3][1] = g[3][2]
            g[3][0] = g[3][1]
            self.pu = [self.phys(s) for s in g]
            nut, kat, L = self.closure(g)
        else:
            self.pu = [self.phys(s) for s in self.u]
        n1, n2, n3, nt = self.nonlinear(L)
        del L
        f, tw, m2 = self.f, 1.0 / self.f, self.m2
        yf, y = col(self.yf - 1.0), col(self.y - 1.0)
        nuk = self.nu * self.k2
        v2 = 0.5 * (cu2 + self.up(cu2))
        adv = lambda c, yy: 1j * c * (m2 * yy * tw * self.kz)   # noqa: E731
        w = np.where(self.dy != 0, 0.5 / np.where(self.dy != 0, self.dy, 1.0), 0.0)
        buoy = col(w) * (cth * col(np.concatenate([[0.0], self.dyf[:-1]])) + self.dn(cth) * col(self.dyf))
        buoy[..., 0, 0] = 0
        cf = [-nuk * cu1 + f * cu3 - adv(cu1, yf) - n1,
              -nuk * cu2 + buoy - adv(cu2, y) - n2,
              -nuk * cu3 - f * cu1 - adv(cu3, yf) - m2 * tw * v2 - n3,
              -nuk * cth - m2 * cu1 - adv(cth, yf) - nt]
        del n1, n2, n3, nt, buoy, v2
        cp = self.cp
        idy = np.where(self.dy != 0, 1.0 / np.where(self.dy != 0, self.dy, 1.0), 0.0)
        gp = [1j * self.kx * cp, (cp - self.dn(cp)) * col(idy), 1j * self.kz * cp, 0.0]
        cr = []
        for e in range(4):
            r = self.u[e] - h * gp[e] + beta * h * cf[e]
            if rk > 0:
                r = r + zeta * h * self.cf[e]
            lo = (self.jst, 2, self.jst, self.jth)[e]
            r[:lo] = 0
            r[n + 1:] = 0
            cr.append(r)
        self.cf = cf
        eqs = ("u1", "u2", "u3", "th")
        if self.les:
            new = [self.solve(eqs[e], self.pu[e], self.phys(cr[e]), h, kat if e == 3 else nut, False) for e in range(4)]
            vel = new[:3]
            self.u = [self.spec(q) for q in new]
        else:
            self.u = [self.solve(eqs[e], self.u[e], cr[e], h) for e in range(4)]
            vel = [self.phys(q) for q in self.u[:3]] if rk == 2 and case.get("variable_dt") else None
        dt = None
        if rk == 2 and case.get("variable_dt"):
            dt = self.courant(vel)
        self.rem_div(self.u[0], self.u[1], self.u[2], h)
        if dt is not None:
            self.dt = dt

    def courant(self, vel):
        j = slice(self.jst, self.ny + 1)
        dx, dz = self.lx / self.nx, self.lx / self.nz
        c3 = self.col(self.m2 / self.f * (self.yf - 1.0))
        m = max(float((vel[0][j].abs() / dx).max()), float((vel[1][j].abs() / self.col(self.dy)[j]).max()),
                float(((vel[2][j] + c3[j]).abs() / dz).max()))
        return min(1.0, 0.5 * min(dx, dz) ** 2 / self.nu, 2.0 * self.pi / self.f / 20.0,
                   float(np.float32(0.1)) * 2.0 * self.pi, 0.5 / m)


def exact(case, seed):
    kind = case["kind"]
    if kind == "fft":
        t = torch.randn((case["ny"] + 2, case["nz"], case["nx"]), generator=_gen(seed), device="cuda", dtype=torch.float64)
        s = torch.fft.rfft2(t)
        s[..., case["nx"] // 3 + 1:] = 0
        s[..., case["nz"] // 3 + 1:case["nz"] - case["nz"] // 3, :] = 0
        return torch.fft.irfft2(s, s=(case["nz"], case["nx"]))
    if kind == "train":
        feat, tgt, params, d = _train_data(case, seed)
        w = torch.tensor(params.astype(np.float64), device="cuda", requires_grad=True)
        box = _Exact.__new__(_Exact)
        mean, std, scale = (torch.tensor(d[k].astype(np.float64), device="cuda") for k in ("mean", "std", "scale"))
        box.net = dict(params=w, mean=mean, std=std, scale=scale)
        opt = torch.optim.Adam([w], lr=1e-3)
        loss = []
        for _ in range(case["steps"]):
            opt.zero_grad()
            v = (box.mlp(feat.double()) - tgt.double()).square().sum(1).mean()
            v.backward()
            opt.step()
            loss.append(v.item())
        return dict(loss=np.array(loss), params=w.detach())
    m2 = np.sqrt(1.0 / _ri(case, seed)) if kind == "ensemble" else None
    sim = _Exact(case, m2)
    sim.start(_initial(case, seed))
    for _ in range(case["steps"]):
        for rk in range(3):
            sim.substep(rk)
    u1, u2, u3, th = sim.u
    out = (u1, u2, u3, sim.cp, th)
    if kind == "ensemble":
        out = [o.transpose(0, 1).contiguous() for o in out]
    return [_to_ref(case, o) for o in out]
