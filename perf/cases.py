"""The work whose speed this repository looks after, as a user's program has it
done through :class:`simson_b200.bla.Channel`.

Kinds of case:

* ``dns``: RK3 steps of the channel without a subgrid model (the nonlinear
  step over xz-planes, the implicit Chebyshev-tau step over pencils), after
  which the resolved state is taken out on the device, as a coupled analysis
  takes it;
* ``les``: the same with a subgrid model (ADM-RT, dynamic Smagorinsky, the
  learned stress);
* ``xys``: samples of the xy statistics of a field and the running sums read;
* ``pressure``: the pressure of a field into page-locked host arrays, as
  before a field is saved.

``exact`` restates each in plain torch at 64 bits: dealiased Fourier products,
Chebyshev tau solves by elimination over the coefficients of all pencils at
once.  Arrays of it are [y][kz][kx], the order ``copy_block`` packs.
"""
import math

import numpy as np
import torch

from simson_b200.bla import Channel

PI = math.pi
RK_A, RK_B = (8 / 15, 5 / 12, 3 / 4), (0.0, -17 / 60, -5 / 12)
MODELS = ("none", "admrt", "smagorinsky", "learned")


def _dns(name, nx, ny, nz, precision, steps, **kw):
    case = dict(name=name, kind="dns", model="none", nx=nx, ny=ny, nz=nz, precision=precision, steps=steps,
                re=9000.0, xl=2 * PI, zl=PI, dt=0.002, rms=0.1)
    case.update(kw)
    return case


def listed():
    config_a = dict(re=4200.0, xl=4 * PI, zl=2 * PI, dt=0.01, rms=0.02)
    config_b = dict(re=4200.0, xl=4 * PI, zl=2 * PI, dt=0.005, rms=0.1)
    les = dict(kind="les", dt=0.005)
    return [
        # a transition study on a small grid: launches and latency count
        _dns("dns 48x65x48 fp64", 48, 65, 48, "fp64", 4, **config_a),
        # a coarse run without a model, the base line of every LES
        _dns("dns 64x97x64 mixed", 64, 97, 64, "mixed", 4, dt=0.005),
        # resolutions chosen for the physics and not for powers of two
        _dns("dns 100x101x90 mixed", 100, 101, 90, "mixed", 4, dt=0.004),
        # Re_tau ~ 200 production DNS, both precisions
        _dns("dns 192x129x160 mixed", 192, 129, 160, "mixed", 2, **config_b),
        _dns("dns 192x129x160 fp64", 192, 129, 160, "fp64", 2, **config_b),
        # Re_tau ~ 395 production DNS, the headline grid, both precisions
        _dns("dns 384x193x384 mixed", 384, 193, 384, "mixed", 2),
        _dns("dns 384x193x384 fp64", 384, 193, 384, "fp64", 2),
        # LES at the grid of the reference's LES configuration
        _dns("les smagorinsky 64x97x64 fp64", 64, 97, 64, "fp64", 2, model="smagorinsky", **les),
        _dns("les admrt 64x97x64 fp64", 64, 97, 64, "fp64", 2, model="admrt", **les),
        _dns("les learned 64x97x64 mixed", 64, 97, 64, "mixed", 2, model="learned", **les),
        # statistics of a production run: some samples, then the sums
        _dns("xys 192x129x160 mixed", 192, 129, 160, "mixed", 4, kind="xys", **config_b),
        # the pressure that goes with a saved field
        _dns("pressure 192x129x160 fp64", 192, 129, 160, "fp64", 1, kind="pressure", **config_b),
    ]


def _smooth(n):
    for f in (2, 3, 5):
        while n % f == 0:
            n //= f
    return n == 1


_NX = [n for n in range(16, 385, 4) if _smooth(n)]          # nx % 4 == 0
_NZ = [n for n in range(16, 385, 2) if _smooth(n)]          # nz even
_NY = [n + 1 for n in range(16, 257, 2) if _smooth(n)]      # ny - 1 even


def _near(rng, sizes, lo, hi):
    """A size of the list, log-uniform between lo and hi."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(sizes, key=lambda n: abs(n - x))


def draw(rng):
    kind = rng.choices(("dns", "les", "xys", "pressure"), (6, 3, 1, 1))[0]
    precision = rng.choice(("fp64", "mixed"))
    model = rng.choice(MODELS[1:]) if kind == "les" else "none"
    hi = {"dns": 384, "les": 96, "xys": 192, "pressure": 192}[kind]
    lo = 16 if kind == "dns" else 32
    nx = _near(rng, _NX, lo, hi)
    nz = _near(rng, [n for n in _NZ if kind != "les" or n % 4 == 0], lo, hi)
    ny = _near(rng, _NY, max(17, lo), {384: 257, 96: 129}.get(hi, 193))
    while nx * ny * nz > 384 * 193 * 384:
        ny = _NY[_NY.index(ny) - 1]
    xl, zl = (2 * PI, PI) if rng.random() < 0.5 else (4 * PI, 2 * PI)
    points = nx * ny * nz
    steps = {"dns": 4 if points < 1_500_000 else 2, "les": 2, "xys": rng.randint(2, 4), "pressure": 1}[kind]
    return dict(kind=kind, model=model, nx=nx, ny=ny, nz=nz, precision=precision, steps=steps,
                re=9000.0 if min(nx, nz) >= 96 else 4200.0, xl=xl, zl=zl,
                dt=0.08 * min(xl / nx, zl / nz * 4), rms=rng.choice((0.05, 0.1)))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _modes(case):
    """alpha over the stored kx, beta over kz (the last half negative)."""
    nx, nz = case["nx"], case["nz"]
    al = 2 * PI / case["xl"] * torch.arange(nx // 2, dtype=torch.float64)
    kz = torch.arange(nz, dtype=torch.float64)
    kz[nz // 2 + 1:] -= nz
    kz[nz // 2] = -(nz // 2)
    return al.to(_device()), (2 * PI / case["zl"] * kz).to(_device())


def _velocity(case, seed):
    """u, v, w [3][y][kz][kx] of a seeded, divergence-free field that meets
    the walls: every stored mode, amplitudes falling off with the wavenumber
    as those of a developed flow do, four wall-normal shapes per mode, on the
    laminar profile."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dev, g = _device(), torch.Generator().manual_seed(int(seed))
    c = torch.randn((2, 4, nz, nx // 2, 2), generator=g, dtype=torch.float64)
    c = torch.view_as_complex(c)
    al, be = _modes(case)
    kx = torch.arange(nx // 2, dtype=torch.float64)
    kz = (be.cpu() * case["zl"] / (2 * PI))
    c = c * (1 + (kx[None, :] ** 2 + kz[:, None] ** 2) / 16.0) ** -1.75
    back = (-torch.arange(nz)) % nz
    c[..., 0] = 0.5 * (c[..., 0] + c[..., back, 0].conj())  # kx = 0: a real field
    c[..., 0, 0] = 0
    c[..., nz // 2, :] = 0                                   # the oddball mode
    y = np.cos(PI * np.arange(ny) / (ny - 1))
    wall = np.polynomial.Polynomial([1, 0, -1]) ** 2
    shapes = [wall * np.polynomial.Chebyshev.basis(q).convert(kind=np.polynomial.Polynomial) * (1 / (1 + q))
              for q in range(4)]
    b = torch.tensor(np.stack([s(y) for s in shapes]), device=dev).to(torch.complex128)
    db = torch.tensor(np.stack([s.deriv()(y) for s in shapes]), device=dev).to(torch.complex128)
    c = c.to(dev)
    v = torch.einsum("qzx,qy->yzx", c[0], b)
    dv = torch.einsum("qzx,qy->yzx", c[0], db)
    om = torch.einsum("qzx,qy->yzx", c[1], b)
    k2 = al[None, :] ** 2 + be[:, None] ** 2
    k2[0, 0] = 1.0
    ia, ib = 1j * al[None, :] / k2, 1j * be[:, None] / k2
    vel = torch.stack([ia * dv - ib * om, v, ib * dv + ia * om])
    e = vel.abs() ** 2
    e[..., 1:] *= 2
    wy = torch.tensor(np.sin(PI * np.arange(ny) / (ny - 1)) * PI / (ny - 1) / 2, device=dev)
    vel *= case["rms"] / math.sqrt(float((e.sum((0, 2, 3)) * wy).sum()) / 3)
    vel[0, :, 0, 0] += torch.tensor(1 - y * y, device=dev)
    return vel


def _weights(seed):
    """A network of the learned stress, its weights representable in BF16."""
    rng = np.random.default_rng(int(seed))
    w = {"w1": rng.standard_normal((64, 10)) / math.sqrt(10.0), "b1": 0.1 * rng.standard_normal(64),
         "w2": rng.standard_normal((64, 64)) / 8.0, "b2": 0.1 * rng.standard_normal(64),
         "w3": rng.standard_normal((6, 64)) / 8.0, "b3": 0.1 * rng.standard_normal(6)}
    return {k: torch.tensor(v).to(torch.bfloat16).float().numpy() for k, v in w.items()}


MLP_SCALES = dict(s_in=0.1, s_y=1.0, s_out=1e-4)


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    ch = Channel(nx, ny, nz, case["re"], case["xl"], case["zl"], case["dt"], precision=case["precision"])
    if case["model"] == "admrt":
        ch.set_les(iles=1)
    elif case["model"] == "smagorinsky":
        ch.set_les(iles=2)
    elif case["model"] == "learned":
        ch.set_sgs_mlp(_weights(seed), **MLP_SCALES)
    vel = _velocity(case, seed).permute(0, 2, 1, 3)  # the host layout: [slot][kz][y][kx]
    re, im = vel.real.contiguous().cpu(), vel.imag.contiguous().cpu()
    ch.upload_raw(re.data_ptr(), im.data_ptr(), 3)
    ch.start()
    s.ch = ch
    # the two blocks of kz planes around the oddball mode, which carries nothing
    s.blocks = [(0, nz // 2), (nz // 2 + 1, nz)]
    s.bufs = []
    if case["kind"] in ("dns", "les"):
        for lo, hi in s.blocks:
            s.bufs.append(torch.empty(ch.copy_block(0, 7, 0, ny, lo, hi), dtype=torch.uint8, device="cuda"))
    elif case["kind"] == "pressure":
        s.p = [torch.empty((nz, ny, nx // 2), dtype=torch.float64, pin_memory=True) for _ in range(2)]
    ch.sync()
    return s


def run(s):
    ch, case = s.ch, s.case
    if case["kind"] == "pressure":
        ch.pressure_raw(s.p[0].data_ptr(), s.p[1].data_ptr())
        return list(s.p)
    if case["kind"] == "xys":
        ch.xys_reset()
        for _ in range(case["steps"]):
            ch.xys_sample()
        sums, weight = ch.xys()
        return _xys_groups(sums) + [weight]
    ch.step(case["steps"])
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    out = []
    for (lo, hi), buf in zip(s.blocks, s.bufs):
        ch.copy_block(0, 7, 0, ny, lo, hi, buf.data_ptr(), nosync=True)
        split = 5 * ny * (hi - lo) * (nx // 2) * (8 if case["precision"] == "mixed" else 16)
        f = buf[:split].view(torch.float32 if case["precision"] == "mixed" else torch.float64)
        f = f.view(5, ny, hi - lo, nx // 2, 2)
        p = buf[split:].view(torch.float64).view(2, ny, hi - lo, nx // 2, 2)
        out += [f[:3], f[3:], p]  # velocity, vorticity, the next stage's right-hand sides
    return out


def _xys_groups(x):
    """The entries of the reference's numbering in groups of like size."""
    cuts = (0, 3, 6, 9, 12, 15, 24, 27, 30, 42, 44, 45, 51, 62, 72, 74, 96)
    return [x[a:b] for a, b in zip(cuts, cuts[1:])]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    modes = nx // 2 * ny * nz
    size = 8 if case["precision"] == "mixed" else 16
    fft_x, fft_z = 2.5 * 1.5 * nx * math.log2(1.5 * nx), 5 * 1.5 * nz * math.log2(1.5 * nz)
    plane = lambda inv, fwd: ny * (1.5 * nz * (inv + fwd) * fft_x + nx / 2 * (inv + fwd) * fft_z)  # noqa: E731
    if case["kind"] == "pressure":  # five fields read, the pressure written
        return {"bytes": modes * (5 * size + 16), "flops": plane(6, 4)}
    if case["kind"] == "xys":  # five fields read a sample; the sums out once
        per = ny * (nz * 16 * 2.5 * nx * math.log2(nx) + nx / 2 * 16 * 5 * nz * math.log2(nz) + 160 * nx * nz)
        return {"bytes": case["steps"] * 5 * modes * size + 96 * nx * ny * 8, "flops": case["steps"] * per}
    # a substep: five fields to physical space and H back; H, both right-hand
    # sides in and the five fields, both right-hand sides out
    bytes_ = modes * (16 * size + 4 * 16)
    flops = plane(6, 3) + modes * (8 * 5 * math.log2(2 * ny) + 400)
    if case["model"] != "none":  # the stress and its force, or the filtered velocity, once each way
        bytes_ += modes * 6 * 16
        flops += {"admrt": modes * 3 * 6 * 40, "smagorinsky": 3.0 * plane(6, 3),
                  "learned": nx * ny * nz * 10240 + 1.0 * plane(6, 3)}[case["model"]]
    n = 3 * case["steps"]
    return {"bytes": n * bytes_, "flops": n * flops}


def tolerance(case):
    """About four times the distance from ``exact`` that was seen.  The mixed
    path's is that of FP32 storage under two to four wall-normal derivatives,
    the FP64 path's that of the stiff tau solves (larger with ny), the learned
    stress's that of BF16 weights and activations."""
    mixed = case["precision"] == "mixed"
    if case["kind"] == "xys":  # seen: 1.1e-7 mixed
        return {"rel": 5e-7 if mixed else 1e-11}
    if case["kind"] == "pressure":  # seen: 5.4e-7 (3.3e-6 on another grid) mixed, 2e-12
        return {"rel": 1e-5 if mixed else 1e-10}
    if case["model"] == "learned":  # seen: 4.8e-3
        return {"rel": 2e-2}
    return {"rel": 1.2e-5 if mixed else 1e-8}  # seen: 2.8e-6 mixed, 2.3e-10 (ny up to 193)


# ---------------------------------------------------------------------------
# the same in plain torch at 64 bits
# ---------------------------------------------------------------------------
class _Exact:
    """Chebyshev, Fourier and tau tools of one case's grid."""

    def __init__(self, case):
        self.case, self.dev = case, _device()
        n = self.n = case["ny"]
        j = np.arange(n)
        cb = np.where((j == 0) | (j == n - 1), 2.0, 1.0)
        cos = np.cos(PI * np.outer(j, j) / (n - 1))
        self.to_phys = self._mat(cos)
        self.to_cheb = self._mat(2 / (n - 1) * cos / np.outer(cb, cb))
        d = np.zeros((n, n))
        for k in range(1, n):
            d[k - 1::-2, k] = 2.0 * k
        d[0] *= 0.5
        self.d = self._mat(d)
        self.al, self.be = _modes(case)
        self.k2 = self.al[None, :] ** 2 + self.be[:, None] ** 2

    def _mat(self, a):
        return torch.tensor(a, device=self.dev)

    def y(self, m, f):
        """A real matrix along y of complex fields [..., y, kz, kx]."""
        return torch.view_as_complex(torch.einsum("jk,...kzxc->...jzxc", m, torch.view_as_real(f)).contiguous())

    def phys(self, f, nx, nz):
        """Spectral [y, kz, kx] on an nx x nz grid, unnormalised, oddball dropped."""
        h = self.case["nz"] // 2
        g = torch.zeros((self.n, nz, nx // 2 + 1), dtype=torch.complex128, device=self.dev)
        g[:, :h, :f.shape[2]] = f[:, :h]
        g[:, nz - h + 1:, :f.shape[2]] = f[:, h + 1:]
        return torch.fft.irfft2(g, s=(nz, nx), dim=(1, 2), norm="forward")

    def spec(self, p):
        """Back, divided by the number of points; the oddball plane zero."""
        h = self.case["nz"] // 2
        g = torch.fft.rfft2(p, dim=(1, 2), norm="forward")[:, :, :self.case["nx"] // 2]
        out = torch.zeros((self.n, 2 * h, g.shape[2]), dtype=torch.complex128, device=self.dev)
        out[:, :h] = g[:, :h]
        out[:, h + 1:] = g[:, g.shape[1] - h + 1:]
        return out

    def tau(self, lam, f, neumann=None):
        """(D^2 - lam) x = f by the tau method: rows of the twice integrated
        equation, x = 0 at the walls, or D x = neumann[0], [1] at y = +1, -1
        (lam and f over [kz, kx], f leading in y)."""
        n, x = self.n, torch.zeros_like(f)
        resp = [None, None]
        for par in (0, 1):
            js = list(range(par, n, 2))
            rows = []
            for j in js[1:]:
                m = j - 1  # 1-based row i = j + 1, m = i - 2
                i = j + 1
                c = (-0.25 if m == 1 else -0.25 / (m * (m + 1))) * lam
                d = 1 + 0.5 / (m * (m + 2)) * lam if i <= n - 2 else torch.ones_like(lam)
                e = -0.25 / ((m + 1) * (m + 2)) * lam if i <= n - 4 else None
                r = (0.25 if j == 2 else 0.25 / ((i - 2) * (i - 1))) * f[j - 2]
                if i <= n - 2:
                    r = r - 0.5 / ((i - 2) * i) * f[j]
                if i <= n - 4:
                    r = r + 0.25 / ((i - 1) * i) * f[j + 2]
                rows.append([c, d, e, r])
            # from the last row up: x_j = u_j + w_j x_{j-2}
            u, w = [None] * len(rows), [None] * len(rows)
            for q in range(len(rows) - 1, -1, -1):
                c, d, e, r = rows[q]
                if e is not None and q + 1 < len(rows):
                    d = d + e * w[q + 1]
                    r = r - e * u[q + 1]
                u[q], w[q] = r / d, -c / d
            # all of them as P + y0 Q of the class's first unknown
            p, s = torch.zeros_like(f[0]), torch.ones_like(lam)
            ps, qs = [p], [s]
            for q in range(len(rows)):
                p, s = u[q] + w[q] * p, w[q] * s
                ps.append(p)
                qs.append(s)
            if neumann is None:
                y0 = -sum(ps) / sum(qs)
            else:
                k2 = [float(j * j) for j in js]
                rhs = (neumann[0] - neumann[1]) / 2 if par == 0 else (neumann[0] + neumann[1]) / 2
                y0 = (rhs - sum(a * b for a, b in zip(k2, ps))) / sum(a * b for a, b in zip(k2, qs))
            for q, j in enumerate(js):
                x[j] = ps[q] + y0 * qs[q]
            resp[par] = (js, qs)
        return x, resp

    def curl(self, vel):
        """omega_x, omega_y, omega_z of Chebyshev coefficients."""
        ia, ib = 1j * self.al, 1j * self.be[:, None]
        u, v, w = vel
        return self.y(self.d, w) - ib * v, ib * u - ia * w, ia * v - self.y(self.d, u)

    def products(self, st):
        """u x omega and |u|^2 / 2 on the dealiased grid, back in Fourier space."""
        u, v, w, ox, oz = st
        oy = 1j * self.be[:, None] * u - 1j * self.al * w
        nx, nz = 3 * self.case["nx"] // 2, 3 * self.case["nz"] // 2
        u, v, w, ox, oy, oz = (self.phys(q, nx, nz) for q in (u, v, w, ox, oy, oz))
        return (self.spec(v * oz - w * oy), self.spec(w * ox - u * oz), self.spec(u * oy - v * ox),
                self.spec((u * u + v * v + w * w) / 2))

    def gradients(self, st):
        """du_i/dx_j, i-major, from velocity and vorticity in physical y."""
        u, v, w, ox, oz = st
        ia, ib = 1j * self.al, 1j * self.be[:, None]
        return [ia * u, ia * v - oz, ib * u, ia * v, -(ia * u + ib * w), ib * v, ia * w, ox + ib * v, ib * w]

    def force(self, tau):
        """sigma_i = d tau_ij / dx_j of tau (11 12 13 22 23 33), physical y."""
        ia, ib = 1j * self.al, 1j * self.be[:, None]
        t = [self.y(self.to_cheb, q) for q in tau]
        dy = lambda q: self.y(self.to_phys, self.y(self.d, q))  # noqa: E731
        t11, t12, t13, t22, t23, t33 = range(6)
        return [ia * tau[t11] + ib * tau[t13] + dy(t[t12]), ia * tau[t12] + ib * tau[t23] + dy(t[t22]),
                ia * tau[t13] + ib * tau[t33] + dy(t[t23])]

    def smagorinsky(self, st):
        """The dynamic model's stress: z-averaged coefficient, clipped at zero."""
        nx, nz = self.case["nx"], self.case["nz"]
        g = [self.phys(q, nx, nz) for q in self.gradients(st)]
        s = [g[0], (g[1] + g[3]) / 2, (g[2] + g[6]) / 2, g[4], (g[5] + g[7]) / 2, g[8]]
        u = [self.phys(q, nx, nz) for q in st[:3]]
        mag = lambda t: torch.sqrt(2 * (t[0] ** 2 + t[3] ** 2 + t[5] ** 2)  # noqa: E731
                                   + 4 * (t[1] ** 2 + t[2] ** 2 + t[4] ** 2))
        keep_z = torch.ones(nz, device=self.dev)
        keep_z[nz // 4 + 1:nz - nz // 4] = 0

        def cut(p):
            f = torch.fft.rfft2(p, dim=(1, 2)) * keep_z[None, :, None]
            f[:, :, nx // 4:] = 0
            return torch.fft.irfft2(f, s=(nz, nx), dim=(1, 2))

        eta = np.cos(PI * np.arange(self.n) / (self.n - 1))
        dy = np.full(self.n, 1 - eta[1])
        dy[1:-1] = np.sqrt((eta[2:] - eta[1:-1]) * (eta[1:-1] - eta[:-2]))
        d2 = self._mat((self.case["xl"] / nx * self.case["zl"] / nz * dy) ** (2 / 3))[:, None, None]
        sab = mag(s)
        ub, sb = [cut(q) for q in u], [cut(q) for q in s]
        pairs = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))
        lij = [ub[i] * ub[j] - cut(u[i] * u[j]) for i, j in pairs]
        sbm = mag(sb)
        mij = [4 ** (2 / 3) * d2 * sbm * sb[q] - cut(d2 * sab * s[q]) for q in range(6)]
        dot = lambda a, b: (a[0] * b[0] + a[3] * b[3] + a[5] * b[5]  # noqa: E731
                            + 2 * (a[1] * b[1] + a[2] * b[2] + a[4] * b[4])).sum(1, keepdim=True)
        c = (0.5 * dot(mij, lij) / dot(mij, mij)).clamp_min(0)
        c[0] = c[-1] = 0
        return [self.spec(-2 * c * d2 * sab * q) for q in s]

    def learned(self, st, w):
        """The learned model's stress, the network evaluated at 64 bits."""
        nx, nz, sc = self.case["nx"], self.case["nz"], MLP_SCALES
        g = [self.phys(q, nx, nz) * sc["s_in"] for q in self.gradients(st)]
        wall = 1 - torch.cos(PI * torch.arange(self.n, device=self.dev, dtype=torch.float64) / (self.n - 1)).abs()
        x = torch.stack(g + [(sc["s_y"] * wall)[:, None, None].expand_as(g[0])], -1)
        w = {k: torch.tensor(v, device=self.dev).double() for k, v in w.items()}
        h = torch.tanh(x @ w["w1"].T + w["b1"])
        h = torch.tanh(h @ w["w2"].T + w["b2"])
        t = sc["s_out"] * (h @ w["w3"].T + w["b3"])
        return [self.spec(t[..., q]) for q in range(6)]

    def high_pass(self):
        """The ADM-RT filter of a field: (wall-normal high pass)^6 in y, the
        uniform-grid transfer functions in x and z (cut-off 2/3, order 5)."""
        cutoff, order, n = 1 / 1.5, 5, self.n

        def explicit(x, s, centred):
            x = np.asarray(x) / np.max(np.abs(x))
            s = np.asarray(s)
            rows = [np.ones(5), x, x * x, (-1.0) ** s]
            if not centred:
                return np.linalg.solve(np.stack(rows + [x ** 3]), [1, 0, 0, 0, 0.0])
            last = np.array([0, 0, 0, 0, 1.0])
            c0, c1 = (np.linalg.solve(np.stack(rows + [last]), [1, 0, 0, 0, float(t)]) for t in (0, 1))
            nul = c1 - c0
            a = np.array([c0[4] - c0[0], c0[3] - c0[1]])
            b = np.array([nul[4] - nul[0], nul[3] - nul[1]])
            return c0 - nul * (a @ b) / (b @ b) if b @ b > 1e-30 else c0

        def implicit(b, s, centre):
            z = (b * np.exp(1j * np.asarray(s) * PI * cutoff)).sum()
            al, be, ga = abs(z - 1) ** 2, 2 * (z.real - 1), 1 - 4 * abs(z) ** 2
            a = (-be - math.sqrt(be * be - 4 * al * ga)) / (2 * al) * b
            a[centre] = 0
            a[centre] = 1 - a.sum()
            return a

        y = np.cos(PI * np.arange(n) / (n - 1))
        lhs, rhs = np.eye(n), np.zeros((n, n))
        for k in range(1, n - 1):
            first = min(max(k - 2, 0), n - 5)
            s = np.arange(first, first + 5) - k
            b = explicit(y[k] - y[first:first + 5], s, 2 <= k <= n - 3)
            a = implicit(b, s, k - first)
            lhs[k, first:first + 5], rhs[k, first:first + 5] = a, a - b
        h = np.linalg.matrix_power(np.linalg.solve(lhs, rhs), order + 1)
        s = np.arange(-2, 3)
        b = explicit(s.astype(float), s, True)
        a = implicit(b, s, 2)

        def transfer(m):
            k = np.arange(m + 1) * PI / m
            e = np.exp(1j * np.outer(k, s))
            return ((e @ b) / (e @ a)).real

        nx, nz = self.case["nx"], self.case["nz"]
        gx, gz = transfer(nx // 2)[:nx // 2], transfer(nz // 2)
        gz = gz[np.minimum(np.arange(nz), nz - np.arange(nz))]
        low = self._mat(1 - (1 - np.outer(gz, gx)) ** (order + 1))
        h = self._mat(h)
        return lambda f: f - low * (f - self.y(h, f))

    def steps(self, seed, nsteps):
        """The state after nsteps RK3 steps: the five fields in physical y,
        the two right-hand sides in Chebyshev space."""
        case, re = self.case, self.case["re"]
        al, be, k2 = self.al, self.be[:, None], self.k2
        ia, ib = 1j * al, 1j * be
        dd = self.d @ self.d
        vel = _velocity(case, seed)
        a = [case["dt"] * q for q in RK_A]
        b = [case["dt"] * q for q in RK_B]
        cv = [self.y(self.to_cheb, q) for q in vel]
        ox, oy, oz = self.curl(cv)
        lam = k2 - 2 * re / a[0]
        phi = self.y(dd, cv[1]) - k2 * cv[1]
        pw = lam * oy - self.y(dd, oy)
        pv = lam * phi - self.y(dd, phi)
        mean = lambda q: q[:, 0, 0].real  # noqa: E731
        puw = [-2 * re / a[0] * mean(q) - dd @ mean(q) for q in (cv[0], cv[2])]
        st = list(vel) + [self.y(self.to_phys, ox), self.y(self.to_phys, oz)]
        if nsteps == 0:
            return st, [pv, pw]
        px = -2 / re
        filt = self.high_pass() if case["model"] == "admrt" else None
        inv_k2 = torch.where(k2 > 0, 1 / k2.clamp_min(1e-300), torch.zeros_like(k2))
        ones = torch.ones((1, 1), device=self.dev, dtype=torch.float64)
        even = torch.arange(0, self.n, 2, device=self.dev, dtype=torch.float64)
        for sub in range(3 * nsteps):
            h = list(self.products(st)[:3])
            if case["model"] == "admrt":
                h = [q - 0.2 * filt(f) for q, f in zip(h, st[:3])]
            elif case["model"] != "none":
                t = self.smagorinsky(st) if case["model"] == "smagorinsky" else self.learned(st, _weights(seed))
                h = [q - f for q, f in zip(h, self.force(t))]
            for q in h:
                q[:, case["nz"] // 2] = 0
            h = [self.y(self.to_cheb, q) for q in h]
            an, bn, a1, b1 = a[sub % 3], b[sub % 3], a[(sub + 1) % 3], b[(sub + 1) % 3]
            c0, c1n, c2 = 2 * re / (an + bn), 2 * re / (a1 + b1), 2 * re * b1 / (a1 + b1)
            hv = -(self.y(self.d, ia * h[0] + ib * h[2]) + k2 * h[1])
            hom = ib * h[0] - ia * h[2]
            lam = k2 + c0
            phi, resp = self.tau(lam, pv - c0 * an * hv)
            om, _ = self.tau(lam, pw - c0 * an * hom)
            # v from phi; the class solutions of phi with unit wall values add
            # what makes D v vanish at the walls
            v, _ = self.tau(k2, phi)
            for par in (0, 1):
                js, qs = resp[par]
                ph = torch.zeros(phi.shape, dtype=torch.float64, device=self.dev)
                tot = sum(qs)
                for j, q in zip(js, qs):
                    ph[j] = q / tot
                vh, _ = self.tau(k2, ph)
                kk = torch.arange(self.n, device=self.dev, dtype=torch.float64) ** 2
                sel = torch.zeros_like(kk)
                sel[par::2] = 1
                slope_v = torch.einsum("k,kzx->zx", (kk * sel).to(torch.complex128), v)
                slope_h = torch.einsum("k,kzx->zx", kk * sel, vh)
                v = v - slope_v / slope_h * vh
                del ph, vh
            dv = self.y(self.d, v)
            phi = self.y(self.d, dv) - k2 * v
            dom = self.y(self.d, om)
            new = [(ia * dv - ib * om) * inv_k2, v, (ib * dv + ia * om) * inv_k2,
                   (ia * dom + ib * phi) * inv_k2, (ib * dom - ia * phi) * inv_k2]
            pv = (k2 - c1n) * phi - self.y(dd, phi) - c2 * hv
            pw = (k2 - c1n) * om - self.y(dd, om) - c2 * hom
            # the mean flow, its pressure gradient set by the mass flux 4/3
            fm = [puw[q] - c0 * an * mean(h[2 * q]) for q in (0, 1)]
            solve = lambda f: self.tau(c0 * ones, f[:, None, None])[0][:, 0, 0]  # noqa: E731
            unit = torch.zeros_like(fm[0])
            unit[0] = 2 * re
            base, one = solve(fm[0]), solve(unit)
            flux = lambda q: -(q[::2] * 2 / (even * even - 1)).sum()  # noqa: E731
            px = (4 / 3 - flux(base)) / flux(one)
            um, wm = base + px * one, solve(fm[1])
            for q, f in zip(new, (um, 0, wm, self.d @ wm, -(self.d @ um))):
                q[:, 0, 0] = f
            pv[:, 0, 0] = 0
            pw[:, 0, 0] = 0
            puw = [-(dd @ q) - c1n * q - c2 * mean(h[2 * i]) for i, q in enumerate((um, wm))]
            st = [self.y(self.to_phys, q) for q in new]
        return st, [pv, pw]

    def pressure(self, seed):
        st, _ = self.steps(seed, 0)
        h1, h2, h3, e = self.products(st)
        ia, ib = 1j * self.al, 1j * self.be[:, None]
        c = lambda q: self.y(self.to_cheb, q)  # noqa: E731
        ch2, cv = c(h2), c(st[1])
        ddv = self.y(self.to_phys, self.y(self.d @ self.d, cv)) - self.k2 * st[1]
        bc = [h2[q] + ddv[q] / self.case["re"] for q in (0, -1)]
        k2 = self.k2.clone()
        k2[0, 0] = 1.0
        x, _ = self.tau(k2, c(ia * h1 + ib * h3) + self.y(self.d, ch2), bc)
        # the mean: the integral of H2, its value at y = -1 that of |u|^2 / 2
        t = ch2[:, 0, 0].real.clone()
        t[-1] = 0
        m, k = torch.zeros_like(t), torch.arange(self.n, device=self.dev, dtype=torch.float64)
        m[1:-1] = (t[:-2] - t[2:]) / (2 * k[1:-1])
        m[1] += t[0] / 2
        m[-1] = t[-2] / (2 * k[-1])
        sign = torch.where(k % 2 == 0, 1.0, -1.0)
        m[0] = e[-1, 0, 0].real - (sign * m).sum()
        x[:, 0, 0] = m
        p = self.y(self.to_phys, x) - e
        p[:, self.case["nz"] // 2] = 0
        p = p.permute(1, 0, 2)
        return [p.real.contiguous(), p.imag.contiguous()]

    def xys(self, seed):
        st, _ = self.steps(seed, 0)
        nx, nz, count = self.case["nx"], self.case["nz"], self.case["steps"]
        oy = 1j * self.be[:, None] * st[0] - 1j * self.al * st[2]
        u = [self.phys(q, nx, nz) for q in st[:3]]
        o = [self.phys(q, nx, nz) for q in (st[3], oy, st[4])]
        g = [self.phys(q, nx, nz) for q in self.gradients(st)]
        out = torch.zeros((96, self.n, nx), dtype=torch.float64, device=self.dev)
        weight = count * self.case["dt"]

        def put(at, *fields):
            for q, f in enumerate(fields):
                out[at - 1 + q] = weight * f.mean(1)

        s = [g[0], (g[3] + g[1]) / 2, (g[6] + g[2]) / 2, g[4], (g[5] + g[7]) / 2, g[8]]
        dot = lambda i, j: sum(g[3 * i + q] * g[3 * j + q] for q in range(3))  # noqa: E731
        put(1, *u)
        put(4, *(q * q for q in u))
        put(7, *o)
        put(10, *(q * q for q in o))
        put(13, u[0] * u[1], u[0] * u[2], u[1] * u[2])
        put(25, dot(0, 0), dot(1, 1), dot(2, 2), dot(0, 1), dot(0, 2), dot(1, 2))
        d = u[0] - u[0].mean(1, keepdim=True)
        out[42], out[43] = d.amin(1).clamp_max(0), d.amax(1).clamp_min(0)
        put(45, s[0] ** 2 + s[3] ** 2 + s[5] ** 2 + 2 * (s[1] ** 2 + s[2] ** 2 + s[4] ** 2), *s)
        put(63, *(q ** 3 for q in u))
        put(66, u[0] ** 2 * u[1], u[0] ** 2 * u[2], u[1] ** 2 * u[0], u[1] ** 2 * u[2], u[2] ** 2 * u[0],
            u[2] ** 2 * u[1], u[0] * u[1] * u[2])
        put(75, *(q ** 4 for q in u))
        return _xys_groups(out) + [weight]


def exact(case, seed):
    x = _Exact(case)
    if case["kind"] == "pressure":
        return x.pressure(seed)
    if case["kind"] == "xys":
        return x.xys(seed)
    st, p = x.steps(seed, case["steps"])
    nz, out = case["nz"], []
    for lo, hi in ((0, nz // 2), (nz // 2 + 1, nz)):
        for fields in (st[:3], st[3:], p):
            out.append(torch.view_as_real(torch.stack([q[:, lo:hi] for q in fields])))
    return out
