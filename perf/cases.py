"""What a user of this framework has it compute, as cases that can be timed and compared.

Every case is honeycomb graphene (nearest-neighbour hopping -2.7 eV, Anderson on-site
disorder), the model of the benchmark configurations and of the tests, and goes through the
package's public entry points:

  moments      device.cheb_moments: one vector set, two sets, or both products of one pass
               (rec_A_tab, rec_A_tab2v, rec_A_tab2v_2), complex128 or complex64
  dos          observables_gpu.kpm_dos_gpu on host arrays, from the matrix to rho(E)
  evolve       device.time_evolve: U and U_c advanced by the exp(-i H t) series
  batch        batched.BatchedELL.moments: disorder instances of uneven size together
  mu_nm        kubo.mu_nm: the Kubo-Greenwood moment matrix
  grad_dos     adjoint.kpm_dos and its gradient (a training step on on-site terms, hoppings)
  grad_sigma   adjoint.kpm_sigma and its gradient (the same for the conductivity)
  time_sigma   device.time_sigma: the commutator series and the time-domain correlator

The 64-bit values of `exact` are formed on the [ny, nx] cell grid with torch.roll, without
ELL arrays and without this package.
"""
import math

import numpy as np
import torch

from minijclsquant_gb300 import adjoint, batched, device, kubo, lattice, observables_gpu

T_HOP = -2.7
A_CC = 0.14199929870718847  # nm, carbon-carbon distance


def listed():
    return [
        # the smallest calls: one vector on a flake of a thousand sites, a user trying things out
        dict(name="moments_small", kind="moments", nx=24, ny=22, R=1, M=128, W=0.5, dtype="c128", pair="one",
             peierls=0.0, periodic=True),
        # the whole drop-in call of the 8,192-site configuration, host arrays in and rho(E) out
        dict(name="dos_64x64", kind="dos", nx=64, ny=64, R=4, M=512, W=0.5, n_energies=1024),
        # one random vector on a lattice with odd sides, as the reference's own interface passes them
        dict(name="moments_one_vector", kind="moments", nx=301, ny=173, R=1, M=512, W=1.0, dtype="c128", pair="one",
             peierls=0.0, periodic=True),
        # local DOS with separate bra and ket under a vector potential: complex hoppings, open edges
        dict(name="moments_two_sided", kind="moments", nx=389, ny=517, R=2, M=128, W=1.0, dtype="c128", pair="both",
             peierls=1.3, periodic=False),
        # the large plain DOS: 8.4M sites, eight random vectors advanced together
        dict(name="moments_large", kind="moments", nx=2048, ny=2048, R=8, M=64, W=1.0, dtype="c128", pair="one",
             peierls=0.0, periodic=True),
        # the same work in mixed precision on a lattice of medium size
        dict(name="moments_c64", kind="moments", nx=1024, ny=1024, R=4, M=256, W=1.0, dtype="c64", pair="one",
             peierls=0.0, periodic=True),
        # time evolution of U and U_c by two steps of the exp(-i H t) series
        dict(name="evolve", kind="evolve", nx=1024, ny=1024, R=2, M=64, steps=2, W=1.0, dtype="c128"),
        # an ensemble of disorder instances, sides from 32 to 512 cells as in the batched configuration
        dict(name="batch", kind="batch", n_inst=20, lo=32, hi=512, sides_seed=42, R=2, M=256, dtype="c64"),
        # the Kubo-Greenwood configuration
        dict(name="mu_nm", kind="mu_nm", nx=1024, ny=1024, R=4, Nm=256, W=1.0),
        # a training step on a DOS: forward, loss, gradients
        dict(name="grad_dos", kind="grad_dos", nx=256, ny=256, R=4, M=512, n_energies=512, ckpt=32),
        # a training step on a conductivity
        dict(name="grad_sigma", kind="grad_sigma", nx=256, ny=256, R=2, Nm=256, n_energies=64),
        # the time-domain conductivity: Fermi-Dirac commutator series, then the correlator
        dict(name="time_sigma", kind="time_sigma", nx=512, ny=384, R=1, M=256, M2=17, len_t=16, W=1.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo_cells, hi_cells):
    """Two sides whose product lies between the bounds, of any parity, aspect up to about 3."""
    cells = _log(rng, lo_cells, hi_cells)
    nx = max(4, int(round(math.sqrt(cells) * math.exp(rng.uniform(-0.5, 0.5)))))
    return nx, max(4, cells // nx)


def draw(rng):
    kind = rng.choice(["moments", "moments", "moments", "dos", "evolve", "batch", "mu_nm", "grad_dos", "grad_sigma",
                       "time_sigma"])
    if kind == "moments":
        nx, ny = _sides(rng, 400, 4000000)
        R = rng.choice([1, 1, 2, 3, 4, 8])
        top = min(600, int(2 * 2048 * 2048 * 8 * 64 / (2 * nx * ny * R)))
        return dict(kind=kind, nx=nx, ny=ny, R=R, M=_log(rng, 16, max(17, top)), W=rng.uniform(0.2, 2.0),
                    dtype=rng.choice(["c128", "c128", "c64"]), pair=rng.choice(["one", "one", "two", "both"]),
                    peierls=rng.choice([0.0, 0.0, 1.3]), periodic=rng.random() < 0.7)
    if kind == "dos":
        nx, ny = _sides(rng, 400, 60000)
        return dict(kind=kind, nx=nx, ny=ny, R=rng.choice([1, 2, 4]), M=_log(rng, 32, 512), W=rng.uniform(0.2, 1.0),
                    n_energies=_log(rng, 100, 1024))
    if kind == "evolve":
        nx, ny = _sides(rng, 1000, 1000000)
        return dict(kind=kind, nx=nx, ny=ny, R=rng.choice([1, 2, 2, 4]), M=_log(rng, 12, 64), steps=rng.choice([1, 2]),
                    W=rng.uniform(0.2, 2.0), dtype=rng.choice(["c128", "c128", "c64"]))
    if kind == "batch":
        lo, hi = _log(rng, 16, 64), _log(rng, 100, 512)
        cells = (hi ** 3 - lo ** 3) / (3.0 * (hi - lo))
        return dict(kind=kind, n_inst=max(2, min(64, int(_log(rng, 100000, 1800000) / cells))), lo=lo, hi=hi,
                    sides_seed=rng.randrange(1 << 20), R=rng.choice([1, 2, 2, 4]), M=_log(rng, 32, 128),
                    dtype=rng.choice(["c64", "c64", "c128"]))
    if kind == "mu_nm":
        nx, ny = _sides(rng, 2000, 800000)
        return dict(kind=kind, nx=nx, ny=ny, R=rng.choice([1, 2, 3, 4]), Nm=_log(rng, 32, 256), W=rng.uniform(0.2, 2.0))
    if kind == "grad_dos":
        nx, ny = _sides(rng, 400, 60000)
        return dict(kind=kind, nx=nx, ny=ny, R=rng.choice([1, 2, 4]), M=_log(rng, 32, 512),
                    n_energies=_log(rng, 64, 512), ckpt=rng.choice([8, 16, 32]))
    if kind == "grad_sigma":
        nx, ny = _sides(rng, 400, 60000)
        return dict(kind=kind, nx=nx, ny=ny, R=rng.choice([1, 2]), Nm=_log(rng, 24, 256), n_energies=_log(rng, 16, 64))
    nx, ny = _sides(rng, 1000, 190000)
    return dict(kind="time_sigma", nx=nx, ny=ny, R=1, M=_log(rng, 32, 256), M2=rng.randrange(10, 18),
                len_t=_log(rng, 2, 16), W=rng.uniform(0.2, 2.0))


# ---- inputs, from the seed alone ------------------------------------------------------------
def _phases(R, n, seed):
    """R random-phase vectors on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    ph = torch.rand((R, n), generator=g, dtype=torch.float64, device="cuda") * (2 * math.pi)
    return torch.polar(torch.ones_like(ph), ph)


def _onsite(n, W, seed):
    return W * (2 * np.random.default_rng(seed).random(n) - 1)


def _bound(W):
    """Symmetric spectral bound: three hoppings and the largest on-site term, with one percent."""
    return (3 * abs(T_HOP) + W) * 1.01


def _displacements():
    """x_j - x_i, y_j - y_i of the three A -> B bonds."""
    a = math.sqrt(3.0) * A_CC
    a1, a2 = np.array([a, 0.0]), np.array([a / 2, a * math.sqrt(3.0) / 2])
    d = (a1 + a2) / 3.0
    return np.stack([d, d - a1, d - a2])


def _bessel_series(t, M):
    """[J_0(t), 2 (-i)^m J_m(t)], the Chebyshev coefficients of exp(-i H t), from the integral
    J_m(t) = (1 / pi) int_0^pi cos(m x - t sin x) dx by the trapezoidal rule."""
    x = (np.arange(4096) + 0.5) * (math.pi / 4096)
    m = np.arange(M)[:, None]
    j = np.cos(m * x[None, :] - t * np.sin(x)[None, :]).mean(axis=1)
    c = 2 * (-1j) ** np.arange(M) * j
    c[0] = j[0]
    return c


def _jackson(M):
    n = np.arange(M)
    g = (M - n + 1) * np.cos(np.pi * n / (M + 1)) + np.sin(np.pi * n / (M + 1)) / np.tan(np.pi / (M + 1))
    return g / (M + 1)


def _fermi_series(M):
    """Jackson-damped Chebyshev coefficients of the Fermi step at E = 0."""
    n = np.arange(1, M)
    c = np.concatenate(([0.5], -2 * np.sin(n * math.pi / 2) / (n * math.pi)))
    return (c * _jackson(M)).astype(np.complex128)


def _batch_sides(case):
    return np.random.default_rng(case["sides_seed"]).integers(case["lo"], case["hi"] + 1, size=case["n_inst"])


def _batch_W(case, seed):
    return np.random.default_rng(seed).uniform(0.0, 2.0, size=case["n_inst"])


def _learnable(case, seed):
    """On-site terms and hoppings of a training step, and the data it is fitted to."""
    rng = np.random.default_rng(seed)
    cells = case["nx"] * case["ny"]
    on, hop = rng.uniform(-0.5, 0.5, 2 * cells), T_HOP + rng.uniform(-0.1, 0.1, 3 * cells)
    E = np.linspace(-1, 1, case["n_energies"])
    shape = (1 - E ** 2) * (1 + 0.2 * rng.uniform(-1, 1, case["n_energies"]))
    return on, hop, shape * (2 * cells / 20.0 if case["kind"] == "grad_dos" else 1.0)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "batch":
        datas, idxs = [], []
        sides, Ws = _batch_sides(case), _batch_W(case, seed)
        for k, (side, W) in enumerate(zip(sides, Ws)):
            n = 2 * int(side) ** 2
            arr = lattice.honeycomb_arrays(int(side), int(side), t=T_HOP, onsite=_onsite(n, W, seed + 1 + k),
                                           with_geometry=False)
            datas.append(arr["data"] / _bound(W))
            idxs.append(arr["indices"])
        s["op"] = batched.BatchedELL(datas, idxs, 4)
        s["v"] = _phases(case["R"], int(2 * (sides.astype(np.int64) ** 2).sum()), seed)
        return s
    nx, ny = case["nx"], case["ny"]
    n = 2 * nx * ny
    if kind in ("grad_dos", "grad_sigma"):
        on, hop, target = _learnable(case, seed)
        if kind == "grad_dos":
            s["plan"] = adjoint.DosPlan(nx, ny, case["M"], R=case["R"], n_energies=case["n_energies"],
                                        ckpt=case["ckpt"], onsite0=on, vector_seed=seed)
        else:
            s["plan"] = adjoint.KuboPlan(nx, ny, case["Nm"], R=case["R"], n_energies=case["n_energies"], onsite0=on,
                                         vector_seed=seed)
        s["onsite"] = torch.tensor(on, device="cuda", requires_grad=True)
        s["hopping"] = torch.tensor(hop, device="cuda", requires_grad=True)
        s["target"] = torch.tensor(target, device="cuda")
        return s
    eps, b = _onsite(n, case["W"], seed), _bound(case["W"])
    bounds = np.array([-b, b])
    if kind == "dos":
        s["H"] = lattice.honeycomb(nx, ny, t=T_HOP, onsite=eps, bounds=bounds)
        s["v"] = _phases(case["R"], n, seed).cpu().numpy()
        return s
    s["v"] = _phases(case["R"], n, seed)
    geometry = kind in ("mu_nm", "time_sigma") or bool(case.get("peierls"))
    g = lattice.honeycomb_device(nx, ny, t=T_HOP, onsite=eps, bounds=bounds, geometry=geometry,
                                 periodic=case.get("periodic", True))
    s["op"] = g.op
    if kind == "moments":
        if case["peierls"]:
            s["op"] = device.DeviceELL(g.data_kpm * torch.exp(1j * case["peierls"] * (g.dx + 0.5 * g.dy)), g.indices,
                                       g.len_row)
        if case["pair"] != "one":
            s["vl"] = _phases(case["R"], n, seed + 1)
    elif kind == "evolve":
        s["c"] = _bessel_series(4.0, case["M"])
    elif kind == "mu_nm":
        s["V"] = device.DeviceELL(-1j * g.data * g.dx, g.indices, g.len_row)
    else:
        s["V1"] = device.DeviceELL(-1j * g.data * g.dy, g.indices, g.len_row)
        s["V2"] = device.DeviceELL(g.data_kpm * g.dx, g.indices, g.len_row)
        s["cu"], s["cfd"] = _bessel_series(0.8, case["M2"]), _fermi_series(case["M"])
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "moments":
        if c["pair"] == "both":
            return device.cheb_moments(s["op"], c["M"], s["v"], v_l=s["vl"], dtype=c["dtype"], both=True)
        return device.cheb_moments(s["op"], c["M"], s["v"], v_l=s.get("vl"), dtype=c["dtype"])
    if kind == "dos":
        return observables_gpu.kpm_dos_gpu(s["H"], c["M"], s["v"], n_energies=c["n_energies"])
    if kind == "evolve":
        return device.time_evolve(s["op"], c["M"], s["c"], c["steps"], s["v"], dtype=c["dtype"])
    if kind == "batch":
        return s["op"].moments(c["M"], s["v"], dtype=c["dtype"])
    if kind == "mu_nm":
        return kubo.mu_nm(s["op"], s["V"], c["Nm"], s["v"])
    if kind == "time_sigma":
        return device.time_sigma(s["op"], s["V1"], s["V2"], s["cu"], c["M2"], s["cfd"], c["M"], c["len_t"], s["v"])
    fn = adjoint.kpm_dos if kind == "grad_dos" else adjoint.kpm_sigma
    out = fn(s["onsite"], s["hopping"], s["plan"])
    loss = torch.sum((out - s["target"]) ** 2)
    g_on, g_hop = torch.autograd.grad(loss, (s["onsite"], s["hopping"]))
    return out.detach(), g_on, g_hop


def work(case):
    """Inputs read once, outputs written once; the recursion's arithmetic."""
    kind = case["kind"]
    if kind == "batch":
        sites = int(2 * (_batch_sides(case).astype(np.int64) ** 2).sum())
        out = case["n_inst"] * case["R"] * case["M"] * 16
    else:
        sites, out = 2 * case["nx"] * case["ny"], 0
    R, cplx = case["R"], bool(case.get("peierls"))
    op = sites * 4 * (20 if cplx else 12)
    vec = sites * R * 16
    spmv = sites * R * (4 * (8 if cplx else 4) + 2)
    if kind in ("moments", "dos", "batch"):
        pairs = 2 if case.get("pair") == "both" else 1
        vecs = 2 if case.get("pair", "one") != "one" else 1
        out = out or case.get("n_energies", R * case["M"] * pairs) * 16
        return dict(bytes=op + vecs * vec + out, flops=case["M"] * (spmv + pairs * 8 * sites * R))
    if kind == "evolve":
        return dict(bytes=op + 2 * vec, flops=case["steps"] * case["M"] * (spmv + 8 * sites * R))
    if kind == "mu_nm":
        Nm = case["Nm"]
        return dict(bytes=op + sites * 4 * 16 + vec + Nm * Nm * 16,
                    flops=2 * Nm * spmv + Nm * sites * R * 32 + 8 * Nm * Nm * sites * R)
    if kind == "time_sigma":
        steps = case["len_t"] - 1
        return dict(bytes=op + 2 * sites * 4 * 16 + vec + case["len_t"] * 16,
                    flops=case["M"] * (3 * spmv) + steps * case["M2"] * 2 * (spmv + 8 * sites) + case["len_t"] * 2 * spmv)
    grads = sites * 5 * 8
    if kind == "grad_dos":
        return dict(bytes=vec + 2 * grads, flops=case["M"] * (2 * spmv + 16 * sites * R + 16 * sites * R))
    Nm = case["Nm"]
    gemm = 8 * Nm * Nm * sites * R
    return dict(bytes=vec + 2 * grads, flops=2 * gemm + Nm * (4 * spmv + 96 * sites * R))


# ---- the same quantities in 64 bits on the cell grid ----------------------------------------
class _Grid:
    """y = H x for x [..., 2, ny, nx]: site (ix, iy, s) is entry 2 (iy nx + ix) + s of a vector; bond k
    of cell A(ix, iy) leads to B(ix, iy), B(ix - 1, iy), B(ix, iy - 1)."""

    def __init__(self, nx, ny, eps, hop, periodic=True):
        dev = torch.device("cuda")
        self.nx, self.ny = nx, ny
        eps = eps if isinstance(eps, torch.Tensor) else torch.tensor(eps, dtype=torch.float64, device=dev)
        self.eps = self.split(eps)
        if not isinstance(hop, torch.Tensor):
            hop = torch.tensor(np.asarray(hop), device=dev).reshape(3, 1, 1).repeat(1, ny, nx)
        if not periodic:
            hop = hop.clone()
            hop[1, :, 0] = 0
            hop[2, 0, :] = 0
        self.hop = hop

    def split(self, x):
        return x.reshape(x.shape[:-1] + (self.ny, self.nx, 2)).movedim(-1, -3)

    def flat(self, x):
        return x.movedim(-3, -1).reshape(x.shape[:-3] + (2 * self.nx * self.ny,))

    def bonds(self, h, g, x):
        """The hopping part: h on A -> B, g on the reverse bonds (stored at the A cell)."""
        A, B = x[..., 0, :, :], x[..., 1, :, :]
        ya = h[0] * B + h[1] * torch.roll(B, 1, -1) + h[2] * torch.roll(B, 1, -2)
        yb = g[0] * A + torch.roll(g[1] * A, -1, -1) + torch.roll(g[2] * A, -1, -2)
        return torch.stack((ya, yb), dim=-3)

    def mul(self, x):
        return self.eps * x + self.bonds(self.hop, self.hop.conj(), x)

    def weighted(self, d, x):
        """(H o d) x with the displacement d[k] of bond k (its negative on the way back)."""
        w = torch.tensor(d, dtype=torch.float64, device=x.device).reshape(3, 1, 1)
        return self.bonds(w * self.hop, -w * self.hop.conj(), x)


def _cheb(mul, v, M):
    t0, t1 = v, mul(v)
    yield t0
    for _ in range(M - 1):
        yield t1
        t0, t1 = t1, 2 * mul(t1) - t0


def _dot(a, b):
    return (a.conj() * b).sum(dim=(-3, -2, -1))


def _exact_moments(mul, v, vl, M):
    return torch.stack([_dot(vl, t) for t in _cheb(mul, v, M)], dim=-1)


def _plan_bound(case, on):
    """The plans' spectral bound: Gershgorin over the columns of the initial operator (summed by
    ascending row), one percent."""
    nx, ny = case["nx"], case["ny"]
    iy, ix = np.meshgrid(np.arange(ny), np.arange(nx), indexing="ij")
    site = lambda x, y, s: 2 * ((y % ny) * nx + x % nx) + s  # noqa: E731
    a = np.stack([site(ix, iy, 0)] + [site(ix - dx, iy - dy, 1) for dx, dy in ((0, 0), (1, 0), (0, 1))], axis=-1)
    b = np.stack([site(ix, iy, 1)] + [site(ix + dx, iy + dy, 0) for dx, dy in ((0, 0), (1, 0), (0, 1))], axis=-1)
    cols = np.stack((a, b), axis=2).reshape(-1, 4)
    w = np.full(cols.shape, abs(T_HOP))
    w[:, 0] = np.abs(on)
    radius = np.bincount(cols.reshape(-1), weights=w.reshape(-1), minlength=on.size) - np.abs(on)
    return max(abs(np.min(on - radius)), abs(np.max(on + radius))) * 1.01


def _host_phases(R, n, seed):
    """The plans' random-phase vectors."""
    v = [np.exp(1j * np.random.default_rng(seed + r).uniform(0, 2 * np.pi, n)) for r in range(R)]
    return torch.tensor(np.stack(v), device="cuda")


def _bond_order(nx, ny):
    """Position, in a plan's list of hoppings, of bond k of cell (iy, ix): the bonds are numbered by
    the smaller of their two slots (four slots a row, the on-site one first)."""
    iy, ix = np.meshgrid(np.arange(ny), np.arange(nx), indexing="ij")
    owner = np.empty((3, ny, nx), dtype=np.int64)
    for k, (dx, dy) in enumerate(((0, 0), (1, 0), (0, 1))):
        a = 2 * (iy * nx + ix)
        b = 2 * (((iy - dy) % ny) * nx + (ix - dx) % nx) + 1
        owner[k] = np.minimum(4 * a + 1 + k, 4 * b + 1 + k)
    rank = np.empty(owner.size, dtype=np.int64)
    rank[np.argsort(owner.reshape(-1), kind="stable")] = np.arange(owner.size)
    return torch.tensor(rank.reshape(3, ny, nx), device="cuda")


class _Symmetric(torch.autograd.Function):
    """y = (e + hopping h) x of a real symmetric operator, differentiated by hand so that a long
    recursion keeps one copy of x and no more."""

    @staticmethod
    def forward(ctx, x, eps, hop, grid):
        ctx.save_for_backward(x, eps, hop)
        ctx.grid = grid
        return eps * x + grid.bonds(hop, hop, x)

    @staticmethod
    def backward(ctx, gy):
        x, eps, hop = ctx.saved_tensors
        gx = eps * gy + ctx.grid.bonds(hop, hop, gy)
        dims = tuple(range(gy.dim() - 3))
        pair = lambda p, q: (p.real * q.real + p.imag * q.imag)  # noqa: E731
        ge = pair(gy, x)
        A, B, gA, gB = x[..., 0, :, :], x[..., 1, :, :], gy[..., 0, :, :], gy[..., 1, :, :]
        gh = []
        for sh, ax in ((0, -1), (1, -1), (1, -2)):
            gh.append(pair(gA, torch.roll(B, sh, ax)) + pair(torch.roll(gB, sh, ax), A))
        gh = torch.stack(gh, dim=-3)
        return gx, ge.sum(dim=dims) if dims else ge, gh.sum(dim=dims) if dims else gh, None


def _exact_grad(case, seed):
    nx, ny, R = case["nx"], case["ny"], case["R"]
    on, hop, target = _learnable(case, seed)
    a = _plan_bound(case, on)
    order = _bond_order(nx, ny)
    p_on = torch.tensor(on, device="cuda", requires_grad=True)
    p_hop = torch.tensor(hop, device="cuda", requires_grad=True)
    g = _Grid(nx, ny, on, [T_HOP] * 3)
    eps, h = g.split(p_on), p_hop[order]
    v = g.split(_host_phases(R, 2 * nx * ny, seed))
    mul = lambda x: _Symmetric.apply(x, eps / a, h / a, g)  # noqa: E731
    if case["kind"] == "grad_dos":
        M = case["M"]
        E = np.linspace(-a + 1e-3, a - 1e-3, case["n_energies"]) / a
        tab = 2 * np.cos(np.arange(M)[None, :] * np.arccos(E)[:, None])
        tab[:, 0] = 1.0
        tab = tab / (math.pi * np.sqrt(1 - E[:, None] ** 2)) * _jackson(M)[None, :]
        mu = torch.stack([_dot(v, t).real.mean() for t in _cheb(mul, v, M)])
        out = torch.tensor(tab, device="cuda") @ mu
        loss = torch.sum((out - torch.tensor(target, device="cuda")) ** 2)
        return (out.detach(),) + torch.autograd.grad(loss, (p_on, p_hop))
    Nm = case["Nm"]
    E = np.linspace(-0.9 * a, 0.9 * a, case["n_energies"]) / a
    w = np.cos(np.arange(Nm)[None, :] * np.arccos(E)[:, None]) * (_jackson(Nm) * np.where(np.arange(Nm) == 0, 1.0, 2.0))
    lat = math.sqrt(3.0) * A_CC
    omega = nx * ny * lat ** 2 * math.sqrt(3.0) / 2
    pref = torch.tensor(2.0 / (omega * a * a * (1.0 - E * E)), device="cuda")
    w = torch.tensor(w, device="cuda")
    d = torch.tensor(_displacements()[:, 0], device="cuda").reshape(3, 1, 1)

    def vel(x, hh):  # V x, V = -i H o dx
        return -1j * g.bonds(d * hh, -d * hh, x)

    # mu_nm = <T_n V v | V T_m v> / R, vector by vector; the loss is differentiated through its value
    def mu_of(r, ee, hh):
        m1 = lambda x: _Symmetric.apply(x, ee / a, hh / a, g)  # noqa: E731
        tv = torch.stack(list(_cheb(m1, v[r], Nm)))
        tu = torch.stack(list(_cheb(m1, vel(v[r], hh), Nm)))
        return tu.reshape(Nm, -1).conj() @ vel(tv, hh).reshape(Nm, -1).T / R

    with torch.no_grad():
        mu = sum(mu_of(r, eps, h) for r in range(R)).real
        out = pref * torch.einsum("en,nm,em->e", w, mu, w)
        gw = (2 * (out - torch.tensor(target, device="cuda")) * pref)[:, None] * w
        C = w.T @ gw
    g_on, g_hop = torch.zeros_like(p_on), torch.zeros_like(p_hop)
    for r in range(R):
        F = (C * mu_of(r, g.split(p_on), p_hop[order]).real).sum()
        go, gh = torch.autograd.grad(F, (p_on, p_hop))
        g_on += go
        g_hop += gh
    return out, g_on, g_hop


@torch.no_grad()
def _exact_plain(case, seed):
    kind = case["kind"]
    if kind == "batch":
        sides, Ws = _batch_sides(case), _batch_W(case, seed)
        v, off, out = _phases(case["R"], int(2 * (sides.astype(np.int64) ** 2).sum()), seed), 0, []
        for k, (side, W) in enumerate(zip(sides, Ws)):
            n, b = 2 * int(side) ** 2, _bound(W)
            g = _Grid(int(side), int(side), _onsite(n, W, seed + 1 + k) / b, [T_HOP / b] * 3)
            x = g.split(v[:, off:off + n])
            out.append(_exact_moments(g.mul, x, x, case["M"]))
            off += n
        return torch.stack(out)
    nx, ny = case["nx"], case["ny"]
    n, b = 2 * nx * ny, _bound(case["W"])
    d = _displacements()
    hop = [T_HOP / b] * 3
    if case.get("peierls"):
        hop = [x * np.exp(1j * case["peierls"] * (d[k, 0] + 0.5 * d[k, 1])) for k, x in enumerate(hop)]
    g = _Grid(nx, ny, _onsite(n, case["W"], seed) / b, hop, case.get("periodic", True))
    v = g.split(_phases(case["R"], n, seed))
    if kind == "moments":
        vl = v if case["pair"] == "one" else g.split(_phases(case["R"], n, seed + 1))
        mu = _exact_moments(g.mul, v, vl, case["M"])
        return (mu, _exact_moments(g.mul, v, v, case["M"])) if case["pair"] == "both" else mu
    if kind == "dos":
        M = case["M"]
        mu = _exact_moments(g.mul, v, v, M).mean(dim=0).real.cpu().numpy()
        E = np.linspace(-b + 1e-3, b - 1e-3, case["n_energies"])
        tab = 2 * np.cos(np.arange(M)[None, :] * np.arccos(E / b)[:, None])
        tab[:, 0] = 1.0
        rho = (tab / (math.pi * np.sqrt(1 - (E / b)[:, None] ** 2)) * _jackson(M)[None, :]) @ mu
        return np.stack((E, rho), axis=1)
    if kind == "evolve":
        c = _bessel_series(4.0, case["M"])
        for _ in range(case["steps"]):
            v = sum(complex(ck) * t for ck, t in zip(c, _cheb(g.mul, v, case["M"])))
        return g.flat(v)
    if kind == "mu_nm":
        Nm = case["Nm"]
        vel = lambda x: -1j * b * g.weighted(d[:, 0], x)  # noqa: E731
        mu = torch.zeros((Nm, Nm), dtype=torch.complex128, device="cuda")
        for r in range(case["R"]):
            L = torch.stack([t.reshape(-1) for t in _cheb(g.mul, vel(v[r]), Nm)])
            Rm = torch.stack([vel(t).reshape(-1) for t in _cheb(g.mul, v[r], Nm)])
            mu += L.conj() @ Rm.T
        return mu / case["R"]
    # time_sigma: V1 = -i H o dy, V2 = (H / b) o dx
    V1 = lambda x: -1j * b * g.weighted(d[:, 1], x)  # noqa: E731
    V2 = lambda x: g.weighted(d[:, 0], x)  # noqa: E731
    cu, cf = _bessel_series(0.8, case["M2"]), _fermi_series(case["M"])
    t0, t1, c0, c1 = v, g.mul(v), torch.zeros_like(v), V2(v)
    uc = complex(cf[1]) * c1
    for m in range(2, case["M"]):
        c0, c1 = c1, 2 * g.mul(c1) - c0 + 2 * V2(t1)
        t0, t1 = t1, 2 * g.mul(t1) - t0
        uc = uc + complex(cf[m]) * c1
    out, u = [], v
    for j in range(case["len_t"]):
        if j:
            u = sum(complex(ck) * t for ck, t in zip(cu, _cheb(g.mul, u, case["M2"])))
            uc = sum(complex(ck) * t for ck, t in zip(cu, _cheb(g.mul, uc, case["M2"])))
        out.append(_dot(uc, V1(u)))
    return torch.stack(out, dim=-1)


def exact(case, seed):
    return _exact_grad(case, seed) if case["kind"].startswith("grad") else _exact_plain(case, seed)
