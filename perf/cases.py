"""What the speed of this framework is measured on.

A user's program holds one target (its context: D matrix, FFT plans, work
buffers) and asks it for matvecs, for solves of the incident polarisations or
directions, and for far fields; or it sends targets to the request loop.  The
cases are those four calls, through the package's public entry points, from a
target of 16 dipoles across to one of 256, on grids with and without
compile-time FFT plans, in FP32, FP64 and mixed precision.

A case is a dict:
  op         matvec | solve | farfield | serve
  shape      ellipsoid | box, ex x ey x ez dipoles (serve: the largest edge)
  nmat       1, or 2 for a core of a second material
  precision  fp32 | fp64 | mixed
  nrhs       right-hand sides of one call (serve: requests)
  policy     the FFT grid's: "reference" (DDAParams' default) or "tuned"
  kd, re, im wave number times dipole spacing; refractive index
  solver, eps, host, iters   (solve) iters: matvecs a solve takes, about
  ndir       (farfield) directions
"""
import math

import numpy as np
import torch

import dda_b200
from dda_b200.serve import Server

UNIT_UM = 0.1  # dipole spacing: only kd enters the equations


def _case(name, op, shape, ex, ey, ez, precision, nrhs, **more):
    c = {"op": op, "shape": shape, "ex": ex, "ey": ey, "ez": ez, "nmat": 1, "precision": precision, "nrhs": nrhs,
         "policy": "reference", "kd": 0.5, "re": 1.5, "im": 0.1}
    if name:
        c["name"] = name
    c.update(more)
    return c


def listed():
    return [
        # a small particle, one polarisation: launches and latency
        _case("matvec_tiny_fp32", "matvec", "ellipsoid", 16, 16, 16, "fp32", 1),
        # the reference's README sphere (40 dipoles across, grid 80^3), FP64
        _case("matvec_sphere40_fp64", "matvec", "ellipsoid", 40, 40, 40, "fp64", 1, kd=0.5236),
        # the README box (250 000 dipoles, grid 200 x 100 x 100), both polarisations
        _case("matvec_box_fp32", "matvec", "box", 100, 50, 50, "fp32", 2, kd=0.10472),
        # the same in FP64
        _case("matvec_box_fp64", "matvec", "box", 100, 50, 50, "fp64", 2, kd=0.10472),
        # a particle of uneven extents and two materials on the grid the
        # reference's rule gives it (150 x 108 x 126): no edge has a length
        # of the tuned set
        _case("matvec_ragged_fp32", "matvec", "ellipsoid", 75, 54, 63, "fp32", 2, nmat=2, kd=0.4),
        # many incident directions of one target as a block: the 48 x 32 x 32
        # spheroid, 64 directions x 2 polarisations
        _case("matvec_spheroid_128rhs", "matvec", "ellipsoid", 96, 64, 64, "fp32", 128, kd=0.40919, re=1.33, im=0.01),
        # the largest grid, 512^3, both polarisations
        _case("matvec_sphere256_fp32", "matvec", "ellipsoid", 256, 256, 256, "fp32", 2, kd=0.46875, re=1.6, im=0.01),
        # the README box solved end to end from host fields (complex float,
        # pinned) to host polarisations: the headline benchmark's call
        _case("solve_box_bicgstab_fp32", "solve", "box", 100, 50, 50, "fp32", 2, kd=0.10472, solver="bicgstab",
              eps=1e-5, host=True, iters=35),
        # the README sphere with the reference's default solver in FP64
        _case("solve_sphere40_qmr_fp64", "solve", "ellipsoid", 40, 40, 40, "fp64", 2, kd=0.5236, solver="qmr",
              eps=1e-5, host=False, iters=107),
        # eight directions x 2 polarisations of the spheroid, mixed precision
        _case("solve_spheroid_16rhs_mixed", "solve", "ellipsoid", 96, 64, 64, "mixed", 16, kd=0.40919, re=1.33,
              im=0.01, solver="qmr", eps=1e-5, host=False, iters=245),
        # far field of both polarisations of the README sphere on the default
        # angle grid (91 x 61 directions)
        _case("farfield_sphere40_fp64", "farfield", "ellipsoid", 40, 40, 40, "fp64", 2, kd=0.5236, ndir=5551),
        # four small targets sent to the request loop together
        _case("serve_4_requests", "serve", "ellipsoid", 40, 30, 24, "mixed", 4, policy="tuned", kd=0.35, solver="qmr",
              eps=1e-5, iters=39),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _extents(rng, lo, hi):
    e = _log_int(rng, lo, hi)
    return e, max(4, int(round(e * rng.uniform(0.5, 1.0)))), max(4, int(round(e * rng.uniform(0.5, 1.0))))


def draw(rng):
    op = rng.choice(["matvec"] * 5 + ["solve"] * 3 + ["farfield", "serve"])
    shape = rng.choice(["ellipsoid", "ellipsoid", "box"])
    more = {"policy": rng.choice(["reference", "reference", "tuned"]), "nmat": rng.choice([1, 1, 2]),
            "kd": round(rng.uniform(0.1, 0.5), 4), "re": round(rng.uniform(1.2, 1.7), 3),
            "im": round(rng.uniform(0.0, 0.2), 3)}
    if op == "matvec":
        precision = rng.choice(["fp32", "fp32", "fp64"])
        ex, ey, ez = _extents(rng, 10, 160)
        nrhs = rng.choice([1, 2, 2, 2, 3, 8])
        return _case(None, op, shape, ex, ey, ez, precision, nrhs, **more)
    if op == "solve":
        # the FP32 solver at a tolerance and an index that FP32 recurrences reach
        precision = rng.choice(["fp32", "fp64", "mixed"])
        solver = "bicgstab" if precision == "fp32" else rng.choice(["qmr", "bicgstab"])
        ex, ey, ez = _extents(rng, 10, 64)
        more.update(kd=round(rng.uniform(0.1, 0.3), 4), re=round(rng.uniform(1.2, 1.5), 3), solver=solver, eps=1e-5,
                    host=rng.random() < 0.3 and precision != "mixed", iters=30)
        return _case(None, op, shape, ex, ey, ez, precision, rng.choice([1, 2, 2, 4]), **more)
    if op == "farfield":
        ex, ey, ez = _extents(rng, 10, 64)
        return _case(None, op, shape, ex, ey, ez, rng.choice(["fp32", "fp64"]), rng.choice([1, 2]),
                     **dict(more, ndir=_log_int(rng, 30, 6000)))
    ex, ey, ez = _extents(rng, 10, 40)
    more.update(policy="tuned", kd=round(rng.uniform(0.1, 0.3), 4), re=round(rng.uniform(1.2, 1.5), 3), nmat=1,
                solver="qmr", eps=1e-5, iters=30)
    return _case(None, op, "ellipsoid", ex, ey, ez, "mixed", rng.choice([1, 2, 3, 4]), **more)


# ------------------------------------------------------------------ targets --
def _cells(case, scale=1.0):
    """Dipole positions [nv][3] (z slowest, as the framework takes them) and
    materials [nv], on the GPU."""
    e = [max(4, int(round(case[k] * scale))) for k in ("ex", "ey", "ez")]
    ax = [torch.arange(n, device="cuda", dtype=torch.float64) for n in e]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    r = sum(((v + 0.5 - n / 2) / (n / 2)) ** 2 for v, n in ((x, e[0]), (y, e[1]), (z, e[2])))
    keep = r <= 1 if case["shape"] == "ellipsoid" else torch.ones_like(r, dtype=torch.bool)
    pos = torch.stack([x[keep], y[keep], z[keep]], dim=1).to(torch.int32)
    mat = (r[keep] < 0.3).to(torch.uint8) * (case["nmat"] - 1)
    return pos - pos.min(dim=0).values, mat


def _indices(case):
    m = complex(case["re"], case["im"])
    return [m, complex(1.2, 0.02)][:case["nmat"]]


def _wavelength_um(case):
    return "%.17gum" % (2 * math.pi * UNIT_UM / case["kd"])


def _params(case):
    pos, mat = _cells(case)
    g = dda_b200.Geometry.from_arrays(pos.cpu().numpy().astype(np.uint32), mat.cpu().numpy(), "%gum" % UNIT_UM)
    return dda_b200.DDAParams(g, _indices(case), _wavelength_um(case), grid_policy=case["policy"])


def _directions(seed, n):
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def _incidences(case, seed):
    """(direction, polarisation) of every right-hand side."""
    d = _directions(seed, (case["nrhs"] + 1) // 2)
    return [(tuple(d[r // 2]), 1 + r % 2) for r in range(case["nrhs"])]


def _complex_normal(shape, seed, dtype):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.complex128).to(dtype)


def _vectors(case, nv, seed):
    """[nrhs][3 nvs] Krylov-like vectors, the padding zero."""
    nvs = (nv + 15) // 16 * 16
    dtype = torch.complex64 if case["precision"] == "fp32" else torch.complex128
    x = torch.zeros(case["nrhs"], 3, nvs, dtype=dtype, device="cuda")
    for r in range(case["nrhs"]):
        x[r, :, :nv] = _complex_normal((3, nv), 1000 * seed + r, dtype)
    return x.reshape(case["nrhs"], 3 * nvs)


def _pinned(a, dtype):
    t = torch.empty(a.shape, dtype=dtype, pin_memory=True)
    t.copy_(torch.as_tensor(a))
    return t.numpy()


# ------------------------------------------------------------------ the path --
def prepare(case, seed):
    op, nrhs = case["op"], case["nrhs"]
    if op == "serve":
        targets = []
        d = _directions(seed, nrhs)
        for i in range(nrhs):  # the requests' targets: of one shape, each smaller than the last
            pos, _ = _cells(case, 1.0 - 0.15 * i)
            targets.append((pos.cpu().numpy().astype(np.uint32), tuple(d[i])))
        torch.cuda.synchronize()
        return {"case": case, "server": Server(budget_bytes=8 << 30, max_active=4), "targets": targets}
    p = _params(case)
    mv = dda_b200.CudaMatVec(p, case["precision"], max_rhs=nrhs)
    rhs = _incidences(case, seed)
    for r, (prop, pol) in enumerate(rhs):
        mv.set_couple_constants(dda_b200.CoupleConstants(p, prop, pol, "ldr"), rhs=r)
    s = {"case": case, "mv": mv, "params": p}
    if op == "matvec":
        s["x"] = _vectors(case, p.nv, seed)
        s["y"] = torch.empty_like(s["x"])
    elif op == "farfield":
        # the polarisations of an earlier run, from its file
        s["pol"] = _pinned(_vectors(dict(case, precision="fp64"), p.nv, seed).cpu(), torch.complex128)
        s["dirs"] = _directions(seed + 1, case["ndir"])
    else:
        einc = np.stack([p.einc(prop, pol) for prop, pol in rhs])
        s["solver"] = dda_b200.CudaSolver(mv, case["solver"])
        single = case["precision"] == "fp32"
        if case["host"]:
            s["einc"] = _pinned(einc, torch.complex64 if single else torch.complex128)
            s["pol"] = _pinned(np.zeros_like(s["einc"]), torch.complex64 if single else torch.complex128)
        else:
            s["einc"] = torch.as_tensor(einc, device="cuda").to(torch.complex64 if single else torch.complex128)
            s["pol"] = torch.empty_like(s["einc"])
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    op, nrhs = case["op"], case["nrhs"]
    if op == "matvec":
        s["mv"].apply_device(s["x"].data_ptr(), s["y"].data_ptr(), nrhs=nrhs)
        return s["y"]
    if op == "solve":
        if case["host"]:
            return s["solver"].get_pol_vec(s["einc"], case["eps"], out=s["pol"])
        s["solver"].get_pol_vec_device(s["einc"].data_ptr(), s["pol"].data_ptr(), nrhs, case["eps"])
        return s["pol"]
    if op == "farfield":
        return s["mv"].far_field(s["dirs"], nrhs=nrhs, pol=s["pol"])
    srv = s["server"]
    for i, (pos, prop) in enumerate(s["targets"]):
        srv.submit(pos, None, _indices(case), "%gum" % UNIT_UM, _wavelength_um(case), prop=prop,
                   solver=case["solver"], precision=case["precision"], eps=case["eps"], keep_pol=True, tag=i,
                   grid_policy=case["policy"])
    done = {d["tag"]: d for d in srv.drain()}
    if any(d["status"] != 0 for d in done.values()):
        raise RuntimeError(str([d["error"] for d in done.values()]))
    return [{"pol": done[i]["pol"], "cext": np.array(done[i]["cext"])} for i in range(nrhs)]


# ---------------------------------------------------------------------- work --
def _smooth(n):
    """Smallest even length >= n with no prime factor above 7."""
    n += n % 2
    while True:
        m = n
        for q in (2, 3, 5, 7):
            while m % q == 0:
                m //= q
        if m == 1:
            return n
        n += 2


def _matvec_work(ex, ey, ez, nv, nrhs, s):
    """One matvec of nrhs right-hand sides: vectors in and out, the D matrix's
    octant and the geometry once; zero-padded FFT lines and the 3 x 3
    products."""
    gx, gy, gz = (_smooth(2 * e) for e in (ex, ey, ez))
    octant = (gx // 2 + 1) * (gy // 2 + 1) * (gz // 2 + 1)
    byte = nrhs * s * 3 * nv * 2 + 6 * octant * s + 13 * nv
    line = lambda n: 5 * n * math.log2(n)  # noqa: E731
    flop = nrhs * (2 * 3 * (ey * ez * line(gx) + gx * ey * line(gz) + gx * gz * line(gy)) + 66 * gx * gy * gz)
    return byte, flop


def work(case):
    e = case["ex"], case["ey"], case["ez"]
    fill = math.pi / 6 if case["shape"] == "ellipsoid" else 1.0
    nv = int(fill * e[0] * e[1] * e[2])
    n, s = case["nrhs"], 8 if case["precision"] == "fp32" else 16
    if case["op"] == "matvec":
        b, f = _matvec_work(*e, nv, n, s)
    elif case["op"] == "farfield":
        b = n * 48 * nv + case["ndir"] * (24 + n * 48)
        f = 24.0 * n * nv * case["ndir"]
    elif case["op"] == "solve":
        # mixed precision: the convolution's data in FP32
        b, f = _matvec_work(*e, nv, n, 8 if case["precision"] == "mixed" else s)
        b, f = case["iters"] * b, case["iters"] * f
    else:
        b = f = 0.0
        for i in range(n):
            k = 1.0 - 0.15 * i
            t = _matvec_work(*[max(4, int(round(v * k))) for v in e], int(nv * k ** 3), 2, 8)
            b, f = b + case["iters"] * t[0], f + case["iters"] * t[1]
    return {"bytes": b, "flops": f}


# ----------------------------------------------------------------- tolerance --
def tolerance(case):
    if case["op"] in ("matvec", "farfield"):
        # four times the distance from exact(): FP32 5.2e-8 to 1.3e-7 (a far
        # field has its polarisations rounded), FP64 1e-16 to 3.7e-16 for a
        # matvec and 2.3e-15 for a far field, whose phases reach hundreds of
        # radians
        if case["precision"] == "fp32":
            return {"rel": 6e-7, "max": 2e-5}
        return {"rel": 2e-15, "max": 1e-13} if case["op"] == "matvec" else {"rel": 1e-14, "max": 1e-12}
    # any vector within the relative residual eps answers a solve, and where
    # an iteration more or less leaves it is up to the rounding of the sums:
    # 2.1 eps from exact() at most
    return {"rel": 8 * case["eps"], "max": 400 * case["eps"]}


# --------------------------------------------------------- the same in 64 bits --
def _beam(prop, pol):
    """The plane wave's direction and polarisation vector."""
    p = np.asarray(prop) / np.linalg.norm(prop)
    if abs(p[2]) >= 1 - 1e-6:
        x, y = np.array([p[2], 0, 0]), np.array([0, 1.0, 0])
    else:
        t = math.sqrt(1 - p[2] ** 2)
        x, y = np.array([p[0] * p[2] / t, p[1] * p[2] / t, -t]), np.array([-p[1] / t, p[0] / t, 0])
    return p, (y if pol == 1 else x)


def _ldr(case, prop, pol):
    """sqrt of the lattice-dispersion-relation polarisability per material,
    in units of d^3."""
    p, inc = _beam(prop, pol)
    s = float(np.sum(p ** 2 * inc ** 2))
    kd, out = case["kd"], []
    for m in _indices(case):
        m2 = m * m
        cm = 3 / (4 * math.pi) * (m2 - 1) / (m2 + 2)
        t = 2j / 3 * kd ** 3 + (1.8915316 + (-0.1648469 + 1.7700004 * s) * m2) * kd ** 2
        out.append(np.sqrt(cm / (1 - cm * t)))
    return torch.tensor(out, dtype=torch.complex128, device="cuda")


class _Operator:
    """y = x - sqrt(cc) G * (sqrt(cc) x) on the dipoles, G the Green's tensor,
    by zero-padded FFTs in 64 bits (torch.fft)."""

    PAIRS = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))

    def __init__(self, pos, kd):
        self.box = [int(v) + 1 for v in pos.max(dim=0).values]
        self.n = [_smooth(2 * b) for b in self.box]  # x, y, z
        self.kd = kd
        x, y, z = (pos[:, i].long() for i in range(3))
        self.at = (z * self.n[1] + y) * self.n[0] + x
        self.kept = None
        if self.n[0] * self.n[1] * self.n[2] < 2 ** 25:
            self.kept = [self._tensor(a, b) for a, b in self.PAIRS]

    def _tensor(self, a, b):
        n = self.n
        off = [torch.arange(m, device="cuda", dtype=torch.float64) for m in n]
        off = [torch.where(v <= m // 2, v, v - m) for v, m in zip(off, n)]
        r = [off[0][None, None, :], off[1][None, :, None], off[2][:, None, None]]
        rho = torch.sqrt(r[0] ** 2 + r[1] ** 2 + r[2] ** 2)
        inside = ((r[0].abs() < self.box[0]) & (r[1].abs() < self.box[1]) & (r[2].abs() < self.box[2]) & (rho > 0))
        rho = torch.where(inside, rho, torch.ones_like(rho))
        q, kr = r[a] * r[b] / rho ** 2, self.kd * rho
        d = 1.0 if a == b else 0.0
        g = torch.complex((3 - kr ** 2) * q + d * (kr ** 2 - 1), kr * (d - 3 * q))
        g = g * torch.polar(1 / rho ** 3, kr)
        return torch.fft.fftn(torch.where(inside, g, torch.zeros_like(g)))

    def conv(self, v):
        """[3][nv] -> [3][nv]."""
        n = self.n[::-1]
        f = []
        for c in range(3):
            g = torch.zeros(n[0] * n[1] * n[2], dtype=torch.complex128, device="cuda")
            g[self.at] = v[c]
            f.append(torch.fft.fftn(g.reshape(n)))
        out = [torch.zeros_like(f[0]) for _ in range(3)]
        for k, (a, b) in enumerate(self.PAIRS):
            t = self.kept[k] if self.kept else self._tensor(a, b)
            out[a].addcmul_(t, f[b])
            if a != b:
                out[b].addcmul_(t, f[a])
        del f
        return torch.stack([torch.fft.ifftn(out[c]).reshape(-1)[self.at] for c in range(3)])

    def apply(self, x, cs):
        return x - cs * self.conv(cs * x)

    def solve(self, b, cs, eps):
        """BiCGStab."""
        x, r = torch.zeros_like(b), b.clone()
        rt, p, v = r.clone(), torch.zeros_like(b), torch.zeros_like(b)
        rho = alpha = om = torch.ones((), dtype=torch.complex128, device="cuda")
        dot = lambda u, w: torch.sum(u.conj() * w)  # noqa: E731
        goal = float(torch.linalg.vector_norm(b)) * eps
        for _ in range(400):
            rho1 = dot(rt, r)
            beta = rho1 / rho * alpha / om
            p = r + beta * (p - om * v)
            v = self.apply(p, cs)
            alpha = rho1 / dot(rt, v)
            s = r - alpha * v
            t = self.apply(s, cs)
            om = dot(t, s) / dot(t, t)
            x = x + alpha * p + om * s
            r, rho = s - om * t, rho1
            if float(torch.linalg.vector_norm(r)) < goal:
                return x
        return None


def _einc(pos, box, kd, prop, pol):
    p, inc = _beam(prop, pol)
    r = pos.double() - (torch.tensor(box, device="cuda", dtype=torch.float64) - 1) / 2
    ph = kd * (r @ torch.tensor(p, device="cuda"))
    return torch.polar(torch.ones_like(ph), ph)[None, :] * torch.tensor(inc, device="cuda")[:, None]


def _solution(case, op, pos, mat, prop, pol):
    """Polarisations [3][nv] of one incidence, in SI units, and Cext."""
    e = _einc(pos, op.box, case["kd"], prop, pol)
    cs = _ldr(case, prop, pol)[mat.long()]
    x = op.solve(cs * e, cs, 1e-11)
    if x is None:
        return None, None
    d = UNIT_UM * 1e-6
    P = cs * x * d ** 3
    cext = 4 * math.pi * case["kd"] / d * float(torch.sum(P * e.conj()).imag)
    return P, cext


def exact(case, seed):
    if case["op"] == "serve":
        out, d = [], _directions(seed, case["nrhs"])
        for i in range(case["nrhs"]):
            pos, mat = _cells(case, 1.0 - 0.15 * i)
            op = _Operator(pos, case["kd"])
            nv, nvs = len(pos), (len(pos) + 15) // 16 * 16
            pols, cext = torch.zeros(2, 3, nvs, dtype=torch.complex128), []
            for r in range(2):
                P, c = _solution(case, op, pos, mat, tuple(d[i]), 1 + r)
                pols[r, :, :nv] = P.cpu()
                cext.append(c)
            out.append({"pol": pols.reshape(2, -1).numpy(), "cext": np.array(cext)})
        return out
    pos, mat = _cells(case)
    nv, nvs, n = len(pos), (len(pos) + 15) // 16 * 16, case["nrhs"]
    rhs = _incidences(case, seed)
    if case["op"] == "farfield":
        v = _vectors(dict(case, precision="fp64"), nv, seed).reshape(n, 3, nvs)[:, :, :nv]
        dirs = torch.tensor(_directions(seed + 1, case["ndir"]), device="cuda")
        d = UNIT_UM * 1e-6
        k = case["kd"] / d
        box = pos.max(dim=0).values.double() + 1
        out = torch.empty(case["ndir"], n, 3, dtype=torch.complex128, device="cuda")
        for i in range(0, case["ndir"], 256):
            u = dirs[i:i + 256]
            ph = -case["kd"] * (u @ (pos.double() - (box - 1) / 2).T)
            S = torch.einsum("dj,ncj->dnc", torch.polar(torch.ones_like(ph), ph), v)
            nS = torch.einsum("dc,dnc->dn", u.to(S.dtype), S)
            out[i:i + 256] = 1j * k * k * (S - u[:, None, :] * nS[:, :, None])
        return out.cpu().numpy()
    if case["op"] == "solve" and nv * case["nrhs"] > 1000000:
        return None  # some 500 matvecs for each right-hand side: over a minute
    op = _Operator(pos, case["kd"])
    out = torch.zeros(n, 3, nvs, dtype=torch.complex128, device="cuda")
    if case["op"] == "matvec":
        x = _vectors(case, nv, seed).reshape(n, 3, nvs)
        for r, (prop, pol) in enumerate(rhs):
            out[r, :, :nv] = op.apply(x[r, :, :nv].to(torch.complex128), _ldr(case, prop, pol)[mat.long()])
        return out.reshape(n, 3 * nvs)
    for r, (prop, pol) in enumerate(rhs):
        P, _ = _solution(case, op, pos, mat, prop, pol)
        if P is None:
            return None
        out[r, :, :nv] = P
    out = out.reshape(n, 3 * nvs)
    return out.cpu().numpy() if case["host"] else out
