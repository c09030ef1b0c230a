"""Performance cases of the package: what its users run, through the public
entry points, with the inputs such a program has in hand.

Sizes come from the package's own workloads (the N=64 / 180-angle demo
problem, paralleltomo N=512 with 360 angles, fanlineartomo N=1024, the N=256
Kaczmarz and CART problems, the uneven batch, the N=256 / 60-angle warm-start
geometry and its U-Net).  Data are analytic line integrals of random ellipses
(centres U[-0.6,0.6]^2, semi-axes U[0.05,0.4], intensities U[0.02,0.2], so that sums stay near [0,1])
plus seeded Gaussian noise, so they do not depend on the code that is measured.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import airtoolsii_b200 as airt
from airtoolsii_b200.batch import sirt_multi_device
from airtoolsii_b200.testprobs import fan_tables, parallel_operator, parallel_tables

DEV = "cuda"
F64 = torch.float64


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # one interactive call on the demo problem: default options, so rho is
        # estimated inside the call; latency and launches count
        dict(name="sirt_demo", kind="sirt", N=64, angles=180, rays=91, method="cimmino",
             iters=50, box=True, level=0.0, rho=False),
        # an ordinary reconstruction to the discrepancy principle, odd sizes
        dict(name="sirt_dp", kind="sirt", N=201, angles=123, rays=283, method="sart", iters=500,
             box=True, level=0.04, rho=False),
        # the large stored system: 120 M nonzeros, read from HBM twice per iteration
        dict(name="sirt_large", kind="sirt", N=512, angles=360, rays=724, method="cimmino",
             iters=200, box=True, level=0.0, rho=True),
        # the same toolbox call on the matrix-free handle (isMatrix = 0)
        dict(name="mf_parallel", kind="mf", geom="parallel", N=512, angles=180, rays=724,
             method="sart", iters=20, box=True),
        # matrix-free fan beam, where A would be the largest
        dict(name="mf_fan", kind="mf", geom="fan", N=1024, angles=180, rays=1448, method="sart",
             iters=10, box=True),
        # row-action sweeps in the reference's order with nonnegativity
        dict(name="kaczmarz", kind="art", N=256, angles=180, rays=362, method="kaczmarz", iters=5),
        # column-action sweeps
        dict(name="columnaction", kind="cart", N=256, angles=60, rays=362, iters=3),
        # start of a session: build A for new angles, project an image, reconstruct with fbp
        dict(name="build_fbp", kind="build", N=512, angles=180, rays=724, filter="hamming"),
        # many uneven problems, each to its own discrepancy-principle stop
        dict(name="batch_dp", kind="batch", count=64, nmax=256, amin=30, amax=180,
             method="cimmino", iters=400, level=0.04),
        # many sinograms of one geometry, each to its own stop
        dict(name="multi_dp", kind="multi", N=256, angles=60, rays=362, count=250,
             method="cimmino", iters=400, level=0.04),
        # warm-start inference on a batch of back projections
        dict(name="unet_infer", kind="unet", N=256, base=32, levels=4, batch=40, chunk=16,
             train=False),
        # one training gradient of that network
        dict(name="unet_train", kind="unet", N=256, base=32, levels=4, batch=16, chunk=16,
             train=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sirt", "sirt", "sirt", "mf", "mf", "art", "cart", "build", "batch", "multi",
                       "unet"])
    if kind == "sirt":
        N = _log_int(rng, 48, 512)
        dp = rng.random() < 0.4
        return dict(kind="sirt", N=N, angles=_log_int(rng, 30, 360),
                    rays=int(round(math.sqrt(2) * N)) + rng.randrange(0, 2),
                    method=rng.choice(["cimmino", "sart", "landweber"]),
                    iters=300 if dp else rng.randrange(20, 150), box=rng.random() < 0.7,
                    level=0.05 if dp else 0.0, rho=rng.random() < 0.5)
    if kind == "mf":
        N = _log_int(rng, 64, 640)
        return dict(kind="mf", geom=rng.choice(["parallel", "fan"]), N=N,
                    angles=_log_int(rng, 30, 180), rays=int(round(math.sqrt(2) * N)) + rng.randrange(0, 3),
                    method=rng.choice(["sart", "cimmino"]), iters=rng.randrange(5, 21),
                    box=rng.random() < 0.7)
    if kind == "art":
        N = _log_int(rng, 48, 256)
        return dict(kind="art", N=N, angles=_log_int(rng, 30, 180), rays=int(round(math.sqrt(2) * N)),
                    method=rng.choice(["kaczmarz", "symkaczmarz", "randkaczmarz"]),
                    iters=2 * rng.randrange(1, 3))
    if kind == "cart":
        N = _log_int(rng, 48, 256)
        return dict(kind="cart", N=N, angles=_log_int(rng, 20, 60), rays=int(round(math.sqrt(2) * N)),
                    iters=rng.randrange(1, 4))
    if kind == "build":
        N = _log_int(rng, 48, 512)
        return dict(kind="build", N=N, angles=_log_int(rng, 30, 180),
                    rays=int(round(math.sqrt(2) * N)) + rng.randrange(0, 2),
                    filter=rng.choice(["ram-lak", "shepp-logan", "hamming", "hann"]))
    if kind == "batch":
        return dict(kind="batch", count=_log_int(rng, 4, 64), nmax=rng.choice([96, 128, 192, 256]),
                    amin=30, amax=rng.randrange(60, 181), method=rng.choice(["cimmino", "sart"]),
                    iters=400, level=0.05)
    if kind == "multi":
        N = _log_int(rng, 64, 256)
        return dict(kind="multi", N=N, angles=_log_int(rng, 30, 60), rays=int(round(math.sqrt(2) * N)),
                    count=_log_int(rng, 5, 250), method=rng.choice(["cimmino", "sart"]), iters=400,
                    level=0.05)
    base = rng.choice([16, 32])
    return dict(kind="unet", N=rng.choice([64, 96, 128, 192, 256]), base=base, levels=rng.choice([3, 4]),
                batch=rng.randrange(1, 17), chunk=16, train=rng.random() < 0.5)


# ------------------------------------------------------------------ the data
def _angles(case, rng):
    """Equispaced angles over the half or full turn with a random start."""
    full = 360.0 if case.get("geom") == "fan" else 180.0
    step = full / case["angles"]
    return np.arange(case["angles"]) * step + rng.uniform(0.05, 0.95) * step


def _rays(case, theta):
    """(x0, y0, dx, dy) of every ray as device FP64 vectors, angle-major."""
    N, p = case["N"], case["rays"]
    t = lambda v: torch.as_tensor(np.asarray(v), dtype=F64, device=DEV)  # noqa: E731
    if case.get("geom") == "fan":
        _, _, R, _, _, ct, st, cw, sw = fan_tables(N, theta, p)
        c, s, cw, sw = t(ct)[:, None], t(st)[:, None], t(cw)[None], t(sw)[None]
        x0, y0 = -s * R, c * R
        a1, a2 = -x0 / R, -y0 / R
        return [v.expand(len(theta), p).reshape(-1) for v in
                (x0, y0, cw * a1 - sw * a2, sw * a1 + cw * a2)]
    _, _, _, ct, st, off = parallel_tables(N, theta, p)
    c, s, o = t(ct)[:, None], t(st)[:, None], t(off)[None]
    return [v.expand(len(theta), p).reshape(-1) for v in (c * o, s * o, -s, c)]


def _ellipses(rng, count):
    """count x 6: amplitude, semi-axes, centre, angle (unit square [-1,1]^2)."""
    return np.stack([rng.uniform(0.02, 0.2, count), rng.uniform(0.05, 0.4, count),
                     rng.uniform(0.05, 0.4, count), rng.uniform(-0.6, 0.6, count),
                     rng.uniform(-0.6, 0.6, count), rng.uniform(0, math.pi, count)], axis=-1)


def _integrals(N, rays, ell):
    """Line integrals of the ellipse sum along every ray; ell (..., count, 6)
    gives (..., rays)."""
    x0, y0, dx, dy = rays
    h = 0.5 * N
    E = torch.as_tensor(ell, dtype=F64, device=DEV)
    out = torch.zeros(E.shape[:-2] + x0.shape, dtype=F64, device=DEV)
    for k in range(E.shape[-2]):
        amp, a, b, cx, cy, phi = [E[..., k, q, None] for q in range(6)]
        c, s = torch.cos(phi), torch.sin(phi)
        px, py = x0 - cx * h, y0 - cy * h
        ux, uy = (c * px + s * py) / (a * h), (c * py - s * px) / (b * h)
        vx, vy = (c * dx + s * dy) / (a * h), (c * dy - s * dx) / (b * h)
        A, B, C = vx * vx + vy * vy, ux * vx + uy * vy, ux * ux + uy * uy - 1.0
        out += amp * 2.0 * torch.sqrt(torch.clamp(B * B - A * C, min=0.0)) / A
    return out


def _noisy(b, eta, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    e = torch.randn(b.shape, generator=g, dtype=F64, device=DEV)
    return b + e * (eta * torch.linalg.norm(b, dim=-1, keepdim=True)
                    / torch.linalg.norm(e, dim=-1, keepdim=True))


def _data(case, seed, count=None):
    """(theta, rays, noisy sinogram) of the case's geometry for this seed."""
    rng = np.random.default_rng(seed)
    theta = _angles(case, rng)
    rays = _rays(case, theta)
    if count is None:
        ell = _ellipses(rng, 20)
    else:
        ell = np.stack([_ellipses(rng, 10) for _ in range(count)])
    return theta, rays, _noisy(_integrals(case["N"], rays, ell), 0.02, seed)


def _image(case, seed):
    """A smooth positive image of N x N pixels (host, x(:) order)."""
    rng = np.random.default_rng(seed + 1)
    v = np.linspace(-1, 1, case["N"])
    X, Y = np.meshgrid(v, v)
    img = np.zeros_like(X)
    for amp, a, b, cx, cy, _ in _ellipses(rng, 12):
        img += amp * np.exp(-((X - cx) / a) ** 2 - ((Y - cy) / b) ** 2)
    return np.ascontiguousarray(img.ravel(order="F"))


def _batch_problems(case, seed):
    """Sizes, angle lists and sinograms of the uneven batch."""
    rng = np.random.default_rng(seed)
    sizes = [n for n in (64, 96, 128, 192, 256) if n <= case["nmax"]]
    out = []
    for k in range(case["count"]):
        # an even spread of sizes and angle counts, so that the work does not
        # hang on the seed; their pairing does
        na = case["amin"] + ((k * 37) % case["count"]) * (case["amax"] - case["amin"]) // case["count"]
        c = dict(N=sizes[k % len(sizes)], angles=int(na))
        c["rays"] = int(round(math.sqrt(2) * c["N"]))
        th = _angles(c, rng)
        rays = _rays(c, th)
        b = _noisy(_integrals(c["N"], rays, _ellipses(rng, 10)), 0.02, seed + 7 * k)
        out.append((c, th, rays, b))
    return out


def _unet_shapes(case):
    b, L = case["base"], case["levels"]
    shapes = []
    for lv in range(L):
        shapes += [(1 if lv == 0 else b << (lv - 1), b << lv, lv), (b << lv, b << lv, lv)]
    for lv in range(L - 2, -1, -1):
        shapes += [((b << (lv + 1)) + (b << lv), b << lv, lv), (b << lv, b << lv, lv)]
    return shapes


def _unet_data(case, seed):
    """He-initialised parameters (the packed order of UNet.set_params) and
    images: smooth bumps as inputs, sharper ones as targets."""
    rng = np.random.default_rng(seed)
    prm = []
    for cin, cout, _ in _unet_shapes(case):
        prm += [rng.standard_normal(cout * 9 * cin) * math.sqrt(2.0 / (9 * cin)),
                0.05 * rng.standard_normal(cout)]
    prm += [rng.standard_normal(case["base"]) / math.sqrt(case["base"]), np.zeros(1)]
    prm = np.concatenate(prm).astype(np.float32)
    N, B = case["N"], case["batch"]
    v = torch.linspace(-1, 1, N, dtype=F64, device=DEV)
    E = torch.as_tensor(np.stack([_ellipses(rng, 8) for _ in range(B)]), dtype=F64, device=DEV)
    u = torch.zeros(B, N, N, dtype=F64, device=DEV)
    t = torch.zeros_like(u)
    for k in range(8):
        amp, a, b, cx, cy, _ = [E[:, k, q, None, None] for q in range(6)]
        r = ((v[None, :, None] - cx) / a) ** 2 + ((v[None, None, :] - cy) / b) ** 2
        u += amp * torch.exp(-r)
        t += amp * torch.exp(-r ** 4)
    return prm, u.reshape(B, -1), t.reshape(B, -1)


# ------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind in ("sirt", "mf", "art", "cart"):
        theta, _, b = _data(case, seed)
        if case.get("geom") == "fan":
            A = _fan_handle(case, theta)
        else:
            _, _, _, ct, sn, off = parallel_tables(case["N"], theta, case["rays"])
            A = parallel_operator(case["N"], ct, sn, off, matrix_free=kind == "mf")
        st.update(A=A, b=b.cpu().numpy())
        opts = {}
        if case.get("box"):
            opts.update(lbound=0.0, ubound=1.0)
        if kind in ("art", "cart"):
            opts["lbound"] = 0.0
        if case.get("level"):
            opts["stoprule"] = dict(type="DP", taudelta=case["level"] * float(np.linalg.norm(st["b"])))
        if case.get("rho"):
            # a program that knows its geometry keeps rho; a rough upper value will do
            opts["rho"] = _rho_bound(case)
        st["opts"] = opts
    elif kind == "build":
        rng = np.random.default_rng(seed)
        st.update(theta=_angles(case, rng), x=_image(case, seed))
    elif kind == "batch":
        pr = _batch_problems(case, seed)
        st["batch"] = airt.ParallelBatch([c["N"] for c, _, _, _ in pr], [th for _, th, _, _ in pr],
                                         [c["rays"] for c, _, _, _ in pr])
        st["b"] = [b.cpu().numpy() for _, _, _, b in pr]
        st["td"] = np.array([case["level"] * np.linalg.norm(b) for b in st["b"]])
    elif kind == "multi":
        theta, _, B = _data(case, seed, case["count"])
        _, _, _, ct, sn, off = parallel_tables(case["N"], theta, case["rays"])
        st["A"] = parallel_operator(case["N"], ct, sn, off)
        st["B"] = B.contiguous()
        st["X"] = torch.empty(case["count"], case["N"] ** 2, dtype=F64, device=DEV)
        st["td"] = case["level"] * torch.linalg.norm(B, dim=1).cpu().numpy()
    else:
        prm, u, t = _unet_data(case, seed)
        net = airt.UNet(case["N"], case["N"], case["base"], case["levels"],
                        max_batch=min(case["chunk"], case["batch"]), seed=0)
        net.set_params(prm)
        st["net"] = net
        if case["train"]:
            st.update(u=u.float().contiguous(), t=t.float().contiguous())
        else:
            st.update(u=u.contiguous(), out=torch.empty_like(u))
    torch.cuda.synchronize()
    return st


def _fan_handle(case, theta):
    from airtoolsii_b200.testprobs import fan_operator
    _, _, R, _, _, ct, sn, cw, sw = fan_tables(case["N"], theta, case["rays"])
    return fan_operator(case["N"], ct, sn, cw, sw, R, matrix_free=True)


def _rho_bound(case):
    """An estimate of the largest eigenvalue of D*A'*M*A from the continuous
    operator: A'A acts on constant images as nearly (angles * N) per pixel."""
    N, nA, m = case["N"], case["angles"], case["angles"] * case["rays"]
    if case["method"] == "cimmino":
        return 1.35 * nA * N / m / N
    if case["method"] == "landweber":
        return 1.1 * nA * N * 1.1
    return 1.0


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind in ("sirt", "mf"):
        K = sorted({max(1, case["iters"] // 4), case["iters"]})
        X, info = airt.sirt(case["method"], st["A"], st["b"], K, None, st["opts"])
        return dict(X=X, resnorms=info["resnorms"], finaliter=info["finaliter"])
    if kind == "art":
        X, info = airt.art(case["method"], st["A"], st["b"], case["iters"], None, st["opts"])
        return dict(X=X, resnorms=info["resnorms"])
    if kind == "cart":
        X, info = airt.columnaction(st["A"], st["b"], case["iters"], None, st["opts"])
        return dict(X=X, resnorms=info["resnorms"])
    if kind == "build":
        _, _, _, ct, sn, off = parallel_tables(case["N"], st["theta"], case["rays"])
        A = parallel_operator(case["N"], ct, sn, off)
        b = A(st["x"], "notransp")
        return dict(b=b, x=airt.fbp(A, b, st["theta"], case["filter"]), nnz=A.nnz)
    if kind == "batch":
        xs, info = st["batch"].sirt(case["method"], st["b"], case["iters"], taudelta=st["td"],
                                    lbound=0.0)
        return dict(x=np.concatenate(xs), finaliter=info["finaliter"])
    if kind == "multi":
        info = sirt_multi_device(st["A"], case["method"], st["B"].data_ptr(), st["X"].data_ptr(),
                                 case["count"], case["iters"], taudelta=st["td"], lbound=0.0)
        return dict(X=st["X"], finaliter=info["finaliter"])
    if case["train"]:
        loss = st["net"].gradients(st["u"].data_ptr(), st["t"].data_ptr(), case["batch"])
        return dict(loss=loss, grads=st["net"].get_grads())
    st["net"].forward_f64(st["u"].data_ptr(), st["out"].data_ptr(), case["batch"],
                          torch.cuda.current_stream().cuda_stream)
    return st["out"]


# ------------------------------------------------------------------ the work
def _nnz(case):
    """Nonzeros of A: every ray covers its chord at 4/pi pixels per unit."""
    N = case["N"]
    spacing = 1.0 if case.get("geom") != "fan" else (2.5 * N / case["rays"]) * (2.0 / 3.0)
    return case["angles"] * N * N * 4.0 / math.pi / spacing


def work(case):
    kind = case["kind"]
    if kind == "unet":
        mac = sum(9 * ci * co * (case["N"] >> lv) ** 2 for ci, co, lv in _unet_shapes(case))
        px = case["batch"] * case["N"] ** 2
        nw = sum(9 * ci * co + co for ci, co, _ in _unet_shapes(case))
        return {"bytes": px * (8 if case["train"] else 16) + nw * (8 if case["train"] else 2),
                "flops": 2.0 * mac * case["batch"] * (3 if case["train"] else 1)}
    if kind == "batch":
        sizes = [n for n in (64, 96, 128, 192, 256) if n <= case["nmax"]]
        na = 0.5 * (case["amin"] + case["amax"])
        nnz = case["count"] * na * np.mean([n * n for n in sizes]) * 4 / math.pi
        it = 25  # typical iterations to the stop
        return {"bytes": 16.0 * nnz * it, "flops": 4.0 * nnz * it}
    nnz, n, m = _nnz(case), case["N"] ** 2, case["angles"] * case["rays"]
    if kind == "multi":
        it, K = 15, case["count"]
        return {"bytes": it * (16.0 * nnz + K * (20.0 * n + 12.0 * m)), "flops": 4.0 * nnz * it * K}
    if kind == "build":
        return {"bytes": 16.0 * nnz + 8.0 * nnz + 16.0 * (m + n), "flops": 4.0 * nnz + 20.0 * nnz}
    it = case["iters"] if not case.get("level") else 20
    if kind == "mf":
        return {"bytes": it * 28.0 * (m + n), "flops": it * 2 * 12.0 * nnz}
    if kind in ("art", "cart"):
        return {"bytes": it * (8.0 * nnz + 16.0 * (m + n)), "flops": it * 4.0 * nnz}
    return {"bytes": it * (16.0 * nnz + 28.0 * n + 24.0 * m), "flops": it * 4.0 * nnz}


# ------------------------------------------------------------------ 64-bit answers
def _entries(N, rays):
    """(row, col, length) of A in FP64: the crossings of every ray with the
    grid lines sorted along it, one entry per positive piece inside."""
    h = 0.5 * N
    g = torch.arange(N + 1, dtype=F64, device=DEV) - h
    R = rays[0].numel()
    chunk = max(1, 24_000_000 // (2 * N + 2))
    rows, cols, vals = [], [], []
    for r0 in range(0, R, chunk):
        x0, y0, a, b = [v[r0:r0 + chunk, None] for v in rays]
        t = torch.cat([(g - x0) / a, (g - y0) / b], dim=1)
        t = torch.nan_to_num(t, nan=math.inf, posinf=math.inf, neginf=-math.inf).sort(dim=1).values
        norm = torch.sqrt(a * a + b * b)
        mid = 0.5 * (t[:, 1:] + t[:, :-1])
        ln = (t[:, 1:] - t[:, :-1]) * norm
        ix = torch.floor(x0 + a * mid + h)
        iy = torch.floor(y0 + b * mid + h)
        ok = (ix >= 0) & (ix < N) & (iy >= 0) & (iy < N) & (ln > 1e-10) & torch.isfinite(ln)
        r, k = ok.nonzero(as_tuple=True)
        rows.append((r + r0).int())
        cols.append((ix[r, k] * N + (N - 1 - iy[r, k])).int())
        vals.append(ln[r, k])
        del t, mid, ln, ix, iy, ok, r, k
    return torch.cat(rows), torch.cat(cols), torch.cat(vals)


def _csr(rows, cols, vals, m, n, transpose=False):
    if transpose:
        order = torch.sort(cols, stable=True).indices
        rows, cols, vals = cols[order], rows[order], vals[order]
        m, n = n, m
    ptr = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.bincount(rows, minlength=m).cumsum(0)
    return torch.sparse_csr_tensor(ptr.int(), cols, vals, size=(m, n))


def _system(case, rays):
    m, n = rays[0].numel(), case["N"] ** 2
    e = _entries(case["N"], rays)
    return _csr(*e, m, n), _csr(*e, m, n, transpose=True)


def _weights64(method, A, At):
    m, n = A.shape
    one = lambda k: torch.ones(k, dtype=F64, device=DEV)  # noqa: E731
    inv = lambda v: torch.where(v > 0, 1.0 / v, torch.zeros_like(v))  # noqa: E731
    if method == "landweber":
        return one(m), one(n)
    if method == "sart":
        return inv(A @ one(n)), inv(At @ one(m))
    sq = torch.sparse_csr_tensor(A.crow_indices(), A.col_indices(), A.values() ** 2, size=A.shape)
    return inv(sq @ one(n)) / m, one(n)


def _rho64(A, At, M, D):
    """Largest eigenvalue of D^(1/2) A' M A D^(1/2): Lanczos, full basis kept."""
    n = A.shape[1]
    sd = torch.sqrt(D)
    V = [torch.full((n,), 1.0 / math.sqrt(n), dtype=F64, device=DEV)]
    al, be, th = [], [], 0.0
    for _ in range(min(120, n)):
        w = sd * (At @ (M * (A @ (sd * V[-1]))))
        al.append(float(V[-1] @ w))
        B = torch.stack(V)
        for _ in range(2):
            w = w - B.T @ (B @ w)
        T = np.diag(al) + np.diag(be, 1) + np.diag(be, -1)
        prev, th = th, float(np.linalg.eigvalsh(T)[-1])
        be.append(float(torch.linalg.norm(w)))
        if be[-1] < 1e-12 * th or abs(th - prev) < 1e-14 * th:
            break
        V.append(w / be[-1])
    return th


def _sirt64(A, At, b, method, K, lo, hi, td, rho=None):
    """SIRT in FP64; K the iterations kept (an iterable) or the last one;
    b (rows,) or (rows, count) with td a number or one per column."""
    M, D = _weights64(method, A, At)
    rho = 1.0 if method == "sart" else rho if rho is not None else _rho64(A, At, M, D)
    many = b.dim() == 2
    if many:
        M, D = M[:, None], D[:, None]
    lam = 1.9 / rho
    kmax = max(K)
    x = torch.zeros((A.shape[1],) + b.shape[1:], dtype=F64, device=DEV)
    r = b.clone()
    fin = torch.full(b.shape[1:], kmax, dtype=torch.int64, device=DEV)
    nr = torch.linalg.norm(r, dim=0)
    res, kept = [nr], []
    live = torch.ones(b.shape[1:], dtype=torch.bool, device=DEV)
    for k in range(0, kmax + 1):
        if k > 0:
            xn = x + lam * (D * (At @ (M * r)))
            if lo is not None:
                xn = xn.clamp(min=lo)
            if hi is not None:
                xn = xn.clamp(max=hi)
            x = torch.where(live, xn, x)
            r = b - A @ x
            nr = torch.linalg.norm(r, dim=0)
            res.append(nr)
        if td is not None:
            stop = live & (nr <= td)
            fin[stop] = k
            live = live & ~stop
        if k in K:
            kept.append(x)
        if not live.any():
            break
    if not many and int(fin) not in K:
        kept = kept[:sum(1 for q in K if q < int(fin))] + [x]
    return x, fin, torch.stack(res), kept


def exact(case, seed):
    kind = case["kind"]
    if kind == "art" and case["method"] == "randkaczmarz":
        return None  # its row stream is the entry point's own
    if kind in ("sirt", "mf"):
        _, rays, b = _data(case, seed)
        A, At = _system(case, rays)
        lo, hi = (0.0, 1.0) if case["box"] else (None, None)
        td = case["level"] * float(torch.linalg.norm(b)) if case.get("level") else None
        K = sorted({max(1, case["iters"] // 4), case["iters"]})
        _, fin, res, kept = _sirt64(A, At, b, case["method"], K, lo, hi, td,
                                    _rho_bound(case) if case.get("rho") else None)
        return dict(X=torch.stack(kept, dim=1), resnorms=res, finaliter=int(fin))
    if kind in ("art", "cart"):
        return _sweeps64(case, seed)
    if kind == "build":
        rng = np.random.default_rng(seed)
        theta = _angles(case, rng)
        A, At = _system(case, _rays(case, theta))
        b = A @ torch.as_tensor(_image(case, seed), device=DEV)
        q = _fbp64(case, b)
        return dict(b=b, x=At @ q * (math.pi / (2 * case["angles"])), nnz=None)
    if kind == "batch":
        xs, fins = [], []
        for c, _, rays, b in _batch_problems(case, seed):
            A, At = _system(c, rays)
            x, fin, _, _ = _sirt64(A, At, b, case["method"], [case["iters"]], 0.0, None,
                                   case["level"] * float(torch.linalg.norm(b)))
            xs.append(x)
            fins.append(int(fin))
        return dict(x=torch.cat(xs), finaliter=np.array(fins))
    if kind == "multi":
        _, rays, B = _data(case, seed, case["count"])
        A, At = _system(case, rays)
        x, fin, _, _ = _sirt64(A, At, B.T.contiguous(), case["method"], [case["iters"]], 0.0, None,
                               case["level"] * torch.linalg.norm(B, dim=1))
        return dict(X=x.T.contiguous(), finaliter=fin)
    return _unet64(case, seed)


def _fbp64(case, b):
    """Every projection times the windowed ramp in the frequency domain."""
    p, na = case["rays"], case["angles"]
    order = max(64, 1 << math.ceil(math.log2(2 * p)))
    n = np.arange(order // 2 + 1) / (order // 2)
    f = n.copy()
    f[0] = 0.4 / order
    f[-1] = 1.0 - f[0]
    w = math.pi * n[1:]
    win = {"ram-lak": np.ones_like(w), "shepp-logan": np.sin(w / 2) / (w / 2),
           "hamming": 0.54 + 0.46 * np.cos(w), "hann": (1 + np.cos(w)) / 2}
    f[1:] *= win[case["filter"]]
    f = torch.as_tensor(np.concatenate([f, f[-2:0:-1]]), device=DEV)
    B = torch.zeros(na, order, dtype=F64, device=DEV)
    B[:, :p] = b.reshape(na, p)
    return torch.fft.ifft(torch.fft.fft(B) * f).real[:, :p].reshape(-1).contiguous()


def _sweeps64(case, seed):
    """Kaczmarz rows or CART columns one after the other, nonnegative."""
    _, rays, b = _data(case, seed)
    m, n = rays[0].numel(), case["N"] ** 2
    rows, cols, vals = _entries(case["N"], rays)
    cart = case["kind"] == "cart"
    W = _csr(rows, cols, vals, m, n, transpose=cart)
    ptr, idx, val = [v.cpu().numpy() for v in (W.crow_indices(), W.col_indices(), W.values())]
    A = _csr(rows, cols, vals, m, n)
    b, x, r = b.cpu().numpy(), np.zeros(n), b.cpu().numpy().copy()
    seg = [(i, idx[ptr[i]:ptr[i + 1]], val[ptr[i]:ptr[i + 1]]) for i in range(n if cart else m)
           if ptr[i + 1] > ptr[i]]
    seg = [(i, c, v, float(v @ v)) for i, c, v in seg]
    sym = case.get("method") == "symkaczmarz"
    order = seg + seg[::-1] if sym else seg
    res = [float(np.linalg.norm(b))]
    for _ in range(case["iters"] // 2 if sym else case["iters"]):
        if cart:
            for j, c, v, s in order:
                od = max(0.25 * float(v @ r[c]) / s, -x[j])
                x[j] += od
                r[c] -= od * v
            res.append(float(np.linalg.norm(r)))
        else:
            for i, c, v, s in order:
                xc = x[c]
                x[c] = np.maximum(xc + ((b[i] - float(v @ xc)) / s) * v, 0.0)
            rr = b - (A @ torch.as_tensor(x, device=DEV)).cpu().numpy()
            res.append(float(np.linalg.norm(rr)))
    return dict(X=x[:, None], resnorms=np.array(res))


def _unet64(case, seed):
    """The network in FP64 (no BF16 rounding), gradients by autograd."""
    F = torch.nn.functional
    prm, u, t = _unet_data(case, seed)
    p = torch.as_tensor(prm, device=DEV).double().requires_grad_(case["train"])
    N, B, L = case["N"], case["batch"], case["levels"]
    views, off = [], 0
    for cin, cout, _ in _unet_shapes(case):
        w = p[off:off + 9 * cin * cout].reshape(cout, 3, 3, cin).permute(0, 3, 1, 2)
        off += 9 * cin * cout
        views.append((w, p[off:off + cout]))
        off += cout
    hw, hb = p[off:off + case["base"]], p[off + case["base"]]

    def net(x):
        it = iter(views)
        conv = lambda v: F.relu(F.conv2d(v, *next(it), padding=1))  # noqa: E731
        skips = []
        for lv in range(L):
            x = conv(conv(x if lv == 0 else F.max_pool2d(x, 2)))
            skips.append(x)
        for lv in range(L - 2, -1, -1):
            x = conv(conv(torch.cat([F.interpolate(x, scale_factor=2.0), skips[lv]], dim=1)))
        return torch.einsum("bchw,c->bhw", x, hw) + hb

    def img(v):  # column-major images: row index first
        return v.reshape(-1, N, N).transpose(1, 2)

    loss = 0.0
    outs = []
    step = 2 if case["train"] else 4
    for q in range(0, B, step):
        x = img(u[q:q + step].float().double() if case["train"] else u[q:q + step])[:, None]
        if case["train"]:
            part = ((net(x) - img(t[q:q + step].float().double())) ** 2).sum() / (B * N * N)
            part.backward()
            loss += float(part.detach())
        else:
            with torch.no_grad():
                outs.append(net(x).transpose(1, 2).reshape(-1, N * N))
    if case["train"]:
        return dict(loss=loss, grads=p.grad)
    return torch.cat(outs)
