"""What a user of this framework has it do, as measurable cases.

Every case is one job of the kernel-polynomial path through the Python API (each call one C-ABI
entry point): a Hamiltonian from a geometry, moments, densities. The sizes are those of the
benchmark workloads, the example inputs and the tests, and what lies between them:

  cell    one k point of a k-sampled supercell job: assembly, local moments, one density per target
  dos     density of states of a matrix in hand, random-phase vectors (cells and flakes, FP32 or FP64)
  ldos    local moments of a few orbitals of a flake in hand
  field   random-phase moments of a flake in a magnetic field (complex Hamiltonian)
  job     a whole job from the geometry: assembly, spectral bounds, moments, density on an energy grid
  kubo    Kubo moments of a flake by random-phase vectors, and the conductivity on an energy grid
  batch   many flakes together (one handle, replayed with other vectors)
  sites   the network's sum over all sites of a flake (inference)
  grad    one loss and gradient of the network on a batch of rows (forward and backward)

An FP32 recursion's moments carry single precision (only their sums are FP64), so they are handed on
as float32; FP64 recursions, and transforms of moments that came from the host, stay float64.
The seed moves the twist angle (or the layer distance of a commensurate cell) by up to a part in a
thousand and sets the vectors, the targets and the Bloch vector.
"""
import math
import random

import numpy as np
import torch

import leo2d_gb300 as L

A0 = 2.46                                  # simple model's lattice constant (A)
CELL_AREA = A0 * A0 * math.sqrt(3.0) / 2   # area of a graphene cell, two orbitals
PER_ROW = 67.0                             # stored entries per row of the simple model's bilayer
ON_CHIP = 100e6                            # bytes that stay in L2 between Chebyshev steps


def listed():
    return [
        # the smallest call: a k point of a (3,2) cell (76 orbitals), real targets, as the k-path examples
        {"name": "cell_76_kpoint", "kind": "cell", "m": 3, "model": "simple", "P": 400, "targets": 4, "k": True},
        # a mid-size commensurate cell with the reference's graphene model, Gamma point, one line of targets
        {"name": "cell_2k_ldos", "kind": "cell", "m": 13, "model": "ref", "P": 1000, "targets": 12, "k": False},
        # benchmark: the 1.05 degree (31,32) cell, 11,908 orbitals, P = 4096, 64 vectors
        {"name": "cell_12k_dos", "kind": "dos", "m": 31, "n": 0, "theta": 0.0, "P": 4096, "R": 64, "fp64": False},
        # benchmark: the 5.09 degree flake, 52k orbitals, FP64 recursion, P = 1000, 16 vectors
        {"name": "flake_52k_fp64", "kind": "dos", "m": 0, "n": 52000, "theta": 5.09, "P": 1000, "R": 16, "fp64": True},
        # local density at the centre sites of a flake
        {"name": "flake_200k_ldos", "kind": "ldos", "n": 200000, "theta": 1.47, "P": 1000, "targets": 8},
        # benchmark headline's matrix in hand: 10M orbitals, P = 1024, the 13 vectors it needs
        {"name": "flake_10M_dos", "kind": "dos", "m": 0, "n": 10000000, "theta": 0.5, "P": 1024, "R": 13, "fp64": False},
        # a whole job at the headline's stacking, from the geometry to the density
        {"name": "flake_2M_job", "kind": "job", "n": 2400000, "theta": 0.5, "model": "simple", "P": 256, "R": 13},
        # magnetic field: complex matrix, 16 complex vectors
        {"name": "flake_400k_field", "kind": "field", "n": 400000, "theta": 0.9, "B": 20.0, "P": 512, "R": 16},
        # Kubo moments and conductivity
        {"name": "flake_150k_kubo", "kind": "kubo", "n": 150000, "theta": 1.5, "P": 256, "R": 16, "energies": 1001},
        # benchmark: flakes of mixed sizes in one batch
        {"name": "batch_10_flakes", "kind": "batch", "flakes": 10, "n": 20000, "n_max": 200000, "P": 512, "R": 32},
        # the network over every site of a flake
        {"name": "network_1M_sites", "kind": "sites", "n": 1000000, "theta": 1.05},
        # one gradient of the network
        {"name": "network_grad_8k", "kind": "grad", "rows": 8192},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cell", "cell", "dos", "dos", "ldos", "field", "job", "kubo", "batch", "sites", "grad"])
    order = lambda lo, hi: 4 * max(1, _log(rng, lo, hi) // 4)  # poly_order is a multiple of 4
    if kind == "cell":
        return {"kind": kind, "m": rng.randint(3, 20), "model": rng.choice(["simple", "ref"]), "P": order(64, 2000),
                "targets": _log(rng, 1, 40), "k": rng.random() < 0.5}
    if kind == "dos":
        where = rng.random()
        if where < 0.35:
            return {"kind": kind, "m": rng.randint(8, 31), "n": 0, "theta": 0.0, "P": order(256, 4096),
                    "R": _log(rng, 2, 64), "fp64": False}
        if where < 0.55:
            return {"kind": kind, "m": 0, "n": _log(rng, 5000, 60000), "theta": rng.uniform(2.0, 6.0), "P": order(200, 1000),
                    "R": _log(rng, 1, 16), "fp64": True}
        return {"kind": kind, "m": 0, "n": _log(rng, 20000, 5000000), "theta": rng.uniform(0.5, 3.0), "P": order(200, 1024),
                "R": _log(rng, 4, 32), "fp64": False}
    if kind == "ldos":
        return {"kind": kind, "n": _log(rng, 20000, 1000000), "theta": rng.uniform(0.8, 6.0), "P": order(200, 1000),
                "targets": _log(rng, 1, 48)}
    if kind == "field":
        return {"kind": kind, "n": _log(rng, 50000, 1000000), "theta": rng.uniform(0.5, 3.0), "B": rng.uniform(1.0, 40.0),
                "P": order(200, 512), "R": _log(rng, 1, 32)}
    if kind == "job":
        return {"kind": kind, "n": _log(rng, 50000, 3000000), "theta": rng.uniform(0.5, 5.0),
                "model": rng.choice(["simple", "ref"]), "P": order(128, 512), "R": _log(rng, 4, 16)}
    if kind == "kubo":
        return {"kind": kind, "n": _log(rng, 10000, 300000), "theta": rng.uniform(1.0, 5.0), "P": order(64, 256),
                "R": _log(rng, 4, 32), "energies": _log(rng, 301, 2001)}
    if kind == "batch":
        lo = _log(rng, 10000, 50000)
        return {"kind": kind, "flakes": rng.randint(2, 24), "n": lo, "n_max": lo * rng.randint(2, 8), "P": order(128, 512),
                "R": rng.choice([8, 16, 24, 32])}
    if kind == "sites":
        return {"kind": kind, "n": _log(rng, 100000, 4000000), "theta": rng.uniform(0.5, 4.0)}
    return {"kind": kind, "rows": _log(rng, 300, 16000)}


# ---------------------------------------------------------------- inputs

def _radius(n):
    return math.sqrt(n * CELL_AREA / (4.0 * math.pi))  # two sheets, two orbitals a cell


def _rescale(case):
    return 20.0 if case.get("model") == "ref" else 10.5


def _moved(case, seed):
    """(random source, twist in degrees, layer distance) of one seed."""
    r = random.Random(1000003 * int(seed) + 17)
    u = r.uniform(-1e-3, 1e-3)
    return r, case.get("theta", 0.0) * (1.0 + u), 3.35 * (1.0 + u)


def _flake_geom(n, theta, h=3.35, rescale=10.5, model="simple", b_field=0.0):
    R = _radius(n)
    size = int(math.ceil(R / A0 * (1.0 + 1.0 / math.sqrt(3.0)))) + 4
    return L.make_geom(model=L.MODEL_REF if model == "ref" else L.MODEL_SIMPLE, size=size, max_R=R, heights=(0.0, h),
                       angles_deg=(0.0, theta), energy_rescale=rescale, b_field=b_field)


def _cell_geom(m, h, rescale=10.5, model="simple", k_vec=None):
    # (m, m-1) below the benchmark's (31, 32), as the examples' (3, 2)
    mn = (31, 32) if m == 31 else (m, m - 1)
    return L.make_geom(model=L.MODEL_REF if model == "ref" else L.MODEL_SIMPLE, boundary_condition=1, size=2 * m + m + 6,
                       supercell_mn=mn, heights=(0.0, h), energy_rescale=rescale, k_vec=k_vec)


def _k_vec(r):
    return (r.uniform(0.005, 0.2), r.uniform(0.005, 0.2))


def _cell_orbitals(m):
    a, b = (31, 32) if m == 31 else (m, m - 1)
    return 4 * (a * a + a * b + b * b)


def _batch_sizes(case):
    f = case["flakes"]
    return [int(case["n"] * (case["n_max"] / case["n"]) ** (i / (f - 1))) for i in range(f)]


def _network(seed):
    """Random parameters (W0 [256][64], b0, W1 [256][256], b1, W2, b2, W3, b3) of the usual scale."""
    g = np.random.default_rng(seed)
    return np.concatenate([np.concatenate([(g.standard_normal((256, d)) * math.sqrt(1.6 / d)).ravel(),
                                           0.05 * g.standard_normal(256)]) for d in (16 * 4, 256, 256, 256)]).astype(np.float32)


def _rows(case, seed):
    g = np.random.default_rng(seed + 5)
    ph = 2 * math.pi * g.random((case["rows"], 2))
    x = np.stack([np.cos(ph[:, 0]), np.sin(ph[:, 0]), np.cos(ph[:, 1]), np.sin(ph[:, 1]), np.cos(ph.sum(1)), np.sin(ph.sum(1)),
                  np.cos(ph[:, 0] - ph[:, 1]), np.sin(ph[:, 0] - ph[:, 1]), np.cos(2 * ph[:, 0]), np.sin(2 * ph[:, 0]),
                  np.cos(2 * ph[:, 1]), np.sin(2 * ph[:, 1]), 0.3 * np.ones(len(ph)), g.integers(0, 2, len(ph)),
                  g.integers(0, 2, len(ph)), np.ones(len(ph))], 1)
    return x.astype(np.float32), (0.3 * g.standard_normal((case["rows"], 256))).astype(np.float32)


def _centre_targets(n, count, r):
    """Orbitals spread over both sheets (the targets of a local job)."""
    return sorted(r.sample(range(n), min(count, n)))


def prepare(case, seed):
    ctx = L.Context(0)
    r, theta, h = _moved(case, seed)
    s = {"case": case, "ctx": ctx, "seed": int(seed)}
    kind = case["kind"]
    if kind == "cell":
        k = _k_vec(r) if case["k"] else None
        s["geom"] = ctx.prepare(_cell_geom(case["m"], h, _rescale(case), case["model"], k))
        s["targets"] = _centre_targets(_cell_orbitals(case["m"]), case["targets"], r)
        s["cfg"] = L.kpm_cfg(case["P"])
    elif kind == "dos":
        g = _cell_geom(case["m"], h) if case["m"] else _flake_geom(case["n"], theta)
        s["csr"] = ctx.build_csr(g)
        s["cfg"] = L.kpm_cfg(case["P"], R=case["R"], seed=seed, precision=L.FP64 if case["fp64"] else L.FP32)
    elif kind == "ldos":
        s["csr"] = ctx.build_csr(_flake_geom(case["n"], theta))
        s["targets"] = _centre_targets(s["csr"].n, case["targets"], r)
        s["cfg"] = L.kpm_cfg(case["P"])
    elif kind == "field":
        s["csr"] = ctx.build_csr(_flake_geom(case["n"], theta, b_field=case["B"]))
        s["cfg"] = L.kpm_cfg(case["P"], R=case["R"], seed=seed)
    elif kind == "job":
        s["geom"] = ctx.prepare(_flake_geom(case["n"], theta, rescale=1.0, model=case["model"]))
        s["cfg"] = L.kpm_cfg(case["P"], R=case["R"], seed=seed)
    elif kind == "kubo":
        s["csr"] = ctx.build_csr(_flake_geom(case["n"], theta))
        s["cfg"] = L.kpm_cfg(case["P"], R=case["R"], seed=seed)
        s["E"] = _energies(case["energies"])
    elif kind == "batch":
        s["csrs"] = [ctx.build_csr(_flake_geom(n, 1.0 + 0.1 * i + theta + 1e-3 * r.random()))
                     for i, n in enumerate(_batch_sizes(case))]
        s["batch"] = L.Batch(ctx, s["csrs"], L.kpm_cfg(case["P"], R=case["R"], seed=seed))
    elif kind == "sites":
        s["csr"] = ctx.build_csr(_flake_geom(case["n"], theta))
        s["theta"] = theta
        s["net"] = L.Mlp(ctx)
        s["net"].set_params(_network(seed))
    else:
        s["net"] = L.Mlp(ctx)
        s["net"].set_params(_network(seed))
        s["x"], s["t"] = _rows(case, seed)
    return s


def _energies(count):
    return 10.5 * (-0.98 + 1.96 * (np.arange(count) + 0.5) / count)


def run(s):
    case, ctx, kind = s["case"], s["ctx"], s["case"]["kind"]
    if kind == "cell":
        csr = ctx.build_csr(s["geom"])
        mu = csr.kpm_ldos(s["cfg"], s["targets"])
        dos = [ctx.dos_transform(row, case["P"], _rescale(case), 0.0)[0] for row in mu]
        csr.close()
        return {"mu": mu.astype(np.float32), "dos": np.array(dos, np.float32)}
    if kind == "dos":
        mu = s["csr"].kpm_dos(s["cfg"])
        return mu if case["fp64"] else mu.astype(np.float32)
    if kind == "ldos":
        return s["csr"].kpm_ldos(s["cfg"], s["targets"]).astype(np.float32)
    if kind == "field":
        return s["csr"].kpm_dos(s["cfg"]).astype(np.float32)
    if kind == "job":
        csr = ctx.build_csr(s["geom"])
        lo, hi = csr.bounds()
        a, b = 1.01 * (hi - lo) / 2, (hi + lo) / 2
        csr.rescale(a, -b)
        mu = csr.kpm_dos(s["cfg"])
        dos = ctx.dos_reconstruct(mu.mean(axis=0), b + a * (-1.0 + 2.0 * (np.arange(4001) + 0.5) / 4001), a, b, 1.0 / csr.n)
        csr.close()
        return {"bounds": np.array([lo, hi]), "mu": mu.astype(np.float32), "dos": dos.astype(np.float32)}
    if kind == "kubo":
        mu = s["csr"].kpm_cond(s["cfg"])
        return {"mu": mu.astype(np.float32), "sigma": ctx.cond_sigma(mu, s["E"], 10.5, 0.0).astype(np.float32)}
    if kind == "batch":
        return s["batch"].run(seed=s["seed"]).astype(np.float32)
    if kind == "sites":
        return s["net"].site_sum(s["csr"], s["theta"]).astype(np.float32)
    loss, grad = s["net"].grad(s["x"], s["t"])
    return {"loss": np.float32(loss), "grad": grad}


# ---------------------------------------------------------------- what a pass cannot do without

def _recursion(n, cols, P, entry_bytes, item, per_row=PER_ROW, complex_h=False):
    """Bytes and flops of P/2 Chebyshev steps of `cols` real columns: the matrix, T_n and T_{n-1} read
    and T_{n+1} written once a step, or once in all where they stay on the chip."""
    matrix, vectors = n * per_row * entry_bytes, n * cols * item
    one = matrix + 3 * vectors
    steps = P // 2
    return {"bytes": one if matrix + 2 * vectors < ON_CHIP else one * steps,
            "flops": steps * n * cols * (per_row * (4 if complex_h else 2) + 6)}


def work(case):
    kind = case["kind"]
    if kind == "cell":
        n, c = _cell_orbitals(case["m"]), 2 if case["k"] else 1
        per_row = PER_ROW if case["model"] == "simple" else 160.0
        w = _recursion(n, c * case["targets"], case["P"], 4 + 4 * c, 4, per_row, case["k"])
        return {"bytes": w["bytes"] + n * per_row * (4 + 8 * c), "flops": w["flops"] + 60 * n * per_row}
    if kind == "dos":
        n = _cell_orbitals(case["m"]) if case["m"] else case["n"]
        return _recursion(n, 2 * case["R"], case["P"], 12 if case["fp64"] else 8, 8 if case["fp64"] else 4)
    if kind == "ldos":
        return _recursion(case["n"], case["targets"], case["P"], 8, 4)
    if kind == "field":
        return _recursion(case["n"], 2 * case["R"], case["P"], 12, 4, complex_h=True)
    if kind == "job":
        per_row = PER_ROW if case["model"] == "simple" else 160.0
        w = _recursion(case["n"], 2 * case["R"], case["P"], 8, 4, per_row)
        return {"bytes": w["bytes"] + case["n"] * per_row * 12, "flops": w["flops"] + 60 * case["n"] * per_row}
    if kind == "kubo":
        n, P, c = case["n"], case["P"], 2 * case["R"]
        w = _recursion(n, c, 2 * P, 8, 4)  # P steps of the B side; as many with two products on the A side
        return {"bytes": 2 * w["bytes"] + 4.0 * n * c * P * 4, "flops": 3 * w["flops"] + 2.0 * P * P * n * c}
    if kind == "batch":
        ws = [_recursion(n, 2 * case["R"], case["P"], 8, 4) for n in _batch_sizes(case)]
        return {"bytes": sum(w["bytes"] for w in ws), "flops": sum(w["flops"] for w in ws)}
    mac = 64 * 256 + 3 * 256 * 256
    if kind == "sites":
        return {"bytes": case["n"] * 16.0 + 4.0 * mac, "flops": 2.0 * mac * case["n"]}
    return {"bytes": case["rows"] * 272 * 4.0 + 8.0 * mac, "flops": 6.0 * mac * case["rows"]}


# ---------------------------------------------------------------- the same in 64 bits, by torch alone

_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_F = torch.float64


def _grid(lo, hi):
    """Cells (i, j) and orbital of a sheet's lattice in its enumeration order, with positions in its own frame."""
    i, j, l = torch.meshgrid(torch.arange(lo[0], hi[0], device=_DEV), torch.arange(lo[1], hi[1], device=_DEV),
                             torch.arange(2, device=_DEV), indexing="ij")
    i, j, l = i.reshape(-1), j.reshape(-1), l.reshape(-1)
    x = i.to(_F) * A0 + j.to(_F) * (0.5 * A0) + l.to(_F) * (0.5 * A0)
    y = j.to(_F) * (0.866025403784438646764 * A0) + l.to(_F) * (0.288675134594812882255 * A0)
    return i, j, l, x, y


def _turn(x, y, t):
    return x * math.cos(t) - y * math.sin(t), x * math.sin(t) + y * math.cos(t)


def _hop(dx, dy, h):
    r = torch.sqrt(dx * dx + dy * dy + h * h)
    return torch.where(r < 8.0, 0.33 * torch.exp(-(r - 3.35) / 0.45), torch.zeros_like(r))


def _phase(v, x1, y1, x2, y2, B, k):
    if not B and k is None:
        return v
    ph = 3.14e-5 * B * (x2 - x1) * 0.5 * (y1 + y2)
    if k is not None:
        ph = ph + k[0] * (x2 - x1) + k[1] * (y2 - y1)
    return torch.polar(v, ph)


def _flake_h(n_want, theta, h=3.35, B=0.0, velocity=False):
    """(crow, col, values[, velocities], x, y) of a simple-model flake, unrescaled."""
    R, th = _radius(n_want), [0.0, 2 * math.pi * theta / 360.0]
    size = int(math.ceil(R / A0 * (1.0 + 1.0 / math.sqrt(3.0)))) + 4
    sheets, base = [], 0
    for s in range(2):
        i, j, l, x, y = _grid((-size, -size), (size, size))
        keep = x * x + y * y < R * R
        index = torch.full((2 * size, 2 * size, 2), -1, dtype=torch.int64, device=_DEV)
        i, j, l, x, y = i[keep], j[keep], l[keep], x[keep], y[keep]
        index[i + size, j + size, l] = base + torch.arange(len(i), device=_DEV)
        base += len(i)
        sheets.append((i, j, l, *_turn(x, y, th[s]), index))
    X, Y = torch.cat([s[3] for s in sheets]), torch.cat([s[4] for s in sheets])
    counts, cols, vals, vels = [], [], [], []
    window = torch.arange(-5, 6, device=_DEV)
    for s in range(2):
        i, j, l, x, y, index = sheets[s]
        other = sheets[1 - s][5]
        for c0 in range(0, len(i), 100000):
            cut = slice(c0, c0 + 100000)
            ii, jj, ll, xx, yy = i[cut], j[cut], l[cut], x[cut], y[cut]
            step = torch.where(ll == 1, 1, -1)  # orbital 0 meets orbital 1 of cells (0,0), (-1,0), (0,-1)
            near = torch.stack([index[(ii + size), (jj + size), 1 - ll], index[(ii + step + size), (jj + size), 1 - ll],
                                index[(ii + size), (jj + step + size), 1 - ll]], 1)
            u, v = _turn(xx, yy, -th[1 - s])
            b = torch.floor(v / (0.866025403784438646764 * A0))
            a = torch.floor(u / A0 - 0.5 * v / (0.866025403784438646764 * A0))
            oi = (a.long()[:, None, None, None] + window[None, :, None, None] + size).expand(-1, 11, 11, 2)
            oj = (b.long()[:, None, None, None] + window[None, None, :, None] + size).expand(-1, 11, 11, 2)
            inside = (oi >= 0) & (oi < 2 * size) & (oj >= 0) & (oj < 2 * size)
            far = other[oi.clamp(0, 2 * size - 1), oj.clamp(0, 2 * size - 1),
                        torch.arange(2, device=_DEV).expand(oi.shape)]
            far = torch.where(inside, far, -1).reshape(len(ii), -1)
            cand = torch.cat([near, far], 1)
            at = cand.clamp(min=0)
            t = torch.where(cand >= 0, _hop(X[at] - xx[:, None], Y[at] - yy[:, None], h), 0.0)
            t[:, :3] = -2.7 * (cand[:, :3] >= 0).to(_F)
            hit = t != 0
            at, x1, y1 = at[hit], xx[:, None].expand_as(t)[hit], yy[:, None].expand_as(t)[hit]
            counts.append(hit.sum(1))
            cols.append(at)
            vals.append(_phase(t[hit], x1, y1, X[at], Y[at], B, None))
            if velocity:
                vels.append(t[hit] * (x1 - X[at]))
    crow = torch.zeros(len(X) + 1, dtype=torch.int64, device=_DEV)
    crow[1:] = torch.cumsum(torch.cat(counts), 0)
    return crow, torch.cat(cols), torch.cat(vals), torch.cat(vels) if velocity else None, X, Y


def _cell_h(m, h, k=None):
    M, N = (31, 32) if m == 31 else (m, m - 1)
    th = math.acos((N * N + 4 * N * M + M * M) / (2.0 * (N * N + N * M + M * M)))
    th = -th if M < N else th
    size = 2 * m + m + 6
    a1, a2 = np.array([A0, 0.0]), np.array([0.5 * A0, 0.866025403784438646764 * A0])
    xs, ys, sheet, cell = [], [], [], None
    for s, (p, q, u, v) in enumerate(((N, M, -M, M + N), (M, N, -N, M + N))):
        sc = np.array([p * a1 + q * a2, u * a1 + v * a2])
        cell = sc if s == 0 else cell
        det = sc[0, 0] * sc[1, 1] - sc[0, 1] * sc[1, 0]
        _, _, _, x, y = _grid((-size, -size), (size, size))
        f0, f1 = (x * sc[1, 1] - y * sc[1, 0]) / det, (-x * sc[0, 1] + y * sc[0, 0]) / det
        keep = (f0 >= -1e-6) & (f0 < 1 - 1e-6) & (f1 >= -1e-6) & (f1 < 1 - 1e-6)
        x, y = _turn(x[keep], y[keep], th * s)
        xs.append(x)
        ys.append(y)
        sheet.append(torch.full((len(x),), s, device=_DEV))
    X, Y, S = torch.cat(xs), torch.cat(ys), torch.cat(sheet)
    rows, cols, vals = [], [], []
    for a in (-1, 0, 1):
        for b in (-1, 0, 1):
            dx = X[None, :] + a * cell[0, 0] + b * cell[1, 0] - X[:, None]
            dy = Y[None, :] + a * cell[0, 1] + b * cell[1, 1] - Y[:, None]
            r2 = dx * dx + dy * dy
            same = S[None, :] == S[:, None]
            t = torch.where(same, -2.7 * ((r2 > 1.0) & (r2 < 2.5)).to(_F), _hop(dx, dy, h))
            i, j = torch.nonzero(t, as_tuple=True)
            rows.append(i)
            cols.append(j)
            vals.append(_phase(t[i, j], 0.0, 0.0, dx[i, j], dy[i, j], 0.0, k))
    i, j, v = torch.cat(rows), torch.cat(cols), torch.cat(vals)
    return torch.sparse_coo_tensor(torch.stack([i, j]), v, (len(X), len(X))).coalesce().to_sparse_csr(), len(X)


def _csr(crow, col, val):
    n = len(crow) - 1
    return torch.sparse_csr_tensor(crow, col, val, (n, n)), n


def _mul32(m, c):
    """High and low words of m c for 32-bit words held in int64."""
    p0, p1 = m * (c & 0xFFFF), m * (c >> 16)
    return (p1 + (p0 >> 16)) >> 16, (((p1 & 0xFFFF) << 16) + p0) & 0xFFFFFFFF


def _phases(n, R, seed):
    """Random phases of Philox4x32-10 (counter: row, vector; key: seed), as float32 cosines and sines."""
    out = torch.empty((n, R), dtype=_F, device=_DEV)
    for v in range(R):
        c = [torch.arange(n, device=_DEV), torch.zeros(n, dtype=torch.int64, device=_DEV),
             torch.full((n,), v, dtype=torch.int64, device=_DEV), torch.zeros(n, dtype=torch.int64, device=_DEV)]
        k0, k1 = seed & 0xFFFFFFFF, seed >> 32
        for _ in range(10):
            h0, l0 = _mul32(0xD2511F53, c[0])
            h1, l1 = _mul32(0xCD9E8D57, c[2])
            c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
            k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
        out[:, v] = (c[0] >> 8).to(_F) * (2 * math.pi / 16777216.0)
    return torch.cos(out).float().to(_F), torch.sin(out).float().to(_F)


def _moments(H, a, T0, P):
    """Re <T_0|T_n(H / a)|T_0> per column, n < P."""
    out = torch.empty((P, T0.shape[1]), dtype=_F, device=_DEV)
    t0, t1 = T0, (H @ T0) / a
    dot = lambda x, y: (x.conj() * y).real.sum(0)
    for k in range(P // 2):
        d0, d1 = dot(t0, t0), dot(t1, t0)
        out[2 * k], out[2 * k + 1] = (d0, d1) if k == 0 else (2 * d0 - out[0], 2 * d1 - out[1])
        t0, t1 = t1, 2 * (H @ t1) / a - t0
    return out.T


def _trace(H, n, a, case, seed):
    c, s = _phases(n, case["R"], seed)
    if H.dtype.is_complex:
        return _moments(H, a, torch.complex(c, s), case["P"]).cpu().numpy()
    return sum(_moments(H, a, x, case["P"]) for x in (c, s)).cpu().numpy()


def _units(n, targets, dtype):
    T = torch.zeros((n, len(targets)), dtype=dtype, device=_DEV)
    T[torch.tensor(targets, device=_DEV), torch.arange(len(targets), device=_DEV)] = 1
    return T


def _jackson(P):
    i = np.arange(P)
    return ((P - i) * np.cos(np.pi * i / P) + np.sin(np.pi * i / P) / np.tan(np.pi / P)) / P


def _density(mu, x, a):
    """Jackson-damped density of moments mu at the scaled energies x."""
    g = mu * _jackson(len(mu))
    w = np.full(len(mu), 2.0)
    w[0] = 1.0
    return np.cos(np.outer(np.arccos(x), np.arange(len(mu)))) @ (w * g) / (np.pi * a * np.sqrt(1 - x * x))


def _kubo(case, theta, seed):
    crow, col, val, vel, X, _ = _flake_h(case["n"], theta, velocity=True)
    (H, n), (D, _) = _csr(crow, col, val / 10.5), _csr(crow, col, vel / 10.5)
    P, mu = case["P"], torch.zeros((case["P"], case["P"]), dtype=_F, device=_DEV)
    for part in _phases(n, case["R"], seed):
        for v0 in range(0, case["R"], 8):
            r = part[:, v0:v0 + 8].contiguous()
            right = torch.empty((P,) + tuple(r.shape), dtype=_F, device=_DEV)
            left = torch.empty_like(right)
            t = [r, -(D @ r)]
            for out, f, x in ((right, lambda y: y, r), (left, lambda y: D @ y, t[1])):
                t0, t1 = x, H @ x
                for k in range(P):
                    out[k] = f(t0)
                    t0, t1 = t1, 2 * (H @ t1) - t0
            mu += left.reshape(P, -1) @ right.reshape(P, -1).T
    mu = (mu / case["R"]).cpu().numpy()
    x = _energies(case["energies"]) / 10.5
    g = _jackson(P) * np.where(np.arange(P) == 0, 1.0, 2.0)
    T = np.cos(np.outer(np.arccos(x), np.arange(P))) * g
    return {"mu": mu, "sigma": np.einsum("ea,ab,eb->e", T, mu, T, optimize=True) / (np.pi ** 2 * (1 - x * x))}


def _gelu(z):
    # the network's activation: erf as Abramowitz & Stegun 7.1.27 gives it
    x = z.abs() / math.sqrt(2.0)
    q = 1 + x * (0.278393 + x * (0.230389 + x * (0.000972 + x * 0.078108)))
    return 0.5 * z * (1 + torch.sign(z) * (1 - q ** -4))


def _layers(p):
    out, at = [], 0
    for d in (64, 256, 256, 256):
        out.append((p[at:at + 256 * d].reshape(256, d), p[at + 256 * d:at + 256 * d + 256]))
        at += 256 * d + 256
    return out


def _forward(p, x):
    a = torch.nn.functional.pad(x, (0, 64 - x.shape[1]))
    for k, (W, b) in enumerate(_layers(p)):
        a = a @ W.T + b
        a = _gelu(a) if k < 3 else a
    return a


def _site_features(n_want, theta):
    """Stacking features of every site: the other sheet's fractional cell coordinates of its cell's origin."""
    R, th = _radius(n_want), [0.0, 2 * math.pi * theta / 360.0]
    size = int(math.ceil(R / A0 * (1.0 + 1.0 / math.sqrt(3.0)))) + 4
    out = []
    for s in range(2):
        i, j, l, x, y = _grid((-size, -size), (size, size))
        keep = x * x + y * y < R * R
        i, j, l = i[keep], j[keep], l[keep]
        x, y = i.to(_F) * A0 + j.to(_F) * (0.5 * A0), j.to(_F) * (0.866025403784438646764 * A0)
        u, v = _turn(*_turn(x, y, th[s]), -th[1 - s])
        q = 2 * math.pi * v / (0.866025403784438646764 * A0)
        p = 2 * math.pi * u / A0 - 0.5 * q
        one = torch.ones_like(p)
        out.append(torch.stack([p.cos(), p.sin(), q.cos(), q.sin(), (p + q).cos(), (p + q).sin(), (p - q).cos(), (p - q).sin(),
                                (2 * p).cos(), (2 * p).sin(), (2 * q).cos(), (2 * q).sin(), one * (theta / 3.0), one * s,
                                l.to(_F), one], 1))
    return torch.cat(out)


def exact(case, seed):
    r, theta, h = _moved(case, seed)
    kind = case["kind"]
    if case.get("model") == "ref":
        return None  # the fitted graphene model's tables exist in this repository only
    if kind == "cell":
        k = _k_vec(r) if case["k"] else None
        H, n = _cell_h(case["m"], h, k)
        mu = _moments(H, 10.5, _units(n, _centre_targets(n, case["targets"], r), H.dtype), case["P"]).cpu().numpy()
        P = case["P"]
        x = np.cos((np.arange(P) + 0.5) * np.pi / P)
        return {"mu": mu, "dos": np.array([_density(row, x, 10.5) for row in mu])}
    if kind == "dos":
        if case["m"]:
            H, n = _cell_h(case["m"], h)
        elif case["n"] * case["R"] * case["P"] > 3e9:
            return None  # minutes in 64 bits
        else:
            crow, col, val, _, _, _ = _flake_h(case["n"], theta)
            H, n = _csr(crow, col, val)
        return _trace(H, n, 10.5, case, seed)
    if kind == "ldos":
        crow, col, val, _, _, _ = _flake_h(case["n"], theta)
        H, n = _csr(crow, col, val)
        return _moments(H, 10.5, _units(n, _centre_targets(n, case["targets"], r), _F), case["P"]).cpu().numpy()
    if kind == "field":
        if case["n"] * case["R"] * case["P"] > 4e9:
            return None
        crow, col, val, _, _, _ = _flake_h(case["n"], theta, B=case["B"])
        H, n = _csr(crow, col, val)
        return _trace(H, n, 10.5, case, seed)
    if kind == "job":
        if case["n"] * case["R"] * case["P"] > 9e9:
            return None
        crow, col, val, _, _, _ = _flake_h(case["n"], theta)
        H, n = _csr(crow, col, val)
        row = torch.repeat_interleave(torch.arange(n, device=_DEV), crow[1:] - crow[:-1])
        top = float(torch.zeros(n, dtype=_F, device=_DEV).index_add_(0, row, val.abs()).max())
        mu = _trace(H, n, 1.01 * top, case, seed)
        x = -1.0 + 2.0 * (np.arange(4001) + 0.5) / 4001
        return {"bounds": np.array([-top, top]), "mu": mu, "dos": _density(mu.mean(axis=0), x, 1.01 * top) / n}
    if kind == "kubo":
        return _kubo(case, theta, seed)
    if kind == "batch":
        out = []
        for i, n in enumerate(_batch_sizes(case)):
            crow, col, val, _, _, _ = _flake_h(n, 1.0 + 0.1 * i + theta + 1e-3 * r.random())
            out.append(_trace(*_csr(crow, col, val), 10.5, case, seed))
        return np.array(out)
    p = torch.from_numpy(_network(seed)).to(_DEV, _F)
    if kind == "sites":
        x = _site_features(case["n"], theta)
        return sum(_forward(p, x[c:c + 200000]).sum(0) for c in range(0, len(x), 200000)).cpu().numpy()
    x, t = (torch.from_numpy(v).to(_DEV, _F) for v in _rows(case, seed))
    p.requires_grad_(True)
    loss = ((_forward(p, x) - t) ** 2).sum() / case["rows"]
    loss.backward()
    return {"loss": float(loss), "grad": p.grad.cpu().numpy()}
