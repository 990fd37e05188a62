"""Workloads of the Hamiltonian build for timing and for comparing outputs.

Every case goes through the package's public classes as a program does: the handle
(tables, device buffers, network weights) is made once by prepare(), and run() is one
pass from reset to the matrix, the energies, the thermal sums or the gradient.

  build     HBuild: reset, accumulate (device Sobol points, or host normals as with -r),
            read-out of Mout.  FP64 forms return float64; the split forms return the
            float32 values that the sM_*.h5 dump stores.
  batch     Batch: several clusters in one accumulate, every cluster's Mout read.
  energies  PES.energies / energies_grad of a batch of host geometries.
  scp1      SCP1Average.sums: one thermal average of the effective-Hessian iteration.
  network   MLP.loss_and_grad: one training batch of the learned surrogate.

exact() restates each of them in 64 bits with torch; the published Sobol direction
numbers and Partridge-Schwenke coefficients are read as data from their tables."""
import math
import os
import re

import numpy as np
import torch

import scp3_b200
from scp3_b200 import constants as C
from scp3_b200 import inputs, modes, surrogate

HERE = os.path.dirname(os.path.abspath(scp3_b200.__file__))
CLUSTERS = {2: "cluster_2_800", 3: "cluster_3_700", 4: "cluster_4_900", 5: "cluster_5_1401", 6: "cluster_6_100",
            7: "cluster_7_500", 8: "cluster_8_0"}


def build(name, input, pes, precision, estimator, n2, n3, n, nm=0, points="sobol", read="device"):
    """nm: the nm highest-frequency modes (0: all); n2, n3: modes with doubles, triples."""
    return {"name": name, "kind": "build", "input": input, "pes": pes, "precision": precision, "estimator": estimator,
            "nm": nm, "n2": n2, "n3": n3, "n": n, "points": points, "read": read}


def listed():
    return [
        # the dimer with the reference's read-out period (E0_sd.dat every 2^14 points), plain form
        build("dimer_fp64", "dimer_qtip4pf", "qtip4pf", "fp64", "direct", 12, 0, 1 << 14, read="host"),
        # a trimer with a few triples on the command line's default (gradient) estimator, same period
        build("trimer_gradient_fp64", CLUSTERS[3], "ttm3f", "fp64", "gradient", 21, 5, 1 << 14, read="host"),
        # the hexamer prism, doubles basis: one dump period (2^17 points) in the package's default precision
        build("hexamer_fp64", "prism_qtip4pf", "qtip4pf", "fp64", "direct", 48, 0, 1 << 17),
        # the same basis on the default estimator, default precision
        build("hexamer_gradient_fp64", "prism_qtip4pf", "qtip4pf", "fp64", "gradient", 48, 0, 1 << 16),
        # the benchmark's step: 2^20 points in the split form
        build("hexamer_bf16x3", "prism_qtip4pf", "qtip4pf", "bf16x3", "direct", 48, 0, 1 << 20),
        # the default estimator in the split form
        build("hexamer_gradient_bf16x3", "prism_qtip4pf", "qtip4pf", "bf16x3", "gradient", 48, 0, 1 << 18),
        # scrambled normals from the host (-r), a ragged count, Mout back on the host
        build("hexamer_normals_bf16x3", "prism_qtip4pf", "qtip4pf", "bf16x3", "direct", 48, 0, 300007,
              points="normals32", read="host"),
        # TTM3-F with triples over half the modes
        build("hexamer_triples_ttm3f", "prism_ttm3f", "ttm3f", "bf16x3", "direct", 48, 24, 1 << 16),
        # sixteen random clusters of two to eight waters built together
        {"name": "batch_16_clusters", "kind": "batch", "count": 16, "precision": "bf16x3", "n": 1 << 18},
        # a finite-difference Hessian's gradients: 2 x 54 geometries
        {"name": "hessian_gradients_ttm3f", "kind": "energies", "input": "prism_ttm3f", "pes": "ttm3f", "grad": True, "n": 108},
        # one thermal average of the hexamer's effective-Hessian iteration
        {"name": "scp1_hexamer", "kind": "scp1", "input": "prism_qtip4pf", "pes": "qtip4pf", "n": 1 << 18},
        # one training batch of the surrogate
        {"name": "surrogate_batch", "kind": "network", "n_in": 48, "hidden": 256, "n": 1 << 14},
    ]


def log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["build"] * 6 + ["batch", "energies", "scp1", "network"])
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(2, 16), "precision": rng.choice(["bf16x3", "f16x3"]), "n": log_int(rng, 1 << 12, 1 << 18)}
    if kind == "network":
        return {"kind": kind, "n_in": 9 * rng.randint(2, 8) - 6, "hidden": 64 * rng.randint(1, 4), "n": 64 * log_int(rng, 16, 256)}
    pes, nw = rng.choice(["qtip4pf", "qtip4pf", "ttm3f"]), rng.randint(2, 8)
    if kind == "energies":
        return {"kind": kind, "input": CLUSTERS[nw], "pes": pes, "grad": rng.random() < 0.5, "n": log_int(rng, 1, 20000)}
    if kind == "scp1":
        return {"kind": kind, "input": CLUSTERS[nw], "pes": pes, "n": log_int(rng, 1 << 12, 1 << (18 if pes == "qtip4pf" else 16))}
    estimator = rng.choice(["direct", "gradient"])
    precision = rng.choice(["fp64", "fp64", "bf16x3", "bf16x3", "bf16x3_pes64"] + (["f16x3"] if estimator == "direct" else []))
    nm = rng.randint(6, 9 * nw - 6)
    n2 = rng.randint(nm // 2, nm)
    n3 = rng.randint(2, min(n2, 14)) if rng.random() < 0.4 else 0
    n = log_int(rng, 1000, 1 << (17 if precision == "fp64" else 19))
    c = build("", CLUSTERS[nw], pes, precision, estimator, n2, n3, n, nm=nm,
              points=rng.choice(["sobol", "sobol", "normals32", "normals64"]), read=rng.choice(["device", "host"]))
    del c["name"]
    most = 1.5e11 if precision == "fp64" else 4e11
    c["n"] = min(n, 1 << 16 if pes == "ttm3f" else n, max(1000, int(most / (work(c)["flops"] / n))))
    return c


# ---------------------------------------------------------------- inputs

_loaded = {}


def molecule(name):
    if name not in _loaded:
        _loaded[name] = inputs.load(name, build_if_missing=False)
    return _loaded[name]


def selected(case):
    nm0 = molecule(case["input"])[3].size
    nm = case["nm"] or nm0
    return np.arange(nm0 - nm, nm0, dtype=np.int32)


def first_index(seed):
    return (1 << 20) + 7919 * (seed % 1000003)


def host_normals(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype = torch.float32 if case["points"] == "normals32" else torch.float64
    y = torch.randn(case["n"], molecule(case["input"])[3].size, generator=g, device="cuda", dtype=dtype)
    return torch.empty(y.shape, dtype=dtype, pin_memory=True).copy_(y)


def thermal_geometries(case, seed):
    """Angstrom geometries of the harmonic ground state around the input's minimum."""
    _, x0, MUa, omega = molecule(case["input"])
    g = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.randn(case["n"], omega.size, generator=g, device="cuda", dtype=torch.float64).cpu().numpy() / math.sqrt(2)
    return C.bohr * (x0 + q @ MUa.T)


def harmonic_density(case):
    """(q, d, isqrtM_U) of the SCP1 iteration at the input's Hessian, kT = 0."""
    species, mass, x0, H = modes.read_input(os.path.join(inputs.DATA, case["input"] + ".dat"))
    _, mass, x0, H = modes.ohhohh(mass, x0, H)
    w2, U = np.linalg.eigh(H)
    omega = np.sqrt(np.abs(w2))
    d = np.where(omega < 50.0 / C.autocm, 0.0, 0.5 / np.maximum(omega, 1e-12))
    return x0, d, U / np.sqrt(mass)[:, None]


def network_data(case, seed):
    """Weights, normal coordinates and targets of one batch."""
    g = torch.Generator().manual_seed(seed)
    h, parts = case["hidden"], []
    for o, i in ((h, case["n_in"]), (h, h), (h, h), (1, h)):
        parts += [torch.randn(o * i, generator=g) / math.sqrt(i), 0.1 * torch.randn(o, generator=g)]
    q = torch.randn(case["n"], case["n_in"], generator=g) / math.sqrt(2)
    t = 0.3 * q.square().sum(1) / math.sqrt(case["n_in"]) + 0.1 * torch.randn(case["n"], generator=g)
    return torch.cat(parts).numpy(), q.numpy(), t.numpy()


def batch_members(case):
    if ("batch", case["count"]) not in _loaded:
        _loaded["batch", case["count"]] = inputs.batch_clusters(case["count"], build_if_missing=False)
    return _loaded["batch", case["count"]]


class State:
    pass


def prepare(case, seed):
    s, kind = State(), case["kind"]
    s.case, s.index0 = case, first_index(seed)
    if kind == "build":
        nw, x0, MUa, omega = molecule(case["input"])
        s.hb = scp3_b200.HBuild(nw, x0, MUa, omega, modes=selected(case), n2=case["n2"], n3=case["n3"], pes=case["pes"],
                                precision=case["precision"], estimator=case["estimator"])
        if case["points"] != "sobol":
            s.keep = host_normals(case, seed)
            s.normals = s.keep.numpy()
        if case["read"] == "device":
            s.M = torch.empty(s.hb.nb, s.hb.nb, dtype=torch.float64, device="cuda")
            s.stream = torch.cuda.ExternalStream(s.hb.stream)
    elif kind == "batch":
        s.batch = scp3_b200.Batch(batch_members(case), precision=case["precision"])
    elif kind == "energies":
        s.pes, s.crd = scp3_b200.PESFromString(case["pes"]), thermal_geometries(case, seed)
    elif kind == "scp1":
        s.density = harmonic_density(case)
        s.average = scp3_b200.SCP1Average(case["pes"], s.density[0].size // 9)
    else:
        p, s.q, s.t = network_data(case, seed)
        s.net = surrogate.MLP(case["n_in"], hidden=case["hidden"], max_batch=case["n"])
        s.net.set_params(p)
    return s


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "build":
        s.hb.reset()
        if case["points"] == "sobol":
            s.hb.accumulate(s.index0, case["n"])
        else:
            s.hb.accumulate_normals(s.normals)
        if case["read"] == "host":
            M = s.hb.read(1)
            return M if case["precision"] == "fp64" else M.astype(np.float32)
        s.hb.read_dev(s.M.data_ptr(), s.hb.nb, 1)
        torch.cuda.current_stream().wait_stream(s.stream)
        return s.M if case["precision"] == "fp64" else s.M.float()
    if kind == "batch":
        s.batch.reset()
        s.batch.accumulate(s.index0, case["n"])
        return [s.batch.read(k, 1).astype(np.float32) for k in range(s.batch.ncl)]
    if kind == "energies":
        return s.pes.energies_grad(s.crd) if case["grad"] else s.pes.energies(s.crd)
    if kind == "scp1":
        return s.average.sums(*s.density, s.index0, 0, case["n"])
    return s.net.loss_and_grad(s.q, s.t)


# ---------------------------------------------------------------- what a pass cannot do without


def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "build":
        nm0 = molecule(case["input"])[3].size
        nb, size = modes.basis_size(case["nm"] or nm0, case["n2"], case["n3"]), 8 if case["precision"] == "fp64" else 4
        pairs = nb * (nb + 1)
        if case["estimator"] == "gradient":   # one product per term: a (mode, function) row against every function
            rows = 1 + sum(len(f) for f in functions(case["nm"] or nm0, case["n2"], case["n3"]))
            pairs = 2 * rows * nb
        host = {"sobol": 0, "normals32": 4, "normals64": 8}[case["points"]] * n * nm0
        return {"bytes": size * nb * nb + host, "flops": n * (pairs + 2.0 * nm0 * (nm0 + 6) + potential_flops(case, nm0))}
    if kind == "batch":
        flops = nbytes = 0.0
        for c in batch_members(case):
            nb, nm0 = modes.basis_size(c["n2"], c["n2"], 0), c["omega"].size
            flops += n * (nb * (nb + 1) + 2.0 * nm0 * (nm0 + 6) + potential_flops({"pes": "qtip4pf"}, nm0))
            nbytes += 4.0 * nb * nb
        return {"bytes": nbytes, "flops": flops}
    if kind == "network":
        h, k = case["hidden"], case["n_in"]
        weights = k * h + 2 * h * h + h
        return {"bytes": 4.0 * (n * (k + 1) + 2 * (weights + 3 * h + 1)), "flops": n * (6.0 * weights - 2.0 * k * h)}
    dim = molecule(case["input"])[1].size
    if kind == "energies":
        return {"bytes": 8.0 * n * (dim * (2 if case["grad"] else 1) + 1), "flops": float(n * potential_flops(case, dim - 6))}
    return {"bytes": 8.0 * (2 * dim * dim + 3 * dim + 1), "flops": n * (4.0 * dim * dim + 2 * potential_flops(case, dim - 6))}


def potential_flops(case, nm0):
    """Ten site pairs for every pair of waters, about 12 operations each; TTM3-F also has its
    245-term monomer polynomials, three times the work per pair and the dipoles of a 3 nw system."""
    nw = (nm0 + 6) // 9
    return 60 * nw * (nw - 1) + 60 * nw if case["pes"] == "qtip4pf" else 180 * nw * (nw - 1) + 2000 * nw + 20 * 18 * nw * nw


# ---------------------------------------------------------------- the same in 64 bits


def table(file, name):
    """A numeric table of one of the package's data headers, flat."""
    with open(os.path.join(HERE, "csrc", file)) as f:
        body = re.search(r"\b%s(?:\[\d+\])+ = \{(.*?)\};" % name, f.read(), re.S).group(1)
    return np.array([float(x) for x in re.findall(r"[-+.\deE]+", body)])


def cuda(x):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device="cuda")


def sobol_normals(dims, index0, n):
    """Bratley-Fox direction numbers, Gray-code points, Beasley-Springer-Moro normals."""
    poly = table("sobol_dirnum.h", "scp3_sobol_poly").astype(int)
    init = table("sobol_dirnum.h", "scp3_sobol_vinit").astype(int).reshape(-1, 13)
    idx = torch.arange(index0, index0 + n, device="cuda", dtype=torch.int64)
    gray = idx ^ (idx >> 1)
    u = torch.empty(n, dims, dtype=torch.float64, device="cuda")
    for d in range(dims):
        m = int(poly[d]).bit_length() - 1
        v = [1] * 62 if d == 0 else [int(x) for x in init[d][:m]]
        while len(v) < 62:
            j, w = len(v), v[len(v) - m]
            for k in range(m):
                if poly[d] >> (m - 1 - k) & 1:
                    w ^= (2 << k) * v[j - k - 1]
            v.append(w)
        x = torch.zeros_like(gray)
        for b in range((index0 + n).bit_length()):
            x ^= (gray >> b & 1) * (v[b] << (61 - b))
        u[:, d] = x.double() * 2.0 ** -62
    y = u - 0.5
    r = y * y
    mid = y * (((-25.44106049637 * r + 41.39119773534) * r + -18.61500062529) * r + 2.50662823884) / (
        (((3.13082909833 * r + -21.06224101826) * r + 23.08336743743) * r + -8.47351093090) * r + 1)
    r = torch.log(-torch.log(torch.where(y > 0, 1 - u, u)))
    t = torch.zeros_like(r)
    for c in (0.0000003960315187, 0.0000002888167364, 0.0000321767881768, 0.0003951896511919, 0.0038405729373609,
              0.0276438810333863, 0.1607979714918209, 0.9761690190917186, 0.3374754822726147):
        t = t * r + c
    return torch.where(y.abs() < 0.42, mid, torch.where(y < 0, -t, t))


CHARGE = 18.22234397655801030455


def geometry(x):
    """x: n x nw x 3 x 3 (O H H)."""
    a, b = x[:, :, 1] - x[:, :, 0], x[:, :, 2] - x[:, :, 0]
    return a, b, a.norm(dim=-1), b.norm(dim=-1)


def distances(a, b):
    return (a[:, :, None, :] - b[:, None, :, :]).square().sum(-1)


def qtip4pf(crd):
    x = crd.reshape(crd.shape[0], -1, 3, 3)
    nw = x.shape[1]
    a, b, ra, rb = geometry(x)
    e = 0.0
    for r in (ra, rb):
        z = 2.287 * (r - 0.9419)
        e = e + (z * z * (1.0 - z * (1.0 - (7.0 / 12.0) * z)) * 116.09).sum(1)
    th = torch.acos((a * b).sum(-1) / ra / rb) - 107.4 * math.pi / 180
    e = e + 0.5 * 87.85 * th.square().sum(1)
    if nw == 1:
        return e
    gamma = 0.73612
    m = gamma * x[:, :, 0] + 0.5 * (1 - gamma) * (x[:, :, 1] + x[:, :, 2])
    qm = -1.1128 * CHARGE
    site, q = torch.stack([x[:, :, 1], x[:, :, 2], m], 2).reshape(x.shape[0], -1, 3), cuda([-qm / 2, -qm / 2, qm] * nw)
    i, j = np.triu_indices(3 * nw, 1)
    keep = i // 3 != j // 3
    i, j = i[keep], j[keep]
    e = e + (q[i] * q[j] / (site[:, i] - site[:, j]).norm(dim=-1)).sum(1)
    i, j = np.triu_indices(nw, 1)
    s6 = (3.1589 ** 2 / (x[:, i, 0] - x[:, j, 0]).square().sum(-1)) ** 3
    return e + (4 * 0.1852 * s6 * (s6 - 1.0)).sum(1)


def ps_tables():
    t = {k: table("ps_coeffs.h", "scp3_ps_" + k) for k in ("c5zA", "cbasis", "ccore", "crest", "coefD", "idx1", "idx2",
                                                           "idx3", "idxD0", "idxD1", "idxD2")}
    c = 0.999677885 * t["c5zA"] + 0.15860145369897 * t["cbasis"] + -1.6351695982132 * t["ccore"] + t["crest"]
    ints = {k: torch.as_tensor(v.astype(np.int64) - 1, device="cuda").clamp(min=0) for k, v in t.items() if k.startswith("idx")}
    return cuda(c), cuda(t["coefD"]), ints


def ps_monomer(x, tab):
    """Partridge-Schwenke energy and the TTM3-F dipole-surface charges of every water."""
    c, cd, ix = tab
    a, b, r1, r2 = geometry(x)
    rhh = (x[:, :, 1] - x[:, :, 2]).norm(dim=-1)
    cos = (a * b).sum(-1) / (r1 * r2)
    e1, e2 = (torch.exp(-2.587949757553683 * (r - 0.9519607159623009)) for r in (r1, r2))
    e = 0.999677885 * 42290.92019288289 * (e1 * (e1 - 2) + e2 * (e2 - 2))
    e = e + 0.999677885 * 16.94879431193463 * math.exp(12.66426998162947) * torch.exp(-12.66426998162947 * rhh)
    powers = [torch.stack([z ** k for k in range(15)], -1) for z in ((r1 - 0.958649) / 0.958649, (r2 - 0.958649) / 0.958649,
                                                                     cos + .24780227221366464506)]
    f = lambda p, k: powers[p][..., ix[k][1:]]   # noqa: E731
    g = torch.exp(-2.0 * ((r1 - 0.958649) ** 2 + (r2 - 0.958649) ** 2))
    poly = ((f(0, "idx1") * f(1, "idx2") + f(0, "idx2") * f(1, "idx1")) * f(2, "idx3")) @ c[1:]
    e = (e + 2 * c[0] + g * poly + 0.44739574026257) * 0.00285914375100642899
    g = torch.exp(-((r1 - 0.958649) ** 2 + (r2 - 0.958649) ** 2))
    p1 = (f(0, "idxD0") * f(1, "idxD1") * f(2, "idxD2")) @ cd[1:]
    p2 = (f(0, "idxD1") * f(1, "idxD0") * f(2, "idxD2")) @ cd[1:]
    pc = 0.2999 * (r1 ** -0.6932 + r2 ** -0.6932) * (1.0099 - 0.1801 * cos + 0.0892 * 0.5 * (3 * cos * cos - 1)) * 0.529177249
    ang = torch.atan2(torch.linalg.cross(a, b).norm(dim=-1) / (r1 * r2), cos) - 1.82400520401572996557
    h1 = cd[0] + p1 * g + pc + 0.5 * (r1 - 0.9578) + 0.012 * ang
    h2 = cd[0] + p2 * g + pc + 0.5 * (r2 - 0.9578) + 0.012 * ang
    return e.sum(1), h1, h2


def ttm3f(crd, tab):
    x = crd.reshape(crd.shape[0], -1, 3, 3)
    n, nw = x.shape[:2]
    e, h1, h2 = ps_monomer(x, tab)
    gamma = 0.46
    m = (1 - gamma) * x[:, :, 0] + 0.5 * gamma * (x[:, :, 1] + x[:, :, 2])
    t = 0.5 * gamma / (1 - gamma)
    q = CHARGE * torch.stack([h1 + t * (h1 + h2), h2 + t * (h1 + h2), -(h1 + h2) / (1 - gamma)], 2).reshape(n, -1)
    site = torch.stack([x[:, :, 1], x[:, :, 2], m], 2).reshape(n, -1, 3)
    if nw == 1:
        return e
    pol = np.tile([0.496, 0.496, 0.837], nw)
    i, j = np.triu_indices(3 * nw, 1)
    keep = i // 3 != j // 3
    i, j = i[keep], j[keep]
    AA, aX = cuda((pol[i] * pol[j]) ** (1 / 6)), 0.175
    R = site[:, i] - site[:, j]
    r = R.norm(dim=-1)
    w = aX * (r / AA) ** 3
    ex = torch.exp(-w)
    gq = torch.special.gammaincc(torch.full_like(w, 2 / 3), w) * 1.354117939426400
    ts0 = (1 - ex + aX ** (1 / 3) * r / AA * gq) / r
    ts1 = (1 - ex) / r ** 3
    e = e + (q[:, i] * q[:, j] * ts0).sum(1)
    field = torch.zeros_like(site)
    field = field.index_add(1, torch.as_tensor(i, device="cuda"), (q[:, j] * ts1)[..., None] * R)
    field = field.index_add(1, torch.as_tensor(j, device="cuda"), -(q[:, i] * ts1)[..., None] * R)[:, 2::3].reshape(n, -1)
    mm = (i % 3 == 2) & (j % 3 == 2)
    ts2 = (ts1[:, mm] - ex[:, mm] * aX / AA[mm] ** 3) / r[:, mm] ** 2
    eye = torch.eye(3 * nw, device="cuda", dtype=torch.float64)
    D = 3 * ts2[..., None, None] * R[:, mm, :, None] * R[:, mm, None, :] - ts1[:, mm, None, None] * eye[:3, :3]
    T = torch.zeros(n, nw * nw, 3, 3, dtype=torch.float64, device="cuda")
    wi, wj = torch.as_tensor(i[mm] // 3, device="cuda"), torch.as_tensor(j[mm] // 3, device="cuda")
    T = T.index_add(1, wi * nw + wj, D).index_add(1, wj * nw + wi, D)
    T = T.reshape(n, nw, nw, 3, 3).permute(0, 1, 3, 2, 4).reshape(n, 3 * nw, 3 * nw)
    dip = torch.linalg.solve(eye / 1.444 - T, field)
    e = e - 0.5 * (dip * field).sum(1)
    i, j = np.triu_indices(nw, 1)
    r = (x[:, i, 0] - x[:, j, 0]).norm(dim=-1)
    return e + (-0.72298855E+03 / r ** 6 + 0.10211829E+06 * torch.exp(-0.37170376E+01 * r)).sum(1)


def potential(pes, crd, grad):
    """(kcal/mol, kcal/mol/A) of Angstrom geometries, a few thousand at a time."""
    tab, E, G = ps_tables() if pes == "ttm3f" else None, [], []
    for x in crd.split(4096):
        x = x.detach().requires_grad_(grad)
        e = ttm3f(x, tab) if pes == "ttm3f" else qtip4pf(x)
        if grad:
            G.append(torch.autograd.grad(e.sum(), x)[0])
        E.append(e.detach())
    return torch.cat(E), torch.cat(G) if grad else None


def functions(nm, n2, n3):
    """Basis functions as lists of (mode, level)."""
    f = [[]] + [[(m, 1)] for m in range(nm)] + [[(m, 2)] for m in range(n2)]
    f += [[(m, 1), (k, 1)] for m in range(n2) for k in range(m + 1, n2)] + [[(m, 3)] for m in range(n3)]
    for m in range(n3):
        for k in range(m + 1, n3):
            f += [[(m, 2), (k, 1)], [(m, 1), (k, 2)]]
    return f + [[(m, 1), (k, 1), (l, 1)] for m in range(n3) for k in range(m + 1, n3) for l in range(k + 1, n3)]


def hermite(q):
    """Levels 0..3 of every mode: h, h(0), dh/dq, d = (h - h(0)) / q, dd/dq, each n x 4 x modes."""
    o, z, s2, s3 = torch.ones_like(q), torch.zeros_like(q), math.sqrt(2), math.sqrt(3)
    rows = [(o, s2 * q, (2 * q * q - 1) / s2, (2 * q * q - 3) * q / s3), (o, z, o / -s2, z),
            (z, s2 * o, 2 * s2 * q, (6 * q * q - 3) / s3), (z, s2 * o, s2 * q, (2 * q * q - 3) / s3), (z, z, s2 * o, 4 * q / s3)]
    return [torch.stack(r, 1) for r in rows]


def factor_columns(fs, nm, without=-1):
    """Column of each of a function's three factors in the n x (4 nm) table of levels."""
    idx = np.zeros((3, len(fs)), dtype=np.int64)
    for k, f in enumerate(fs):
        for p, (m, l) in enumerate(f):
            if m != without:
                idx[p, k] = l * nm + m
    return torch.as_tensor(idx, device="cuda")


def product(h, idx):
    h = h.reshape(h.shape[0], -1)
    return h[:, idx[0]] * h[:, idx[1]] * h[:, idx[2]]


def direct_sum(q, v, nm, n2, n3):
    idx, M = factor_columns(functions(nm, n2, n3), nm), 0.0
    for qs, vs in zip(q.split(8192), v.split(8192)):
        phi = product(hermite(qs)[0], idx)
        M = M + phi.T @ (phi * vs[:, None])
    return M


def stein_sum(q, v, vq, nm, n2, n3):
    """The gradient estimator: every mode either function excites gives one term, averaged."""
    fs = functions(nm, n2, n3)
    nb, M, count = len(fs), torch.zeros(len(fs), len(fs), dtype=torch.float64, device="cuda"), torch.zeros(len(fs), len(fs), device="cuda")
    level = np.zeros((nm, nb), dtype=np.int64)
    for k, f in enumerate(fs):
        for m, l in f:
            level[m, k] = l
    step = max(512, (1 << 23) // nb)
    for m in range(nm):
        idx, has = factor_columns(fs, nm, m), np.flatnonzero(level[m])
        cols = {b: torch.as_tensor(np.flatnonzero(level[m] == b), device="cuda") for b in range(4) if (level[m] == b).any()}
        rows = torch.as_tensor(has, device="cuda")
        on = torch.as_tensor(level[m] > 0, device="cuda")
        count += (on[:, None] | on[None, :]).float()
        for qs, vs, gs in zip(q.split(step), v.split(step), vq.split(step)):
            h, h0, dh, d, dd = hermite(qs)
            R = product(h, idx)
            h, h0, dh, d, dd = (t[:, :, m] for t in (h, h0, dh, d, dd))
            x = qs[:, m]
            for b, cb in cols.items():
                K = []
                for a in range(4):
                    u = h0[:, a] * h0[:, b] + 0.5 * (dd[:, a] * h[:, b] + d[:, a] * dh[:, b] + h0[:, a] * dd[:, b])
                    if a == b == 3:      # the reference's own formula for this element
                        u = (2 * x * x - 3) * (x * x - 3) / 6
                    K.append(u * vs + 0.5 * (d[:, a] * h[:, b] + h0[:, a] * d[:, b]) * gs[:, m])
                K = torch.stack(K, 1)[:, torch.as_tensor(level[m][has], device="cuda")]
                T = (R[:, rows] * K).T @ R[:, cb]
                M[rows[:, None], cb[None, :]] += T
                if b == 0:
                    M[cb[:, None], rows[None, :]] += T.T
    M[0, 0] = v.sum() * 1.0
    count[0, 0] = 1
    return M / count


def exact_build(pes, input, sel, n2, n3, normals, gradient):
    _, x0, MUa, omega = molecule(input)
    MUa, w, sel = cuda(MUa), cuda(omega), torch.as_tensor(sel.astype(np.int64), device="cuda")
    q = normals.double() / math.sqrt(2)
    E, G = potential(pes, C.bohr * (cuda(x0) + q @ MUa.T), gradient)
    v = E / C.autokcalpmol - 0.5 * (q * w * q).sum(1)
    nm = sel.numel()
    if gradient:
        vq = (G * (C.bohr / C.autokcalpmol)) @ MUa - w * q
        M = stein_sum(q[:, sel], v, vq[:, sel], nm, n2, n3)
    else:
        M = direct_sum(q[:, sel], v, nm, n2, n3)
    ws = omega[sel.cpu().numpy()]
    diag = [0.5 * omega.sum() + sum(l * ws[m] for m, l in f) for f in functions(nm, n2, n3)]
    return M / q.shape[0] + torch.diag(cuda(diag))


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "build":
        nm0 = molecule(case["input"])[3].size
        y = sobol_normals(nm0, first_index(seed), n) if case["points"] == "sobol" else host_normals(case, seed).cuda()
        return exact_build(case["pes"], case["input"], selected(case), case["n2"], case["n3"], y, case["estimator"] == "gradient")
    if kind == "batch":
        return [exact_build("qtip4pf", c["name"], c["modes"], c["n2"], 0, sobol_normals(c["omega"].size, first_index(seed), n), False)
                for c in batch_members(case)]
    if kind == "energies":
        E, G = potential(case["pes"], cuda(thermal_geometries(case, seed)), case["grad"])
        return (E, G) if case["grad"] else E
    if kind == "scp1":
        x0, d, U = harmonic_density(case)
        dq = (sobol_normals(d.size, first_index(seed), n) * cuda(np.sqrt(d))) @ cuda(U).T
        E, G = potential(case["pes"], C.bohr * (cuda(x0) + dq), True)
        G = G * (C.bohr / C.autokcalpmol)
        return float(E.sum() / C.autokcalpmol), G.sum(0), G.T @ dq
    return exact_network(case, seed)


def exact_network(case, seed):
    """Float64 with the network's stored types: BF16 weights and layer inputs."""
    p, q, t = network_data(case, seed)
    h, at, W, B = case["hidden"], 0, [], []
    p = cuda(p)
    for o, i in ((h, case["n_in"]), (h, h), (h, h), (1, h)):
        W.append(p[at:at + o * i].reshape(o, i))
        B.append(p[at + o * i:at + o * i + o])
        at += o * i + o
    bf = lambda x: x.float().bfloat16().double()   # noqa: E731
    x, Z, X = cuda(q), [], []
    for l in range(3):
        X.append(bf(x))
        Z.append(X[l] @ bf(W[l]).T + B[l])
        x = torch.nn.functional.gelu(Z[l])
    x = bf(x)
    off = x @ W[3][0] + B[3][0] - cuda(t)
    dy = 2 * off / case["n"]
    gW, gB = [None] * 3 + [(dy @ x)[None]], [None] * 3 + [dy.sum()[None]]
    dh = dy[:, None] * W[3]
    for l in (2, 1, 0):
        z = Z[l]
        dz = dh * (0.5 * (1 + torch.erf(z / math.sqrt(2))) + z * torch.exp(-0.5 * z * z) / math.sqrt(2 * math.pi))
        gW[l], gB[l] = dz.T @ X[l], dz.sum(0)
        dh = dz @ W[l]
    return float(off.square().mean()), torch.cat([v.reshape(-1) for l in range(4) for v in (gW[l], gB[l])])
