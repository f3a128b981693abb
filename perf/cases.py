"""Performance cases: the work that users of this library have it do.

Kinds of case:

* ``run``: a resident handle advances ``steps`` time steps, then the program
  reads the PGV map and the free-surface snapshot (what a time loop that
  writes a snapshot every IT_SKIP steps does);
* ``batch``: several scenarios of uneven size advance together as one batch
  with CUDA graphs, then each one's maps are read (what the serving loop does
  between two rounds);
* ``propagate``: the one-call drop-in, host buffers in and out, from the model
  upload to the seismograms;
* ``stage``: one RK4 time step on device buffers that the caller owns
  (four cgfdm_stage_noalloc calls), the form for hosts that cannot allocate.

Models have the shape that the reference's own generators give them: layered
media with a perturbation per cell, a terrain-following grid (``grid`` =
"terrain": stretched in z only, as every grid built from a run directory is)
or, through the array interface, a grid that is skewed in x and y as well
("skewed").  Every state starts from a smooth random wavefield that fills the
volume, so that each point, slab and layer has work that shows in the result.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "cgfdm-fp16_sve_sme_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import cgfdm  # noqa: E402
from cgfdm import _lib  # noqa: E402

DH, DT = 100.0, 0.008
PREC = {"fp32": cgfdm.FP32, "fp16": cgfdm.FP16, "bf16": cgfdm.BF16, "fp64": cgfdm.FP64}
STORE = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16,
         "fp64": torch.float64}
BYTES = {"fp32": 4, "fp16": 2, "bf16": 2, "fp64": 8}
# velocity, stress and buoyancy scaling of the 16-bit storage forms (macro.h:65-73)
CV, CS, CRHO = 5.0e3, 1.0e-6, 1.0e6
# MacCormack signs of step it, (it mod 8); all flip after every RK stage (propagate.cpp:105-117)
FB = [(-1, -1, -1), (1, 1, -1), (1, 1, 1), (-1, -1, 1), (-1, 1, -1), (1, -1, -1), (1, -1, 1),
      (-1, 1, 1)]
LAYERS = [(2000.0, 2600.0, 4500.0, 2300.0), (8000.0, 3350.0, 5800.0, 2600.0),
          (1e9, 3750.0, 6500.0, 2800.0)]  # bottom depth, Vs, Vp, density
NT_MAX = 400000  # a handle's configured number of steps: a long run's


def _case(name, kind, precision, nx, ny, nz, npml, steps, source="point", graph=False,
          grid="terrain", members=1):
    c = {"kind": kind, "precision": precision, "nx": nx, "ny": ny, "nz": nz, "npml": npml,
         "steps": steps, "source": source, "graph": graph, "grid": grid, "members": members}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the default params.json: a first try, a regression run; launch latency counts
        _case("run fp32 64x64x48 graph", "run", "fp32", 64, 64, 48, 12, 50, graph=True),
        # the half-space accuracy configuration
        _case("run fp32 161x161x101", "run", "fp32", 161, 161, 101, 12, 20),
        # the Gaussian-hill configuration: 20-cell PML, a middle-sized production run
        _case("run fp32 401x401x201", "run", "fp32", 401, 401, 201, 20, 4),
        # the same in scaled FP16 storage
        _case("run fp16 401x401x201", "run", "fp16", 401, 401, 201, 20, 4),
        # the PerformanceTest shape with its finite fault, FP32 and FP16
        _case("run fp32 601x601x401 fault", "run", "fp32", 601, 601, 401, 12, 2, source="fault"),
        _case("run fp16 601x601x401 fault", "run", "fp16", 601, 601, 401, 12, 2, source="fault"),
        # BF16 storage on a ragged middle-sized grid
        _case("run bf16 225x187x133", "run", "bf16", 225, 187, 133, 12, 10, graph=True),
        # the FP64 accuracy reference
        _case("run fp64 121x121x101", "run", "fp64", 121, 121, 101, 12, 8),
        # the serving loop's batch of small and middle-sized scenarios
        _case("batch fp32 4 scenarios", "batch", "fp32", 181, 161, 121, 12, 10, graph=True,
              members=4),
        # the one-call drop-in with host buffers and seismograms
        _case("propagate fp32 161x161x101", "propagate", "fp32", 161, 161, 101, 12, 120),
        # one step on caller-owned device buffers: a skewed grid in FP32, FP16 storage
        _case("stage fp32 225x225x201 skewed", "stage", "fp32", 225, 225, 201, 12, 1,
              grid="skewed"),
        _case("stage fp16 201x161x121", "stage", "fp16", 201, 161, 121, 12, 1),
    ]


def draw(rng):
    kind = rng.choice(["run"] * 6 + ["batch", "propagate", "stage", "stage"])
    precision = rng.choice(["fp32"] * 5 + ["fp16"] * 3 + ["bf16"] * 2 +
                           (["fp64"] if kind == "run" else []))
    most = {"run": 100e6, "batch": 8e6, "propagate": 4e6, "stage": 30e6}[kind]
    if precision == "fp64":
        most = 4e6
    size = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    while True:
        nx, ny, nz = size(48, 601), size(48, 601), size(40, 401)
        if nx * ny * nz <= most:
            break
    npml = rng.choice([0, 6, 8, 10, 12, 12, 12, 16, 20])
    if kind == "propagate":
        steps = min(rng.randint(60, 120), int(250e6 / (nx * ny * nz)))
    elif kind == "stage":
        steps = 1
    else:
        steps = max(2, min(50, int(30e6 / (nx * ny * nz))))
    return _case(None, kind, precision, nx, ny, nz, npml, steps,
                 source=rng.choice(["point", "point", "fault"]),
                 graph=kind == "batch" or (kind == "run" and rng.random() < 0.5),
                 grid=rng.choice(["terrain", "terrain", "terrain", "skewed"]),
                 members=rng.randint(2, 5) if kind == "batch" else 1)


# ---- inputs ---------------------------------------------------------------

def _members(case):
    """The grids of a case: the case's own, and for a batch smaller ones beside it."""
    for q in range(case["members"]):
        f = 1.0 - 0.5 * q / max(1, case["members"])
        yield dict(case, nx=max(40, int(case["nx"] * f)), ny=max(40, int(case["ny"] * f) | 1),
                   nz=max(36, int(case["nz"] * f)))


def _scales(case):
    return (CV, CS, CRHO) if case["precision"] in ("fp16", "bf16") else (1.0, 1.0, 1.0)


def _model(c, seed):
    """cjm [13, nz_, ny_, nx_] and rdz [2, ny_, nx_, 9], float32 on the GPU."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)
    r = np.random.default_rng(seed)
    nx_, ny_, nz_ = c["nx"] + 6, c["ny"] + 6, c["nz"] + 6
    f64 = dict(dtype=torch.float64, device=dev)
    x = ((torch.arange(nx_, **f64) - 3) * DH)[None, :]
    y = ((torch.arange(ny_, **f64) - 3) * DH)[:, None]
    s = ((torch.arange(nz_, **f64) - 3) / (c["nz"] - 1))[:, None, None]
    depth = (c["nz"] - 1) * DH
    h = torch.zeros(ny_, nx_, **f64)
    hx, hy = torch.zeros_like(h), torch.zeros_like(h)
    for _ in range(4):  # hills
        x0, y0 = r.uniform(0, c["nx"] * DH), r.uniform(0, c["ny"] * DH)
        w = r.uniform(0.15, 0.4) * min(c["nx"], c["ny"]) * DH
        e = r.uniform(-0.2, 0.5) * min(0.25 * depth, 0.15 * w, 1500.0) * torch.exp(
            -((x - x0) ** 2 + (y - y0) ** 2) / w ** 2)
        h, hx, hy = h + e, hx - 2 * (x - x0) / w ** 2 * e, hy - 2 * (y - y0) / w ** 2 * e
    # lateral skew x = X + f(Y), y = Y + g(X): x_eta = fy, y_xi = gx
    k = 0.05 if c["grid"] == "skewed" else 0.0
    fy = k * torch.sin(2 * math.pi * y / (c["ny"] * DH) + r.uniform(0, 6)) * torch.ones_like(x)
    gx = k * torch.sin(2 * math.pi * x / (c["nx"] * DH) + r.uniform(0, 6)) * torch.ones_like(y)
    dj = 1.0 - fy * gx
    xi, et = (1 / dj, -fy / dj), (-gx / dj, 1 / dj)  # (xi_x, xi_y), (eta_x, eta_y); no z part
    a = ((h + depth) / depth)  # z_zeta, the same at every height
    cv, cs, crho = _scales(c)
    cjm = torch.empty(13, nz_, ny_, nx_, dtype=torch.float32, device=dev)
    one = torch.ones(nz_, 1, 1, **f64)
    for q, v in enumerate([xi[0], xi[1], torch.zeros_like(h), et[0], et[1], torch.zeros_like(h)]):
        cjm[q] = v + 0.0  # +0: no negative zeros
    zx, zy = hx * xi[0] + hy * et[0], hx * xi[1] + hy * et[1]
    cjm[6] = (-s * (zx / a)).float()
    cjm[7] = (-s * (zy / a)).float()
    cjm[8] = ((1 / a) * one).float()
    cjm[9] = ((a * dj) * one).float()
    below = (h + depth) * (1 - s)  # depth under the surface
    below = below.float()
    med = [torch.full_like(below, LAYERS[-1][q]) for q in (1, 2, 3)]
    for q in (0, 1, 2):
        for lay in reversed(LAYERS[:-1]):
            med[q][below < lay[0]] = lay[1 + q]
    del below
    for q in (0, 1):
        med[q] *= 1 + 0.1 * (torch.rand(nz_, ny_, nx_, generator=g, device=dev) - 0.5)
    rho = med[2] * (cs / cv)
    cjm[10] = rho * med[0] ** 2
    cjm[11] = rho * (med[1] ** 2 - 2 * med[0] ** 2)
    cjm[12] = 1.0 / rho / crho
    # V_zeta at the free surface from V_xi and V_eta: no traction on zeta = const
    top = cjm[:, nz_ - 4].double()
    mu, lam = top[10], top[11]

    def traction(b):  # sum over directions of A(zeta, b) V_b, as matrices [ny_, nx_, 3, 3]
        z = torch.stack([top[6], top[7], top[8]], -1)
        m = lam[..., None, None] * z[..., :, None] * b[..., None, :]
        m = m + mu[..., None, None] * b[..., :, None] * z[..., None, :]
        return m + (mu * (z * b).sum(-1))[..., None, None] * torch.eye(3, **f64)

    dz = torch.linalg.inv(traction(torch.stack([top[6], top[7], top[8]], -1)))
    rdz = torch.stack([-(dz @ traction(torch.stack([top[3 * d], top[3 * d + 1], top[3 * d + 2]], -1)))
                       for d in (0, 1)])
    return cjm, rdz.reshape(2, ny_, nx_, 9).float().contiguous()


def _state(c, seed):
    """A smooth random wavefield [9, nz_, ny_, nx_] in storage units, zero in the halo."""
    dev = torch.device("cuda")
    r = np.random.default_rng(seed + 77)
    cv, cs, _ = _scales(c)
    W = torch.zeros(9, c["nz"] + 6, c["ny"] + 6, c["nx"] + 6, dtype=torch.float32, device=dev)
    for v in range(9):
        amp = 0.1 * cv if v < 3 else 1e6 * cs
        for _ in range(2):
            p = []
            for n in (c["nz"], c["ny"], c["nx"]):
                k = 2 * math.pi / r.uniform(12.0, 40.0)
                p.append(torch.sin(k * torch.arange(n, device=dev, dtype=torch.float32) +
                                   r.uniform(0, 6)))
            W[v, 3:-3, 3:-3, 3:-3] += (0.5 * amp * r.uniform(0.5, 1.5)) * (
                p[0][:, None, None] * p[1][None, :, None] * p[2][None, None, :])
    return W


def _source(c, seed):
    """The point source's padded cell, or the finite fault's cells and moment rates."""
    r = np.random.default_rng(seed + 78)
    if c["source"] == "point":
        return {"point": tuple(int(n * r.uniform(0.35, 0.65)) + 3 for n in
                               (c["nx"], c["ny"], c["nz"])), "rickerfc": float(r.uniform(0.5, 3.0))}
    # a plane of cells across the middle; scaled moment rates, smooth in time
    n0, n1 = min(80, c["nx"] // 2), min(40, c["nz"] // 3)
    i = c["nx"] // 4 + np.arange(n0) + 3
    k = c["nz"] // 3 + np.arange(n1) + 3
    K, I = np.meshgrid(k, i, indexing="ij")
    J = c["ny"] // 2 + (K - k[0]) // 2 + 3
    idx = (I + J * (c["nx"] + 6) + K * (c["nx"] + 6) * (c["ny"] + 6)).reshape(-1)
    nt = 64
    shape = np.sin(np.linspace(0, math.pi, nt))[:, None, None] ** 2
    rate = (shape * r.normal(size=(1, idx.size, 6)) * 1e6 * _scales(c)[1]).astype(np.float32)
    return {"src_index": idx.astype(np.int64), "moment_rate": rate, "src_nt": nt, "src_dt": 1.0}


def _stations(c, seed):
    """25 surface stations on a lattice and 25 borehole ones, padded indices."""
    r = np.random.default_rng(seed + 79)
    n = (c["nx"], c["ny"], c["nz"])
    top = [[n[0] * (a + 1) // 6 + 3, n[1] * (b + 1) // 6 + 3, n[2] + 2] for a in range(5)
           for b in range(5)]
    deep = [[int(r.integers(0, m)) + 3 for m in n] for _ in range(25)]
    return np.array(top + deep, np.int32)


def _host(t):
    """A host copy in page-locked memory, where such a program keeps its model."""
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out.numpy()


def _desc(c, nt):
    return cgfdm.make_desc(c["nx"], c["ny"], c["nz"], c["npml"], DH, DT, nt, PREC[c["precision"]])


def _handle(c, seed):
    sim = cgfdm.Simulation(_desc(c, NT_MAX))
    cjm, rdz = _model(c, seed)
    sim.set_model(_host(cjm), _host(rdz))
    del cjm, rdz
    sim.set_state(0, W=_host(_state(c, seed)))
    src = _source(c, seed)
    if c["source"] == "point":
        sim.set_point_source(*src["point"], src["rickerfc"])
    else:
        sim.set_fault_source(src["src_index"], src["moment_rate"], src["src_nt"], src["src_dt"])
    return sim


def _slab_sizes(c):
    n, p = (c["nx"], c["ny"], c["nz"]), c["npml"]
    return [9 * n[0] * n[1] * n[2] // n[ax] * p for ax in (0, 1, 2, 0, 1)]


def prepare(case, seed):
    if case["kind"] in ("run", "batch"):
        sims = [_handle(c, seed + 1000 * q) for q, c in enumerate(_members(case))]
        if case["kind"] == "batch":
            return {"kind": "batch", "steps": case["steps"], "sims": sims,
                    "batch": cgfdm.Batch(sims, graph=case["graph"])}
        if case["graph"]:
            sims[0].set_graph(True)
        return {"kind": "run", "steps": case["steps"], "sim": sims[0]}
    cjm, rdz = _model(case, seed)
    if case["kind"] == "propagate":
        return {"kind": "propagate", "desc": _desc(case, case["steps"]), "cjm": _host(cjm),
                "rdz": _host(rdz), "stations": _stations(case, seed),
                "source": _source(case, seed)}
    # the caller's own device buffers
    L = cgfdm.hbm_layout(case["nx"], case["ny"], case["nz"], BYTES[case["precision"]])
    dev, dtype = torch.device("cuda"), STORE[case["precision"]]

    def buffer(nf, src=None):
        b = torch.zeros(nf * L["fs"], dtype=dtype, device=dev)
        v = b.view(nf, L["fs"])[:, :L["nz_"] * L["plane"]].view(
            nf, L["nz_"], L["ny_"], L["px"])[..., L["xoff"]:L["xoff"] + L["nx_"]]
        if src is not None:
            v.copy_(src)
        return b, v

    A, X, Y, T, B = buffer(9, _state(case, seed)), buffer(9), buffer(9), buffer(9), buffer(9)
    C = buffer(13, cjm)
    naux = max(64, sum(_slab_sizes(case)))
    aux = [torch.zeros(naux, device=dev) for _ in range(5)]  # step start, X, Y, t, step end
    if case["npml"]:  # a step in mid-run: auxiliaries of the size of the fields they damp
        g = torch.Generator(device=dev).manual_seed(seed + 80)
        cv, cs, _ = _scales(case)
        o = 0
        for n9 in _slab_sizes(case):
            part = aux[0][o:o + n9].view(9, -1)
            part.copy_(torch.randn(part.shape, generator=g, device=dev))
            part[:3] *= 0.02 * cv
            part[3:] *= 2e5 * cs
            o += n9
    stages, ins, outs = [], (A, X, Y, X), (X, Y, X, B)
    aux_in, aux_out = (0, 1, 2, 1), (1, 2, 1, 4)
    for irk in range(4):
        s = -1 if irk % 2 else 1
        stages.append(_lib.StageBuffers(
            nx=case["nx"], ny=case["ny"], nz=case["nz"], npml=case["npml"], dh=DH, dt=DT,
            precision=PREC[case["precision"]], irk=irk, fb1=s * FB[0][0], fb2=s * FB[0][1],
            fb3=s * FB[0][2], w_in=ins[irk][0].data_ptr(), w_out=outs[irk][0].data_ptr(),
            w_m=A[0].data_ptr(), t=T[0].data_ptr(), cjm=C[0].data_ptr(), rdz=rdz.data_ptr(),
            aux_in=aux[aux_in[irk]].data_ptr(), aux_out=aux[aux_out[irk]].data_ptr(),
            aux_m=aux[0].data_ptr(), aux_t=aux[3].data_ptr()))
    return {"kind": "stage", "stages": stages, "wave": B[1], "aux": aux[4],
            "keep": (A, X, Y, T, C, rdz, aux)}


def _maps(sim):
    return {"pgv": sim.pgv(), "free_surface": sim.free_surface()}


def run(state):
    if state["kind"] == "run":
        state["sim"].run(state["steps"])
        return _maps(state["sim"])
    if state["kind"] == "batch":
        state["batch"].run(state["steps"])
        state["batch"].synchronize()
        return [_maps(s) for s in state["sims"]]
    if state["kind"] == "propagate":
        sta, pgv, fs = cgfdm.propagate(state["desc"], state["cjm"], state["rdz"],
                                       stations=state["stations"], **state["source"])
        return {"stations": sta, "pgv": pgv, "free_surface": fs}
    stream = torch.cuda.current_stream().cuda_stream
    for b in state["stages"]:
        cgfdm.stage_noalloc(b, stream, wait=False)
    return {"wave": state["wave"], "aux": state["aux"]}


# ---- what a pass cannot do without ----------------------------------------

def work(case):
    """Per step and stage: the wavefield that it differentiates and the 12
    coefficients read, its result written; the combination of the four stages
    reads the step's start in the three later ones and two stage results once.
    Per slab point: the same for the 9 auxiliaries, in 32 bits (64 in FP64)."""
    b = BYTES[case["precision"]]
    r = 8 if case["precision"] == "fp64" else 4
    total = flops = 0.0
    for c in _members(case):
        pts = c["nx"] * c["ny"] * c["nz"]
        slab = sum(_slab_sizes(c)) // 9
        fields = 4 * (9 + 12 + 9) + 3 * 9 + 2 * 9
        total += case["steps"] * (pts * fields * b + slab * 9 * r * (4 * 2 + 3 + 2))
        flops += case["steps"] * 4 * (pts * (27 * 9 + 90 + 36) + slab * 9 * 10)
        if case["kind"] == "propagate":  # the model comes from the host
            total += 4.0 * 13 * (c["nx"] + 6) * (c["ny"] + 6) * (c["nz"] + 6)
    return {"bytes": float(total), "flops": float(flops)}


def tolerance(case):
    """About four times the distance from ``exact`` that the listed and some
    drawn cases showed (FP32 4e-7 and below, FP16 2e-3 over 50 steps, BF16
    9e-3 over 10); FP64 from the order of its sums alone."""
    return {"fp32": {"rel": 2e-6, "max": 1e-4}, "fp16": {"rel": 8e-3, "max": 0.1},
            "bf16": {"rel": 3e-2, "max": 0.5}, "fp64": {"rel": 1e-12, "max": 1e-11}}[case["precision"]]


# ---- the same in 64 bits --------------------------------------------------

_f = lambda v: float(np.float32(v))
A5 = [_f(v) for v in (-0.30874, -0.6326, 1.2330, -0.3334, 0.04168)]  # taps -1 .. +3
C3 = [_f(v) for v in (-1.16666667, 1.33333333, -0.16666667)]
B_RK, A_RK = [_f(v) for v in (0.16666667, 0.33333333, 0.33333333, 0.16666667)], (0.5, 0.5, 1.0)


def _profiles(c):
    """alpha, beta, d of each axis over the padded grid (init_pml_para.cpp:99-234)."""
    out = []
    for ax, n in enumerate((c["nx"], c["ny"], c["nz"])):
        p = c["npml"]
        l = np.full(n + 6, -1.0)
        if p:
            length = DH * (p - 1)
            i = np.arange(3, n + 3)
            l[3:3 + p] = (3 + p - 1 - i[:p]) * DH
            if ax != 2:
                l[n + 3 - p:n + 3] = (i[n - p:] - (n + 3 - p)) * DH
            big = _f(10.0 ** (-(math.log10(p) - 1) / math.log10(2.0) - 3))
            q = np.where(l < 0, 0.0, l / length)
            on = l >= 0
            beta = 1 + 2 * q ** 2
            d0 = -3 * 6000.0 / (2 * length) * math.log(big)
            out.append([np.where(on, 3.141592657 * 0.5 * (1 - q), 0.0), 1 / beta, d0 * q ** 2 / beta])
        else:
            out.append([np.zeros(n + 6), np.ones(n + 6), np.zeros(n + 6)])
    return [[torch.from_numpy(v).to("cuda") for v in p] for p in out]


class _Exact:
    """The time step in 64 bits, plain torch, whole arrays at a time."""

    def __init__(self, c, cjm, rdz, W):
        store = STORE[c["precision"]]
        self.c, self.W = c, W.to(store).double()
        self.C = cjm.to(store).double()
        self.rdz = rdz.double().reshape(2, c["ny"] + 6, c["nx"] + 6, 3, 3)
        self.bu = _scales(c)[2]
        self.prof = _profiles(c)
        self.rDH, self.dt = _f(1.0 / DH), _f(DT)
        n, p = [c["nx"], c["ny"], c["nz"]], c["npml"]
        self.slabs, self.aux = [], []
        for s, ax in enumerate((0, 1, 2, 0, 1) if p else ()):
            box = [[3, n[q] + 3] for q in range(3)]
            box[ax] = [3, 3 + p] if s < 3 else [n[ax] + 3 - p, n[ax] + 3]
            self.slabs.append((ax, box))
            self.aux.append(torch.zeros([9] + [b - a for a, b in box[::-1]], dtype=torch.float64,
                                        device="cuda"))

    def cut(self, f, box, ax=None, o=0):
        b = [[x, y] for x, y in box]
        if ax is not None:
            b[ax] = [b[ax][0] + o, b[ax][1] + o]
        return f[..., b[2][0]:b[2][1], b[1][0]:b[1][1], b[0][0]:b[0][1]]

    def diff(self, f, box, ax, fb):
        r = A5[1] * self.cut(f, box)
        for k, o in ((0, -1), (2, 1), (3, 2), (4, 3)):
            r += A5[k] * self.cut(f, box, ax, fb * o)
        return r.mul_(fb * self.rDH)

    def axis(self, v, ax, box):
        shape = [1, 1, 1]
        shape[2 - ax] = -1
        return v[box[ax][0]:box[ax][1]].reshape(shape)

    def velocity(self, m, L, box, h):
        """Adds one direction's part from the stress derivatives L(q), q = 3..8."""
        b = self.cut(self.C[12], box) * self.bu
        for row, (x, y, z) in enumerate(((3, 6, 7), (6, 4, 8), (7, 8, 5))):
            h[row] += (m[0] * L(x) + m[1] * L(y) + m[2] * L(z)) * b

    def stress(self, m, dv, box, h):
        """Adds one direction's part from the velocity derivatives dv."""
        mu, lam = self.cut(self.C[10], box), self.cut(self.C[11], box)
        div = (m[0] * dv[0] + m[1] * dv[1] + m[2] * dv[2]) * lam
        for q in range(3):
            h[3 + q] += div + 2 * mu * (m[q] * dv[q])
        h[6] += (m[1] * dv[0] + m[0] * dv[1]) * mu
        h[7] += (m[2] * dv[0] + m[0] * dv[2]) * mu
        h[8] += (m[2] * dv[1] + m[1] * dv[2]) * mu

    def surface(self, k, fb, h):
        """The increment of one of the three top layers (freeSurface.cpp:104-256)."""
        c, W, C = self.c, self.W, self.C
        ktop = c["nz"] + 2
        box = [[3, c["nx"] + 3], [3, c["ny"] + 3], [k, k + 1]]
        bx, by = (self.axis(self.prof[a][1], a, box) for a in (0, 1))
        full = [[0, c["nx"] + 6], [0, c["ny"] + 6]]

        def rows(d, kk):  # J (d . T) on the whole padded plane kk
            m = [C[3 * d + q, kk:kk + 1] * C[9, kk:kk + 1] for q in range(3)]
            t = W[:, kk:kk + 1]
            return torch.stack([m[0] * t[3] + m[1] * t[6] + m[2] * t[7],
                                m[0] * t[6] + m[1] * t[4] + m[2] * t[8],
                                m[0] * t[7] + m[1] * t[8] + m[2] * t[5]])

        flat = [full[0], full[1], [0, 1]]
        inner = [[3, c["nx"] + 3], [3, c["ny"] + 3], [0, 1]]
        total = self.diff(rows(0, k), inner, 0, fb[0]) * bx
        total += self.diff(rows(1, k), inner, 1, fb[1]) * by
        ks = ktop - k + 3
        for q, o in ((0, -1), (1, 0), (2, 1), (3, 2), (4, 3)):
            e = 3 + fb[2] * o
            if e != ks:  # the surface row is zero, rows above it mirror those below
                src = e if e < ks else 2 * ks - e
                total += (1 if e < ks else -1) * fb[2] * self.rDH * A5[q] * self.cut(
                    rows(2, k + src - 3), inner)
        h[:3] = total * (self.cut(C[12], box) * self.bu / self.cut(C[9], box))
        dx = [self.diff(W[v], box, 0, fb[0]) * bx for v in range(3)]
        dy = [self.diff(W[v], box, 1, fb[1]) * by for v in range(3)]
        if k == ktop:
            M = self.rdz[:, 3:-3, 3:-3]
            dz = [sum(M[0, :, :, q, v] * dx[v] + M[1, :, :, q, v] * dy[v] for v in range(3))
                  for q in range(3)]
        else:
            taps = [(-1.0, 0), (1.0, 1)] if k == ktop - 1 else list(zip(C3, range(3)))
            dz = [sum(w * self.cut(W[v], box, 2, fb[2] * o) for w, o in taps) * (fb[2] * self.rDH)
                  for v in range(3)]
        h[3:] = 0
        for d, dv in ((0, dx), (1, dy), (2, dz)):
            self.stress([self.cut(C[3 * d + q], box) for q in range(3)], dv, box, h)

    def stage(self, irk, fb):
        c, W = self.c, self.W
        n = [c["nx"], c["ny"], c["nz"]]
        ktop = n[2] + 2
        box = [[3, m + 3] for m in n]
        h = torch.zeros([9] + n[::-1], dtype=torch.float64, device="cuda")
        for d in range(3):
            m = [self.cut(self.C[3 * d + q], box) for q in range(3)]
            beta = self.axis(self.prof[d][1], d, box)
            dv = [self.diff(W[v], box, d, fb[d]) * beta for v in range(3)]
            self.stress(m, dv, box, h)
            del dv
            self.velocity(m, lambda q: self.diff(W[q], box, d, fb[d]) * beta, box, h)
        for k in range(ktop - 2, ktop + 1):
            self.surface(k, fb, h[:, k - 3:k - 2])
        h *= self.dt
        new = []
        for (ax, sb), a in zip(self.slabs, self.aux):
            al, be, dd = (self.axis(v, ax, sb) for v in self.prof[ax])
            t = torch.zeros_like(a)
            m = [self.cut(self.C[3 * ax + q], sb) for q in range(3)]
            self.stress(m, [self.diff(W[v], sb, ax, fb[ax]) * dd for v in range(3)], sb, t)
            self.velocity(m, lambda q: self.diff(W[q], sb, ax, fb[ax]) * dd, sb, t)
            if ax != 2:  # the surface-gradient part (pml_freeSurface.cpp)
                tb = [sb[0], sb[1], [ktop, ktop + 1]]
                M = self.rdz[ax, tb[1][0]:tb[1][1], tb[0][0]:tb[0][1]]
                dl = self.axis(self.prof[ax][2], ax, tb)
                vd = [self.diff(W[v], tb, ax, fb[ax]) * dl for v in range(3)]
                vz = [sum(M[:, :, q, v] * vd[v] for v in range(3)) for q in range(3)]
                self.stress([self.cut(self.C[6 + q], tb) for q in range(3)], vz, tb, t[:, -1:])
            i0 = [slice(x - 3, y - 3) for x, y in sb[::-1]]
            h[(slice(None), *i0)] -= be * a * self.dt
            new.append((t - (dd + al) * a) * self.dt)
        if irk == 0:
            self.m = (self.cut(W, box).clone(), [a.clone() for a in self.aux])
            self.t = (self.m[0].clone(), [a.clone() for a in self.aux])
        for dst, m, t, hh in zip([self.cut(W, box)] + self.aux, [self.m[0]] + self.m[1],
                                 [self.t[0]] + self.t[1], [h] + new):
            t += B_RK[irk] * hh
            dst.copy_(t if irk == 3 else m + A_RK[irk] * hh)

    def step(self, it, src):
        c, W = self.c, self.W
        cv, cs, _ = _scales(c)
        if src and "point" in src:
            sx, sy, sz = src["point"]
            f = src["rickerfc"]
            r = 3.141592657 * f * (it * self.dt - 1.2 / f)
            s = r * (2 * r * r - 3) * math.exp(-r * r) * 2 * 3.141592657 * f * 1e16
            g = torch.arange(-3, 4, dtype=torch.float64, device="cuda")
            g = torch.exp(-(g / 1.5) ** 2) / (1.5 * 1.772453850905516)
            amp = g[:, None, None] * g[None, :, None] * g[None, None, :] / 0.998125703461425
            W[3:6, sz - 3:sz + 4, sy - 3:sy + 4, sx - 3:sx + 4] += (
                -s * amp / (self.C[9, sz, sy, sx] * DH ** 3) * cs * self.dt)
        elif src:
            q = it * self.dt / src["src_dt"]
            k = int(q)
            if k + 1 < src["src_nt"]:
                m = torch.from_numpy(src["moment_rate"]).to("cuda").double()
                at = torch.from_numpy(src["src_index"]).to("cuda")
                W.view(9, -1)[3:, at] -= ((m[k + 1] - m[k]) * (q - k) + m[k]).T * self.dt
        for irk in range(4):
            s = -1 if irk % 2 else 1
            self.stage(irk, [s * f for f in FB[it % 8]])
        v = W[:3, c["nz"] + 2, 3:-3, 3:-3] / cv
        vh = (v[0] ** 2 + v[1] ** 2).sqrt()
        vv = (v ** 2).sum(0).sqrt()
        now = torch.stack([vh, vv], -1)
        self.pgv = now if not hasattr(self, "pgv") else torch.maximum(self.pgv, now)
        self.fs = v


def exact(case, seed):
    if case["kind"] in ("run", "batch"):
        out = []
        for q, c in enumerate(_members(case)):
            e = _Exact(c, *_model(c, seed + 1000 * q), _state(c, seed + 1000 * q))
            src = _source(c, seed + 1000 * q)
            for it in range(case["steps"]):
                e.step(it, src)
            out.append({"pgv": e.pgv.cpu().numpy(), "free_surface": e.fs.cpu().numpy()})
        return out if case["kind"] == "batch" else out[0]
    if case["kind"] == "propagate":
        z = torch.zeros(9, case["nz"] + 6, case["ny"] + 6, case["nx"] + 6, device="cuda")
        e = _Exact(case, *_model(case, seed), z)
        src = _source(case, seed)
        at = torch.from_numpy(_stations(case, seed).astype(np.int64)).to("cuda")
        cv, cs, _ = _scales(case)
        unit = torch.tensor([1 / cv] * 3 + [1 / cs] * 6, dtype=torch.float64, device="cuda")
        rows = []
        for it in range(case["steps"]):
            e.step(it, src)
            rows.append((e.W[:, at[:, 2], at[:, 1], at[:, 0]].T * unit))
        return {"stations": torch.stack(rows, 1).cpu().numpy(), "pgv": e.pgv.cpu().numpy(),
                "free_surface": e.fs.cpu().numpy()}
    s = prepare(case, seed)  # the same inputs, in the storage type
    start = s["keep"][6][0].double()
    e = _Exact(case, *_model(case, seed), _state(case, seed))
    o = 0
    for q, a in enumerate(e.aux):
        e.aux[q] = start[o:o + a.numel()].view(a.shape).clone()
        o += a.numel()
    for irk in range(4):
        e.stage(irk, [(-1 if irk % 2 else 1) * f for f in FB[0]])
    aux = torch.cat([a.reshape(-1) for a in e.aux]) if e.aux else start
    return {"wave": e.W, "aux": aux}
