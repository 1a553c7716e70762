"""Performance cases of the RTM engine: the calls that a migration makes, through psdm_b200.rtm.

A marine migration prepares each shot's traces (band-pass filter, resampling to the propagation
step, cuts and taper), migrates the shot in a window around its streamer (forward pass keeping the
source wavefield, backward pass with the imaging condition) and stacks the window images.  The
cases cover these calls from test-sized windows to the largest window one GPU keeps resident, in
the precisions, statement orders and forms that the engine offers.

`exact` restates the arithmetic in 64-bit torch, independent of the engine: the 6th-order
acoustic stencil with C-PML strips and corners, the free-surface rules, the snapshots, the imaging
condition, the Butterworth filter and the trace conditioning.
"""
import math

import numpy as np
import torch

from psdm_b200 import rtm
from psdm_b200._lib import Conditioning

ACC = 3
PRECISIONS = {"fp32": 0, "fp16": 1, "bf16": 2}


def listed():
    """Sizes are those of the benchmark configurations (200 x 600 cells, 120 channels, 3000 steps;
    1200 x 4000 cells, 480 channels, 8000 steps; 3000 x 16000 cells, 960 channels) and of the
    tests; records are shortened where a full one would take seconds."""
    shallow = dict(ny=200, nrec=120, rec_step=1.25, near=10, pad=51, dd=10.0, dt=1e-3, dpml=40, fs=1, disk=0)
    deep = dict(ny=1200, nrec=480, rec_step=2.0, near=16, pad=81, dd=6.25, dt=5e-4, dpml=50, fs=1, disk=0)
    salt = dict(ny=3000, nrec=960, rec_step=2.5, near=20, pad=101, dd=5.0, dt=4e-4, dpml=50, fs=1, disk=0)
    plain = dict(precision="fp32", ks=1, taper=0)
    half = dict(precision="fp16", ks=4, taper=0)
    return [
        # The smallest shot, host arrays in and out: what a test or a parameter trial runs;
        # launches, synchronisations and host work count.
        dict(name="shot_tiny", kind="shot_host", ny=36, nrec=24, rec_step=2.0, near=4, pad=7, dd=10.0, dt=1e-3,
             nt=260, dpml=8, fs=0, disk=0, **plain),
        # One shot of a shallow line: a small grid and thousands of dependent steps.
        dict(name="shot_shallow", kind="shot", nt=3000, **shallow, **plain),
        # One shot of the benchmark's deep-water line, every snapshot kept: the headline workload.
        dict(name="shot_deep", kind="shot", nt=8000, **deep, **plain),
        # Odd sizes, disk statement order, no free surface, tapered record, host arrays.
        dict(name="shot_ragged", kind="shot_host", ny=331, nrec=77, rec_step=3.0, near=7, pad=43, dd=7.5, dt=8e-4,
             nt=1501, dpml=25, fs=0, disk=1, precision="fp32", ks=1, taper=120),
        # Checkpoints in place of snapshots, the form for shots whose snapshots do not fit.
        dict(name="shot_checkpoint", kind="shot", nt=2000, checkpoint=100, **deep, **plain),
        # The largest window: 16-bit snapshots every 4 steps, wavefield larger than L2.
        dict(name="shot_salt_fp16", kind="shot", nt=2400, **salt, **half),
        # Forward modelling of one gather, the traces returned to the host.
        dict(name="model_deep", kind="model", nt=4000, **deep, **plain),
        # The two solver calls as a Fortran driver binds them, the wavefield through host memory.
        dict(name="solvers_shallow", kind="solvers", nt=600, **shallow, **plain),
        # A rank's shots in one call: small windows in 32 bits.
        dict(name="batch_shallow", kind="batch", nt=3000, shots=4, uneven=0.0, **shallow, **plain),
        # A rank's shots in one call: deep windows, 16-bit snapshots.
        dict(name="batch_deep_fp16", kind="batch", nt=1200, shots=8, uneven=0.0, **deep, **half),
        # Shots whose windows and records differ, as feathering and mutes make them.
        dict(name="batch_uneven_bf16", kind="batch", ny=500, nrec=330, rec_step=2.0, near=16, pad=81, dd=6.25,
             dt=6e-4, nt=1800, dpml=40, fs=1, disk=0, shots=6, uneven=0.11, precision="bf16", ks=4, taper=0),
        # Preparation of one shot's traces: band-pass, resampling, cuts and taper.
        dict(name="prepare_traces", kind="traces", nrec=480, nt_data=2004, dt_data=2e-3, nt=8000, dt=5e-4, band=1),
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["shot", "shot", "shot", "shot_host", "shot_host", "model", "solvers", "batch", "batch", "traces"])
    if kind == "traces":
        nt_data = int(log(500, 3000))
        up = rng.choice([1, 2, 4])
        return dict(kind=kind, nrec=int(log(48, 480)), nt_data=nt_data, dt_data=up * 5e-4, nt=up * nt_data, dt=5e-4,
                    band=rng.randint(0, 1))
    c = dict(kind=kind, ny=int(log(36, 1200)), nrec=0, rec_step=rng.choice([1.0, 1.25, 2.0, 2.5, 3.0]), near=rng.randint(4, 20),
             pad=0, dd=rng.choice([5.0, 6.25, 10.0]), dt=0.0, nt=0, dpml=rng.choice([8, 20, 25, 30, 40, 50]),
             fs=rng.randint(0, 1), disk=rng.randint(0, 1), precision="fp32", ks=1, taper=0)
    c["dt"] = round(0.09e-3 * c["dd"], 7)
    c["pad"] = max(7, c["dpml"] // 2 + rng.randint(4, 30))  # the window is at least as wide as a C-PML strip
    c["nrec"] = max(12, int((log(80, 1136) - 2 * c["pad"] - c["near"]) / c["rec_step"]))
    cells = (c["ny"] + 2 * c["dpml"]) * (c["nrec"] * c["rec_step"] + 2 * c["pad"] + 2 * c["dpml"])
    most = 8000
    if kind == "solvers":  # the wavefield goes through host memory
        c["ny"] = min(c["ny"], 400)
        most = max(100, int(3e7 / cells))
    elif kind == "batch":
        c.update(shots=rng.randint(2, 8), uneven=rng.choice([0.0, 0.05, 0.1]), precision=rng.choice(["fp32", "fp16", "bf16"]))
        most = 3000
    elif kind != "model":
        c["precision"] = rng.choice(["fp32", "fp32", "fp32", "fp16", "bf16"])
        c["taper"] = rng.choice([0, 0, 100])
        if kind == "shot" and c["precision"] == "fp32" and rng.random() < 0.2:
            c["checkpoint"] = rng.randint(50, 150)
    if c["precision"] != "fp32":
        c["ks"] = rng.choice([2, 4])
    most = min(most, int(1.2e10 / cells / c.get("shots", 1)))
    c["nt"] = max(150, int(log(200, max(201, most))))
    return c


# ---- inputs ---------------------------------------------------------------------------------------

def device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def shots_of(case):
    """Channels and record length of each shot of a case."""
    u = case.get("uneven", 0.0)
    return [(max(12, int(case["nrec"] * (1.0 - u * i))), max(150, int(case["nt"] * (1.0 - 0.7 * u * i))))
            for i in range(case.get("shots", 1))]


def ricker(t, f0):
    a = (math.pi * f0 * t) ** 2
    return (1.0 - 2.0 * a) * torch.exp(-a)


def gather(nrec, nt, dt, offsets, f0, g, dev):
    """Reflections of a layered sea floor under low band-limited noise, (nrec, nt) float32."""
    t = torch.arange(nt, device=dev, dtype=torch.float32) * dt
    out = 0.02 * torch.randn((nrec, nt), device=dev, generator=g)
    out = torch.nn.functional.avg_pool1d(out[:, None], 5, 1, 2)[:, 0]
    r = torch.rand(12, generator=g, device=dev).tolist()
    for k in range(6):
        t0 = (0.15 + 0.8 * r[k]) * nt * dt
        v = 1500.0 + 1800.0 * r[6 + k]
        th = torch.sqrt(t0 * t0 + (offsets / v) ** 2)
        out += (1.0 - 0.13 * k) * (-1) ** k * ricker(t[None] - th[:, None], f0)
    return out


def velocity(nx, ny, g, dev):
    """Water over layers whose velocity grows with depth, the sea floor with relief; (nx, ny) float32."""
    r = torch.rand(5, generator=g, device=dev).tolist()
    x = torch.linspace(0, 1, nx, device=dev)[:, None]
    z = torch.linspace(0, 1, ny, device=dev)[None]
    sea = 0.18 + 0.04 * torch.sin(2 * math.pi * (x * (0.6 + r[0]) + r[1])) + 0.02 * torch.sin(2 * math.pi * (x * 3.1 + r[2]))
    v = 1700.0 + 2300.0 * (z - sea) / (1.0 - sea) * (1.0 + 0.05 * torch.sin(7.0 * x + 11.0 * z + 6 * r[3]))
    v = v + 120.0 * torch.floor(6.0 * (z + 0.03 * torch.sin(5.0 * x + r[4])))
    return torch.where(z < sea, torch.full_like(v, 1500.0), v.clamp(1550.0, 4400.0)).contiguous()


def make_shot(case, nrec, nt, g, dev):
    """Geometry (1-based model coordinates), model window, source and conditioned traces of one shot."""
    dd, dt = case["dd"], case["dt"]
    steps = np.floor(np.arange(nrec) * case["rec_step"]).astype(np.int32)
    span = int(steps[-1]) + case["near"]
    shift = int(torch.randint(0, 64, (1,), generator=g, device=dev).item())
    nx = span + 2 * case["pad"] + 96
    sx = case["pad"] + span + 8 + shift
    zs, zr = (2, 2) if case["ny"] < 100 else (2, 3)
    rx = (sx - case["near"] - steps).astype(np.int32)
    rz = np.full(nrec, zr, np.int32)
    space = (case["pad"] - 1) * dd
    nx_w, x_i, _ = rtm.dynamic_window(sx, rx, dd, nx, space)
    f0 = 0.06 * 1500.0 / dd * 1.5
    taper = case.get("taper", 0)
    nt_taper = nt + (taper // 2 if taper else 0)
    off = torch.from_numpy((sx - rx).astype(np.float32)).to(dev) * dd
    data = gather(nrec, nt_taper, dt, off, f0, g, dev)
    data[:, nt:] = 0.0
    t = torch.arange(nt, device=dev, dtype=torch.float32) * dt
    return dict(sx=sx, sz=zs, rx=rx, rz=rz, nx=nx, nx_w=nx_w, x_i=x_i, space=space, nt=nt, nt_taper=nt_taper,
                src=ricker(t - 1.2 / f0, f0).contiguous(), data=data.contiguous(), vp=velocity(nx_w, case["ny"], g, dev))


def make_traces(case, g, dev):
    nrec, n = case["nrec"], case["nt_data"]
    off = torch.arange(nrec, device=dev, dtype=torch.float32) * 12.5 + 100.0
    raw = gather(nrec, n, case["dt_data"], off, 25.0, g, dev)
    raw[nrec // 3] = 0.0  # a dead channel
    r = torch.rand(nrec, generator=g, device=dev).cpu().numpy()
    nt = case["nt"]
    cut = (nt * (0.75 + 0.2 * r)).astype(np.int32)
    cut[-1] = int(0.95 * nt)  # the farthest channel's multiple comes last and sets the record's length
    sea = (nt * (0.05 + 0.1 * r)).astype(np.int32)
    n_taper, n_zeros = 100, 400
    nt2 = int(min(nt, cut.max()))
    return dict(raw=raw.contiguous(), cut=cut, sea=sea, lens=np.array([nt2, nt2 + n_zeros, n_taper, n_zeros], np.int32))


def inputs(case, seed):
    dev = device()
    g = torch.Generator(device=dev).manual_seed(int(seed) * 7919 + 13)
    if case["kind"] == "traces":
        return make_traces(case, g, dev)
    return [make_shot(case, n, nt, g, dev) for n, nt in shots_of(case)]


# ---- calls ----------------------------------------------------------------------------------------

_kept = {}


def engine(checkpoint):
    """The program's engine, on the program's stream (one more for the shots with checkpoints)."""
    if "stream" not in _kept:
        _kept["stream"] = torch.cuda.Stream()
    if checkpoint not in _kept:
        e = rtm.Engine(torch.cuda.current_device())
        e.set_stream(_kept["stream"].cuda_stream)
        if checkpoint:
            e.set_checkpointing(checkpoint)
        _kept[checkpoint] = e
    return _kept[checkpoint]


def prepare(case, seed):
    st = dict(case=case, engine=engine(case.get("checkpoint", 0)))
    if case["kind"] == "traces":
        t = inputs(case, seed)
        st.update(t, work=torch.empty_like(t["raw"]), cond=Conditioning(1, 1, 1, 0.05, 0.2),
                  out=torch.empty((case["nrec"], int(t["lens"][1])), device=device()))
    else:
        st["prm"] = rtm.Params(case["dpml"], case["fs"], 2 if case["disk"] else 1, PRECISIONS[case["precision"]])
        st["shots"] = inputs(case, seed)
        for s in st["shots"]:
            if case["kind"] in ("shot_host", "model", "solvers"):
                for k in ("src", "data", "vp"):
                    s[k] = s[k].cpu().numpy()
                if case["kind"] == "solvers":
                    s["adjoint"] = np.ascontiguousarray(s["data"][:, ::-1])
                    s["fields"] = np.zeros((s["nt"], s["nx_w"], case["ny"]), np.float32)
                    s["synth"] = np.zeros((s["rx"].size, s["nt"]), np.float32)
            else:
                s["image"] = torch.zeros((s["nx_w"], case["ny"]), device=device())
    torch.cuda.synchronize()
    return st


def run(st):
    case, e = st["case"], st["engine"]
    kind = case["kind"]
    if kind == "traces":
        with torch.cuda.stream(_kept["stream"]):
            st["work"].copy_(st["raw"])
            if case["band"]:
                e.freq_filter_device(st["work"].data_ptr(), case["nt_data"], case["dt_data"], case["nrec"], 3, 4.0, 60.0)
            e.condition_traces_device(st["cond"], case["nrec"], st["work"].data_ptr(), case["nt_data"], case["dt_data"],
                                      case["dt"], st["cut"], st["sea"], st["lens"], st["out"].data_ptr())
        return {"filtered": st["work"], "target": st["out"]}
    prm, s = st["prm"], st["shots"][0]
    dd, dt, ny, ks = case["dd"], case["dt"], case["ny"], case["ks"]
    taper = case["taper"]
    options = (1, taper, s["nt_taper"] - s["nt"]) if taper else (0, 1, 0)
    if kind == "shot":
        e.rtm_shot_device(prm, s["sx"], s["sz"], s["rx"], s["rz"], s["src"].data_ptr(), s["data"].data_ptr(), dd, dt, ny,
                          s["nx"], s["nx_w"], s["vp"].data_ptr(), s["space"], ks, s["nt"], s["nt"], s["nt_taper"],
                          *options, s["image"].data_ptr())
        return s["image"]
    if kind == "shot_host":
        return e.rtm_shot(prm, s["sx"], s["sz"], s["rx"], s["rz"], s["src"], s["data"], dd, dt, ny, s["nx"], s["nx_w"],
                          s["vp"], s["space"], ks, s["nt"], s["nt"], s["nt_taper"], *options)
    if kind == "model":
        return e.model_shot(prm, s["sx"], s["sz"], s["rx"], s["rz"], s["src"], dd, dt, ny, s["nx"], s["nx_w"], s["vp"],
                            s["space"], s["nt"])
    if kind == "solvers":
        nt = s["nt"]
        args = (prm, [s["sx"]], [s["sz"]], s["rx"], s["rz"])
        grid = (dd, dt, ny, s["nx"], s["nx_w"], s["vp"], s["space"], 1, nt, nt)
        e.dynamic_window_solver_forward_ram(*args, s["src"], *grid, Fields=s["fields"], Data_synth=s["synth"])
        image = np.zeros((s["nx_w"], ny), np.float32)
        e.dynamic_window_solver_backward_ram(*args, s["adjoint"], *grid, s["fields"], image)
        return {"fields": s["fields"], "traces": s["synth"], "image": image}
    shots = [dict(nxSou=h["sx"], nySou=h["sz"], nxRec=h["rx"], nyRec=h["rz"], nx_w=h["nx_w"], nt_prop2=h["nt"],
                  nt_taper=h["nt_taper"], d_Vp_w=h["vp"].data_ptr(), d_Data_target=h["data"].data_ptr(),
                  d_PSDM_w=h["image"].data_ptr()) for h in st["shots"]]
    longest = max(st["shots"], key=lambda h: h["nt"])
    nx = max(h["nx"] for h in st["shots"])
    e.rtm_batch_device(prm, shots, longest["src"].data_ptr(), dd, dt, ny, nx, s["space"], ks)
    return [h["image"] for h in st["shots"]]


def work(case):
    """Inputs read and outputs written once, the kept source wavefield written once and read once
    (it has to leave the chip), and the arithmetic of the cell updates: 29 operations a cell and
    step, 27 more for each C-PML direction, 3 for a snapshot and 4 for an imaging update."""
    if case["kind"] == "traces":
        n, m = case["nrec"] * case["nt_data"], case["nrec"] * case["nt"]
        fft = 4 * 2 * case["nt_data"] * math.log2(2 * case["nt_data"]) * case["nrec"] * 2.5 if case["band"] else 0.0
        return {"bytes": 4.0 * (2 * n + m), "flops": fft + 30.0 * m}
    total_b = total_f = 0.0
    dn, ny = case["dpml"] + 2 * ACC, case["ny"]
    for nrec, nt in shots_of(case):
        nx_w = int((nrec - 1) * case["rec_step"]) + case["near"] + 2 * case["pad"]
        cells = (ny + (1 if case["fs"] else 2) * dn) * (nx_w + 2 * dn)
        inner = ny * nx_w
        strips = 2 * dn * (ny + (1 if case["fs"] else 2) * dn) + (1 if case["fs"] else 2) * dn * (nx_w + 2 * dn)
        step = 29.0 * cells + 27.0 * strips
        passes = 1 if case["kind"] == "model" else 2
        if case.get("checkpoint"):
            passes += 1
        total_f += passes * nt * step
        total_b += 4.0 * (inner + nt)
        if case["kind"] == "model":
            total_b += 4.0 * nrec * nt
            continue
        total_b += 4.0 * (nrec * nt + inner)
        total_f += 7.0 * inner * nt / case["ks"]
        if case["kind"] == "solvers":
            total_b += 4.0 * nrec * nt
        if not case.get("checkpoint"):
            size = 4.0 if case["precision"] == "fp32" else 2.0
            total_b += 2 * size * inner * (nt // case["ks"])
    return {"bytes": total_b, "flops": total_f}


# ---- 64-bit restatement ---------------------------------------------------------------------------

D1 = (0.0, 3 / 4, -3 / 20, 1 / 60)
D2 = (-49 / 36, 3 / 2, -3 / 20, 1 / 90)


def difference(n, coef, sign, dev):
    """Rows of the 6th-order difference over n points; the first and last 3 rows repeat their neighbour's."""
    m = torch.zeros((n, n), dtype=torch.float64)
    for i in range(n):
        c = min(max(i, ACC), n - 1 - ACC)
        for k in range(4):
            m[i, c + k] += coef[k]
            m[i, c - k] += sign * coef[k]
    return m.to(dev)


class Solver64:
    """One propagation in 64 bits on the padded grid, arrays (x, z)."""

    def __init__(self, case, s, dev):
        self.case, self.dev = case, dev
        self.dd, self.dt = float(np.float32(case["dd"])), float(np.float32(case["dt"]))
        ny, nx, dp = case["ny"], s["nx_w"], case["dpml"]
        dn = dp + 2 * ACC
        self.dn, self.ny, self.nx = dn, ny, nx
        n_x, n_z = nx + 2 * dn, ny + 2 * dn
        self.d2x, self.d2z = difference(n_x, D2, 1, dev), difference(n_z, D2, 1, dev).T.contiguous()
        d1x, d1z = difference(n_x, D1, -1, dev), difference(n_z, D1, -1, dev).T.contiguous()
        self.d1x = [d1x[:dn].contiguous(), d1x[n_x - dn:].contiguous()]
        self.d1z = [d1z[:, :dn].contiguous(), d1z[:, n_z - dn:].contiguous()]
        self.local = difference(dn, D1, -1, dev)
        vp = torch.as_tensor(s["vp"]).to(dev).double()
        c = torch.nn.functional.pad(vp[None, None], (dn, dn, dn, dn), mode="replicate")[0, 0]
        if not case["disk"]:  # RAM solvers pad the top and bottom strips of the first dn interior columns only
            for rows in (slice(0, dn), slice(dn + ny, n_z)):
                c[2 * dn:dn + nx, rows] = 0.0
        self.c2 = c * c * (self.dt * self.dt) / (self.dd * self.dd)
        w = (dp - 1) * self.dd
        r = np.arange(dp) / (dp - 1.0)
        alpha = 30.0 * 3.14159265 * (1.0 - r)
        sigma = -(6000.0 * math.log(1e-5) / (2.0 * w)) * r * r
        f_a, f_b = np.zeros(dn), np.zeros(dn)
        a = np.exp(-(sigma + alpha) * self.dt)
        f_a[ACC:ACC + dp], f_b[ACC:ACC + dp] = a, (a - 1.0) * sigma / (sigma + alpha)
        f_a[ACC + dp:], f_b[ACC + dp:] = f_a[ACC + dp - 1], f_b[ACC + dp - 1]

        def depth(n, inner):
            i = np.arange(n)
            return np.where(i < dn, dn - i, np.where(i >= dn + inner, i - (dn + inner) + 1, 0))

        k = np.maximum(depth(n_x, nx)[:, None], depth(n_z, ny)[None])
        pick = [torch.from_numpy(np.where(k > 0, f[np.maximum(k, 1) - 1], 0.0)).to(dev) for f in (f_a, f_b)]
        self.fx = [[q[:dn].contiguous(), q[n_x - dn:].contiguous()] for q in pick]
        self.fz = [[q[:, :dn].contiguous(), q[:, n_z - dn:].contiguous()] for q in pick]
        self.p1 = torch.zeros((n_x, n_z), dtype=torch.float64, device=dev)
        self.p = torch.zeros_like(self.p1)
        z = torch.zeros
        self.phx = [z((dn, n_z), dtype=torch.float64, device=dev) for _ in range(4)]  # phi left, right, chi left, right
        self.phz = [z((n_x, dn), dtype=torch.float64, device=dev) for _ in range(4)]
        self.side = [z((2 * dn,), dtype=torch.float64, device=dev) for _ in range(2)]  # levels n-1, n

    def step(self, cells, values):
        """One time step with `values` injected at flat interior `cells`; returns p(n+1) - p(n-1) on the interior."""
        dn, n_x, n_z = self.dn, *self.p.shape
        p = self.p
        dxx, dzz = self.d2x @ p, p @ self.d2z
        main = dxx + dzz
        x_part, z_part = (slice(0, dn), slice(n_x - dn, n_x)), (slice(0, dn), slice(n_z - dn, n_z))
        add = []
        for h in range(2):
            d = self.local @ self.phx[h]
            phi = self.fx[0][h] * self.phx[h] + self.fx[1][h] * (self.d1x[h] @ p)
            self.phx[2 + h] = self.fx[0][h] * self.phx[2 + h] + self.fx[1][h] * (dxx[x_part[h]] + d)
            self.phx[h] = phi
            add.append((x_part[h], slice(None), d + self.phx[2 + h]))
        for h in range(2):
            if h == 0 and self.case["fs"]:
                continue
            d = self.phz[h] @ self.local.T
            phi = self.fz[0][h] * self.phz[h] + self.fz[1][h] * (p @ self.d1z[h])
            self.phz[2 + h] = self.fz[0][h] * self.phz[2 + h] + self.fz[1][h] * (dzz[:, z_part[h]] + d)
            self.phz[h] = phi
            add.append((slice(None), z_part[h], d + self.phz[2 + h]))
        for x, zz, v in add:
            main[x, zz] += v
        if len(cells):
            main.view(-1)[cells] += values
        new = 2.0 * p - self.p1 + self.c2 * main
        if self.case["fs"]:
            new[:, :dn] = 0.0  # rows above the free surface are never updated
            if self.case["disk"]:
                new[dn:n_x - dn, dn] = 0.0
            else:  # the side strips keep their own history of the free-surface row
                edge = torch.cat((torch.arange(dn), torch.arange(n_x - dn, n_x))).to(self.dev)
                row = new[edge, dn] + 2.0 * self.side[1] - self.side[0]
                self.side = [self.side[1], row]
                new[:, dn] = 0.0
        change = (new - self.p1)[dn:n_x - dn, dn:n_z - dn]
        self.p1, self.p = p, new
        return change

    def flat(self, xs, zs):
        return (torch.as_tensor(np.asarray(xs) + self.dn - 1) * self.p.shape[1]
                + torch.as_tensor(np.asarray(zs) + self.dn - 1)).to(self.dev)


def forward64(case, s, dev, fields, traces):
    f = Solver64(case, s, dev)
    nt, ks = s["nt"], case["ks"]
    src = torch.as_tensor(s["src"]).to(dev).double()
    cell = f.flat([s["sx"] - s["x_i"] + 1], [s["sz"]])
    rec = f.flat(s["rx"] - s["x_i"] + 1, s["rz"])
    kept = torch.zeros(((nt - 1) // ks, f.nx, f.ny), dtype=torch.float64, device=dev) if fields else None
    out = torch.zeros((len(s["rx"]), nt), dtype=torch.float64, device=dev) if traces else None
    for k in range(2, nt + 1):
        change = f.step(cell, src[k - 2])
        if fields and (k - 1) % ks == 0:
            torch.mul(change, 0.5 / f.dt, out=kept[(k - 1) // ks - 1])
        if traces:
            out[:, k - 2] = f.p.view(-1)[rec]
    if traces:
        out[:, nt - 1] = out[:, nt - 2]
    return kept, out


def backward64(case, s, dev, kept):
    b = Solver64(case, s, dev)
    nt, ks, taper = s["nt_taper"], case["ks"], case["taper"]
    data = torch.as_tensor(s["data"]).to(dev).double()
    where = {}
    for j, (x, z) in enumerate(zip(s["rx"] - s["x_i"] + 1, s["rz"])):
        where[(int(x), int(z))] = j  # of receivers in one cell the last is injected
    cells = b.flat([x for x, _ in where], [z for _, z in where])
    data = data[list(where.values())]
    weight = np.ones(nt)
    if taper:
        n = np.arange(taper)
        weight[s["nt"] - taper:s["nt"]] = 0.5 * (1.0 + np.cos(np.pi * n / taper))
        weight[s["nt"]:] = 0.0
    image = torch.zeros((b.nx, b.ny), dtype=torch.float64, device=dev)
    for k in range(2, nt + 1):
        change = b.step(cells, data[:, nt - k + 1])
        r = nt + 1 - k  # the forward step that this step meets in time
        if r % ks == 0 and 1 <= r // ks <= len(kept) and weight[r - 1] != 0.0:
            image.addcmul_(change, kept[r // ks - 1], value=0.5 * ks * weight[r - 1])
    return image


def shot64(case, s, dev):
    kept, _ = forward64(case, s, dev, True, False)
    return backward64(case, s, dev, kept)


def filter64(raw, dt, f1, f2):
    """Band-pass of filters.f90: an order-6 Butterworth response on 24-fold zero-padded traces."""
    n = raw.shape[1]
    ts = 24 * n
    f = torch.arange(ts // 2 + 1, dtype=torch.float64, device=raw.device) * (1.0 / float(np.float32(dt)) / ts)
    f0, q = math.sqrt(f1 * f2), math.sqrt(f1 * f2) / (f2 - f1)
    s = q * 1j * (f / f0 - f0 / f.clamp(min=1e-300))
    poly = torch.ones_like(s)
    for k in (1, 2, 3):
        poly = poly * (s * s - 2.0 * s * math.cos((2 * k + 5) * math.pi / 12) + 1.0)
    h = 1.0 / poly
    h[0] = 0.0
    out = torch.empty_like(raw)
    for i in range(0, raw.shape[0], 64):
        x = torch.nn.functional.pad(raw[i:i + 64], (ts - n, 0))
        out[i:i + 64] = torch.fft.irfft(torch.fft.rfft(x) * h, n=ts)[:, ts - n:]
    return out


def akima64(y, dx, t):
    """Akima's local cubic through the samples of each row of y at k dx, at the times t."""
    n = y.shape[1]
    m = (y[:, 1:] - y[:, :-1]) / dx
    left = 2 * m[:, :1] - m[:, 1:2]
    right = 2 * m[:, -1:] - m[:, -2:-1]
    m = torch.cat((2 * left - m[:, :1], left, m, right, 2 * right - m[:, -1:]), 1)
    w1, w2 = (m[:, 3:] - m[:, 2:-1]).abs(), (m[:, 1:-2] - m[:, :-3]).abs()
    both = w1 + w2
    d = torch.where(both == 0, 0.5 * (m[:, 1:-2] + m[:, 2:-1]), (w1 * m[:, 1:-2] + w2 * m[:, 2:-1]) / both.clamp(min=1e-300))
    j = (t / dx).floor().long().clamp(0, n - 2)
    u = t - j * dx
    a, b, mj = d[:, j], d[:, j + 1], m[:, j + 2]
    return y[:, j] + u * (a + u * ((3 * mj - 2 * a - b) / dx + u * (a + b - 2 * mj) / (dx * dx)))


def traces64(case, t, dev):
    raw = t["raw"].to(dev).double()
    if case["band"]:
        raw = filter64(raw, case["dt_data"], 4.0, 60.0)
    nt2, nt, n_taper, _ = (int(v) for v in t["lens"])
    dx, dt = float(np.float32(case["dt_data"])), float(np.float32(case["dt"]))
    out = torch.zeros((case["nrec"], nt), dtype=torch.float64, device=dev)
    if case["dt_data"] != case["dt"]:
        out[:, :nt2] = akima64(raw, dx, torch.arange(nt2, dtype=torch.float64, device=dev) * dt)
    else:
        n = min(nt2, raw.shape[1])
        out[:, :n] = raw[:, :n]
    s = torch.arange(1, nt + 1, device=dev)[None]
    cut = torch.from_numpy(np.clip(t["cut"], 1, nt)).to(dev)[:, None]
    out[(s <= torch.from_numpy(t["sea"]).to(dev)[:, None]) | (s >= cut)] = 0.0
    at = s - (cut - n_taper + 1).clamp(min=1)
    ramp = 0.5 * (1.0 + torch.cos(math.pi * at.double() / n_taper))
    out = torch.where((at >= 0) & (s <= cut), out * ramp, out)
    return {"filtered": raw, "target": out}


def exact(case, seed):
    dev = device()
    if case["kind"] == "traces":
        return traces64(case, inputs(case, seed), dev)
    # 64-bit products take about a microsecond per 10^5 cells beside 0.5 ms of launches a step
    steps = sum(nt for _, nt in shots_of(case)) * (1 if case["kind"] == "model" else 2)
    dn, nrec, nt = case["dpml"] + 2 * ACC, case["nrec"], case["nt"]
    n_x, n_z = nrec * case["rec_step"] + 2 * case["pad"] + 2 * dn, case["ny"] + 2 * dn
    seconds = steps * (5e-4 + 2.0 * n_x * n_z * (n_x + n_z) / 2e13)
    kept = 0 if case["kind"] == "model" else 8.0 * case["ny"] * (n_x - 2 * dn) * nt / case["ks"]
    if seconds > 18 or kept > 4e10:
        return None
    shots = inputs(case, seed)
    if case["kind"] == "model":
        return forward64(case, shots[0], dev, False, True)[1]
    if case["kind"] == "solvers":
        s = shots[0]
        fields, traces = forward64(case, s, dev, True, True)
        image = backward64(case, s, dev, fields)
        return {"fields": torch.nn.functional.pad(fields, (0, 0, 0, 0, 0, 1)), "traces": traces, "image": image}
    if case["kind"] != "batch":
        return shot64(case, shots[0], dev)
    longest = max(shots, key=lambda h: h["nt"])
    return [shot64(case, dict(s, src=longest["src"]), dev) for s in shots]
