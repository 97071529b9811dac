"""The work that programs on this framework have it do, as cases that can be timed and checked.

A case is one of three kinds of program:

  layer     one shear layer advanced by some steps: a :class:`Domain`
  ensemble  32 small independent layers advanced together: an :class:`Ensemble`
  train     the closure network's gradient and one training epoch: a :class:`Trainer`

``prepare`` makes the seeded start states on the GPU and the objects a program keeps,
``run`` is one pass of the program, ``exact`` evaluates the same scheme in FP64 with plain
torch operations (a restatement of the documented method, independent of the kernels).

A layer pass restarts from the start state the program holds (device memory through
``set_planes_async``, or pinned host memory through ``upload_state_async``), so that every
pass steps the same flow, and hands the stepped state back the same way.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import freeshearlayer_b200 as fsl

P0, RHO0, GAMMA, RGAS, CV = 1e5, 1.0, 1.4, 287.10, 717.75
DW0 = 1.0  # initial vorticity thickness of the temporal layers

SGS = {"dynamic": fsl.SGS_DYNAMIC, "learned": fsl.SGS_LEARNED, "static": fsl.SGS_STATIC, "none": fsl.SGS_NONE}
RECON = {"char": fsl.RECON_CHARMINMOD, "ppm": fsl.RECON_PPM}


def _layer(L, H, D, steps, precision=64, sgs="dynamic", recon="char", setup="temporal", loop="call", io="device",
           stats=False, amp=1e-3, mach=0.7, reynolds=1000.0):
    return dict(kind="layer", L=L, H=H, D=D, steps=steps, precision=precision, sgs=sgs, recon=recon, setup=setup,
                loop=loop, io=io, stats=stats, amp=amp, mach=mach, reynolds=reynolds)


def listed():
    cases = {
        # The smallest production run: the validation layer of 64x32x32 cells, plain FP64 method, in
        # chunks of 20 steps with the Favre row sums read after each chunk; launches and idle SMs count.
        "validation_64": _layer(64, 32, 32, 20, mach=0.4, reynolds=500.0, stats=True),
        # The reference's shipped case (its layer2.ini grid and physics) as its driver loop runs it:
        # one step, a synchronisation and the printed scalars per step.
        "driver_spatial_100": _layer(100, 80, 35, 10, setup="spatial", loop="driver"),
        # The same physics through the per-phase entry points (a driver that keeps the reference's phases).
        "phased_spatial_96": _layer(96, 72, 40, 4, setup="spatial", loop="phased"),
        # The precision study's plain arm: PPM in FP64 at 256x128x128.
        "ppm64_256": _layer(256, 128, 128, 2, recon="ppm", mach=0.6),
        # The same study's FP32-bulk arm with the learned closure.
        "ppm32_learned_256": _layer(256, 128, 128, 4, precision=32, recon="ppm", sgs="learned", mach=0.6),
        # The plain FP64 method at the production size (the comparison arm of every speed-up).
        "plain64_512": _layer(512, 256, 256, 2),
        # The headline: FP32 bulk with the learned closure at the production size, statistics per output.
        "learned32_512": _layer(512, 256, 256, 4, precision=32, sgs="learned", stats=True),
        # A turbulent layer on a ragged grid, FP32 bulk with the dynamic procedure.
        "turbulent32_ragged": _layer(203, 97, 75, 6, precision=32, amp=5e-2, mach=0.6, reynolds=2e4),
        # The spatially developing case with the static model (the distributed variant's), FP32 bulk, ragged.
        "spatial32_static": _layer(161, 90, 53, 6, precision=32, sgs="static", setup="spatial"),
        # A host program that owns the state: upload, one step, download, from and to pinned memory.
        "host_exchange_128": _layer(128, 64, 64, 1, precision=32, io="host"),
        # The batched study: 32 layers on grids of 48..128 x 32..64 x 32..64, five steps per output.
        "ensemble_32": dict(kind="ensemble", members=32, steps=5),
        # The closure's training: gradient over the sample set, then one epoch of Adam from given weights.
        "train_1m": dict(kind="train", samples=1 << 20, batch=65536),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.random()
    if what < 0.08:
        n = _log(rng, 1 << 15, 1 << 20)
        return dict(kind="train", samples=n, batch=min(n, 128 * _log(rng, 32, 512)))
    if what < 0.16:
        return dict(kind="ensemble", members=rng.randint(4, 32), steps=rng.randint(2, 5))
    L, H, D = _log(rng, 24, 512), _log(rng, 16, 256), _log(rng, 16, 256)
    setup = "spatial" if rng.random() < 0.3 else "temporal"
    precision = rng.choice([64, 32])
    sgs = rng.choice(["dynamic", "dynamic", "static", "none"] if setup == "spatial" else
                     ["dynamic", "dynamic", "learned", "static"])
    recon = rng.choice(["char", "char", "ppm"])
    loops = ["call", "call", "driver"] + (["phased"] if precision == 64 and sgs != "learned" else [])
    loop = rng.choice(loops)
    io = "host" if loop != "phased" and rng.random() < 0.15 and L * H * D < 2000000 else "device"
    amp = 1e-3 if sgs == "learned" else rng.choice([1e-3, 5e-2])
    mach = round(rng.uniform(0.2, 0.8), 3)
    reynolds = round(math.exp(rng.uniform(math.log(300.0), math.log(2e4))), 1)
    heavy = (2 if recon == "ppm" else 1) * (3 if loop == "phased" else 1)
    steps = max(1, min(20, int(2.0e7 / (heavy * L * H * D)))) if L * H * D < 4000000 else 1
    return _layer(L, H, D, steps, precision=precision, sgs=sgs, recon=recon, setup=setup, loop=loop, io=io,
                  stats=rng.random() < 0.3, amp=amp, mach=mach, reynolds=reynolds)


# ---------------------------------------------------------------- inputs
def _velocity_difference(mach):
    return 2.0 * mach * math.sqrt(GAMMA * P0 / RHO0)


def _params(c):
    """The parameter set of a layer case: the shipped physics for the spatial setup, a 2pi x pi x pi
    box at acoustic CFL 0.5 for the temporal one."""
    p = dict(LEN=c["L"], HIG=c["H"], DEP=c["D"], Answer=0, numstep=0, Pr_L=0.72, Pr_T=0.8, Cs=0.01, Ns_min=10,
             Nst=50, f_step=50, nStages=3, seed_X=0.317391239817,
             precision=fsl.PREC_FP32 if c["precision"] == 32 else fsl.PREC_FP64, sgs=SGS[c["sgs"]],
             recon=RECON[c["recon"]])
    if c["setup"] == "spatial":
        p.update(deltaX=1.6666667, deltaY=1.0, deltaZ=1.5, deltaT=0.0007, mu_L=0.253358, BL_HIG=5, Ua=35.0,
                 Va=35.0, Wa=35.0, maxCoNum=0.1, setup=fsl.SETUP_SPATIAL, cfl_mode=fsl.CFL_STREAMWISE)
    else:
        p.update(deltaX=2 * math.pi / c["L"], deltaY=math.pi / c["H"], deltaZ=math.pi / c["D"], deltaT=1e-5,
                 mu_L=_velocity_difference(c["mach"]) * DW0 / c["reynolds"], BL_HIG=0, Ua=0.0, Va=0.0, Wa=0.0,
                 maxCoNum=0.5, setup=fsl.SETUP_TEMPORAL, cfl_mode=fsl.CFL_ACOUSTIC)
    return p


def _two_streams(j, H):
    """The shipped case's inflow velocity of row j."""
    lower = (j < H // 2).to(torch.float64)
    return 76.4 * lower + 200.0 * (1.0 - lower)


def _start(c, seed):
    """The start state [L][H][5][D] on the GPU: the tanh layer with Crocco-Busemann temperature (temporal)
    or the shipped two-stream profile (spatial), with seeded uniform velocity noise of amplitude amp dU."""
    L, H, D = c["L"], c["H"], c["D"]
    p = _params(c)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    f64 = dict(dtype=torch.float64, device="cuda")
    j = torch.arange(H, **f64)
    if c["setup"] == "spatial":
        dU = 200.0 - 76.4
        um = _two_streams(j, H)
        rho = torch.full((H,), RHO0, **f64)
    else:
        dU = _velocity_difference(c["mach"])
        y = (j + 0.5) * p["deltaY"] - 0.5 * H * p["deltaY"]
        um = 0.5 * dU * torch.tanh(2.0 * y / DW0)
        T = P0 / (RGAS * RHO0) + (0.25 * dU * dU - um * um) / (2.0 * CV * GAMMA)
        rho = P0 / (RGAS * T)
    s = torch.empty((L, H, 5, D), **f64)
    n = torch.rand((3, L, H, D), generator=gen, **f64).mul_(2.0).sub_(1.0).mul_(c["amp"] * dU)
    n[0] += um[None, :, None]
    r = rho[None, :, None].expand(L, H, D)
    s[:, :, 0] = r
    for q in range(3):
        s[:, :, 1 + q] = r * n[q]
    s[:, :, 4] = P0 / (GAMMA - 1.0) + 0.5 * r * (n * n).sum(0)
    return s


def _domain(c):
    d = fsl.Domain(_params(c))
    if c["sgs"] == "learned":
        d.closure_set_scales(DW0 / _velocity_difference(c["mach"]), DW0)
        d.closure_set_weights(fsl.closure_weights())
    return d


def _members(case, seed):
    """The batched study's layers: grids, Mach and Reynolds numbers drawn for the study, noise by `seed`."""
    rng = np.random.default_rng(20251203)
    out = []
    for q in range(case["members"]):
        L, H, D = (int(rng.choice(v)) for v in ([48, 64, 96, 128], [32, 48, 64], [32, 48, 64]))
        out.append((_layer(L, H, D, case["steps"], precision=32, mach=float(rng.uniform(0.2, 0.8)),
                           reynolds=float(rng.uniform(300.0, 1000.0))), seed * 1000 + q))
    return out


def _samples(case, seed):
    """Training pairs of a turbulent layer: every cell's eight features and its dynamic Cs^2."""
    side = max(24, int(math.ceil((case["samples"] / 2) ** (1 / 3))) + 4)
    c = _layer(2 * side, side, side, 0, amp=5e-2, mach=0.6, reynolds=2e4)
    m = _Scheme(c, _start(c, seed))
    m.ghost()
    X, _ = m.features(DW0 / _velocity_difference(0.6), DW0)
    m.dynamic()
    X = X.reshape(-1, 8)[: case["samples"]].float()
    Y = m.Cd.reshape(-1)[: case["samples"]].float()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    w = fsl.closure_weights()
    w = w * (1.0 + 0.05 * torch.randn(w.size, generator=gen, device="cuda").cpu().numpy())
    return X, Y, w.astype(np.float32)


def prepare(case, seed):
    if case["kind"] == "ensemble":
        doms, outs = [], []
        for c, s in _members(case, seed):
            d = _domain(c)
            start = _start(c, s)
            d.set_planes(1, c["L"], _ready(start))
            doms.append(d)
            outs.append(torch.empty_like(start))
        e = fsl.Ensemble(doms)
        e.set_chunk(case["steps"])
        return dict(case=case, domains=doms, ensemble=e, outs=outs)
    if case["kind"] == "train":
        X, Y, w = _samples(case, seed)
        t = fsl.Trainer(case["samples"], seed=1)
        t.set_samples(X.cpu().numpy(), Y.cpu().numpy())
        return dict(case=case, trainer=t, weights=w)
    start = _start(case, seed)
    if case["io"] == "host":
        start = start.cpu().pin_memory()
        return dict(case=case, domain=_domain(case), start=start.numpy(),
                    out=torch.empty_like(start, pin_memory=True).numpy())
    return dict(case=case, domain=_domain(case), start=_ready(start), out=torch.empty_like(start))


def _ready(t):
    torch.cuda.current_stream().synchronize()  # the domain reads it on a stream of its own
    return t


# ---------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    if case["kind"] == "ensemble":
        state["ensemble"].step(case["steps"])
        for d, o in zip(state["domains"], state["outs"]):
            d.get_planes_async(1, d.p.LEN, o)
        return state["outs"]
    if case["kind"] == "train":
        t = state["trainer"]
        t.set_weights(state["weights"])
        grad, loss0 = t.gradient()
        loss = t.train(1, case["batch"], 1e-3)
        return {"grad": grad, "loss0": loss0, "weights": t.weights(), "loss": loss}
    d = state["domain"]
    if case["io"] == "host":
        d.upload_state_async(state["start"])
    else:
        d.set_planes_async(1, case["L"], state["start"])
    scalars = []
    if case["loop"] == "driver":
        for _ in range(case["steps"]):
            d.step(1)
            d.sync()
            i = d.info()
            scalars.append((i.maxCo, i.deltaT))
    elif case["loop"] == "phased":
        d.step_phased(case["steps"])
    else:
        d.step(case["steps"])
    out = {"state": state["out"]}
    if case["io"] == "host":
        d.download_state_async(state["out"])
        d.transfer_wait()
    else:
        d.get_planes_async(1, case["L"], state["out"])
    if case["stats"]:
        out["rows"] = d.plane_sums()
    if scalars:
        out["scalars"] = np.array(scalars)
    return out


# ---------------------------------------------------------------- the least work of a pass
def work(case):
    """Bytes: per step and cell each array of the method once (three stages: the stage state and U^n read,
    the new state written, and the SGS viscosity, 128 B in FP64 and 123 B with an FP32 viscosity; the SGS
    model's own read of rho and the momenta and write of the viscosity), the start state in and the stepped
    one out.  Flops: 1120 per cell and stage (1057 in the FP32 bulk's grouping, about 700 more for PPM),
    about 500 per cell for the dynamic procedure, the network's products per cell for the closure."""
    if case["kind"] == "ensemble":
        parts = [work(c) for c, _ in _members(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if case["kind"] == "train":
        macs = 8 * 64 + 2 * 64 * 64 + 64
        n = case["samples"]
        grads = 2 + (n // case["batch"]) * (case["batch"] // 128 * 128) / n
        return {"bytes": grads * n * 36.0, "flops": grads * n * 6.0 * macs}
    cells = float(case["L"] * case["H"] * case["D"])
    fp32 = case["precision"] == 32
    sgs = {"dynamic": 36.0 if fp32 else 40.0, "learned": 36.0 if fp32 else 40.0, "static": 0.0, "none": 0.0}
    flops = 3.0 * ((1057.0 if fp32 else 1120.0) + (700.0 if case["recon"] == "ppm" else 0.0))
    flops += {"dynamic": 500.0, "learned": 2.0 * (8 * 64 + 2 * 64 * 64 + 64), "static": 0.0, "none": 0.0}[case["sgs"]]
    per_step = 3.0 * (122.67 if fp32 else 128.0) + sgs[case["sgs"]]
    return {"bytes": cells * (case["steps"] * per_step + 80.0), "flops": cells * case["steps"] * flops}


# ---------------------------------------------------------------- the scheme in FP64, in plain torch
C1, C2, TWO_THIRDS, SMALL = 0.333333333333333, 0.166666666666667, 0.666666666666667, 1e-30
INNER = slice(1, -1)


def _shift(a, *by):
    """The interior-sized view of a padded field displaced by `by` cells along x, y, z."""
    return a[tuple(slice(1 + o, a.shape[q] - 1 + o) for q, o in enumerate(by))]


def _minmod(x, y):
    y = 4.0 * y
    r = torch.sign(x) * torch.minimum(x.abs(), y.abs())
    return torch.where(x * y <= 0.0, torch.zeros_like(x), r)


def _mc(a, b):
    m = torch.minimum(torch.minimum(0.5 * (a + b).abs(), 2.0 * a.abs()), 2.0 * b.abs())
    return torch.where(a * b <= 0.0, torch.zeros_like(a), torch.sign(a) * m)


class _Scheme:
    """The explicit step on padded fields [5][L+2][H+2][D+2]."""

    def __init__(self, c, start):
        self.c, self.p = c, _params(c)
        self.N = (c["L"], c["H"], c["D"])
        self.spatial = c["setup"] == "spatial"
        self.h = tuple(self.p[k] for k in ("deltaX", "deltaY", "deltaZ"))
        self.DD = (self.h[0] * self.h[1] * self.h[2]) ** TWO_THIRDS
        self.dt = self.p["deltaT"]
        self.X, self.counter, self.block = self.p["seed_X"], 0, (0, 0, 0.0, 0.0, 0.0)
        self.U = start.new_zeros((5,) + tuple(n + 2 for n in self.N))
        self.U[:, INNER, INNER, INNER] = start.permute(2, 0, 1, 3)
        self.mu = start.new_zeros(self.U.shape[1:])

    def state(self):
        return self.U[:, INNER, INNER, INNER].permute(1, 2, 0, 3).contiguous()

    # ghost layer: x, then z over all x, then y over all x and z
    def ghost(self, U=None):
        u = self.U if U is None else U
        L, H, D = self.N
        if self.spatial:
            um = _two_streams(torch.arange(H, device=u.device), H)[:, None]
            inflow = torch.stack([torch.ones_like(um), um, 0 * um, 0 * um, P0 / 0.4 + 0.5 * um * um])
            u[:, 0, INNER, INNER] = inflow.expand(5, H, D)
            e = u[:, L, INNER, INNER].clone()
            e[4] = P0 / 0.4 + 0.5 * (e[1:4] ** 2).sum(0) / e[0]
            u[:, L + 1, INNER, INNER] = e
        else:
            u[:, 0], u[:, L + 1] = u[:, L].clone(), u[:, 1].clone()
        u[..., 0], u[..., D + 1] = u[..., D].clone(), u[..., 1].clone()
        u[:, :, 0], u[:, :, H + 1] = u[:, :, 1].clone(), u[:, :, H].clone()
        if self.spatial:
            u[2, :, 0] *= -1.0
            u[2, :, H + 1] *= -1.0

    # the driver's random disturbance block of the inflow
    def disturb(self):
        def rnd(x):
            x = 11.0 * x + math.pi
            return x - float(int(x))

        if self.counter > 0:
            self.counter -= 1
            return
        p, D, X = self.p, self.N[2], self.X
        X = rnd(X)
        self.counter = int(p["Ns_min"] + p["Nst"] * X)
        X = rnd(X)
        k0 = int(D * X)
        X = rnd(X)
        k1 = int(k0 + D * X)
        k1 -= D if k1 > D else 0
        v = []
        for a in ("Ua", "Va", "Wa"):
            X = rnd(X)
            v.append(p[a] * (1 - X - X))
        self.X, self.block = X, (k0, k1, *v)

    def inflow_faces(self, like):
        """Outer states of the inflow faces [5][H][D]."""
        L, H, D = self.N
        k0, k1, du, dv, dw = self.block
        j = torch.arange(H, device=like.device)[:, None].expand(H, D)
        k = torch.arange(D, device=like.device)[None, :].expand(H, D)
        hit = (k >= k0) & (k < k1) if k1 > k0 else ~((k >= k1) & (k < k0))
        hit &= (j >= H // 2) & (j < H // 2 + self.p["BL_HIG"])
        hit = hit.to(like.dtype)
        u, v, w = _two_streams(j, H) + du * hit, dv * hit, dw * hit
        return torch.stack([torch.ones_like(u), u, v, w, P0 / 0.4 + 0.5 * (u * u + v * v + w * w)])

    # characteristic reconstruction along axis d: states on the upper and the lower face of every cell
    def sweep(self, U, d):
        N = self.N[d]
        u = U[:, INNER, INNER, INNER]
        n, t1, t2 = ((1, 2, 3), (2, 3, 1), (3, 1, 2))[d]
        order = (0, n, t1, t2, 4)
        R = 1.0 / u[0]
        vel = {q: u[q] * R for q in (1, 2, 3)}
        vn, v1, v2 = vel[n], vel[t1], vel[t2]
        ff = vn * vn + v1 * v1 + v2 * v2
        C = torch.sqrt(GAMMA * ((u[4] - 0.5 * u[0] * ff) * 0.4) * R)
        ll = 0.5 / C
        ee = ll / C

        def at(o):
            by = [0, 0, 0]
            by[d] = o
            return [_shift(U[q], *by) for q in order]

        def forward(x, y, s=slice(None)):
            m = [p - q for p, q in zip(x, y)]
            A = 0.2 * ff[s] * m[0] - 0.4 * (vn[s] * m[1] + v1[s] * m[2] + v2[s] * m[3]) + 0.4 * m[4]
            B = C[s] * (m[1] - vn[s] * m[0])
            return [A - C[s] * C[s] * m[0], m[2] - v1[s] * m[0], m[3] - v2[s] * m[0], A + B, A - B]

        def inverse(k, s=slice(None)):
            ks, kd = k[3] + k[4], k[3] - k[4]
            hh = -2.0 * ee[s]
            t2_ee = (vn if d == 2 else v2)[s] * ee[s]  # the reference's z sweep takes w here
            out = [None] * 5
            out[0] = hh * k[0] + ee[s] * ks
            out[n] = vn[s] * hh * k[0] + vn[s] * ee[s] * ks + ll[s] * kd
            out[t1] = v1[s] * hh * k[0] + k[1] + v1[s] * ee[s] * ks
            out[t2] = v2[s] * hh * k[0] + k[2] + t2_ee * ks
            out[4] = (-ff[s] * ee[s] * k[0] + v1[s] * k[1] + v2[s] * k[2] + (0.5 * ff[s] * ee[s] + 1.25) * ks +
                      vn[s] * ll[s] * kd)
            return torch.stack(out)

        c0, fw, bw = at(0), at(1), at(-1)
        M, W = forward(fw, c0), forward(c0, bw)
        a = [_minmod(x, y) for x, y in zip(M, W)]
        b = [_minmod(y, x) for x, y in zip(M, W)]
        hi = u + inverse([x * C1 + y * C2 for x, y in zip(a, b)])
        lo = u - inverse([x * C2 + y * C1 for x, y in zip(a, b)])
        if self.c["recon"] == "ppm" and N > 2:  # cells with two neighbours on either side
            s = tuple(slice(1, -1) if q == d else slice(None) for q in range(3))
            rows = [U[v][tuple(slice(None) if q == d else INNER for q in range(3))] for v in order]

            def cells(o):  # the cells displaced by o from those
                return [q.narrow(d, 2 + o, N - 2) for q in rows]

            Ws = [forward(cells(o + 1), cells(o), s) for o in (-2, -1, 0, 1)]
            qr, ql = [], []
            for w0, w1, w2, w3 in zip(*Ws):
                dm, dc, dp = _mc(w0, w1), _mc(w1, w2), _mc(w2, w3)
                r, l = 0.5 * w2 - (dp - dc) / 6.0, -0.5 * w1 - (dc - dm) / 6.0
                flat = r * l >= 0.0
                big_r = ~flat & (r.abs() > 2.0 * l.abs())
                big_l = ~flat & ~big_r & (l.abs() > 2.0 * r.abs())
                zero = torch.zeros_like(r)
                qr.append(torch.where(flat, zero, torch.where(big_r, -2.0 * l, r)))
                ql.append(torch.where(flat, zero, torch.where(big_l, -2.0 * r, l)))
            at_s = (slice(None),) + s
            hi[at_s] = u[at_s] + inverse(qr, s)
            lo[at_s] = u[at_s] + inverse(ql, s)
        return hi, lo

    def faces(self, U, d):
        """Minus and plus states of the N+1 faces along axis d, boundary faces included."""
        hi, lo = self.sweep(U, d)
        N = self.N[d]
        first, last = (lambda a: a.narrow(d + 1, 0, 1)), (lambda a: a.narrow(d + 1, N - 1, 1))
        if d == 0 and self.spatial:
            outer0 = self.inflow_faces(U)[:, None]
            outerN = last(hi).clone()
            outerN[4] = P0 / 0.4 + 0.5 * (outerN[1:4] ** 2).sum(0) / outerN[0]
        elif d == 1:
            outer0, outerN = first(lo).clone(), last(hi).clone()
            if self.spatial:
                outer0[2] *= -1.0
                outerN[2] *= -1.0
        else:
            outer0, outerN = last(hi), first(lo)
        return torch.cat([outer0, hi], d + 1), torch.cat([lo, outerN], d + 1)

    @staticmethod
    def riemann(A, B, d):
        def side(s):
            v = s[1:4] / s[0]
            P = (s[4] - 0.5 * s[0] * (v * v).sum(0)) * 0.4
            C = torch.sqrt(GAMMA * P / s[0])
            r = P / (s[0] * C)
            return v, C, -0.4 * P, v[d] + r, v[d] - r

        va, Ca, joa, jpa, jma = side(A)
        vb, Cb, job, jpb, jmb = side(B)
        Un, C = 0.5 * (va[d] + vb[d]), 0.5 * (Ca + Cb)
        pp, pm, po = Un + C > 0, Un - C > 0, Un > 0
        al_p = 0.2 * torch.where(pp, jma - jpa, jmb - jpb) / torch.where(pp, joa, job)
        al_m = 0.2 * torch.where(pm, jpa - jma, jpb - jmb) / torch.where(pm, joa, job)
        al_o = 0.7 * torch.where(po, jpa - jma, jpb - jmb)
        al_o = -al_o * al_o
        Jp, Jm, Jo = torch.where(pp, jpa, jpb), torch.where(pm, jma, jmb), torch.where(po, joa, job)
        P = (Jp - Jm) / (al_p - al_m)
        Un = Jp - al_p * P
        rho = (Jo - P) / al_o
        v = torch.where((Un > 0)[None], va, vb)
        v[d] = Un
        return rho, P, v

    def flux(self, U, d):
        rho, P, v = self.riemann(*self.faces(U, d), d)
        V = U[1:4] / U[0]
        T = (U[4] - 0.5 * U[0] * (V * V).sum(0)) * 0.4 / (RGAS * U[0])

        def cell(a, plus, by=(0, 0, 0)):  # the cells on one side of the faces, displaced
            s = [slice(1 + by[q], a.shape[q] - 1 + by[q]) for q in range(3)]
            s[d] = slice(1, None) if plus else slice(0, -1)
            if by[d]:
                raise ValueError("normal displacement")
            return a[tuple(s)]

        g = [[None] * 3 for _ in range(3)]
        for b in range(3):
            if b == d:
                for a in range(3):
                    g[a][b] = (cell(V[a], True) - cell(V[a], False)) / self.h[b]
                continue
            up, dn = [0, 0, 0], [0, 0, 0]
            up[b], dn[b] = 1, -1
            for a in range(3):
                g[a][b] = (cell(V[a], True, up) + cell(V[a], False, up) - cell(V[a], True, dn) -
                           cell(V[a], False, dn)) / (4.0 * self.h[b])
        if self.c["sgs"] == "static":
            rr = 0.5 * (cell(U[0], True) + cell(U[0], False))
            S2 = sum(g[q][q] ** 2 for q in range(3))
            S2 = S2 + 2.0 * sum((0.5 * (g[a][b] + g[b][a])) ** 2 for a, b in ((0, 1), (0, 2), (1, 2)))
            mu_t = rr * self.p["Cs"] * self.DD * torch.sqrt(2.0 * S2)
        elif self.c["sgs"] == "none":
            mu_t = torch.zeros_like(P)
        else:  # the plus cell and its lower x neighbour, on every face
            s = [INNER, INNER, INNER]
            s[d] = slice(1, None)
            m = list(s)
            m[0] = slice(0, -1) if d == 0 else slice(0, self.mu.shape[0] - 2)
            mu_t = 0.5 * (self.mu[tuple(s)] + self.mu[tuple(m)])
        mu = self.p["mu_L"] + mu_t
        div = g[0][0] + g[1][1] + g[2][2]
        s = [TWO_THIRDS * mu * (3.0 * g[d][d] - div) if a == d else mu * (g[a][d] + g[d][a]) for a in range(3)]
        lam = self.p["mu_L"] * CV * GAMMA / self.p["Pr_L"] + mu_t * (CV * GAMMA / self.p["Pr_T"])
        q = -lam * (cell(T, True) - cell(T, False)) / self.h[d]
        m = rho * v[d]
        F = [m] + [m * v[a] - s[a] for a in range(3)]
        F[1 + d] = F[1 + d] + P
        E = v[d] * (3.5 * P + 0.5 * rho * (v * v).sum(0)) + q
        for a in range(3):
            E = E - 0.5 * (cell(V[a], True) + cell(V[a], False)) * s[a]
        return torch.stack(F + [E])

    # box test filter: y, z and x sweeps on buffers whose never written bands are zero
    def filter(self, a):
        L, H, D = self.N
        t1, t2 = torch.zeros_like(a), torch.zeros_like(a)
        t1[: L + 1, 1: H + 1, : D + 1] = (a[: L + 1, : H, : D + 1] + a[: L + 1, 1: H + 1, : D + 1] +
                                          a[: L + 1, 2:, : D + 1]) / 3.0
        t2[: L + 1, : H + 1, 1: D + 1] = (t1[: L + 1, : H + 1, : D] + t1[: L + 1, : H + 1, 1: D + 1] +
                                          t1[: L + 1, : H + 1, 2:]) / 3.0
        t1[1: L + 1, : H + 1, : D + 1] = (t2[:L, : H + 1, : D + 1] + t2[1: L + 1, : H + 1, : D + 1] +
                                          t2[2:, : H + 1, : D + 1]) / 3.0
        return t1

    def strain(self, V):
        """Strain-rate components 11 12 13 22 23 33 of the interior and |S|."""
        def by(q):
            o = [0, 0, 0]
            o[q] = 1
            return o

        g = [[(_shift(V[a], *by(b)) - _shift(V[a], *[-z for z in by(b)])) / (2.0 * self.h[b]) for b in range(3)]
             for a in range(3)]
        S = [g[0][0], 0.5 * (g[0][1] + g[1][0]), 0.5 * (g[0][2] + g[2][0]), g[1][1], 0.5 * (g[1][2] + g[2][1]), g[2][2]]
        mag = torch.sqrt(2.0 * (S[0] ** 2 + S[3] ** 2 + S[5] ** 2 + 2.0 * (S[1] ** 2 + S[2] ** 2 + S[4] ** 2)))
        return S, mag

    def dynamic(self):
        pairs = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))
        V = self.U[1:4] / self.U[0]
        Vf = torch.stack([self.filter(V[q]) for q in range(3)])
        I = (INNER, INNER, INNER)
        Lij = [(self.filter(V[a] * V[b]) - Vf[a] * Vf[b])[I] for a, b in pairs]
        S, mag = self.strain(V)
        Sf, magf = self.strain(Vf)
        M = []
        for s, sf in zip(S, Sf):
            A = torch.zeros_like(self.mu)
            A[I] = mag * s
            M.append(self.DD * (4.0 * magf * sf - self.filter(A)[I]))
        tr = (Lij[0] + Lij[3] + Lij[5]) / 3.0
        for q in (0, 3, 5):
            Lij[q] = Lij[q] - tr
        twice = (1.0, 2.0, 2.0, 1.0, 2.0, 1.0)
        LM = sum(t * l * m for t, l, m in zip(twice, Lij, M))
        MM = sum(t * m * m for t, m in zip(twice, M))
        self.Cd = torch.clamp(-0.5 * LM / (MM + SMALL), 0.0, 0.15)
        self.mu[I] = self.U[0][I] * self.Cd * self.DD * mag

    def features(self, t_ref, len_ref):
        V = self.U[1:4] / self.U[0]
        S, mag = self.strain(V)
        inv = 1.0 / (mag + SMALL)
        rho = self.U[0, INNER, INNER, INNER]
        width = (self.h[0] * self.h[1] * self.h[2]) ** (1.0 / 3.0) / len_ref
        X = [torch.log1p(mag * t_ref), S[0] * inv, S[3] * inv, S[1] * inv, S[2] * inv, S[4] * inv, rho,
             torch.full_like(rho, width)]
        return torch.stack(X, -1), mag

    def learned(self):
        X, mag = self.features(DW0 / _velocity_difference(self.c["mach"]), DW0)
        w = torch.from_numpy(fsl.closure_weights()).to(X)
        X = X.reshape(-1, 8)
        y = torch.cat([_network(w, b) for b in X.split(1 << 20)]).clamp(0.0, 0.15)
        I = (INNER, INNER, INNER)
        self.mu[I] = self.U[0][I] * y.reshape(mag.shape) * self.DD * mag

    def step(self):
        u = self.U[:, INNER, INNER, INNER]
        v = u[1:4] / u[0]
        if self.spatial:
            co = (v[0] * (self.dt / self.h[0])).max()
        else:
            C = torch.sqrt(GAMMA * (u[4] - 0.5 * u[0] * (v * v).sum(0)) * 0.4 / u[0])
            co = sum((v[q].abs() + C) * (self.dt / self.h[q]) for q in range(3)).max()
        self.co = max(0.0, float(co))
        self.dt *= self.p["maxCoNum"] / self.co
        self.disturb()
        self.ghost()
        if self.c["sgs"] == "dynamic":
            self.dynamic()
        elif self.c["sgs"] == "learned":
            self.learned()
        stage, keep = self.U, (0.0, 0.75, 1.0 / 3.0)
        for s in range(3):
            if s:
                self.ghost(stage)
            inc = torch.zeros_like(u)
            for d in range(3):
                F = self.flux(stage, d)
                inc += (self.dt / self.h[d]) * (F.narrow(d + 1, 0, self.N[d]) - F.narrow(d + 1, 1, self.N[d]))
            new = stage.clone() if s == 0 else stage
            I = (slice(None), INNER, INNER, INNER)
            new[I] = keep[s] * self.U[I] + (1.0 - keep[s]) * (stage[I] + inc)
            stage = new
        self.U = stage


def _network(w, X):
    """The 8-64-64-64-1 SiLU network of one parameter vector."""
    W1, b1, W2, b2, W3, b3, w4, b4 = w.split([1024, 64, 4096, 64, 4096, 64, 64, 1])
    a = torch.nn.functional.silu(X @ W1.reshape(64, 16)[:, :8].T + b1)
    a = torch.nn.functional.silu(a @ W2.reshape(64, 64).T + b2)
    a = torch.nn.functional.silu(a @ W3.reshape(64, 64).T + b3)
    return a @ w4 + b4


def _exact_layer(c, seed):
    m = _Scheme(c, _start(c, seed))
    scalars = []
    for _ in range(c["steps"]):
        m.step()
        scalars.append((m.co, m.dt))
    out = {"state": m.state()}
    if c["stats"]:
        u = m.U[:, INNER, INNER, INNER]
        v = u[1:4] / u[0]
        q = [u[0], u[1], u[2], u[3], u[1] * v[0], u[2] * v[1], u[3] * v[2], u[1] * v[1]]
        out["rows"] = torch.stack([x.sum((0, 2)) for x in q], -1)
    if c["loop"] == "driver":
        out["scalars"] = torch.tensor(scalars, dtype=torch.float64)
    return out


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] == "ensemble":
            return [_exact_layer(c, s)["state"] for c, s in _members(case, seed)]
        if case["kind"] == "layer":
            return _exact_layer(case, seed)
    # the gradient of the viscosity-weighted squared error; the trained weights have no exact value
    X, Y, w = _samples(case, seed)
    X, Y = X.double(), Y.double()
    weight = (torch.expm1(X[:, 0]) * X[:, 6]) ** 2
    weight = weight / weight.mean()
    w = torch.from_numpy(w).to(X).requires_grad_()
    loss = 0.0
    for x, y, q in zip(X.split(1 << 18), Y.split(1 << 18), weight.split(1 << 18)):
        part = (q * (_network(w, x) - y) ** 2).sum() / len(X)
        part.backward()
        loss += float(part)
    return {"grad": w.grad, "loss0": loss, "weights": None, "loss": None}
