"""The work that a user of this framework has it do, as cases that can be timed.

A case is a dict of plain values.  Its "kind" names the public entry point:

  map     Engine.get_2d_map(_device): dispersion maps of a model grid, the call
          that every line-search step of an inversion makes
  kernel  Engine.get_1d_kernel_device: dispersion and depth kernels, once per
          iteration
  disp    Engine.surfdisp96_batch: dispersion curves of many layered models in
          host memory (ambient-noise and receiver-side 1-D work, samplers)
  times   SurfTime.travel_time: maps, then fast marching for every station pair
  grad    SurfTime.compute_grad: kernels, marching, rays, the sensitivity rows and
          their product with the residuals
  lsmr    lsmr on such rows: the solve of every iteration
  batch   UnevenBatch: several models of their own shapes in one launch
  train   MLP.train_step: one Adam step of the bracket proposal network

Models are drawn on the GPU: a velocity gradient with smooth perturbations, a
low-velocity zone in a fifth of the columns, and (water) fluid nodes on top of
a tenth of them.  The sizes are those of the repository's configurations (16 x
16 columns of 20 nodes up to 256 x 256 columns of 64 nodes) and what lies
between.
"""
import math

import numpy as np
import torch

from jdsurfg_b200 import learn, mlp, synth
from jdsurfg_b200.batch import UnevenBatch
from jdsurfg_b200.engine import Engine, torch_stream
from jdsurfg_b200.lsmr import DeviceCSR, lsmr
from jdsurfg_b200.surftime import SurfTime

WAVES = ("Rc", "Rg", "Lc", "Lg")
MOST_COST = 65536 * 120 * 64      # columns x root slots x nodes of the largest listed grid
MOST_KERNEL = 65536 * 120 * 64    # columns x output slots x nodes


def listed():
    def grid(name, kind, nx, ny, nz, nt, tmin, tmax, waves, nmode=1, learned=True, water=False, host=False):
        return dict(name=name, kind=kind, nx=nx, ny=ny, nz=nz, nt=nt, tmin=tmin, tmax=tmax, waves=waves, nmode=nmode,
                    learned=learned, water=water, host=host)
    return [
        # a local study's maps, from and to host arrays: the smallest call, all latency
        grid("map_16x16_host", "map", 16, 16, 20, 25, 2.0, 40.0, "Rc Rg", host=True),
        # the reference's example grid: one line-search step's maps
        grid("map_33x36", "map", 33, 36, 41, 19, 4.0, 40.0, "Rc Rg"),
        # the same grid's kernels: one iteration of the example
        grid("kernel_33x36", "kernel", 33, 36, 41, 19, 4.0, 40.0, "Rc Rg"),
        # a regional grid of odd sizes without the proposal networks (an Engine as it is made)
        grid("kernel_97x61_plain", "kernel", 97, 61, 33, 30, 2.0, 50.0, "Rc Lc", learned=False),
        # the production grid: both wave types, phase and group, two modes, coast columns
        grid("kernel_128x128_modes", "kernel", 128, 128, 48, 40, 1.0, 60.0, "Rc Rg Lc Lg", nmode=2, water=True),
        # the grid that the headline figure is quoted on
        grid("kernel_256x256", "kernel", 256, 256, 64, 60, 1.0, 80.0, "Rc Lc"),
        # dispersion curves of a set of 1-D models, as a sampler asks for them
        dict(name="disp_1500x37", kind="disp", nmodel=1500, nlayer=37, nt=21, tmin=1.0, tmax=40.0, iwave=2, mode=1,
             igr=0),
        # a line-search step of the example, maps and every station pair's march
        dict(name="times_33x36", kind="times", nx=33, ny=36, nstation=80, nperiod=19, waves="Rc Rg"),
        # the gradient of an iteration on the same grid with a sparser network
        dict(name="grad_33x36", kind="grad", nx=33, ny=36, nstation=40, nperiod=19, waves="Rc Rg"),
        # the solve of the example's system
        dict(name="lsmr_20000", kind="lsmr", nx=33, ny=36, nz=41, rows=20000, iters=24),
        # an iteration over models of different shapes
        dict(name="batch_6_models", kind="batch", nmodels=6, shapes=3, learned=True),
        # one optimiser step of the proposal network at the training batch
        dict(name="train_4096", kind="train", rows=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _root_slots(c):
    """Periods that the root search runs for: group slots of a kernel take two more each."""
    n = {"R": 0, "L": 0}
    for w in c["waves"].split():
        group = w[1] == "g" and c["kind"] == "kernel"
        n[w[0]] = max(n[w[0]], 3 if group else 1)
    return c["nt"] * c["nmode"] * sum(n.values())


def draw(rng):
    kind = rng.choice(["map", "map", "kernel", "kernel", "kernel", "disp", "times", "grad", "lsmr", "batch", "train"])
    if kind in ("map", "kernel"):
        while True:
            side = math.exp(rng.uniform(math.log(9.0), math.log(256.0)))
            r = rng.uniform(0.6, 1.6)
            waves = rng.choice(["Rc", "Lc", "Rg", "Rc Rg", "Rc Lc", "Lc Lg", "Rc Rg Lc Lg"])
            c = dict(kind=kind, nx=max(5, round(side * r)), ny=max(5, round(side / r)), nz=rng.randint(12, 80),
                     nt=rng.randint(5, 60), tmin=round(rng.uniform(1.0, 5.0), 2), tmax=round(rng.uniform(30.0, 90.0), 1),
                     waves=waves, nmode=rng.choice([1, 1, 2]), learned=rng.random() < 0.7, water=rng.random() < 0.3,
                     host=False)
            c["host"] = kind == "map" and c["nx"] * c["ny"] < 4096 and rng.random() < 0.4
            ncol = c["nx"] * c["ny"]
            cost = ncol * _root_slots(c) * c["nz"] * (1.0 if c["learned"] else 1.6)
            if cost <= 0.5 * MOST_COST and ncol * len(waves.split()) * c["nt"] * c["nmode"] * c["nz"] <= MOST_KERNEL:
                return c
    if kind == "disp":
        return dict(kind=kind, nmodel=_log_int(rng, 20, 6000), nlayer=rng.randint(5, 90), nt=rng.randint(5, 60),
                    tmin=round(rng.uniform(0.5, 4.0), 2), tmax=round(rng.uniform(20.0, 60.0), 1),
                    iwave=rng.choice([1, 2]), mode=rng.choice([1, 1, 2]), igr=rng.choice([0, 0, 1]))
    if kind in ("times", "grad"):
        return dict(kind=kind, nx=rng.randint(14, 40), ny=rng.randint(14, 40), nstation=_log_int(rng, 8, 60),
                    nperiod=rng.randint(2, 19), waves=rng.choice(["Rc", "Rc Rg", "Rg"]))
    if kind == "lsmr":
        return dict(kind=kind, nx=rng.randint(12, 48), ny=rng.randint(12, 48), nz=rng.randint(10, 40),
                    rows=_log_int(rng, 300, 20000), iters=rng.randint(8, 30))
    if kind == "batch":
        return dict(kind=kind, nmodels=rng.randint(2, 8), shapes=rng.randint(0, 9999), learned=rng.random() < 0.6)
    return dict(kind="train", rows=_log_int(rng, 64, 16384))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda", 0)


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed) * 7919 + 17)


def _depth(nz):
    if nz > 24:
        return synth.depth_grid(21, 1.0, nz, 2.5)
    return (np.arange(nz) * 2.0).astype(np.float32)


def _brocher(vs):
    v = vs.double()
    vp = (0.9409 + 2.0947 * v - 0.8206 * v ** 2 + 0.2683 * v ** 3 - 0.0251 * v ** 4).float()
    p = vp.double()
    rho = (1.6612 * p - 0.4721 * p ** 2 + 0.0671 * p ** 3 - 0.0043 * p ** 4 + 0.000106 * p ** 5).float()
    return vp, rho


def _model(c, seed):
    """(vs, vp, rho) as (nz, columns) float32 on the GPU; vp and rho None without water."""
    dev, g = _device(), _generator(seed)
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    depth = torch.from_numpy(_depth(nz)).to(dev)
    coarse = torch.randn((1, 1, nz // 3 + 2, ny // 4 + 2, nx // 4 + 2), device=dev, generator=g)
    f = torch.nn.functional.interpolate(coarse, size=(nz, ny, nx), mode="trilinear", align_corners=True)[0, 0]
    f = f / f.abs().max()
    base = 2.5 + 2.1 * (depth - depth[0]) / (depth[-1] - depth[0])
    vs = (base[:, None, None] * (1.0 + 0.08 * f)).reshape(nz, nx * ny)
    lvz = torch.rand(nx * ny, device=dev, generator=g) < 0.2
    zone = (depth >= 15.0) & (depth <= 25.0)
    vs = torch.where(zone[:, None] & lvz[None, :], vs * 0.9, vs).float().contiguous()
    if not c["water"]:
        return vs, None, None
    vp, rho = _brocher(vs)
    wet = torch.rand(nx * ny, device=dev, generator=g) < 0.1
    nw = torch.randint(1, 4, (nx * ny,), device=dev, generator=g) * wet
    fluid = torch.arange(nz, device=dev)[:, None] < nw[None, :]
    vs = torch.where(fluid, torch.zeros_like(vs), vs)
    vp = torch.where(fluid, torch.full_like(vp, 1.5), vp)
    rho = torch.where(fluid, torch.full_like(rho, 1.03), rho)
    return vs.contiguous(), vp.contiguous(), rho.contiguous()


def _periods(c):
    return np.geomspace(c["tmin"], c["tmax"], c["nt"])


def _tables(c):
    t = np.ascontiguousarray(np.repeat(_periods(c)[:, None], c["nmode"], axis=1))
    return [t if w in c["waves"].split() else None for w in WAVES]


def _layered(c, seed):
    """1-D layered models as host arrays (models, layers)."""
    rng = np.random.default_rng(seed)
    n, m = c["nmodel"], c["nlayer"]
    thk = rng.uniform(0.6, 1.4, (n, m)) * (60.0 / m)
    thk[:, -1] = 0.0
    vs = np.sort(rng.uniform(2.0, 4.7, (n, m)), axis=1) * rng.uniform(0.97, 1.03, (n, m))
    vs[:, -1] = vs.max(axis=1) + 0.1
    vp = 1.75 * vs
    rho = 0.32 * vp + 0.77
    return [np.ascontiguousarray(a, np.float32) for a in (thk, vp, vs, rho)]


def _rays_csr(c, seed):
    """Frechet-shaped CSR rows: the cells near the straight ray of a random
    station pair, at every depth, weighted around the depth that the row's
    period samples, with some scatter."""
    dev, g = _device(), _generator(seed)
    nxi, nyi, nzi, m = c["nx"] - 2, c["ny"] - 2, c["nz"] - 1, c["rows"]
    ends = torch.rand((m, 4), device=dev, generator=g) * torch.tensor([nxi, nyi, nxi, nyi], device=dev)
    x = torch.arange(nxi, device=dev).float()[None, None, :] + 0.5
    y = torch.arange(nyi, device=dev).float()[None, :, None] + 0.5
    rowptr = torch.zeros(m + 1, dtype=torch.int64, device=dev)
    idx, val, near = [], [], []
    peak, width = nzi * torch.rand((2, m), device=dev, generator=g)
    for a in range(0, m, 2048):
        ax, ay, bx, by = (ends[a:a + 2048, i, None, None] for i in range(4))
        dx, dy = bx - ax, by - ay
        t = (((x - ax) * dx + (y - ay) * dy) / (dx * dx + dy * dy + 1e-6)).clamp(0.0, 1.0)
        d2 = (x - ax - t * dx) ** 2 + (y - ay - t * dy) ** 2
        w = torch.where(d2 < 4.0, torch.exp(-d2), torch.zeros_like(d2)).reshape(t.shape[0], -1)
        near.append((w > 0).sum(1) * nzi)
        z = torch.arange(nzi, device=dev).float()[None, :] - peak[a:a + 2048, None]
        depth = 0.01 + torch.exp(-(z / (1.0 + 0.2 * width[a:a + 2048, None])) ** 2)
        full = (w[:, None, :] * depth[:, :, None]).reshape(t.shape[0], -1)
        k = torch.nonzero(full)
        idx.append(k[:, 1].int())
        v = full[k[:, 0], k[:, 1]]
        val.append(v * torch.randn(v.shape, device=dev, generator=g))
    rowptr[1:] = torch.cumsum(torch.cat(near), 0)
    b = torch.randn(m, dtype=torch.float64, device=dev, generator=g)
    return rowptr, torch.cat(idx).contiguous(), torch.cat(val).contiguous(), nxi * nyi * nzi, b


def _training_rows(c, seed):
    """Feature rows as the training set has them: 258 normalised values, zero padding."""
    dev, g = _device(), _generator(seed)
    x = torch.zeros((c["rows"], mlp.IN_DIM), device=dev)
    x[:, :258] = 0.8 + 0.2 * torch.randn((c["rows"], 258), device=dev, generator=g)
    y = 0.3 * torch.randn(c["rows"], device=dev, generator=g)
    return x.bfloat16().contiguous(), y.contiguous()


def _survey(c):
    """Station pairs of the case's network: the same ones for every model."""
    return synth.make_survey("example", seed=7, nx=c["nx"], ny=c["ny"], nstation=c["nstation"], nperiod=c["nperiod"],
                             waves=tuple(c["waves"].split()))


def _shapes(c):
    """Grids, depths and period tables of an uneven batch's models: 8 to 20
    columns a side, 24 to 40 nodes, one or two wave types, one to three modes."""
    rng = np.random.default_rng(c["shapes"])
    models = []
    for _ in range(c["nmodels"]):
        nx, ny = (int(v) for v in rng.integers(8, 21, 2))
        nz, nt, nmode = int(rng.integers(24, 41)), int(rng.integers(15, 61)), int(rng.integers(1, 4))
        some = rng.choice(WAVES, size=int(rng.integers(1, 3)), replace=False)
        waves = [w for w in WAVES if w in some]
        m = dict(kind="kernel", nx=nx, ny=ny, nz=nz, nt=nt, nmode=nmode, waves=" ".join(waves), water=True,
                 tmin=float(rng.uniform(1.0, 5.0)), tmax=float(rng.uniform(30.0, 100.0)))
        models.append(dict(m, depth=_depth(nz), tables=_tables(m)))
    return models


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("map", "kernel"):
        vs, vp, rho = _model(case, seed)
        eng = Engine()
        nets = learn.load_proposals(eng) if case["learned"] else None
        eng.setup(dict(depth=_depth(case["nz"]), tables=_tables(case)))
        ncol, kmax, dev = case["nx"] * case["ny"], eng.kmax, _device()
        s = dict(case=case, eng=eng, nets=nets, vs=vs, vp=vp, rho=rho)
        if case["host"]:
            for k in ("vs", "vp", "rho"):
                s[k] = None if s[k] is None else s[k].cpu().numpy()
            return s
        s["vc"] = torch.zeros((kmax, ncol), dtype=torch.float64, device=dev)
        s["vout"] = torch.zeros_like(s["vc"])
        s["status"] = torch.zeros((kmax, ncol), dtype=torch.int32, device=dev)
        if kind == "kernel":
            s["kernel"] = torch.zeros((kmax, case["nz"], ncol), dtype=torch.float64, device=dev)
        return s
    if kind == "disp":
        return dict(case=case, eng=Engine(), models=_layered(case, seed), t=_periods(case))
    if kind in ("times", "grad"):
        sv = _survey(case)
        nx, ny, lat0, lon0, dlat, dlon = sv["grid"]
        st = SurfTime()
        st.set_model(sv["case"]["depth"], lat0, lon0, dlat, dlon, nx, ny)
        rng = np.random.default_rng(seed)
        vs, _, _ = _model(dict(case, nz=len(sv["case"]["depth"]), water=False), seed)
        st.set_data(sv["tables"], sv["kmax_per_mode"], sv["pairs"],
                    obst=rng.uniform(20.0, 200.0, int(sv["pairs"]["rcv_ptr"][-1])))
        return dict(case=case, st=st, vs=vs.cpu().numpy())
    if kind == "lsmr":
        rowptr, idx, val, n, b = _rays_csr(case, seed)
        return dict(case=case, A=DeviceCSR(rowptr, idx, val, case["rows"], n), b=b)
    if kind == "batch":
        models = _shapes(case)
        for i, m in enumerate(models):
            m["vs"], m["vp"], m["rho"] = (a.cpu().numpy() for a in _model(m, int(seed) * 64 + i))
        return dict(case=case, batch=UnevenBatch(models, learned=case["learned"]))
    x, y = _training_rows(case, seed)
    return dict(case=case, net=mlp.MLP(seed=int(seed) % (1 << 31)), x=x, y=y)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind in ("map", "kernel"):
        eng, nx, ny, nz = state["eng"], c["nx"], c["ny"], c["nz"]
        if c["host"]:
            return eng.get_2d_map(state["vs"], state["vp"], state["rho"], nx=nx, ny=ny)
        stream = torch_stream(_device())
        out = {k: state[k] for k in ("vc", "vout", "status")}
        if kind == "map":
            eng.get_2d_map_device(nx, ny, nz, state["vs"], state["vp"], state["rho"], out["vc"], out["vout"],
                                  out["status"], stream=stream)
            return out
        out["kernel"] = state["kernel"]
        eng.get_1d_kernel_device(nx, ny, nz, state["vs"], state["vp"], state["rho"], out["vc"], out["vout"],
                                 out["kernel"], out["status"], stream=stream)
        return out
    if kind == "disp":
        cg, ierr = state["eng"].surfdisp96_batch(*state["models"], 1, c["iwave"], c["mode"], c["igr"], state["t"])
        return dict(cg=cg, ierr=ierr)
    if kind == "times":
        return dict(ttime=state["st"].travel_time(state["vs"]))
    if kind == "grad":
        data, grad = state["st"].compute_grad(state["vs"])
        return dict(ttime=data, grad=grad)
    if kind == "lsmr":
        x, info = lsmr(state["A"], state["b"], damp=0.1, atol=0.0, btol=0.0, conlim=0.0, itnlim=c["iters"])
        return dict(x=x, normr=info["normr"], normAr=info["normAr"], itn=info["itn"])
    if kind == "batch":
        state["batch"].launch(torch_stream(_device()))
        return [{k: b[k] for k in ("vc", "vout", "st", "ker")} for b in state["batch"].bufs]
    loss = state["net"].train_step(state["x"], state["y"], 1e-3)
    return dict(loss=loss, grads=state["net"].grads(), params=state["net"].params())


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
RAYLEIGH, LOVE = 161.0, 19.0            # FP64 operations per layer of a secular evaluation
RAYLEIGH_EIGEN, LOVE_EIGEN = 675.0, 132.0  # and of an eigenfunction pass
EVALS = 3.0                             # a root takes two evaluations that bracket it and one that refines it


def _grid_work(c):
    ncol, layers, per = c["nx"] * c["ny"], 4 * c["nz"] - 3, c["nt"] * c["nmode"]
    waves = c["waves"].split()
    flops = slots = 0.0
    roots = {"R": 0, "L": 0}
    for w in waves:
        slots += per
        three = w[1] == "g" and c["kind"] == "kernel"
        roots[w[0]] = max(roots[w[0]], 3 if three else 1)
        passes = (3 if three else 1) if c["kind"] == "kernel" else (1 if w[1] == "g" else 0)
        flops += per * passes * layers * (RAYLEIGH_EIGEN if w[0] == "R" else LOVE_EIGEN)
    flops += per * EVALS * layers * (roots["R"] * RAYLEIGH + roots["L"] * LOVE)
    nbytes = ncol * (c["nz"] * 4.0 * (3 if c["water"] else 1) + slots * 20.0)
    if c["kind"] == "kernel":
        nbytes += ncol * slots * c["nz"] * 8.0
    return dict(bytes=nbytes, flops=flops * ncol)


def work(case):
    c, kind = case, case["kind"]
    if kind in ("map", "kernel"):
        return _grid_work(c)
    if kind == "disp":
        roots = c["nt"] * c["mode"] * (2 if c["igr"] else 1)
        per = RAYLEIGH if c["iwave"] == 2 else LOVE
        return dict(bytes=c["nmodel"] * (16.0 * c["nlayer"] + 8.0 * c["nt"] + 4),
                    flops=c["nmodel"] * roots * EVALS * c["nlayer"] * per)
    if kind in ("times", "grad"):
        waves = c["waves"].split()
        pairs = len(waves) * c["nperiod"] * c["nstation"]
        rcv = pairs * 0.18 * (c["nstation"] - 1)
        nodes = (8 * (c["nx"] - 3) + 1) * (8 * (c["ny"] - 3) + 1)  # propagation grid of a march
        g = dict(kind="kernel" if kind == "grad" else "map", nx=c["nx"], ny=c["ny"], nz=41, nt=c["nperiod"], nmode=1,
                 waves=c["waves"], water=False)
        w = _grid_work(g)
        w["flops"] += pairs * (nodes + 129.0 * 129.0) * 4 * 60.0   # four trial times per accepted node
        w["bytes"] += rcv * 16.0 + c["nx"] * c["ny"] * 41 * 4.0
        return w
    if kind == "lsmr":
        per_row = min(c["nx"] - 2, c["ny"] - 2) * 0.55 * 4.0 * (c["nz"] - 1)
        nnz = c["rows"] * per_row
        n = (c["nx"] - 2.0) * (c["ny"] - 2) * (c["nz"] - 1)
        return dict(bytes=c["iters"] * (2 * 8.0 * nnz + 8.0 * (4 * c["rows"] + 10 * n)), flops=c["iters"] * 4.0 * nnz)
    if kind == "batch":
        each = [_grid_work(m) for m in _shapes(c)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    weights = 256.0 * 320 + 3 * 256 * 256 + 256 * 64
    return dict(bytes=c["rows"] * 644.0 + weights * 4 * 8, flops=6.0 * c["rows"] * weights)


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def _rayleigh(c, om, d, a, b, r):
    """Sign-carrying Rayleigh period equation (Dunkin's delta matrix), layers
    first; c and om broadcast against the layer arrays' columns."""
    k = om / c
    k2 = k * k

    def vertical(v):
        q = (k - om / v) * (k + om / v)
        return q, torch.sqrt(q.abs())

    qa, ra = vertical(a[-1])
    qb, rb = vertical(b[-1])
    g = 2.0 * (b[-1] / om) ** 2
    gam = g * k2
    rho = r[-1]
    e = [rho * rho * ((gam - 1) ** 2 - gam * g * ra * rb), -rho * ra, rho * (gam - 1 - g * ra * rb), rho * rb,
         k2 - ra * rb]
    for m in range(d.shape[0] - 2, -1, -1):
        rho = r[m]
        ex, cs, sn_over, sn_times = [], [], [], []
        for v in (a[m], b[m]):
            q, s = vertical(v)
            p = s * d[m]
            dec = torch.exp(-2.0 * p)
            ev = q > 0
            cs.append(torch.where(ev, 0.5 * (1 + dec), torch.cos(p)))
            sn = torch.where(ev, 0.5 * (1 - dec), torch.sin(p))
            sn_over.append(sn / s)
            sn_times.append(torch.where(ev, sn * s, -sn * s))
            ex.append(torch.where(ev, torch.exp(-p), torch.ones_like(p)))
        a0 = ex[0] * ex[1]
        w, y, x, z = sn_over[0], sn_over[1], sn_times[0], sn_times[1]
        cp, cq = cs
        cpcq, cpy, cpz, cqw, cqx = cp * cq, cp * y, cp * z, cq * w, cq * x
        xy, xz, wy, wz = x * y, x * z, w * y, w * z
        g = 2.0 * (b[m] / om) ** 2
        gam = g * k2
        g1 = gam - 1
        tw, gg, gs = gam + g1, gam * g, g1 * g1
        ap = a0 - cpcq
        c11 = cpcq - 2 * gam * g1 * ap - gg * xz - k2 * gs * wy
        c12 = (k2 * cpy - cqx) / rho
        c13 = -(tw * ap + g * xz + k2 * g1 * wy) / rho
        c14 = (cpz - k2 * cqw) / rho
        c15 = -(2 * k2 * ap + xz + k2 * k2 * wy) / (rho * rho)
        c21 = (gg * cpz - gs * cqw) * rho
        c23 = g * cpz - g1 * cqw
        c41 = (gs * cpy - gg * cqx) * rho
        c43 = g1 * cpy - g * cqx
        c51 = -(2 * gg * gs * ap + gg * gg * xz + gs * gs * wy) * rho * rho
        c53 = -(g * g1 * tw * ap + gam * g * g * xz + g1 * gs * wy) * rho
        t = -2 * k2
        c33 = a0 + 2 * (cpcq - c11)
        f = [e[0] * c11 + e[1] * c21 + e[2] * t * c53 + e[3] * c41 + e[4] * c51,
             e[0] * c12 + e[1] * cpcq + e[2] * t * c43 - e[3] * xy + e[4] * c41,
             e[0] * c13 + e[1] * c23 + e[2] * c33 + e[3] * c43 + e[4] * c53,
             e[0] * c14 - e[1] * wz + e[2] * t * c23 + e[3] * cpcq + e[4] * c21,
             e[0] * c15 + e[1] * c14 + e[2] * t * c13 + e[3] * c12 + e[4] * c11]
        top = f[0].abs()
        for v in f[1:]:
            top = torch.maximum(top, v.abs())
        e = [v / top for v in f]
    return e[0]


def _love(c, om, d, a, b, r):
    k = om / c
    s = torch.sqrt(((k - om / b[-1]) * (k + om / b[-1])).abs())
    e1, e2 = r[-1] * s, 1.0 / (b[-1] * b[-1]) + 0.0 * s
    for m in range(d.shape[0] - 2, -1, -1):
        mu = r[m] * b[m] * b[m]
        q = (k - om / b[m]) * (k + om / b[m])
        s = torch.sqrt(q.abs())
        p = s * d[m]
        dec = torch.exp(-2.0 * p)
        ev = q > 0
        cs = torch.where(ev, 0.5 * (1 + dec), torch.cos(p))
        sn = torch.where(ev, 0.5 * (1 - dec), torch.sin(p))
        f1 = e1 * cs + e2 * mu * torch.where(ev, sn * s, -sn * s)
        f2 = e1 * sn / (s * mu) + e2 * cs
        top = torch.maximum(f1.abs(), f2.abs())
        e1, e2 = f1 / top, f2 / top
    return e1


def _fundamental(vs, vp, rho, depth, periods, love):
    """Phase velocities (period, column) of the fundamental mode: 4 sublayers
    per node interval, earth flattening, first sign change of the period
    equation from below, halved until it stands."""
    dev = vs.device
    vs, vp, rho = vs.double(), vp.double(), rho.double()
    dep = torch.as_tensor(depth, dtype=torch.float64, device=dev)
    lay = []
    for v in (vp, vs, rho):
        w = (torch.arange(4, device=dev).double() * 2 + 1) / 8
        sub = v[:-1, None] + w[None, :, None] * (v[1:] - v[:-1])[:, None]
        lay.append(torch.cat([sub.reshape(-1, v.shape[1]), v[-1:]]))
    thk = torch.cat([((dep[1:] - dep[:-1]) / 4).repeat_interleave(4), torch.ones(1, dtype=torch.float64, device=dev)])
    bottom = torch.cumsum(thk, 0)
    r0, r1 = 6370.0 - (bottom - thk), 6370.0 - bottom
    d = 6370.0 * torch.log(r0 / r1)
    s = 2 * 6370.0 / (r0 + r1)
    a, b = lay[0] * s[:, None], lay[1] * s[:, None]
    r = lay[2] * (s[:, None] ** (-5.0 if love else -2.275))
    f = _love if love else _rayleigh
    om = (2 * math.pi / torch.as_tensor(periods, dtype=torch.float64, device=dev))[:, None]
    lo = (0.8 * b.min(0).values)[None, :].expand(len(periods), -1).clone()
    sign = torch.sign(f(lo, om, d, a, b, r))
    found = torch.zeros_like(lo, dtype=torch.bool)
    hi = lo.clone()
    for _ in range(2000):
        nxt = torch.where(found, hi, lo + 0.005)
        change = ~found & (torch.sign(f(nxt, om, d, a, b, r)) != sign)
        hi = torch.where(change, nxt, hi)
        lo = torch.where(found | change, lo, nxt)
        found = found | change
        if bool(found.all()) or bool((lo.min() > b.max())):
            break
    for _ in range(46):
        mid = 0.5 * (lo + hi)
        same = torch.sign(f(mid, om, d, a, b, r)) == sign
        lo, hi = torch.where(same, mid, lo), torch.where(same, hi, mid)
    c = 0.5 * (lo + hi)
    x = (1.5 if love else 0.5) * c / (6371.0 * om)
    return torch.where(found, c / torch.sqrt(1 + x * x), torch.full_like(c, math.nan))


def _exact_maps(c, seed):
    vs, vp, rho = _model(c, seed)
    if vp is None:
        vp, rho = _brocher(vs)
    got = {}
    rows = []
    for w in WAVES:
        if w in c["waves"].split():
            if w[0] not in got:
                got[w[0]] = _fundamental(vs, vp, rho, _depth(c["nz"]), _periods(c), w[0] == "L")
            rows.append(got[w[0]])
    out = dict(vc=torch.cat(rows), vout=None, status=None)
    if not any(w[1] == "g" for w in c["waves"].split()):
        out["vout"] = out["vc"]
    if c["kind"] == "kernel":
        out["kernel"] = None
    return out


def _exact_lsmr(c, seed):
    """The same number of LSMR steps (Fong & Saunders 2011) in 64 bits."""
    rowptr, idx, val, n, b = _rays_csr(c, seed)
    A = torch.sparse_csr_tensor(rowptr, idx.long(), val.double(), size=(c["rows"], n))
    rows = torch.repeat_interleave(torch.arange(c["rows"], device=b.device), torch.diff(rowptr))
    cols, v64 = idx.long(), val.double()
    damp = 0.1

    def at(u):
        return torch.zeros(n, dtype=torch.float64, device=b.device).index_add_(0, cols, v64 * u[rows])

    beta = float(b.norm())
    u = b / beta
    v = at(u)
    alpha = float(v.norm())
    v = v / alpha
    abar, zbar, rho, rbar, cbar, sbar = alpha, alpha * beta, 1.0, 1.0, 1.0, 0.0
    h, hbar, x = v.clone(), torch.zeros_like(v), torch.zeros_like(v)
    for _ in range(c["iters"]):
        u = A @ v - alpha * u
        beta = float(u.norm())
        u = u / beta
        v = at(u) - beta * v
        alpha = float(v.norm())
        v = v / alpha
        ahat = math.hypot(abar, damp)
        rold, rho = rho, math.hypot(ahat, beta)
        cc, ss = ahat / rho, beta / rho
        theta, abar = ss * alpha, cc * alpha
        rbold, thbar, rt = rbar, sbar * rho, cbar * rho
        rbar = math.hypot(rt, theta)
        cbar, sbar = rt / rbar, theta / rbar
        zeta, zbar = cbar * zbar, -sbar * zbar
        hbar = h - (thbar * rho / (rold * rbold)) * hbar
        x = x + (zeta / (rho * rbar)) * hbar
        h = v - (theta / rho) * h
    res = A @ x - b
    normr = math.sqrt(float(res.norm()) ** 2 + damp * damp * float(x.norm()) ** 2)
    return dict(x=x, normr=normr, normAr=float((at(res) + damp * damp * x).norm()), itn=None)


def _exact_train(c, seed):
    """Loss and gradients in 64 bits from the 16-bit weights that the step multiplies with."""
    x, y = _training_rows(c, seed)
    x, y = x.double(), y.double()
    w = torch.from_numpy(mlp.MLP(seed=int(seed) % (1 << 31)).params()).to(x.device)
    parts, h, lay = [], x, mlp.layout()
    for i, (wo, n, k, bo) in enumerate(lay):
        W = w[wo:wo + n * k].bfloat16().double().reshape(n, k).requires_grad_(True)
        bias = w[bo:bo + n].double().requires_grad_(True)
        parts += [(wo, W), (bo, bias)]
        h = h @ W.T + bias
        if i < len(lay) - 1:
            h = torch.nn.functional.gelu(h)
    mu, ls = h[:, 0], h[:, 1].clamp(-12.0, 4.0)
    loss = (0.5 * ((y - mu) * torch.exp(-ls)) ** 2 + ls).mean()
    loss.backward()
    g = torch.zeros(w.numel(), dtype=torch.float64, device=x.device)
    for o, p in parts:
        g[o:o + p.numel()] = p.grad.reshape(-1)
    return dict(loss=float(loss), grads=g, params=None)


def exact(case, seed):
    """Values of run() in 64 bits, where there is a short way to them: the
    fundamental mode's phase velocities of small grids without water, the
    LSMR iterate, the network's loss and gradients."""
    c, kind = case, case["kind"]
    if kind in ("map", "kernel") and c["nmode"] == 1 and not c["water"]:
        slots = c["nx"] * c["ny"] * c["nt"] * len({w[0] for w in c["waves"].split()})
        if slots * c["nz"] <= 3_000_000:
            return _exact_maps(c, seed)
    if kind == "lsmr":
        return _exact_lsmr(c, seed)
    if kind == "train":
        return _exact_train(c, seed)
    return None
