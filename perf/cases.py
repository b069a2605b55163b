"""The work this framework is run for, as cases that can be timed and compared.

A case is a dict of plain values; ``kind`` says which of the public calls a
pass makes, the other values say on what:

  step        one SimPL global iteration of the quadratic path with the FP64
              solve: B2B build anchored at spread positions, Jacobi-PCG of x
              and y to 1e-6, HPWL, occupancy and overflow
  fast_step   the same iteration with the FP32 aggregation-preconditioned PCG
              in FP64 refinement (coarse 2: coupling share, 3: learned vector)
  legalize    look-ahead legalization of lower-bound positions
  batch       x and y systems of several netlists of uneven size, one batch
  spmv        A v for both axes (SparseSystem::multiply)
  train       loss and gradient of the learned coarse vector, both axes
  kraftwerk2  Kraftwerk2's initial placement step

Designs come from the seeded generator (ktplace_b200.synth) in the shapes of
the repository's configurations: 300-cell designs as in the tests, the 12,000-
cell design with pads only, the 211,000-cell design with 550 macros, batches
of 5,000 to 200,000 cells at mean degree 3.5, and a million cells with macros.
"""
import ctypes
import math

import numpy as np
import torch

from ktplace_b200 import grid, netlist, synth
from ktplace_b200._lib import SolveInfo, MixedInfo
from ktplace_b200.gpu import Batch, Context
from ktplace_b200.learned import Learned

TOL = 1e-6           # the configurations' relative residual
MAX_ITER = 100000
COARSE_WEIGHTS = "ktplace_b200/weights/learned_coarse.npy"


def listed():
    return [
        # the smallest design of the tests, on device data: launch and barrier
        # latency of every call of the iteration
        dict(name="step_300", kind="step", cells=300, nets=330, pads=16, rows=12, macros=0,
             bins=16, alpha=0.2, host=False),
        # the 12,000-cell configuration called as a C++ host does, with host
        # arrays in and out of every call
        dict(name="step_12k_host", kind="step", cells=12000, nets=13000, pads=200, rows=120,
             macros=0, bins=128, alpha=0.2, host=True),
        # the 211,000-cell configuration with its 512 x 512 bins, data resident:
        # the framework's headline step
        dict(name="step_211k", kind="step", cells=211000, nets=221000, pads=1000, rows=890,
             macros=550, bins=512, alpha=0.2, host=False),
        # a large design, whose systems no longer fit the L2 cache; early
        # iteration, so a weak anchor and many CG iterations
        dict(name="step_1m", kind="step", cells=1000000, nets=1023000, pads=2000, rows=1950,
             macros=3600, bins=512, alpha=0.05, host=False),
        # the fast solve of the same 211,000-cell iteration, aggregates rebuilt
        # as after every first build of a design
        dict(name="fast_211k", kind="fast_step", cells=211000, nets=221000, pads=1000, rows=890,
             macros=550, bins=512, alpha=0.5, coarse=2, host=False),
        # the learned coarse vector on a mid-size design, host arrays
        dict(name="fast_47k_host", kind="fast_step", cells=47123, nets=51050, pads=397, rows=238,
             macros=0, bins=256, alpha=0.1, coarse=3, host=True),
        # legalization of the upper bound, once per SimPL iteration: a small
        # design through host arrays and the macro design on device data
        dict(name="legalize_12k_host", kind="legalize", cells=12007, nets=13001, pads=200,
             rows=120, macros=0, sweeps=4, host=True),
        dict(name="legalize_211k", kind="legalize", cells=211000, nets=221000, pads=1000, rows=890,
             macros=550, sweeps=3, host=False),
        # the first netlists of the batched-solve configuration: a few pairs
        # large enough for the whole GPU, the rest on clusters
        dict(name="batch_12", kind="batch", first=0, netlists=12, alpha=0.2),
        # the matrix product alone, e.g. for a true residual
        dict(name="spmv_500k", kind="spmv", cells=500000, nets=511500, pads=1500, rows=775,
             macros=0),
        # one training sample of the learned coarse vector (both axes)
        dict(name="train_60k", kind="train", cells=60001, nets=65000, pads=450, rows=268, macros=0,
             vectors=2, alpha=0.1),
        # the other placer's initial step
        dict(name="kraftwerk2_100k", kind="kraftwerk2", cells=100003, nets=105000, pads=600,
             rows=346, macros=0),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "fast_step", "legalize", "batch", "spmv", "train",
                       "kraftwerk2"])
    if kind == "batch":
        return dict(kind=kind, first=rng.randrange(64), netlists=rng.randint(2, 10),
                    alpha=round(rng.uniform(0.1, 0.5), 3))
    lo, hi = {"step": (300, 600000), "fast_step": (300, 400000), "legalize": (2000, 150000),
              "spmv": (1000, 500000), "train": (5000, 100000),
              "kraftwerk2": (1000, 200000)}[kind]
    cells = _log_uniform(rng, lo, hi)
    c = dict(kind=kind, cells=cells, nets=int(cells * rng.uniform(1.02, 1.09)),
             pads=max(16, int(2 * math.sqrt(cells))),
             rows=max(12, int(round(120 * math.sqrt(cells / 12000)))), macros=0)
    if cells > 20000 and rng.random() < 0.5 and kind in ("step", "fast_step", "legalize"):
        c["macros"] = cells // 400
        c["rows"] = int(c["rows"] * 1.75)
    if kind in ("step", "fast_step"):
        c["bins"] = rng.choice([64, 128, 200, 256, 512])
        c["alpha"] = round(rng.uniform(0.05, 1.0), 3)
        c["host"] = rng.random() < 0.5
    if kind == "fast_step":
        c["coarse"] = rng.choice([0, 1, 2, 3])
    if kind == "legalize":
        c["sweeps"] = rng.randint(2, 5)
        c["host"] = rng.random() < 0.5
    if kind == "train":
        c["vectors"] = rng.randint(1, 4)
        c["alpha"] = round(rng.uniform(0.05, 1.0), 3)
    return c


# ---- inputs --------------------------------------------------------------------


def _design(case, seed):
    spec = synth.SynthSpec(num_movable=case["cells"], num_nets=case["nets"], num_pads=case["pads"],
                           num_rows=case["rows"], utilization=0.6 if case["macros"] else 0.7,
                           num_macros=case["macros"], seed=seed)
    return netlist.flatten(synth.generate(spec), kraftwerk2=case["kind"] == "kraftwerk2")


def _uniform(nl, rng):
    lx, ly, ux, uy = nl.die
    return (lx + rng.random(nl.num_movable) * np.maximum(ux - lx - nl.width, 0.0),
            ly + rng.random(nl.num_movable) * np.maximum(uy - ly - nl.height, 0.0))


def _smooth(nl, fields, sweeps):
    """`sweeps` times, every cell's value becomes the mean over its nets of
    their pins' means; `fields` are pairs (values of the movable cells, values
    of the fixed vertices)."""
    N = nl.num_nets
    deg = np.diff(nl.net_start)
    net = np.repeat(np.arange(N), deg)
    var = nl.var_of_vertex[nl.pin_cell]
    mov = var >= 0
    cnt = np.maximum(np.bincount(var[mov], minlength=nl.num_movable), 1)
    out = []
    for pos, fixed in fields:
        for _ in range(sweeps):
            at = fixed[nl.pin_cell]
            at[mov] = pos[var[mov]]
            mean = np.bincount(net, weights=at, minlength=N) / np.maximum(deg, 1)
            pos = np.bincount(var[mov], weights=mean[net[mov]], minlength=nl.num_movable) / cnt
        out.append(pos)
    return out


def _lower_bound(nl, rng, sweeps):
    """Positions like those a quadratic solve leaves: a uniform start, smoothed
    over the nets with the fixed pins holding them apart."""
    x, y = _uniform(nl, rng)
    return _smooth(nl, ((x, nl.fixed_x), (y, nl.fixed_y)), sweeps)


def _spread(pos, size, lo, hi):
    """Anchors as a legalizer leaves them: the order of `pos`, the cells spread
    evenly over the die."""
    order = np.argsort(pos, kind="stable")
    out = np.empty_like(pos)
    out[order] = lo + (np.arange(len(pos)) + 0.5) * ((hi - lo) / len(pos))
    return np.minimum(out, hi - size)


def _iterate(nl, rng):
    x, y = _lower_bound(nl, rng, 2)
    lx, ly, ux, uy = nl.die
    ax, ay = _spread(x, nl.width, lx, ux), _spread(y, nl.height, ly, uy)
    return x, y, ax, ay


class _State:
    pass


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _inputs(case, seed):
    """The netlist and the vectors of one case, as host arrays."""
    nl = _design(case, seed)
    rng = np.random.default_rng(seed + 1)
    kind = case["kind"]
    if kind == "legalize":
        v = dict(zip(("x", "y"), _lower_bound(nl, rng, case["sweeps"])))
    elif kind == "kraftwerk2":
        v = dict(zip(("x", "y"), _uniform(nl, rng)))
    else:
        v = dict(zip(("x", "y", "ax", "ay"), _iterate(nl, rng)))
    if kind == "spmv":
        v["vx"], v["vy"] = rng.standard_normal((2, nl.num_movable))
    if kind == "train":
        # test vectors like the errors a few solver steps leave: smooth over
        # the nets and nothing at the fixed pins
        zero = np.zeros(nl.num_vertices)
        for k in ("ex", "ey"):
            starts = rng.random((case["vectors"], nl.num_movable))
            v[k] = np.stack(_smooth(nl, [(e, zero) for e in starts], 6))
    return nl, v


def _batch_inputs(case, seed):
    out = []
    for k in range(case["netlists"]):
        spec = synth.spec_batch_member(case["first"] + k)
        spec.seed += 1000 * seed
        nl = netlist.flatten(synth.generate(spec))
        out.append((nl,) + _iterate(nl, np.random.default_rng(spec.seed + 1)))
    return out


def prepare(case, seed):
    s = _State()
    s.case, s.kind, s.host = case, case["kind"], case.get("host", False)
    if s.kind == "batch":
        # the plan an autotuner run keeps for these batches: clusters of four
        # CTAs, pairs of at least 44,000 rows on the whole GPU
        s.batch = Batch(0)
        s.stream = torch.cuda.Stream()
        s.batch.set_stream(s.stream.cuda_stream)
        s.rows = []
        ctx = Context(0)
        for nl, x, y, ax, ay in _batch_inputs(case, seed):
            fx, fy = nl.floors()
            ctx.upload_netlist(nl)
            ctx.build_b2b(x, y, case["alpha"], ax, ay, fx, fy)
            s.batch.add_from_context(ctx, x, y)
            s.rows += [nl.num_movable] * 2
        ctx.close()
        s.batch.set_shape(4, 1024)
        s.batch.set_offload(44000, 2, 0)
        return s

    nl, v = _inputs(case, seed)
    s.fx, s.fy = nl.floors()
    s.ctx = ctx = Context(0)
    ctx.upload_netlist(nl)
    s.stream = torch.cuda.Stream()
    ctx.set_stream(s.stream.cuda_stream)
    if s.kind in ("step", "fast_step"):
        ctx.set_grid(grid.build_grid(nl, case["bins"], 1.0))
    if s.kind == "legalize":
        ctx.set_grid(grid.build_grid(nl, grid.default_bins_per_axis(nl.num_movable), 1.0))
        ctx.set_free_space(grid.build_free_space(nl))
    if s.kind == "fast_step":
        ctx.set_option("precond", 2)
        ctx.set_option("coarse", case["coarse"])
    if s.kind == "train" or case.get("coarse") == 3:
        s.net = Learned(0, seed=1)
        s.net.load(COARSE_WEIGHTS)
    if s.kind in ("spmv", "train"):
        ctx.build_b2b(v["x"], v["y"], case.get("alpha", 0.2), v["ax"], v["ay"], s.fx, s.fy)
    if s.host or s.kind == "train":
        for k, a in v.items():
            setattr(s, k, a)
        return s
    for k, a in v.items():
        setattr(s, k, _dev(a))
    s.wx, s.wy = torch.empty_like(s.x), torch.empty_like(s.y)
    if s.kind in ("step", "fast_step"):
        s.occ = torch.zeros(case["bins"] ** 2, dtype=torch.float64, device="cuda")
        s.scal = torch.zeros(2, dtype=torch.float64, device="cuda")
    info = MixedInfo if s.kind == "fast_step" else SolveInfo
    s.info = torch.zeros(ctypes.sizeof(info) // 8, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    return s


# ---- one pass ------------------------------------------------------------------


def run(s):
    return {"step": _run_step, "fast_step": _run_fast, "legalize": _run_legalize,
            "batch": _run_batch, "spmv": _run_spmv, "train": _run_train,
            "kraftwerk2": _run_kraftwerk2}[s.kind](s)


def _run_step(s):
    ctx, alpha = s.ctx, s.case["alpha"]
    if s.host:
        ctx.build_b2b(s.x, s.y, alpha, s.ax, s.ay, s.fx, s.fy)
        r = ctx.solve(s.x, s.y, TOL, MAX_ITER)
        hpwl = ctx.hpwl(r["x"], r["y"])
        occ, overflow = ctx.occupancy(r["x"], r["y"])
        return dict(x=r["x"], y=r["y"], iters=[r["iters"], r["iters_x"], r["iters_y"]], hpwl=hpwl,
                    occ=occ, overflow=overflow)
    with torch.cuda.stream(s.stream):
        s.wx.copy_(s.x)
        s.wy.copy_(s.y)
        ctx.build_b2b_dev(s.x, s.y, alpha, s.ax, s.ay, s.fx, s.fy)
        ctx.solve_dev(s.wx, s.wy, TOL, MAX_ITER, s.info)
        ctx.hpwl_dev(s.wx, s.wy, s.scal[0:1])
        ctx.occupancy_dev(s.wx, s.wy, s.occ, s.scal[1:2])
    # the info's residuals are stopping diagnostics; its counts are outputs
    return dict(x=s.wx, y=s.wy, iters=[s.info[2], s.info[3], s.info[4]], hpwl=s.scal[0],
                occ=s.occ, overflow=s.scal[1])


def _run_fast(s):
    ctx, alpha = s.ctx, s.case["alpha"]
    if s.host:
        ctx.build_b2b(s.x, s.y, alpha, s.ax, s.ay, s.fx, s.fy)
        if s.case["coarse"] == 3:
            s.net.prepare_coarse(ctx)
        r = ctx.solve_mixed(s.x, s.y, TOL)
        hpwl = ctx.hpwl(r["x"], r["y"])
        occ, overflow = ctx.occupancy(r["x"], r["y"])
        return dict(x=r["x"], y=r["y"], iters=list(r["inner"]), hpwl=hpwl, occ=occ,
                    overflow=overflow)
    with torch.cuda.stream(s.stream):
        s.wx.copy_(s.x)
        s.wy.copy_(s.y)
        ctx.build_b2b_dev(s.x, s.y, alpha, s.ax, s.ay, s.fx, s.fy)
        if s.case["coarse"] == 3:
            s.net.prepare_coarse_dev(ctx)
        ctx.solve_mixed_dev(s.wx, s.wy, TOL, info=s.info)
        ctx.hpwl_dev(s.wx, s.wy, s.scal[0:1])
        ctx.occupancy_dev(s.wx, s.wy, s.occ, s.scal[1:2])
    return dict(x=s.wx, y=s.wy, iters=[s.info[2], s.info[3]], hpwl=s.scal[0], occ=s.occ,
                overflow=s.scal[1])


def _run_legalize(s):
    if s.host:
        x, y = s.ctx.lal(s.x, s.y)
        return dict(x=x, y=y)
    with torch.cuda.stream(s.stream):
        s.wx.copy_(s.x)
        s.wy.copy_(s.y)
        s.ctx.lal_dev(s.wx, s.wy)
    return dict(x=s.wx, y=s.wy)


def _run_batch(s):
    s.batch.reset_x()
    s.batch.solve(TOL, MAX_ITER, 1)
    res = s.batch.results()
    return dict(x=[s.batch.get_x(i, n) for i, n in enumerate(s.rows)],
                iters=np.array([r["iters"] for r in res]),
                status=np.array([[r["outer"], r["status"]] for r in res]))


def _run_spmv(s):
    with torch.cuda.stream(s.stream):
        s.ctx.spmv_dev(0, s.vx, s.wx)
        s.ctx.spmv_dev(1, s.vy, s.wy)
    return dict(x=s.wx, y=s.wy)


def _run_train(s):
    lx, gx = s.net.coarse_loss_grad(s.ctx, 0, s.ex)
    ly, gy = s.net.coarse_loss_grad(s.ctx, 1, s.ey)
    return dict(loss=[lx, ly], grad=[gx, gy])


def _run_kraftwerk2(s):
    with torch.cuda.stream(s.stream):
        s.wx.copy_(s.x)
        s.wy.copy_(s.y)
        s.ctx.build_kraftwerk2_dev(s.wx, s.wy, True, s.fx, s.fy)
        s.ctx.kraftwerk2_adjust_dev(None, None, None, 1e-12)
        s.ctx.solve_dev(s.wx, s.wy, 1e-5, 150, s.info)
    return dict(x=s.wx, y=s.wy, iters=[s.info[2], s.info[3], s.info[4]])


# ---- what a pass cannot do without -----------------------------------------------


def _netlist_size(case):
    """Expected pins and off-diagonal entries per axis of a case's design (the
    degree law's means; a net of p pins has 2 p - 3 springs)."""
    mean = synth.mean_degree()
    pins = case["nets"] * mean
    return pins, case["nets"] * 2 * (2 * mean - 3)


def work(case):
    """Inputs read once and outputs written once; the systems, which exist only
    between the calls of a step, count as one write and one read. Operations:
    two per entry and axis of every product a solve needs, at about 150
    iterations of the FP64 solve and 20 of the preconditioned one."""
    if case["kind"] == "batch":
        nbytes = flops = 0.0
        for k in range(case["netlists"]):
            n = synth.spec_batch_member(case["first"] + k).num_movable
            m = n * 13 / 12 * 8.0
            nbytes += 2 * (12.0 * m + 28 * n + 16 * n)
            flops += 2 * 2 * m * 60
        return {"bytes": nbytes, "flops": flops}
    n = case["cells"]
    pins, m = _netlist_size(case)
    if case["kind"] == "spmv":
        return {"bytes": 2 * (12.0 * m + 4 * n + 24 * n), "flops": 4.0 * m + 2 * n}
    if case["kind"] == "legalize":
        return {"bytes": 56.0 * n, "flops": 20.0 * n * math.log2(n)}
    if case["kind"] == "train":
        # three layers, forward and twice that backward, of 64-wide products
        per = 3 * (case["nets"] * 64 * 64 + 2 * n * 64 * 64) + n * 64 * 24
        return {"bytes": 2 * (8.0 * pins + 12 * m + 8 * n * case["vectors"]), "flops": 12.0 * per}
    build = 28.0 * pins + 8 * case["nets"] + 2 * 2 * (12 * m + 20 * n) + 32 * n
    iters = 20 if case["kind"] == "fast_step" else 150
    return {"bytes": build + 32.0 * n + 8 * case.get("bins", 0) ** 2,
            "flops": 2.0 * iters * (2 * m + 12 * n)}


# ---- the same results from plain torch in 64 bits ----------------------------------


class _System:
    """One axis system in plain torch: CSR with the diagonal apart."""

    def __init__(self, n, row, col, val, diag, rhs):
        self.n, self.diag, self.rhs = n, diag, rhs
        order = torch.argsort(row * n + col, stable=True)
        rp = torch.zeros(n + 1, dtype=torch.int64, device=row.device)
        rp[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
        self.off = torch.sparse_csr_tensor(rp, col[order], val[order], (n, n),
                                           dtype=torch.float64)
        self.rowabs = torch.zeros(n, dtype=torch.float64, device=row.device).index_add_(
            0, row, val.abs())

    def mul(self, v):
        return self.diag * v + torch.mv(self.off, v)


class _Exact:
    """A flattened netlist as torch tensors."""

    def __init__(self, nl):
        dev = "cuda" if torch.cuda.is_available() else "cpu"

        def t(a):
            return torch.from_numpy(np.ascontiguousarray(a)).to(dev)
        self.dev, self.nl, self.n, self.N = dev, nl, nl.num_movable, nl.num_nets
        self.deg = t(np.diff(nl.net_start))
        self.start = t(nl.net_start[:-1])
        self.net = torch.repeat_interleave(torch.arange(self.N, device=dev), self.deg)
        self.cell = t(nl.pin_cell).long()
        self.var = t(nl.var_of_vertex).long()[self.cell]
        self.mov = self.var >= 0
        self.fixed = (t(nl.fixed_x)[self.cell], t(nl.fixed_y)[self.cell])
        self.off = (t(nl.off_x), t(nl.off_y))
        self.weight = t(nl.net_weight)
        self.t = t

    def at(self, axis, pos):
        return torch.where(self.mov, pos[self.var.clamp(min=0)], self.fixed[axis])

    def extremes(self, v, last_high):
        """Pin index of each net's lowest and highest pin (first of equals;
        with last_high the last of the highest)."""
        P = v.numel()
        idx = torch.arange(P, device=v.device)
        inf = torch.full((self.N,), math.inf, dtype=torch.float64, device=v.device)
        lov = inf.scatter_reduce(0, self.net, v, "amin")
        hiv = (-inf).scatter_reduce(0, self.net, v, "amax")
        big = torch.full((self.N,), P, dtype=torch.int64, device=v.device)
        lo = big.scatter_reduce(0, self.net, torch.where(v == lov[self.net], idx, P), "amin")
        if last_high:
            hi = (big * 0 - 1).scatter_reduce(0, self.net,
                                              torch.where(v == hiv[self.net], idx, -1), "amax")
        else:
            hi = big.scatter_reduce(0, self.net, torch.where(v == hiv[self.net], idx, P), "amin")
        return lo, hi

    def b2b(self, axis, pos, alpha, anchor, floor, kraftwerk2=False):
        v = self.at(axis, pos) + self.off[axis]
        lo, hi = self.extremes(v, kraftwerk2)
        P = v.numel()
        idx = torch.arange(P, device=v.device)
        base = (2.0 if kraftwerk2 else 1.0) * self.weight / (self.deg - 1).clamp(min=1).double()
        ok = (lo != hi)[self.net] & (self.deg[self.net] > 1)
        to_lo = ok & (idx != lo[self.net])
        to_hi = ok & (idx != lo[self.net]) & (idx != hi[self.net])
        a = torch.cat([idx[to_lo], idx[to_hi]])
        b = torch.cat([lo[self.net[to_lo]], hi[self.net[to_hi]]])
        a, b = torch.cat([a, b]), torch.cat([b, a])
        keep = self.mov[a]
        if kraftwerk2:
            keep &= ~(self.mov[b] & (self.cell[a] == self.cell[b]))
        a, b = a[keep], b[keep]
        w = base[self.net[a]] / (v[a] - v[b]).abs().clamp(min=floor)
        row = self.var[a]
        diag = torch.zeros(self.n, dtype=torch.float64, device=v.device).index_add_(0, row, w)
        off = self.off[axis]
        term = torch.where(self.mov[b], w * (off[b] - off[a]), w * (v[b] - off[a]))
        rhs = torch.zeros_like(diag).index_add_(0, row, term)
        if alpha > 0:
            wa = alpha / (pos - anchor).abs().clamp(min=floor)
            diag = diag + wa
            rhs = rhs + wa * anchor
        diag = diag.clamp(min=1e-12)
        m = self.mov[b]
        return _System(self.n, row[m], self.var[b[m]], -w[m], diag, rhs)

    def hpwl(self, x, y):
        total = 0.0
        for axis, pos in ((0, x), (1, y)):
            v = self.at(axis, pos) + self.off[axis]
            inf = torch.full((self.N,), math.inf, dtype=torch.float64, device=v.device)
            span = (-inf).scatter_reduce(0, self.net, v, "amax") - inf.scatter_reduce(
                0, self.net, v, "amin")
            total = total + span[self.deg > 1].sum()
        return total

    def occupancy(self, g, x, y):
        w, h = self.t(self.nl.width), self.t(self.nl.height)

        def index(c, o, d, k):
            return ((c - o) / d).clamp(min=0.0, max=float(k) - 1e-9).long()
        ix = index(x + 0.5 * w, g.origin_x, g.dx, g.nx)
        iy = index(y + 0.5 * h, g.origin_y, g.dy, g.ny)
        occ = torch.zeros(g.size, dtype=torch.float64, device=x.device).index_add_(
            0, iy * g.nx + ix, w * h)
        over = (occ - g.density_limit * self.t(g.avail)).clamp(min=0.0).sum() / g.total_avail
        return occ, over


def _pcg(S, x, tol, max_iter):
    """Jacobi-PCG: the iterate after the first step whose residual is <= tol."""
    x = x.clone()
    r = S.rhs - S.mul(x)
    z = r / S.diag
    bn = float(S.rhs.norm())
    p, rho = z.clone(), float(r @ z)
    it, resid = 0, float(r.norm()) / bn if bn > 0 else 0.0
    while it < max_iter and bn > 0 and resid > tol:
        it += 1
        ap = S.mul(p)
        pap = float(p @ ap)
        if not pap > 0:
            break
        a = rho / pap
        x += a * p
        r -= a * ap
        z = r / S.diag
        resid = float(r.norm()) / bn
        nxt = float(r @ z)
        if not nxt > 0:
            break
        p = z + (nxt / rho) * p
        rho = nxt
    return x, it


def _exact_axes(E, v, case, floors, tol, max_iter=MAX_ITER, kraftwerk2=False):
    out = []
    for axis, (p, q) in enumerate((("x", "ax"), ("y", "ay"))):
        pos = E.t(v[p])
        S = E.b2b(axis, pos, 0.0 if kraftwerk2 else case.get("alpha", 0.2),
                  None if kraftwerk2 else E.t(v[q]), floors[axis], kraftwerk2)
        out.append(_pcg(S, pos, tol, max_iter))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "legalize":
        return None  # a sequential algorithm: no plain torch form, and no rounding of its own
    if kind == "batch":
        xs = []
        for nl, x, y, ax, ay in _batch_inputs(case, seed):
            E = _Exact(nl)
            sol = _exact_axes(E, dict(x=x, y=y, ax=ax, ay=ay), case, nl.floors(), 1e-12)
            xs += [sol[0][0].cpu(), sol[1][0].cpu()]
        return dict(x=xs, iters=None, status=None)
    nl, v = _inputs(case, seed)
    E = _Exact(nl)
    floors = nl.floors()
    if kind == "spmv":
        return {k: E.b2b(axis, E.t(v[k]), 0.2, E.t(v["a" + k]), floors[axis]).mul(E.t(v["v" + k]))
                for axis, k in enumerate("xy")}
    if kind == "kraftwerk2":
        (x, kx), (y, ky) = _exact_axes(E, v, case, floors, 1e-5, 150, True)
        return dict(x=x, y=y, iters=[max(kx, ky), kx, ky])
    if kind == "train":
        got = [_exact_train(E, case, v, axis, floors) for axis in (0, 1)]
        return dict(loss=[float(g[0]) for g in got], grad=[g[1] for g in got])
    # the FP64 step's outputs are the iterate that meets the tolerance, the
    # refined solve's approximate the solution itself
    fp64 = kind == "step"
    (x, kx), (y, ky) = _exact_axes(E, v, case, floors, TOL if fp64 else 1e-12)
    occ, over = E.occupancy(grid.build_grid(nl, case["bins"], 1.0), x, y)
    return dict(x=x, y=y, iters=[max(kx, ky), kx, ky] if fp64 else None, hpwl=E.hpwl(x, y),
                occ=occ, overflow=over)


def _exact_train(E, case, v, axis, floors):
    """Loss and gradient of the learned coarse vector by automatic
    differentiation: a three-layer mean-aggregation network over the cell-net
    graph (hidden 64) on topology features, a 16-wide head per system, and the
    share of the test vectors' A-energy outside the predicted vector."""
    shapes = [(8, 64), (64,)]
    for _ in range(3):
        shapes += [(64, 64), (64,), (64, 64), (64, 64), (64,)]
    shapes += [(64, 16), (18, 16), (16,), (16,), (1,)]
    flat = E.t(np.load(COARSE_WEIGHTS).astype(np.float64)).requires_grad_(True)
    par, o = [], 0
    for s in shapes:
        k = math.prod(s)
        par.append(flat[o:o + k].reshape(s))
        o += k
    n, N, deg = E.n, E.N, E.deg.double()
    mc, mn = E.var[E.mov], E.net[E.mov]

    def count(i, k, w=None):
        w = torch.ones(i.numel(), dtype=torch.float64, device=i.device) if w is None else w
        return torch.zeros(k, dtype=torch.float64, device=i.device).index_add_(0, i, w)
    nmov, npin = count(mn, N), count(mc, n)
    area = E.t(E.nl.width * E.nl.height)
    fixed = deg - nmov
    invp = torch.where(npin > 0, 1.0 / npin.clamp(min=1), 0.0)
    inv = torch.where(deg >= 2, 1.0 / (deg - 1).clamp(min=1), 0.0)
    feat = torch.stack([torch.ones_like(npin), npin / 8, count(mc, n, (nmov - 1)[mn]) * invp / 8,
                        count(mc, n, fixed[mn]) * invp / 4,
                        count(mc, n, (fixed > 0).double()[mn]) * invp,
                        count(mc, n, inv[mn]) * invp,
                        torch.where(area > 0, area.clamp(min=1e-300).log() / 8, 0.0),
                        torch.log1p(npin) / 2], 1)

    def mean(h, src, dst, k, cnt):
        out = torch.zeros(k, h.shape[1], dtype=torch.float64, device=h.device)
        return out.index_add(0, dst, h[src]) / cnt.clamp(min=1)[:, None]
    h = torch.relu(feat @ par[0] + par[1])
    for layer in range(3):
        wa, ba, wb, wc, bb = par[2 + 5 * layer:7 + 5 * layer]
        e = torch.relu(mean(h, mc, mn, N, nmov) @ wa + ba)
        h = torch.relu(h @ wb + mean(e, mn, mc, n, npin) @ wc + bb)
    p = h @ par[17]
    k = "xy"[axis]
    S = E.b2b(axis, E.t(v[k]), case["alpha"], E.t(v["a" + k]), floors[axis])
    logd = S.diag.log()
    u = torch.cat([p, (S.rowabs / S.diag)[:, None], (logd - logd.mean())[:, None]], 1)
    z = torch.nn.functional.softplus(torch.relu(u @ par[18] + par[19]) @ par[20] + par[21][0])
    es = E.t(v["e" + k])
    ae = torch.stack([S.mul(e) for e in es])
    az = S.mul(z.detach())
    # z^T A z with A symmetric: its gradient is 2 A z
    q = 2 * (z @ az) - float(z.detach() @ az)
    loss = (1 - (ae @ z) ** 2 / (q * (es * ae).sum(1))).mean()
    loss.backward()
    return loss.detach(), flat.grad.float()
