"""The B2B build's tiles (64 rows, 256 pins and 1,024 edges at a time) against
a plain restatement in the reference's order (simpl_lss.cc:11-114 and
kraftwerk2_placer.cc:328-410), bit for bit: row counts around a tile, a row with
hundreds of pins, bound pins of a net longer than a tile's edges, rows without
pins, nets that list a cell twice."""
import dataclasses

import numpy as np
import pytest

from ktplace_b200 import netlist, synth

pytestmark = pytest.mark.gpu


def design(n, seed):
    raw = synth.generate(synth.spec_tiny(seed=seed, macros=0, cells=n, nets=n + 8, pads=8))
    rng = np.random.default_rng(seed)
    movable = np.nonzero(~raw.fixed)[0]
    fixed = np.nonzero(raw.fixed)[0]
    nets = [movable]                                              # one over every cell
    nets += [np.array([movable[0], rng.choice(movable)]) for _ in range(300)]  # a hub's pins
    nets += [rng.choice(movable[: max(1, n - n // 8)], rng.integers(2, 7)) for _ in range(n)]
    nets += [np.concatenate([rng.choice(movable, 2), rng.choice(fixed, 2)]) for _ in range(8)]
    pins = np.concatenate(nets).astype(raw.pin_cell.dtype)
    start = np.concatenate([[0], np.cumsum([len(k) for k in nets])]).astype(raw.net_start.dtype)
    return dataclasses.replace(
        raw, net_start=start, pin_cell=pins, pin_fox=rng.uniform(-2.0, 2.0, len(pins)),
        pin_foy=rng.uniform(-2.0, 2.0, len(pins)), net_weight=rng.uniform(0.5, 2.0, len(nets)))


def restated(nl, pos, axis, alpha, anchor, floor, kraftwerk2):
    fixed, off = (nl.fixed_x, nl.off_x) if axis == 0 else (nl.fixed_y, nl.off_y)
    var = nl.var_of_vertex[nl.pin_cell]
    own = np.where(var >= 0, pos[np.maximum(var, 0)], fixed[nl.pin_cell])
    at = own + off
    row_ptr, col, val, diag, rhs = [0], [], [], [], []
    for i in range(nl.num_movable):
        dg = rh = np.float64(0.0)
        for e in range(nl.pin_start[i], nl.pin_start[i + 1]):
            k, q = nl.pin_net[e], nl.pin_q[e]
            s, t = nl.net_start[k], nl.net_start[k + 1]
            if t - s < 2:
                continue
            lo = int(np.argmin(at[s:t]))
            hi = int(np.argmax(at[s:t]))
            if kraftwerk2:
                hi = int(t - s - 1 - np.argmax(at[s:t][::-1]))
            if lo == hi:
                continue
            base = nl.net_weight[k] / np.float64(t - s - 1)
            base = 2.0 * base if kraftwerk2 else base
            others = [j for j in range(t - s) if j != q] if q in (lo, hi) else [lo, hi]
            mine = at[s + q] - pos[i]
            for j in others:
                p = s + j
                if kraftwerk2 and var[p] == i:
                    continue
                w = base / max(abs(at[s + q] - at[p]), floor)
                dg = dg + w
                if var[p] >= 0:
                    col.append(var[p])
                    val.append(-w)
                    rh = rh + (w * (off[p] - off[s + q]) if kraftwerk2
                               else w * ((at[p] - own[p]) - mine))
                else:
                    rh = rh + w * (at[p] - (off[s + q] if kraftwerk2 else mine))
        if alpha > 0.0 and not kraftwerk2:
            w = alpha / max(abs(pos[i] - anchor[i]), floor)
            dg = dg + w
            rh = rh + w * anchor[i]
        row_ptr.append(len(col))
        diag.append(dg if kraftwerk2 else max(dg, 1e-12))
        rhs.append(rh)
    return dict(row_ptr=row_ptr, col=col, val=val, diag=diag, rhs=rhs)


@pytest.mark.parametrize("kraftwerk2", [False, True])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 257, 1100])
def test_build_at_tile_edges(n, kraftwerk2, gpu_ctx):
    nl = netlist.flatten(design(n, 40 + n), kraftwerk2=kraftwerk2)
    n = nl.num_movable
    rng = np.random.default_rng(n)
    x, y, ax, ay = rng.uniform(0.0, 500.0, (4, n))
    gpu_ctx.upload_netlist(nl)
    if kraftwerk2:
        gpu_ctx.build_kraftwerk2(x, y, True, 3.0, 2.0)
    else:
        gpu_ctx.build_b2b(x, y, 0.3, ax, ay, 3.0, 2.0)
    for axis, (pos, anchor, floor) in enumerate(((x, ax, 3.0), (y, ay, 2.0))):
        want = restated(nl, pos, axis, 0.3, anchor, floor, kraftwerk2)
        got = gpu_ctx.system(axis)
        m = want["row_ptr"][-1]
        for k in ("row_ptr", "diag", "rhs"):
            assert np.array_equal(got[k], np.asarray(want[k])), (axis, k)
        for k in ("col", "val"):
            assert np.array_equal(got[k][:m], np.asarray(want[k])), (axis, k)


def test_pins_listed_twice(gpu_ctx):
    """A cell may list a pin more than once; each listing adds its edges to the
    row, beyond what the nets' pins alone would give."""
    raw = design(65, 9)
    fixed = np.nonzero(raw.fixed)[0].astype(raw.pin_cell.dtype)
    pads = np.tile(fixed[:2], 200)  # nets of fixed pins: room for the listings
    starts = raw.net_start[-1] + 2 * np.arange(1, 201)
    zeros = np.zeros(len(pads))
    raw = dataclasses.replace(
        raw, net_start=np.concatenate([raw.net_start, starts.astype(raw.net_start.dtype)]),
        pin_cell=np.concatenate([raw.pin_cell, pads]),
        pin_fox=np.concatenate([raw.pin_fox, zeros]), pin_foy=np.concatenate([raw.pin_foy, zeros]),
        net_weight=np.concatenate([raw.net_weight, np.ones(200)]))
    nl = netlist.flatten(raw)
    n = nl.num_movable
    times = np.where(np.arange(len(nl.pin_net)) % 3 == 0, 2, 1)
    cell = np.repeat(np.repeat(np.arange(n), np.diff(nl.pin_start)), times)
    nl.pin_net, nl.pin_q = np.repeat(nl.pin_net, times), np.repeat(nl.pin_q, times)
    nl.pin_start = np.concatenate([[0], np.cumsum(np.bincount(cell, minlength=n))])
    x, y, ax, ay = np.random.default_rng(2).uniform(0.0, 500.0, (4, n))
    gpu_ctx.upload_netlist(nl)
    gpu_ctx.build_b2b(x, y, 0.3, ax, ay, 3.0, 2.0)
    for axis, (pos, anchor, floor) in enumerate(((x, ax, 3.0), (y, ay, 2.0))):
        want = restated(nl, pos, axis, 0.3, anchor, floor, False)
        got = gpu_ctx.system(axis)
        for k, v in want.items():
            assert np.array_equal(got[k], np.asarray(v)), (axis, k)


@pytest.mark.parametrize("nets", [2047, 2048, 2049, 4097])
def test_bound_pins_download(nets, gpu_ctx):
    """The first lowest and the first highest pin of every net."""
    raw = design(64, 3)
    rng = np.random.default_rng(nets)
    pins = rng.choice(np.nonzero(~raw.fixed)[0], (nets, 3))
    raw = dataclasses.replace(
        raw, net_start=(3 * np.arange(nets + 1)).astype(raw.net_start.dtype),
        pin_cell=pins.ravel().astype(raw.pin_cell.dtype), pin_fox=rng.uniform(-2.0, 2.0, 3 * nets),
        pin_foy=rng.uniform(-2.0, 2.0, 3 * nets), net_weight=np.ones(nets))
    nl = netlist.flatten(raw, kraftwerk2=True)  # (pins of one cell stay apart)
    n = nl.num_movable
    x, y = rng.uniform(0.0, 500.0, (2, n))
    gpu_ctx.upload_netlist(nl)
    gpu_ctx.build_b2b(x, y, 0.0, None, None, 3.0, 2.0)
    for axis, (pos, off) in enumerate(((x, nl.off_x), (y, nl.off_y))):
        at = (pos[nl.var_of_vertex[nl.pin_cell]] + off).reshape(-1, 3)
        lo, hi = gpu_ctx.bound_pins(axis)
        assert nl.num_nets == nets
        assert np.array_equal(lo, np.argmin(at, 1)) and np.array_equal(hi, np.argmax(at, 1))
