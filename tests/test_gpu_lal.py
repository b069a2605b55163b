"""Look-ahead legalization on the GPU (ktg_lal) against the reference's own
LookAheadLegalizer (oracle/_ref, RefDesign.lal) and the Python restatement
(oracle/lal_ref.py).

Bar: bit-identical positions. Designs: seeded tiny designs with macros (the
restatement and the reference both check), and a 12k-cell design whose cells
start in a tight cluster, so that one region holds every cell and the long
segment sort (chunks + merge passes) runs; uniform starts give many small
clusters and batches. Each case runs with blocks of up to 2048 cells
finished in one CTA (the default), with every level run level by level
(lal_subtree_cells = 0), and with the hand-off at 64 cells; and with the
area sums read off exact integer prefixes (the default for these integer
areas) as well as summed sequentially (lal_exact_sums = 0)."""
import resource

import numpy as np
import pytest

import oracle
from oracle import lal_ref
from ktplace_b200 import grid, netlist, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True, scope="module")
def big_stack():
    # the reference's recursion wants more than the default main-thread stack
    try:
        resource.setrlimit(resource.RLIMIT_STACK, (resource.RLIM_INFINITY, resource.RLIM_INFINITY))
    except (ValueError, OSError):
        pass


def clustered(raw, n, seed, spread):
    """Lower-left positions around the die centre (normal, `spread` of the
    die's extent), so the centre bins are far over their room."""
    rng = np.random.default_rng(seed)
    lx, ly, ux, uy = raw.die
    x = 0.5 * (lx + ux) + spread * (ux - lx) * rng.standard_normal(n)
    y = 0.5 * (ly + uy) + spread * (uy - ly) * rng.standard_normal(n)
    return x, y


def run_gpu(ctx, nl, bins, density, x, y, subtree=2048, exact=1, **opts):
    ctx.set_option("lal_subtree_cells", subtree)
    ctx.set_option("lal_exact_sums", exact)
    ctx.upload_netlist(nl)
    ctx.set_grid(grid.build_grid(nl, bins, density))
    ctx.set_free_space(grid.build_free_space(nl))
    return ctx.lal(x, y, **opts)


def run_oracle(nl, bins, density, x, y, **opts):
    g = grid.build_grid(nl, bins, density)
    fs = grid.build_free_space(nl)
    rows = lal_ref.free_rows(fs.row_y, fs.row_span, fs.spans)
    gd = dict(origin=(g.origin_x, g.origin_y), dx=g.dx, dy=g.dy, nx=g.nx, ny=g.ny, avail=g.avail)
    L = lal_ref.LAL(nl.width, nl.height, gd, rows, nl.obstacles, nl.die, g.density_limit, **opts)
    px, py = L.legalize(x, y)
    return np.array(px), np.array(py)


@pytest.mark.parametrize("exact", [1, 0])
@pytest.mark.parametrize("subtree", [2048, 0, 64])
@pytest.mark.parametrize("seed,cells,macros,bins,density,start", [
    (2, 400, 3, 16, 1.0, "uniform"),
    (5, 900, 4, 24, 1.0, "cluster"),
    (7, 600, 0, 8, 0.8, "uniform"),
    (9, 700, 2, 12, 0.9, "cluster"),
])
def test_lal_tiny_bit_exact(seed, cells, macros, bins, density, start, subtree, exact, gpu_ctx):
    raw = synth.generate(synth.spec_tiny(seed=seed, macros=macros, cells=cells, nets=cells + 30))
    nl = netlist.flatten(raw)
    if start == "uniform":
        x, y = synth.seed_positions(raw, nl.num_movable, seed + 10)
    else:
        x, y = clustered(raw, nl.num_movable, seed + 10, 0.08)
    gx, gy = run_gpu(gpu_ctx, nl, bins, density, x, y, subtree, exact)
    ox, oy = run_oracle(nl, bins, density, x, y)
    assert np.array_equal(gx, ox) and np.array_equal(gy, oy)
    assert np.mean(gx != x) > 0.1  # legalization did move cells
    if oracle.ref_available():
        ref = oracle.RefDesign.from_netlist(nl)
        ref.grid(bins, density)
        rx, ry = ref.lal(x, y)
        assert np.array_equal(gx, rx) and np.array_equal(gy, ry)


@pytest.mark.parametrize("subtree", [2048, 0])
@pytest.mark.parametrize("opts", [dict(max_level=6, min_cells_to_split=2, stripe_area_fraction=0.05),
                                  dict(max_level=30, min_cells_to_split=0, stripe_area_fraction=0.3),
                                  # many stripes: the one-CTA path runs out of stripe slots
                                  # below the top level and hands the blocks back
                                  dict(max_level=20, min_cells_to_split=4,
                                       stripe_area_fraction=0.002)])
def test_lal_options(opts, subtree, gpu_ctx):
    raw = synth.generate(synth.spec_tiny(seed=3, macros=2, cells=500, nets=530))
    nl = netlist.flatten(raw)
    x, y = clustered(raw, nl.num_movable, 21, 0.1)
    gx, gy = run_gpu(gpu_ctx, nl, 16, 1.0, x, y, subtree, **opts)
    ox, oy = run_oracle(nl, 16, 1.0, x, y, max_level=opts["max_level"],
                        min_cells=opts["min_cells_to_split"],
                        stripe_fraction=opts["stripe_area_fraction"])
    assert np.array_equal(gx, ox) and np.array_equal(gy, oy)


@pytest.mark.parametrize("subtree,exact", [(2048, 1), (0, 1), (2048, 0)])
@pytest.mark.parametrize("start", ["uniform", "cluster"])
def test_lal_12k_matches_reference(start, subtree, exact, gpu_ctx):
    if not oracle.ref_available():
        pytest.skip("reference library not built")
    raw = synth.generate(synth.spec_small(seed=3))
    nl = netlist.flatten(raw)
    if start == "uniform":
        x, y = synth.seed_positions(raw, nl.num_movable, 5)
    else:
        x, y = clustered(raw, nl.num_movable, 5, 0.03)
    bins = grid.default_bins_per_axis(nl.num_movable)
    gx, gy = run_gpu(gpu_ctx, nl, bins, 1.0, x, y, subtree, exact)
    ref = oracle.RefDesign.from_netlist(nl)
    ref.grid(bins, 1.0)
    rx, ry = ref.lal(x, y)
    assert np.array_equal(gx, rx) and np.array_equal(gy, ry)


def test_lal_no_overflow_only_clamps(gpu_ctx):
    """Nothing overfilled: positions only clamped to the die."""
    raw = synth.generate(synth.spec_tiny(seed=4, cells=200, nets=220))
    nl = netlist.flatten(raw)
    x, y = synth.seed_positions(raw, nl.num_movable, 1)
    x = x.copy()
    x[:5] = raw.die[2] + 50.0  # outside the die, but their bin is not overfilled
    gx, gy = run_gpu(gpu_ctx, nl, 4, 1.0, x, y)
    ox, oy = run_oracle(nl, 4, 1.0, x, y)
    assert np.array_equal(gx, ox) and np.array_equal(gy, oy)


def test_lal_stats_count_the_work(gpu_ctx):
    raw = synth.generate(synth.spec_tiny(seed=5, macros=4, cells=900, nets=930))
    nl = netlist.flatten(raw)
    x, y = clustered(raw, nl.num_movable, 15, 0.08)
    run_gpu(gpu_ctx, nl, 24, 1.0, x, y)
    st = gpu_ctx.lal_stats()
    assert st["batches"] >= 1 and st["regions"] >= st["batches"]
    assert st["levels"] >= 1 and st["syncs"] >= 2 and st["ms_total"] > 0.0


def test_lal_requires_free_space(gpu_ctx):
    from ktplace_b200.gpu import KtgError
    raw = synth.generate(synth.spec_tiny(seed=4, cells=100, nets=110))
    nl = netlist.flatten(raw)
    gpu_ctx.upload_netlist(nl)
    gpu_ctx.set_grid(grid.build_grid(nl, 8, 1.0))
    x, y = synth.seed_positions(raw, nl.num_movable, 1)
    if getattr(gpu_ctx, "_fs", None) is None:
        with pytest.raises(KtgError):
            gpu_ctx.lal(x, y)
    with pytest.raises(KtgError):
        gpu_ctx.lal(x, y, stripe_area_fraction=0.0)


def test_simpl_mirror_legalizes_in_place(gpu_ctx):
    """simpl.LookAheadLegalizer reads like the reference's (simpl_placer.cc:
    299-310): built from the grid, the free space and the options, legalize()
    updates x and y in place."""
    from ktplace_b200 import simpl
    raw = synth.generate(synth.spec_tiny(seed=5, macros=4, cells=900, nets=930))
    nl = netlist.flatten(raw)
    x, y = clustered(raw, nl.num_movable, 15, 0.08)
    gpu_ctx.set_option("lal_subtree_cells", 2048)
    gpu_ctx.set_option("lal_exact_sums", 1)
    gpu_ctx.upload_netlist(nl)
    legalizer = simpl.LookAheadLegalizer(gpu_ctx, grid.build_grid(nl, 24, 1.0),
                                         grid.build_free_space(nl), simpl.SimplOptions())
    px, py = x.copy(), y.copy()
    legalizer.legalize(px, py)
    ox, oy = run_oracle(nl, 24, 1.0, x, y)
    assert np.array_equal(px, ox) and np.array_equal(py, oy)


@pytest.mark.parametrize("subtree", [0, 2048])
@pytest.mark.parametrize("kind", ["uneven_rows", "many_spans", "many_obstacles"])
def test_lal_profile_branches(kind, subtree, gpu_ctx):
    """Free spaces that take the other branch of the level-by-level kernels:
    rows whose heights do not sum exactly (heights added in order), more steps
    and edges than one round of a CTA takes, more obstacle cuts than it sorts
    in shared memory. Bit-identical positions, as everywhere."""
    raw = synth.generate(synth.spec_tiny(seed=8, macros=2, cells=420, nets=450))
    nl = netlist.flatten(raw)
    x, y = clustered(raw, nl.num_movable, 31, 0.15)
    g = grid.build_grid(nl, 8, 1.0)
    fs = grid.build_free_space(nl)
    rng = np.random.default_rng(4)
    lx, ly, ux, uy = fs.die
    if kind == "uneven_rows":
        edge = np.concatenate([[0.0], np.cumsum(rng.uniform(11.0, 13.0, fs.row_y.shape[0]))])
        fs.row_y = np.stack([edge[:-1], edge[1:]], 1)
    elif kind == "many_spans":
        cut = np.linspace(lx, ux, 421)
        per = np.stack([cut[:-1], cut[1:] - 0.03], 1)
        fs.spans = np.concatenate([per + 0.001 * r for r in range(fs.row_y.shape[0])])
        fs.row_span = np.arange(fs.row_y.shape[0] + 1, dtype=np.int64) * per.shape[0]
    else:
        ox, oy = rng.uniform(lx, ux, 2300), rng.uniform(ly, uy, 2300)
        fs.obstacles = np.stack([ox, oy, ox + 0.5, oy + 0.5], 1)
    gpu_ctx.set_option("lal_subtree_cells", subtree)
    gpu_ctx.set_option("lal_exact_sums", 1)
    gpu_ctx.upload_netlist(nl)
    gpu_ctx.set_grid(g)
    gpu_ctx.set_free_space(fs)
    gx, gy = gpu_ctx.lal(x, y)
    gpu_ctx.set_option("lal_subtree_cells", 2048)
    gd = dict(origin=(g.origin_x, g.origin_y), dx=g.dx, dy=g.dy, nx=g.nx, ny=g.ny, avail=g.avail)
    L = lal_ref.LAL(nl.width, nl.height, gd, lal_ref.free_rows(fs.row_y, fs.row_span, fs.spans),
                    fs.obstacles, fs.die, g.density_limit)
    ox, oy = L.legalize(x, y)
    assert np.array_equal(gx, np.array(ox)) and np.array_equal(gy, np.array(oy))
    assert np.mean(gx != x) > 0.1


@pytest.mark.parametrize("exact", [1, 0])
@pytest.mark.parametrize("cells,subtree", [(2047, 0), (2048, 0), (2049, 0), (2049, 2048),
                                           (4096, 0), (4097, 2048), (6150, 2048)])
def test_lal_level_sorts_at_tile_edges(cells, subtree, exact, gpu_ctx):
    """Level-by-level blocks around one tile of the sort (2048 keys), two and
    three, with many equal centres, and centres a few ulp apart whose distances
    from the cutline round to the same value: those fill by index."""
    raw = synth.generate(synth.spec_tiny(seed=cells, macros=2, cells=cells, nets=cells + 30))
    nl = netlist.flatten(raw)
    n = nl.num_movable
    rng = np.random.default_rng(cells)
    lx, ly, ux, uy = raw.die
    x = lx + 0.12 * (ux - lx) * np.abs(rng.standard_normal(n))
    y = 0.5 * (ly + uy) + 0.08 * (uy - ly) * rng.standard_normal(n)
    x = np.where(rng.random(n) < 0.3, np.round(x / 8.0) * 8.0, x)
    near = rng.random(n) < 0.3
    x[near] = lx + 2.0 + np.spacing(4.0) * rng.integers(0, 60, int(near.sum()))
    gx, gy = run_gpu(gpu_ctx, nl, 8, 1.0, x, y, subtree=subtree, exact=exact)
    gpu_ctx.set_option("lal_subtree_cells", 2048)
    gpu_ctx.set_option("lal_exact_sums", 1)
    ox, oy = run_oracle(nl, 8, 1.0, x, y)
    assert np.array_equal(gx, ox) and np.array_equal(gy, oy)
    assert np.mean(gx != x) > 0.1


@pytest.mark.parametrize("cells,macros,rows,seed,spread", [(60000, 150, 400, 2, 0.05),
                                                           (60000, 150, 400, 2, 0.2),
                                                           (100000, 250, 500, 3, 0.25)])
def test_lal_handed_off_blocks(cells, macros, rows, seed, spread, gpu_ctx):
    """Blocks whose halves go to other CTAs, with macros that leave some halves
    with too few cells to split: bit-identical to the level-by-level path,
    whichever halves are handed off."""
    raw = synth.generate(synth.SynthSpec(num_movable=cells, num_nets=cells + 1000, num_pads=400,
                                         num_rows=rows, utilization=0.6, num_macros=macros,
                                         seed=seed))
    nl = netlist.flatten(raw)
    x, y = clustered(raw, nl.num_movable, seed, spread)
    bins = grid.default_bins_per_axis(nl.num_movable)
    want = run_gpu(gpu_ctx, nl, bins, 1.0, x, y, subtree=0)
    for _ in range(4):
        got = run_gpu(gpu_ctx, nl, bins, 1.0, x, y)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("subtree", [0, 2048])
@pytest.mark.parametrize("kind", ["lx_past_ux", "ly_past_uy", "not_a_number"])
def test_lal_obstacles_with_sides_out_of_order(kind, subtree, gpu_ctx):
    """Obstacles whose lower side lies past their upper one, or is no number,
    inside the blocks: their edges cut stripes as every obstacle's do, so the
    room for stripes has to count them."""
    raw = synth.generate(synth.spec_tiny(seed=8, macros=2, cells=420, nets=450))
    nl = netlist.flatten(raw)
    x, y = clustered(raw, nl.num_movable, 31, 0.15)
    g = grid.build_grid(nl, 8, 1.0)
    fs = grid.build_free_space(nl)
    rng = np.random.default_rng(6)
    lx, ly, ux, uy = fs.die
    px, py = rng.uniform(lx, ux, 1900), rng.uniform(ly, uy, 1900)
    swap = 0.5 * np.array([[1, 0, 0, 1], [0, 1, 1, 0], [0, 0, 1, 1]])[
        ["lx_past_ux", "ly_past_uy", "not_a_number"].index(kind)]
    fs.obstacles = np.stack([px, py, px, py], 1) + swap
    if kind == "not_a_number":
        fs.obstacles[:, 0] = np.nan
    gpu_ctx.set_option("lal_subtree_cells", subtree)
    gpu_ctx.set_option("lal_exact_sums", 1)
    gpu_ctx.upload_netlist(nl)
    gpu_ctx.set_grid(g)
    gpu_ctx.set_free_space(fs)
    try:
        gx, gy = gpu_ctx.lal(x, y)
    finally:
        gpu_ctx.set_option("lal_subtree_cells", 2048)
    gd = dict(origin=(g.origin_x, g.origin_y), dx=g.dx, dy=g.dy, nx=g.nx, ny=g.ny, avail=g.avail)
    L = lal_ref.LAL(nl.width, nl.height, gd, lal_ref.free_rows(fs.row_y, fs.row_span, fs.spans),
                    fs.obstacles, fs.die, g.density_limit)
    ox, oy = L.legalize(x, y)
    assert np.array_equal(gx, np.array(ox)) and np.array_equal(gy, np.array(oy))
    assert np.mean(gx != x) > 0.1


@pytest.mark.parametrize("subtree", [0, 2048])
def test_lal_rows_that_start_at_no_number(subtree, gpu_ctx):
    """Rows whose start is no number break the order that the row searches rely
    on, so a half box can find more of them than its block: the room for its
    profile has to hold. Positions stay finite and inside the die."""
    raw = synth.generate(synth.spec_tiny(seed=8, macros=2, cells=900, nets=950))
    nl = netlist.flatten(raw)
    x, y = clustered(raw, nl.num_movable, 31, 0.15)
    g = grid.build_grid(nl, 8, 1.0)
    fs = grid.build_free_space(nl)
    lx, ly, ux, uy = fs.die
    rows = 4000
    edge = np.linspace(ly, uy, rows + 1)
    fs.row_y = np.stack([edge[:-1], edge[1:]], 1)
    fs.row_y[np.random.default_rng(3).integers(0, rows, rows // 3), 0] = np.nan
    fs.spans = np.tile([[lx, ux]], (rows, 1))
    fs.row_span = np.arange(rows + 1, dtype=np.int64)
    gpu_ctx.set_option("lal_subtree_cells", subtree)
    gpu_ctx.set_option("lal_exact_sums", 1)
    gpu_ctx.upload_netlist(nl)
    gpu_ctx.set_grid(g)
    gpu_ctx.set_free_space(fs)
    try:
        gx, gy = gpu_ctx.lal(x, y)
    finally:
        gpu_ctx.set_option("lal_subtree_cells", 2048)
    assert np.all((gx >= lx) & (gx <= ux) & (gy >= ly) & (gy <= uy))
    assert np.mean(gx != x) > 0.1


def piled(raw, n, seed, ulps):
    """Centres within `ulps` ulp of one x, far from the cutline: thousands of them
    at each rounded distance."""
    rng = np.random.default_rng(seed)
    lx, ly, ux, uy = raw.die
    x = lx + 2.0 + np.spacing(4.0) * rng.integers(0, ulps, n)
    y = 0.5 * (ly + uy) + 0.1 * (uy - ly) * rng.standard_normal(n)
    return x, y


@pytest.mark.parametrize("exact", [1, 0])
@pytest.mark.parametrize("subtree", [0, 2048])
def test_lal_long_runs_of_one_distance(subtree, exact, gpu_ctx):
    raw = synth.generate(synth.spec_tiny(seed=12, macros=2, cells=5200, nets=5230))
    nl = netlist.flatten(raw)
    x, y = piled(raw, nl.num_movable, 3, 60)
    far = np.random.default_rng(4).random(nl.num_movable) < 0.2
    x[far] = clustered(raw, nl.num_movable, 5, 0.2)[0][far]
    gx, gy = run_gpu(gpu_ctx, nl, 8, 1.0, x, y, subtree=subtree, exact=exact)
    gpu_ctx.set_option("lal_subtree_cells", 2048)
    gpu_ctx.set_option("lal_exact_sums", 1)
    ox, oy = run_oracle(nl, 8, 1.0, x, y)
    assert np.array_equal(gx, ox) and np.array_equal(gy, oy)


def test_lal_long_runs_cost_no_square(gpu_ctx):
    """A pile of 150k cells takes at most the time of two legalizations with one
    centre for all of them: only the levels with such runs sort and fill again."""
    raw = synth.generate(synth.SynthSpec(num_movable=150000, num_nets=151000, num_pads=400,
                                         num_rows=500, utilization=0.6, num_macros=0, seed=5))
    nl = netlist.flatten(raw)
    bins = grid.default_bins_per_axis(nl.num_movable)
    ms = {}
    for ulps in (1, 60):
        x, y = piled(raw, nl.num_movable, 7, ulps)
        took = []
        for _ in range(4):
            run_gpu(gpu_ctx, nl, bins, 1.0, x, y)
            took.append(gpu_ctx.lal_stats()["ms_total"])
        ms[ulps] = min(took[1:])
    print(ms)
    assert ms[60] <= 2.0 * ms[1], ms


@pytest.mark.parametrize("cells", [700, 1300, 1900])
def test_lal_halves_go_to_other_ctas(cells, gpu_ctx):
    """The queue is used: every region is one block of the first launch, so more
    one-CTA blocks than regions are halves that were handed off. Without the
    level-by-level path in between, and bit-identical to it."""
    raw = synth.generate(synth.spec_tiny(seed=cells, macros=2, cells=cells, nets=cells + 30))
    nl = netlist.flatten(raw)
    x, y = clustered(raw, nl.num_movable, 3, 0.03)
    want = run_gpu(gpu_ctx, nl, 16, 1.0, x, y, subtree=0)
    gx, gy = run_gpu(gpu_ctx, nl, 16, 1.0, x, y)
    st = gpu_ctx.lal_stats()
    assert st["big_levels"] == 0 and st["subtree_handed_back"] == 0
    assert st["subtree_blocks"] > st["regions"], st
    assert np.array_equal(gx, want[0]) and np.array_equal(gy, want[1])


def test_lal_scratch_of_a_small_design(port_built):
    """A design whose blocks keep a few CTAs busy takes scratch for those, not for
    one on every SM (0.8 MB each)."""
    import torch
    from ktplace_b200.gpu import Context
    raw = synth.generate(synth.spec_tiny(seed=5, macros=2, cells=300, nets=330))
    nl = netlist.flatten(raw)
    x, y = clustered(raw, nl.num_movable, 3, 0.03)
    taken = []
    for _ in range(2):  # the first one also loads the kernels
        with Context(0) as ctx:
            before = torch.cuda.mem_get_info()[0]
            run_gpu(ctx, nl, 16, 1.0, x, y)
            assert ctx.lal_stats()["subtree_blocks"] >= 1
            taken.append(before - torch.cuda.mem_get_info()[0])
    assert taken[1] <= 48 * 2**20, taken


@pytest.mark.parametrize("subtree", [0, 300, 2048])
@pytest.mark.parametrize("cells,seed", [(600, 5), (2500, 6)])
def test_lal_rows_that_overlap(cells, seed, subtree, gpu_ctx):
    """Rows in order of their starts whose ends are not: a search by row end finds
    the oracle's row only over all rows, not over those that a block can meet.
    Bit-identical positions on every path."""
    raw = synth.generate(synth.spec_tiny(seed=seed, macros=2, cells=cells, nets=cells + 30))
    nl = netlist.flatten(raw)
    x, y = clustered(raw, nl.num_movable, 31, 0.15)
    g = grid.build_grid(nl, 8, 1.0)
    fs = grid.build_free_space(nl)
    lx, ly, ux, uy = fs.die
    rng = np.random.default_rng(seed)
    rows = 150
    start = np.linspace(ly, uy, rows + 1)[:-1]
    fs.row_y = np.stack([start, start + rng.uniform(0.1, 3.0, rows) * (uy - ly) / rows], 1)
    fs.spans = np.sort(rng.uniform(lx, ux, (rows, 4)), axis=1).reshape(-1, 2)
    fs.row_span = 2 * np.arange(rows + 1, dtype=np.int64)
    assert np.any(np.diff(fs.row_y[:, 1]) < 0)
    gpu_ctx.set_option("lal_subtree_cells", subtree)
    gpu_ctx.set_option("lal_exact_sums", 1)
    gpu_ctx.upload_netlist(nl)
    gpu_ctx.set_grid(g)
    gpu_ctx.set_free_space(fs)
    try:
        gx, gy = gpu_ctx.lal(x, y)
    finally:
        gpu_ctx.set_option("lal_subtree_cells", 2048)
    gd = dict(origin=(g.origin_x, g.origin_y), dx=g.dx, dy=g.dy, nx=g.nx, ny=g.ny, avail=g.avail)
    L = lal_ref.LAL(nl.width, nl.height, gd, lal_ref.free_rows(fs.row_y, fs.row_span, fs.spans),
                    fs.obstacles, fs.die, g.density_limit)
    ox, oy = L.legalize(x, y)
    assert np.array_equal(gx, np.array(ox)) and np.array_equal(gy, np.array(oy))
    assert np.mean(gx != x) > 0.1
