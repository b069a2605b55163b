"""The sliced FP64 solve (ktg_pcg_sliced.cu, the default form) at the sizes
where its layout changes: rows around the lane-count limits (8, 16, 24 entries
per lane and their doublings up to a warp per row), empty rows, blocks and
slices that are not full, one block against several, and each choice of the
vectors that live in shared memory.

Tolerances: the solve follows the reference's iteration with other summation
orders, so iteration counts are equal and solutions of these well-conditioned
systems (diagonally dominant, fewer than 40 steps) agree far below the 1e-9
that the other solve tests allow."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
TOL, SOL_RTOL = 1e-8, 1e-11


def random_system(n, lengths, seed):
    """Unsymmetric pattern is enough for the products; symmetric values keep PCG
    defined, so entry (i, j) is mirrored. lengths: wanted row lengths, cycled."""
    rng = np.random.default_rng(seed)
    want = np.resize(np.asarray(lengths), n) // 2
    rows = np.repeat(np.arange(n), want)
    cols = rng.integers(0, n, rows.shape[0])
    keep = rows != cols
    rows, cols = rows[keep], cols[keep]
    v = -rng.uniform(0.1, 1.0, rows.shape[0])
    r, c, v = np.concatenate([rows, cols]), np.concatenate([cols, rows]), np.concatenate([v, v])
    order = np.argsort(r, kind="stable")
    r, c, v = r[order], c[order], v[order]
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(r, minlength=n), out=rp[1:])
    diag = np.bincount(r, weights=-v, minlength=n) * 1.3 + rng.uniform(0.5, 1.0, n)
    return dict(row_ptr=rp, col=c.astype(np.int32), val=v, diag=diag, rhs=rng.standard_normal(n))


def check(ctx, n, lengths, seed=0):
    sx, sy = random_system(n, lengths, seed), random_system(n, lengths[::-1], seed + 1)
    rng = np.random.default_rng(seed + 2)
    x0, y0 = rng.standard_normal((2, n))
    ctx.upload_system(0, sx)
    ctx.upload_system(1, sy)
    got = ctx.solve(x0, y0, TOL, 1000)
    again = ctx.solve(x0, y0, TOL, 1000)
    ref = oracle.port_solve_both(sx, x0, sy, y0, TOL, 1000)
    assert got["iters"] == ref["iters"]
    for k in ("x", "y"):
        assert np.linalg.norm(got[k] - ref[k]) <= SOL_RTOL * np.linalg.norm(ref[k])
        assert np.array_equal(got[k], again[k])  # the same from run to run


@pytest.mark.parametrize("n", [1, 2, 31, 33, 300, 511, 512, 513, 640, 1021, 5003])
def test_sizes(n, gpu_ctx, port_built):
    check(gpu_ctx, n, [0, 2, 4, 6, 10, 20])


@pytest.mark.parametrize("lengths", [[0], [8], [9, 7], [16, 17, 1], [24, 25, 23, 48, 49],
                                     [96, 97, 2, 4], [190, 200, 390, 6, 6, 6], [800, 2, 0, 2, 4]])
@pytest.mark.parametrize("n", [450, 2050])
def test_row_lengths(n, lengths, gpu_ctx, port_built):
    check(gpu_ctx, n, lengths, seed=7)


@pytest.mark.parametrize("n", [40_009, 160_001, 290_003, 560_003, 1_050_001])
def test_vector_homes(n, gpu_ctx, port_built):
    """Wider lanes from 2,048 rows a block; 4, 2, 1 and 0 vectors in shared
    memory (about 3.8k, 7.4k and 14.1k rows a block)."""
    check(gpu_ctx, n, [2, 6, 2, 4, 8, 40], seed=3)


def test_axes_apart(gpu_ctx, port_built):
    """One axis done before the other, one that never starts (b = 0) and one
    that is not positive definite."""
    n = 2000
    sx, sy = random_system(n, [4, 8], 1), random_system(n, [4, 8], 2)
    rng = np.random.default_rng(5)
    x0, y0 = rng.standard_normal((2, n))
    for kind in ("zero", "solved", "indefinite"):
        s = dict(sy)
        y = y0.copy()
        if kind == "zero":
            s["rhs"] = np.zeros(n)
        elif kind == "solved":
            y = oracle.port_pcg_axis(sy, y0, 1e-5, 1000)["x"]
        else:
            s["val"] = -3.0 * sy["val"]
        gpu_ctx.upload_system(0, sx)
        gpu_ctx.upload_system(1, s)
        got = gpu_ctx.solve(x0, y, TOL, 200)
        ref = oracle.port_solve_both(sx, x0, s, y, TOL, 200)
        assert got["iters"] == ref["iters"], kind
        assert np.linalg.norm(got["x"] - ref["x"]) <= SOL_RTOL * np.linalg.norm(ref["x"]), kind
        scale = max(np.linalg.norm(ref["y"]), 1e-300)
        assert np.linalg.norm(got["y"] - ref["y"]) <= 1e-9 * scale, kind


@pytest.mark.parametrize("tol", [-3e-2, -1.0, 0.0])
@pytest.mark.parametrize("n", [300, 2050])
def test_tolerance_that_nothing_meets(n, tol, gpu_ctx, port_built):
    """Zero and negative tolerances run all the iterations that are allowed."""
    sx, sy = random_system(n, [2, 6, 10], 11), random_system(n, [4, 8], 12)
    x0, y0 = np.random.default_rng(13).standard_normal((2, n))
    gpu_ctx.upload_system(0, sx)
    gpu_ctx.upload_system(1, sy)
    got = gpu_ctx.solve(x0, y0, tol, 6)
    ref = oracle.port_solve_both(sx, x0, sy, y0, tol, 6)
    assert ref["iters"] == 6 and got["iters"] == 6
    for k in ("x", "y"):
        assert np.linalg.norm(got[k] - ref[k]) <= SOL_RTOL * np.linalg.norm(ref[k])


def test_scratch_follows_the_blocks(port_built):
    """The copy is padded per block of the solve, so a small design's context takes
    little memory; rows may outgrow it when the entries do not."""
    import torch
    from ktplace_b200 import netlist, synth
    from ktplace_b200.gpu import Context
    nl = netlist.flatten(synth.generate(synth.spec_tiny(seed=1, cells=300, nets=330)))
    taken = []
    for _ in range(2):  # the first one also loads the library
        with Context(0) as ctx:
            before = torch.cuda.mem_get_info()[0]
            ctx.upload_netlist(nl)
            taken.append(before - torch.cuda.mem_get_info()[0])
    assert taken[1] <= 6 * 2**20, taken
    with Context(0) as ctx:
        check(ctx, 300, [100, 200, 60])
        check(ctx, 24_001, [0, 2], seed=4)
        check(ctx, 160_001, [0, 2, 0, 0], seed=5)
        check(ctx, 300, [100, 200, 60])


@pytest.mark.parametrize("n", [9_999, 10_000, 24_003, 110_001, 720_007])
def test_solves_of_few_iterations(n, gpu_ctx, port_built):
    """Either side of the line below which a capped solve runs on the systems
    themselves: the iterates are the same ones."""
    sx, sy = random_system(n, [2, 6, 10], 21), random_system(n, [4, 8], 22)
    x0, y0 = np.random.default_rng(23).standard_normal((2, n))
    gpu_ctx.upload_system(0, sx)
    gpu_ctx.upload_system(1, sy)
    for steps in (0, 1, 2, 4, 5, 7, 8):
        got = gpu_ctx.solve(x0, y0, TOL, steps, hist_cap=8)
        ref = oracle.port_solve_both(sx, x0, sy, y0, TOL, steps)
        assert got["iters"] == ref["iters"] == steps
        for k in ("x", "y"):
            assert np.linalg.norm(got[k] - ref[k]) <= SOL_RTOL * np.linalg.norm(ref[k])


def test_few_iterations_need_no_copy(gpu_ctx, port_built):
    """A solve that may take no step costs the first residual, two and a half steps
    at most; making the sliced copy takes more than four."""
    import time
    import torch
    n = 1_000_000
    sx = random_system(n, [6, 8, 10], 31)
    gpu_ctx.upload_system(0, sx)
    gpu_ctx.upload_system(1, sx)
    x0, y0 = np.random.default_rng(32).standard_normal((2, n))
    dx, dy = torch.tensor(x0, device="cuda"), torch.tensor(y0, device="cuda")
    took = {}
    for steps in (0, 10, 20):
        for rep in range(6):
            torch.cuda.synchronize()
            t = time.perf_counter()
            gpu_ctx.solve_dev(dx, dy, 0.0, steps)
            torch.cuda.synchronize()
            if rep:
                took[steps] = min(took.get(steps, 1.0), time.perf_counter() - t)
    assert took[0] <= 2.5 * (took[20] - took[10]) / 10, took
