"""Failure detection without a GPU fault: a bounded wait is made to run out
(one block of a cooperative launch never arrives), the kernel reports
KTG_ERR_TIMEOUT through the status word, and the same context then solves
normally. Host-side failures (bad arguments, calls out of order) return
error codes."""
import ctypes
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(HERE, "golden"))

from cases import build_case, TOL, MAX_ITER  # noqa: E402

pytestmark = pytest.mark.gpu


def test_wait_timeout_is_reported_and_context_survives(gpu_ctx):
    from ktplace_b200 import _lib
    st = ctypes.c_int(0)
    rc = gpu_ctx.lib.ktg_selftest_wait_timeout(gpu_ctx.h, 50_000_000, ctypes.byref(st))
    assert rc == 0
    assert st.value == _lib.KTG_ERR_TIMEOUT
    raw, nl, x, y, ax, ay, alpha, _ = build_case("tiny_macros")
    gpu_ctx.upload_netlist(nl)
    fx, fy = nl.floors()
    gpu_ctx.build_b2b(x, y, alpha, ax, ay, fx, fy)
    r = gpu_ctx.solve(x, y, TOL, MAX_ITER)
    assert r["iters"] > 0 and max(r["resid"]) <= TOL


def test_host_side_errors(gpu_ctx):
    from ktplace_b200 import _lib
    from ktplace_b200._lib import KtgError
    with pytest.raises(KtgError) as e:
        gpu_ctx.set_option("pcg_lanes", 3)
    assert e.value.code == _lib.KTG_ERR_ARG
    st = ctypes.c_int(0)
    assert gpu_ctx.lib.ktg_selftest_wait_timeout(gpu_ctx.h, 0, ctypes.byref(st)) == _lib.KTG_ERR_ARG
    x = np.zeros(4)
    with pytest.raises(KtgError):
        gpu_ctx.solve_mixed(x, x, TOL, inner_tol=1.5)


def test_out_of_memory_leaves_no_system_behind(port_built):
    """A larger system that does not fit takes the smaller one with it (its arrays
    had to make way): no later call runs on what is left, and the context takes
    systems again."""
    import torch
    import oracle
    from ktplace_b200 import _lib
    from ktplace_b200._lib import KtgError
    from ktplace_b200.gpu import Context
    from test_gpu_sliced import random_system
    n = 500
    small = [random_system(n, [2, 6, 10], k) for k in (1, 2)]
    m = 8_000_000
    rng = np.random.default_rng(3)
    large = dict(row_ptr=np.linspace(0, m, n + 1).astype(np.int64),
                 col=rng.integers(0, n, m).astype(np.int32), val=np.full(m, -1e-3),
                 diag=np.full(n, 1e3), rhs=np.ones(n))
    x0, y0 = rng.standard_normal((2, n))
    ref = oracle.port_solve_both(small[0], x0, small[1], y0, TOL, 1000)
    with Context(0) as ctx:
        for axis in (0, 1):
            ctx.upload_system(axis, small[axis])
        ctx.solve(x0, y0, TOL, 1000)
        torch.cuda.empty_cache()
        room = torch.cuda.mem_get_info()[0] - 300 * 2**20
        held = torch.empty(room, dtype=torch.uint8, device="cuda")
        try:
            with pytest.raises(KtgError):
                ctx.upload_system(0, large)
            for call in (lambda: ctx.solve(x0, y0, TOL, 10), lambda: ctx.spmv(0, x0),
                         lambda: ctx.solve_mixed(x0, y0, TOL)):
                with pytest.raises(KtgError) as e:
                    call()
                assert e.value.code == _lib.KTG_ERR_STATE
        finally:
            del held
            torch.cuda.empty_cache()
        for axis in (0, 1):
            ctx.upload_system(axis, small[axis])
        got = ctx.solve(x0, y0, TOL, 1000)
        assert got["iters"] == ref["iters"]
        for k in ("x", "y"):
            assert np.linalg.norm(got[k] - ref[k]) <= 1e-9 * np.linalg.norm(ref[k])


def test_scratch_from_one_design_to_the_next():
    """The solvers' scratch stays with the context from one netlist or system to
    another where it is large enough, with the results of a fresh context, and goes
    back where it is far larger than what the next one needs."""
    import torch
    from ktplace_b200 import netlist, synth
    from ktplace_b200.gpu import Context
    from test_gpu_sliced import random_system

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    def run(ctx, design):
        if isinstance(design, list):
            n = len(design[0]["diag"])
            for axis in (0, 1):
                ctx.upload_system(axis, design[axis])
        else:
            n = design.num_movable
            ctx.upload_netlist(design)
            x, y = 100.0 * np.random.default_rng(n).random((2, n))
            ctx.build_b2b(x, y, 0.2, y, x)
        x0, y0 = np.random.default_rng(n + 1).standard_normal((2, n))
        out = []
        for precond in (0, 2):
            ctx.set_option("precond", precond)
            got = ctx.solve(x0, y0, 1e-7, 500), ctx.solve_mixed(x0, y0, 1e-6)
            out += [v for g in got for v in (g["x"], g["y"])]
        return out

    raw = [synth.generate(synth.spec_tiny(seed=k, macros=0, cells=n, nets=n + 20))
           for k, n in enumerate((300, 3000))]
    designs = [netlist.flatten(raw[0]), [random_system(20_000, [2, 6, 10], k) for k in (1, 2)],
               netlist.flatten(raw[0]), netlist.flatten(raw[1]),
               [random_system(777, [0, 4, 300], k) for k in (3, 4)], netlist.flatten(raw[0])]
    with Context(0) as ctx:
        for design in designs:
            got = run(ctx, design)
            with Context(0) as fresh:
                for a, b in zip(got, run(fresh, design)):
                    assert np.array_equal(a, b)
        n, m = 500, 30_000_000
        ctx.upload_system(0, dict(row_ptr=np.linspace(0, m, n + 1).astype(np.int64),
                                  col=np.resize(np.arange(n, dtype=np.int32), m),
                                  val=np.full(m, -1e-6), diag=np.ones(n), rhs=np.ones(n)))
        before = free()
        run(ctx, designs[0])
        assert free() - before > 1_500_000_000  # of 0.72 GB of systems, 1.2 GB of scratch
