"""The bench's line on standard output: short enough to be read back whole, with
the step's figures and the last leg's."""
import json

import bench


def full_line():
    clocks = {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "samples": 66, "reasons": ["sw_power_cap"]}
    long = [{"hpwl": 322413208.70273274 + k, "ms": 1.2345678901234567} for k in range(400)]
    line = {k: 4.187654321012345 for k in bench.HEADLINE}
    line.update(metric=bench.METRIC, unit=bench.UNIT, data="synthetic " * 8, clocks=clocks,
                config={"workload": bench.WORKLOAD, "cells": 211000, "nets": 221000,
                        "pins": 865422, "grid": 512},
                roofline={"kernel": "k" * 100, "bound": "hbm", "achieved": 2.5e3, "peak": 6.5e3,
                          "unit": "GB/s", "frac": 0.38, "peak_kind": "measured", "traffic": 3.8e9,
                          "algorithmic_bytes": 1.4e10, "note": "n" * 300, "limiter": "l" * 300},
                e2e={"value": 5.1, "unit": bench.UNIT, "h2d_bytes_per_step": 16880000,
                     "d2h_bytes_per_step": 5473224},
                cpu_baseline=None, simpl_report=long, batch={"ms_per_batch": 27.1, "all": long},
                kraftwerk2={"gpu_ms": 2.6}, bookshelf=None, lal={"gpu_ms": 12.0, "e2e_ms": 13.0},
                learned_step={"ms": 1.9, "e2e_ms": 2.4},
                solve_variants={f"variant_{k}": {"ms": 1.2345678901234567, "x": long}
                                for k in range(7)})
    return line


def test_headline_is_short_and_complete():
    line = full_line()
    out = bench.headline(line)
    assert len(json.dumps(out)) <= 3000 < len(json.dumps(line))
    for k in bench.HEADLINE:
        if k != "roofline":
            assert out[k] == line[k]
    assert out["roofline"]["frac"] == 0.38 and "limiter" not in out["roofline"]
    assert out["legs"]["batch"] == {"ms_per_batch": 27.1} and "bookshelf" not in out["legs"]
    assert len(out["legs"]["solve_ms"]) == 7


def test_nothing_but_the_headline_on_standard_output():
    import inspect
    src = inspect.getsource(bench.run_ours)
    assert src.count("print(") == 2 and "file=sys.stderr" in src
