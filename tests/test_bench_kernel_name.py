"""The bench line names the solver kernel that the timed arm launched."""
import importlib.util
import os
from types import SimpleNamespace

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def name(tuned=None, **kw):
    spec = importlib.util.spec_from_file_location("bench_mod", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    args = dict(schedule="persistent", block_threads=0, blocks_per_sm=0, placement="", precision="fp64", parity=False)
    args.update(kw)
    if tuned is not None:
        tuned = {"chosen": dict(dict(schedule=1, block_threads=128, placement=0, min_blocks=1, cells_per_thread=1), **tuned)}
    return bench.solver_kernel_name(tuned, SimpleNamespace(**args))


@pytest.mark.parametrize("kw,start", [
    (dict(), "k_rosenbrock_wide<0> "),
    (dict(parity=True, schedule="static"), "k_rosenbrock_wide<1> "),
    (dict(placement="lu-tmem-wide", block_threads=128), "k_rosenbrock_wide<0> "),
    (dict(tuned=dict(placement=10)), "k_rosenbrock_wide<0> "),
    (dict(tuned=dict(placement=10), parity=True), "k_rosenbrock_wide<1> "),
    (dict(block_threads=128), "k_rosenbrock ("),
    (dict(blocks_per_sm=1), "k_rosenbrock ("),
    (dict(precision="fp32lu"), "k_rosenbrock ("),
    (dict(placement="lu-tmem", block_threads=256), "k_rosenbrock ("),
    (dict(tuned=dict(placement=4, block_threads=256)), "k_rosenbrock ("),
    (dict(tuned=dict(cells_per_thread=2)), "k_rosenbrock ("),
    (dict(tuned=dict(schedule=2, block_threads=256), parity=True), "k_rosenbrock_coopx_g8 "),
])
def test_kernel_name(kw, start):
    assert name(**kw).startswith(start)
