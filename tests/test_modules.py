"""The update passes' kernels stay out of the module that a context's creation
loads: the runtime loads a module whole, and the passes of every precision,
tile shape and place of the chains beside the persistent sweep made a process's
first context take 58 ms to create instead of 3."""
import glob
import os
import re
import subprocess

import pytest

from lceqcd_b200 import build

PASSES = re.compile(r"\b(higgs|link|link3|higgs_fin)_kernel<")


def kernels(obj):
    return [s for s in subprocess.run(["nm", "-C", obj], capture_output=True, text=True, check=True).stdout.splitlines()
            if PASSES.search(s)]


def test_pass_kernels_are_in_modules_of_their_own():
    objs = {os.path.basename(o): o for o in glob.glob(os.path.join(build.BUILD, "*.o"))}
    if "lce_update.o" not in objs:
        pytest.skip("no objects of a build here")
    for r, real in (("f32", "float"), ("f64", "double")):
        for i, place in enumerate(("table", "one", "many")):  # lce_passes.cuh: Chains
            names = kernels(objs[f"lce_passes_{r}_{place}.o"])
            assert names and all(f"<{real}, " in n for n in names)
            assert all(re.search(rf", (\(lce::Chains\))?{i}>|higgs_fin_kernel", n) for n in names), names[0]
    for name, obj in objs.items():
        if not name.startswith("lce_passes_"):
            assert not kernels(obj), name
