"""Non-coherent loads (__ldg) need data that nothing writes while the kernel
lives. The passes of an update are launched while the pass before them, which
writes what they read, may still run, so none of them may use one."""
import os
import re

import what_irregularity_costs_b200 as package

CSRC = os.path.join(os.path.dirname(package.__file__), "csrc")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//.*", "", f.read())


def test_passes_launched_early_use_coherent_loads():
    early = [f for f in sorted(os.listdir(CSRC)) if f.endswith(".cu") and "launch_after(" in _code(f)]
    assert early == ["band_kernels.cu", "finish_kernels.cu"]
    # Helpers of the shared header that load through the read-only path.
    header = _code("tsdf_device.cuh")
    helpers = [m.group(1) for m in re.finditer(r"__forceinline__ \w+ (\w+)\([^)]*\) \{(?:(?!\n\}).)*?__ldg", header, re.S)]
    assert helpers == ["weight_at", "mean_from"]
    for name in early:
        for load in ["__ldg", "ld.global.nc"] + helpers:
            assert not re.search(r"\b" + re.escape(load) + r"\b", _code(name)), f"{load} in {name}"
