"""Kernels launched with an early start (launch_after) run from before their wait for the
step before them, which still writes their input.  So they read what steps write with
coherent loads: no __ldg of populations, moments or adjoint fields, and no const __restrict__
parameter that the compiler could read on that path.  Flags, links and the inlet profile,
which no step writes, may be read so.  A check of the sources, on the CPU."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "myfluidsimulation_b200", "csrc")
CONSTANT = {"flags", "links", "uin"}


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def test_early_kernels_read_the_state_with_coherent_loads():
    files = ["lbm_aa.cu", "lbm_pair.cu", "lbm_push.cu", "lbm_home.cu", "lbm_adjoint.cu"]
    early = {}
    for f in files:
        for k in re.findall(r"launch_after\((\w+)", source(f)):
            early[k] = f
    assert {"aa_even", "aa_odd", "aa_odd_rows", "aa_pair", "pair_solids", "ref_push", "home_step", "adj_fwd", "adj_bwd"} <= set(early)
    for k, f in early.items():
        sig = re.search(r"__global__[^;{]*?\b%s\((.*?)\)\s*\{" % k, source(f), re.S).group(1)
        for par in sig.split(","):
            if "const" in par and "__restrict__" in par:
                assert par.split()[-1].lstrip("*") in CONSTANT, (k, par)
    for f in files + ["lbm_common.cuh", "lbm_vec.cuh"]:
        for arg in re.findall(r"__ldg\(([^;]*)", source(f)):
            assert re.match(r"(reinterpret_cast<const uint16_t\*>\()?p\.(flags|links)\b", arg), (f, arg)
