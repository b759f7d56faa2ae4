"""Calls that step two at a time, replayed as graphs and with the set-up changed between them:
the same bits as one step per call of the same solver."""
import numpy as np
import pytest

from myfluidsimulation_b200 import workloads as W
from myfluidsimulation_b200.solvers import BC_DUCT, BC_PERIODIC, METHOD_HYBRID, METHOD_LEGACY, Solver

pytestmark = pytest.mark.gpu


def fields(dims, seed):
    rng = np.random.default_rng(seed)
    f = [(1 + 1e-3 * rng.standard_normal(dims[::-1])).astype(np.float32)]
    return f + [(0.02 * rng.standard_normal(dims[::-1])).astype(np.float32) for _ in range(3)]


def obstacles(dims, seed):
    rng = np.random.default_rng(seed)
    return W.duct_mask(*dims, (rng.random(dims[::-1]) < 0.01).astype(np.uint8))


def results(s):
    return [s.state(), *s.macros(), np.array(list(s.stats().values()))]


def run(dims, method, bc, how, script):
    s = Solver(*dims, 0.57, (1e-5, 2e-6, 0.0), method=method, bc=bc, inlet_u=0.03 if bc == BC_DUCT else 0.0)
    out = []
    for act in script(s):
        if act is None:
            out.append(results(s))
        elif how == "graph":
            s.step_graph(act)
        elif how == "call":
            s.step(act)
        else:
            for _ in range(act):
                s.step(1)
    s.close()
    return out


def same(dims, method, bc, script):
    want = run(dims, method, bc, "single", script)
    for how in ("call", "graph"):
        for a, b in zip(run(dims, method, bc, how, script), want, strict=True):
            for x, y in zip(a, b, strict=True):
                np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("dims", [(64, 24, 13), (61, 16, 20)])
@pytest.mark.parametrize("method", [METHOD_LEGACY, METHOD_HYBRID])
def test_graphs_and_changed_rates_without_solid_cells(gpu, method, dims):
    def script(s):
        s.reinit_from_host(*fields(dims, 3))
        s.enable_stats(True)
        yield from (10, 10, 10, None)
        s.set_force(-2e-5, 0.0, 1e-5)
        if method == METHOD_HYBRID:
            s.set_shear_omega(1.2)
        yield from (7, 7, 7, 7, None)      # both parities of a graph
        s.enable_stats(False)
        s.set_macro_output(False)
        yield from (8, 8)
        s.set_macro_output(True)
        s.enable_stats(True)
        yield from (6, None)
        s.reinit_from_host(*fields(dims, 4))
        yield from (9, None)

    same(dims, method, BC_PERIODIC, script)


@pytest.mark.parametrize("bc", [BC_PERIODIC, BC_DUCT])
@pytest.mark.parametrize("method", [METHOD_LEGACY, METHOD_HYBRID])
def test_masks_and_bands_changed_between_calls(gpu, method, bc):
    dims = (193, 121, 120)      # beyond L2: pairs with and without solid cells

    def script(s):
        s.reinit_from_host(*fields(dims, 5))
        s.enable_stats(True)
        assert s.step_passes(9) < 9
        yield from (9, None)
        s.set_solid_mask(obstacles(dims, 6))      # at an odd parity
        if method == METHOD_HYBRID:
            s.build_band(2)
        yield from (10, 10, None)
        s.set_solid_mask(obstacles(dims, 7))      # cells turn solid and fluid
        if method == METHOD_HYBRID:
            s.build_band(4)
            s.set_shear_omega(1.3)
        yield from (11, None)
        s.set_solid_mask(np.zeros(dims[::-1], np.uint8))
        yield from (10, None)

    same(dims, method, bc, script)
