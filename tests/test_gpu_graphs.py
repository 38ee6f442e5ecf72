"""Captured steps start from either ping-pong buffer: calls of an odd number of steps alternate between two
graphs, calls with other counts or parameters in between replace them, and every sequence equals the same
steps one by one."""
import numpy as np
import pytest

from openaerolab_alpha_01_b200 import _capi as capi
from openaerolab_alpha_01_b200.cases import entropic_taylor_green_case, sphere_channel_case
from openaerolab_alpha_01_b200.solver import Geometry, Level

pytestmark = pytest.mark.gpu

CALLS = [[1, 1, 1, 1], [3, 3, 2, 3, 3], [5, 1, 5, 1], [2, 2, 3]]


def compare(make, params, calls):
    a, b = make(), make()
    for i, n in enumerate(calls):
        p = capi.StepParams.from_buffer_copy(params)
        if i == len(calls) - 1:
            p.tau = params.tau + 0.05  # new parameters on a parity that already has a graph
        a.execute_timestep_batch(p, n)
        for _ in range(n):
            b.perform_timestep(p)
    for x, y in zip(a.state(), b.state()):
        assert np.array_equal(x, y)
    a.close()
    b.close()


@pytest.mark.parametrize("calls", CALLS)
@pytest.mark.parametrize("operator", ["cumulant", "entropic"])
def test_odd_calls_equal_single_steps(oal, operator, calls):
    case = (sphere_channel_case(40, 24, 24, diameter=6.0, centre_x=12.0, re=100.0) if operator == "cumulant"
            else entropic_taylor_green_case(16))
    g = Geometry(case.dom)

    def make():
        L = Level(g, operator, storage="f16" if operator == "cumulant" else "f32")
        L.init_equilibrium(case.rho, case.vel)
        return L

    compare(make, case.params, calls)
    g.close()


@pytest.mark.parametrize("calls", CALLS)
def test_odd_hierarchy_calls_equal_single_steps(oal, calls):
    from openaerolab_alpha_01_b200.amr import Hierarchy, blocks_in_box, level_taus, refine
    from openaerolab_alpha_01_b200.solver import build_box, default_step_params
    coarse = build_box(5, 4, 4)
    doms = [coarse, refine(coarse, blocks_in_box(coarse, (16, 8, 8), (24, 24, 24)))]
    P = [default_step_params(tau=t, c_wale=0.2, u_inlet=0.05) for t in level_taus(0.53, 2)]
    trees = [Hierarchy(doms, storage="f32") for _ in range(2)]
    r = np.random.default_rng(3)
    for l, d in enumerate(doms):
        vel = 0.05 + 0.005 * r.standard_normal((3, d.n_blocks, 512))
        for t in trees:
            t.level(l).init_equilibrium(np.ones((d.n_blocks, 512)), vel)
    for n in calls:
        trees[0].advance(P, n)
        for _ in range(n):
            trees[1].advance(P, 1)
    for l in range(2):
        for x, y in zip(trees[0].level(l).state(), trees[1].level(l).state()):
            assert np.array_equal(x, y)
    for t in trees:
        t.close()


def two_levels(n_trees=1):
    from openaerolab_alpha_01_b200.amr import Hierarchy, blocks_in_box, level_taus, refine
    from openaerolab_alpha_01_b200.solver import build_box, default_step_params
    coarse = build_box(5, 4, 4)
    doms = [coarse, refine(coarse, blocks_in_box(coarse, (16, 8, 8), (24, 24, 24)))]
    P = [default_step_params(tau=t, c_wale=0.2, u_inlet=0.05) for t in level_taus(0.53, 2)]
    trees = [Hierarchy(doms, storage="f32") for _ in range(n_trees)]
    r = np.random.default_rng(3)
    for l, d in enumerate(doms):
        vel = 0.05 + 0.005 * r.standard_normal((3, d.n_blocks, 512))
        for t in trees:
            t.level(l).init_equilibrium(np.ones((d.n_blocks, 512)), vel)
    return doms, P, trees


# (coarse steps, outlet setting before them): on, changed and off between calls of counts that have a
# captured graph from either buffer
ON, CHANGED, OFF = dict(p_target=1.0 / 3.0), dict(p_target=0.34, sigma_relax=0.5, all_blocks=True), dict(enabled=False)
OUTLET = [[(1, None), (1, None), (1, ON), (1, None), (1, CHANGED), (1, None), (1, OFF), (1, None)],
          [(2, ON), (2, None), (2, CHANGED), (2, OFF), (2, None), (2, ON)],
          [(3, ON), (1, None), (3, CHANGED), (3, None), (1, OFF), (3, None), (3, None)]]


@pytest.mark.parametrize("calls", OUTLET)
def test_hierarchy_calls_see_the_outlet_as_it_is_set(oal, calls):
    from openaerolab_alpha_01_b200.amr import Hierarchy
    doms, P, (tree,) = two_levels()
    outlet = OFF
    for n, change in calls:
        if change is not None:
            outlet = change
            tree.level(0).set_nscbc(**change)
        fresh = Hierarchy(doms, storage="f32")  # the same state and outlet, no captured steps
        for l in range(2):
            fresh.level(l).set_state(*tree.level(l).state())
        fresh.level(0).set_nscbc(**outlet)
        tree.advance(P, n)
        fresh.advance(P, n)
        for l in range(2):
            for x, y in zip(tree.level(l).state(), fresh.level(l).state()):
                assert np.array_equal(x, y), (n, change, l)
        fresh.close()
    tree.close()


@pytest.mark.parametrize("calls", [[1, 1, 1], [1, 1, 1, 1, 1], [3, 3, 3]])
def test_hierarchy_with_steps_of_a_refined_level_between(oal, calls):
    """A refined level stepped on its own interpolates from the parent as the last coarse step left it, whether
    that step was captured or replayed; the coarse steps after it start from the buffer it ended on."""
    _, P, (a, b) = two_levels(2)
    for n in calls:
        a.advance(P, n)
    b.advance(P, sum(calls))
    for _ in range(2):
        for t in (a, b):
            t.level(1).perform_timestep(P[1])
        a.level(1).execute_timestep_batch(P[1], 2)
        for _ in range(2):
            b.level(1).perform_timestep(P[1])
        a.advance(P, 1)
        b.advance(P, 1)
        for l in range(2):
            for x, y in zip(a.level(l).state(), b.level(l).state()):
                assert np.array_equal(x, y)
    a.close()
    b.close()
