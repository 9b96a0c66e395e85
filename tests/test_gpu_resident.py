"""The resident solve (the system in shared memory: one CTA, one cluster, the
whole grid) against the solve graph on the same systems.

Gaps and the residual of given multipliers take no sum over rows, and the
first step's length is 1 / bound, so after 0 and 1 iterations the two agree
bit for bit.  From the second step on the step length is a ratio of FP64 sums
taken in another order, which rounds to FP32: at most one unit in the last
place (6e-8) a step, each step moving a multiplier by at most a step length
times its gap."""

import numpy as np
import pytest

from microsimulator_b200 import abi, workloads
from microsimulator_b200.backend import B200Backend
from microsimulator_b200.sweep import ColonyBatch
from microsimulator_b200.types import ContactDynamicsParameters, ContactSolveParameters, ContactSystem
from tests.systems import LAWS, mixed_system, multipliers_for

pytestmark = pytest.mark.gpu


@pytest.fixture
def forms(backend):
    yield backend
    backend.set_relaxation(B200Backend.RELAXATION_AUTOMATIC)


def solve_both(backend, system, initial, iterations, automatic=None):
    """The automatic form's solve (which ran as `automatic`) and the graph's."""
    out, ran = [], []
    for form in (B200Backend.RELAXATION_AUTOMATIC, B200Backend.RELAXATION_GRAPH):
        backend.set_relaxation(form)
        out.append(backend.solve_contact_forces(system, initial, ContactSolveParameters(1e-9, iterations)))
        ran.append(backend.last_step_solve_forms()[-1])
    assert ran[1] == "slots" and (automatic is None or ran[0] == automatic)
    return out


# (bodies, rows): one CTA (two rows, fewer bodies than a group, a full
# group and one more, the largest), one cluster, the grid.
SIZES = [(3, 2), (7, 5), (8, 30), (9, 30), (300, 1100), (350, 1300), (2000, 4000), (9000, 21000), (20000, 40000),
         (90000, 200000)]


@pytest.mark.parametrize("bodies,rows", SIZES)
@pytest.mark.parametrize("law", range(3))
def test_agrees_with_the_graph(forms, bodies, rows, law):
    system = mixed_system(bodies + law, bodies, rows, LAWS[law])
    initial = multipliers_for(system, rows)
    form = "one cta" if rows <= 1300 else "cluster" if rows <= 21000 else "grid"
    for iterations in (0, 1):
        resident, graph = solve_both(forms, system, initial, iterations, form)
        assert resident.report == graph.report
        assert np.array_equal(resident.multipliers, graph.multipliers)
    resident, graph = solve_both(forms, system, initial, 6)
    assert resident.report.status == graph.report.status
    assert resident.report.iterations == graph.report.iterations
    scale = np.max(np.abs(graph.multipliers))
    assert np.max(np.abs(resident.multipliers - graph.multipliers)) <= 1e-5 * scale


def hub_system(degree: int, bodies: int = 400) -> ContactSystem:
    """A chain whose middle body also touches every tenth of `degree` others."""
    system = mixed_system(degree, bodies, bodies - 1, LAWS[0], walls=0.0)
    system.rows["first_slot"] = np.arange(bodies - 1)
    system.rows["second_slot"] = np.arange(1, bodies)
    hub = np.resize(system.rows, degree - 2)
    hub["first_slot"], hub["second_slot"] = bodies // 2, np.arange(degree - 2)
    system.rows = np.concatenate([system.rows, hub]).astype(abi.CONTACT_ROW_DTYPE)
    return system


@pytest.mark.parametrize("degree", [61, 62, 63, 64, 150])
def test_bodies_of_many_rows(forms, degree):
    # Up to 62 entries a body the system is resident; beyond it takes the graph.
    system = hub_system(degree)
    initial = multipliers_for(system, 3)
    resident, graph = solve_both(forms, system, initial, 1, "one cta" if degree <= 62 else "slots")
    assert resident.report == graph.report
    assert np.array_equal(resident.multipliers, graph.multipliers)


def test_empty_bodies_and_profile_hook(forms):
    # Bodies without rows are evaluated too; the timing hook goes on from the
    # resident solve's iterate.
    system = mixed_system(5, 5000, 300, LAWS[2])
    initial = multipliers_for(system, 1)
    resident, graph = solve_both(forms, system, initial, 1)
    assert np.array_equal(resident.multipliers, graph.multipliers)
    forms.set_relaxation(B200Backend.RELAXATION_AUTOMATIC)
    forms.solve_contact_forces(system, initial, ContactSolveParameters(1e-9, 1))
    assert forms.profile_iterations(2)["rows"] == 300


def test_waits_that_run_out_fail_the_call(forms):
    """With no polls allowed the grid's CTAs do not wait for one another: the
    solve and a batch's gangs (whose CTAs then count as late, not as misfits)
    fail, and the next calls are sound."""
    system = mixed_system(1, 20000, 40000, LAWS[0])
    initial = multipliers_for(system, 1)
    parameters = ContactSolveParameters(1e-9, 3)
    sizes = [300, 12000, 9000]
    batch = ColonyBatch([workloads.sweep_colony(n, seed=n) for n in sizes], np.full(3, 1.0), np.full(3, 1.0e4))
    p = ContactDynamicsParameters(overlap_tolerance=5e-4)

    def step():
        cells = batch.concatenated()
        forms.advance_contact_dynamics_batch(cells, batch.counts(), batch.drag, batch.stiffness, 0.002, p)
        return cells.geometry()

    forms.set_relaxation(B200Backend.RELAXATION_AUTOMATIC)
    step()
    expected = forms.solve_contact_forces(system, initial, parameters).multipliers, step()
    forms.set_wait_limit(0)
    try:
        with pytest.raises(abi.NativeError, match="wait of the resident solve ran out"):
            forms.solve_contact_forces(system, initial, parameters)
        with pytest.raises(abi.NativeError, match="wait of the batched resident solve ran out"):
            step()
    finally:
        forms.set_wait_limit()
    assert np.array_equal(forms.solve_contact_forces(system, initial, parameters).multipliers, expected[0])
    assert np.array_equal(step(), expected[1])


@pytest.mark.parametrize("cells", [13000, 30000])
@pytest.mark.parametrize("flat", [True, False])
def test_steps_in_spatial_order(forms, cells, flat):
    """Steps whose solves spread over the grid in spatial order (a colony in
    the plane, one whose cells share one x, where every key is of y alone):
    within four solve tolerances, as two solves of one system may differ."""
    world = workloads.jammed(cells, seed=cells)
    if not flat:
        world.position_z, world.position_x = world.position_x.copy(), np.zeros(cells, np.float32)
        world.direction_z, world.direction_x = world.direction_x.copy(), np.zeros(cells, np.float32)
    p = ContactDynamicsParameters(overlap_tolerance=5e-4)
    results = []
    for form in (B200Backend.RELAXATION_AUTOMATIC, B200Backend.RELAXATION_GRAPH):
        forms.set_relaxation(form)
        stepped = world.copy()
        report = forms.advance_contact_dynamics(stepped, None, 0.02, p).report
        results.append((stepped, report))
        assert set(forms.last_step_solve_forms()) == {"slots" if form == B200Backend.RELAXATION_GRAPH else "grid"}
    (a, ra), (b, rb) = results
    assert ra.substeps == rb.substeps and ra.halvings == rb.halvings
    assert np.max(np.abs(a.geometry() - b.geometry())) <= 4 * p.overlap_tolerance


def test_first_batch_of_a_context_runs_as_the_second(backend):
    """Gangs from the first call on, without a launch shape tuned for clusters
    that no colony needs: the same solves and the same bits."""
    sizes = [40, 900, 12000]
    batch = ColonyBatch([workloads.sweep_colony(n, seed=n) for n in sizes], np.full(3, 1.0), np.full(3, 1.0e4))
    p = ContactDynamicsParameters(overlap_tolerance=5e-4)
    results = []
    with B200Backend(0) as b:
        for call in range(3):
            if call == 2:
                b.tune_batch()
            cells = batch.concatenated()
            _, colonies = b.advance_contact_dynamics_batch(cells, batch.counts(), batch.drag, batch.stiffness, 0.002, p)
            results.append((cells.geometry(), colonies["iterations"]))
            assert set(b.last_step_solve_forms()) == {"gangs"}
    for geometry, iterations in results[1:]:
        assert np.array_equal(geometry, results[0][0])
        assert np.array_equal(iterations, results[0][1])


def test_batch_by_gangs_steps_as_by_clusters(backend):
    """Colonies held by one CTA, by gangs of several and (one body touching
    more than 62 rows) by none, against the clusters' solve: the same rows,
    geometry within four solve tolerances."""
    sizes = [1, 2, 40, 300, 900, 3000, 12000]
    worlds = [workloads.sweep_colony(n, seed=n) for n in sizes]
    star = workloads.sweep_colony(120, seed=9)
    star.position_x[:], star.position_y[:] = star.position_x * 0.02, star.position_y * 0.02
    batch = ColonyBatch([*worlds, star], np.full(8, 1.0), np.full(8, 1.0e4))
    p = ContactDynamicsParameters(overlap_tolerance=5e-4)
    counts = batch.counts()
    results, ran = [], []
    with B200Backend(0) as b:
        for form in (B200Backend.RELAXATION_AUTOMATIC, B200Backend.RELAXATION_GRAPH):
            b.set_relaxation(form)
            cells = batch.concatenated()
            report, colonies = b.advance_contact_dynamics_batch(cells, counts, batch.drag, batch.stiffness, 0.002, p)
            results.append((cells.geometry(), report, colonies))
            ran.append(set(b.last_step_solve_forms()))
    assert "gangs and clusters" in ran[0] and ran[1] == {"clusters"}
    (a, ra, ca), (g, rg, cg) = results
    assert ra.substeps == rg.substeps
    assert np.array_equal(ca["rows"], cg["rows"])
    assert np.array_equal(ca["status"], cg["status"])
    assert np.max(np.abs(a - g)) <= 4 * p.overlap_tolerance
