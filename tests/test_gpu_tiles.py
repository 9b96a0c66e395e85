"""The tiled solve of systems too large to be resident, against the solve
graph: bit for bit on the same systems after 0 and 1 iterations, which take no
sum over rows (test_gpu_resident.py states why later ones may differ in the
last bits); on steps the same substeps, and geometry within four solve
tolerances (two solves of one system may differ by that)."""

import numpy as np
import pytest

from microsimulator_b200 import abi, workloads
from microsimulator_b200.backend import B200Backend
from microsimulator_b200.sweep import ColonyBatch
from microsimulator_b200.types import (
    ContactDynamicsParameters,
    ContactSolveParameters,
    ContactSystem,
    GrowthLoadResponse,
)
from microsimulator_b200.world import WorldState
from tests.systems import LAWS, mixed_system, multipliers_for

pytestmark = pytest.mark.gpu


@pytest.fixture
def forms(backend):
    yield backend
    backend.set_relaxation(B200Backend.RELAXATION_AUTOMATIC)


def step_both(backend, world, constraints=None, dt=0.002, tiled=True, **parameters):
    p = ContactDynamicsParameters(overlap_tolerance=5e-4, **parameters)
    results = []
    ran = []
    for form in (B200Backend.RELAXATION_AUTOMATIC, B200Backend.RELAXATION_GRAPH):
        backend.set_relaxation(form)
        stepped = world.copy()
        result = backend.advance_contact_dynamics(stepped, constraints, dt, p)
        results.append((stepped, result.report))
        ran.append(set(backend.last_step_solve_forms()))
        if form == B200Backend.RELAXATION_AUTOMATIC and tiled:
            assert any(name.startswith("tiles") for name in ran[0])
            # The timing hook runs on the system of the last solve, by its form.
            timed = backend.profile_iterations(2)
            assert timed["bodies"] == len(world) and timed["rows"] == backend.last_step_solves()["rows"][-1]
    assert ran[1] == {"slots"}
    (a, ra), (b, rb) = results
    assert ra.substeps == rb.substeps and ra.halvings == rb.halvings
    assert np.max(np.abs(a.geometry() - b.geometry())) <= 4 * p.overlap_tolerance
    return ra


def neighbours_system(seed: int, bodies: int, rows: int, law) -> tuple[ContactSystem, np.ndarray]:
    """A mixed system whose pair rows join bodies at most 20 apart along a
    hidden order (returned), so that most rows lie within a tile."""
    system = mixed_system(seed, bodies, rows, law)
    rng = np.random.default_rng(seed + 1)
    order = rng.permutation(bodies)
    pairs = system.rows["second_slot"] != abi.INVALID_SLOT
    first = rng.integers(0, bodies, rows)
    second = np.clip(first + rng.integers(1, 21, rows) * rng.choice([-1, 1], rows), 0, bodies - 1)
    second = np.where(second == first, (first + 1) % bodies, second)
    system.rows["first_slot"] = order[first]
    system.rows["second_slot"] = np.where(pairs, order[second], abi.INVALID_SLOT)
    return system, order


def solve_both_ways(backend, system, order, blocks, initial, iterations):
    parameters = ContactSolveParameters(1e-9, iterations)
    tiled = backend.solve_by_tiles(system, order, blocks, initial, parameters)
    form = backend.last_step_solve_forms()[-1]
    backend.set_relaxation(B200Backend.RELAXATION_GRAPH)
    return tiled, backend.solve_contact_forces(system, initial, parameters), form


# One tile (its rows all within it, no boundary rows), a last tile of one body,
# of all but one; drift and constraint rows in each.
@pytest.mark.parametrize("bodies,rows", [(3, 2), (5, 7), (255, 500), (256, 256), (257, 260), (1000, 1000), (5119, 5000)])
@pytest.mark.parametrize("blocks", [1, 2, 3, 4])
@pytest.mark.parametrize("law", range(3))
def test_agrees_with_the_graph(forms, bodies, rows, blocks, law):
    system, order = neighbours_system(bodies + law, bodies, rows, LAWS[law])
    initial = multipliers_for(system, rows)
    for iterations in (0, 1):
        tiled, graph, form = solve_both_ways(forms, system, order, blocks, initial, iterations)
        assert form == f"tiles {blocks}"
        assert tiled.report == graph.report
        assert np.array_equal(tiled.multipliers, graph.multipliers)
    tiled, graph, _ = solve_both_ways(forms, system, order, blocks, initial, 6)
    assert tiled.report.iterations == graph.report.iterations
    assert np.max(np.abs(tiled.multipliers - graph.multipliers)) <= 1e-5 * np.max(np.abs(graph.multipliers))


# Rows between random bodies, nearly all of them between tiles: more guests
# than the two that a thread fetches ahead, tiles with an odd first row.
@pytest.mark.parametrize("bodies,rows,fit", [(2000, 2000, 4), (3001, 9000, 3), (2000, 8000, 2), (2049, 12000, 1)])
def test_many_rows_between_tiles(forms, bodies, rows, fit):
    system = mixed_system(bodies, bodies, rows, LAWS[1])
    order = np.random.default_rng(rows).permutation(bodies)
    initial = multipliers_for(system, 1)
    for iterations in (0, 1):
        tiled, graph, form = solve_both_ways(forms, system, order, fit, initial, iterations)
        assert form == f"tiles {fit}"
        assert tiled.report == graph.report
        assert np.array_equal(tiled.multipliers, graph.multipliers)


# A last tile of one body, of all its bodies, of all but one.
@pytest.mark.parametrize("cells", [768 * 256 + 1, 640 * 256, 641 * 256 - 1])
@pytest.mark.parametrize("law", [0, 2])
def test_steps_by_tiles(forms, cells, law):
    world = workloads.jammed(cells, seed=cells)
    step_both(forms, world, growth=GrowthLoadResponse(law, 0.0, 0.2, 3.0))


def test_walls_by_tiles(forms):
    world, walls = workloads.trap_colony(180_000, seed=3)
    world.position_y *= np.float32(1.15)  # into the side walls
    step_both(forms, world, walls)


@pytest.mark.parametrize("cells", [20_000, 180_000])
def test_a_body_of_many_rows(forms, cells):
    """A long capsule over a colony touches more than 62 cells: neither the
    resident nor the tiled solve holds it, and the graph does."""
    world = workloads.jammed(cells, seed=4)
    middle = float(world.position_x.mean())
    fields = {name: getattr(world, name) for name in WorldState.FIELDS}
    long = WorldState.from_arrays(
        np.stack([np.append(fields["position_x"], middle), np.append(fields["position_y"], middle),
                  np.append(fields["position_z"], 0.995)], axis=1),
        np.stack([np.append(fields["direction_x"], 1.0), np.append(fields["direction_y"], 0.0),
                  np.append(fields["direction_z"], 0.0)], axis=1),
        np.append(fields["lengths"], 120.0), 0.5, growth_rates=0.5)
    step_both(forms, long, tiled=False)
    forms.set_relaxation(B200Backend.RELAXATION_AUTOMATIC)
    forms.advance_contact_dynamics(long.copy(), None, 0.002, ContactDynamicsParameters(overlap_tolerance=5e-4))
    assert "slots" in forms.last_step_solve_forms()


def forms_of(backend, world, dt=0.002, tolerance=5e-4):
    backend.set_relaxation(B200Backend.RELAXATION_AUTOMATIC)
    backend.advance_contact_dynamics(world.copy(), None, dt, ContactDynamicsParameters(overlap_tolerance=tolerance))
    return list(zip(backend.last_step_solve_forms(), backend.last_step_solves()["iterations"].tolist()))


def test_solves_that_gain_nothing_by_tiles_go_by_slot(forms):
    """Sparse colonies (under two rows a body) and solves of up to 4
    iterations; after a long solve the next starts by tiles."""
    sparse = forms_of(forms, workloads.jammed(330_000, area_fraction=0.3, seed=2))
    assert max(its for _, its in sparse) > 4
    assert {form for form, _ in sparse} == {"slots"}
    dense = workloads.jammed(170_001, seed=6)
    seen = set()
    for dt, tolerance in ((0.02, 5e-4), (0.002, 0.4)):
        log = forms_of(forms, dense, dt, tolerance)
        for k, (form, its) in enumerate(log):
            tiled = its > 4 or (k > 0 and log[k - 1][1] >= 64)
            assert form.startswith("tiles") == tiled, (k, log)
            seen.add(tiled)
    assert seen == {True, False}


def hold_all_but(free_bytes):
    torch = pytest.importorskip("torch")
    torch.cuda.synchronize()
    return torch.empty(torch.cuda.mem_get_info()[0] - free_bytes, dtype=torch.uint8, device="cuda")


def test_tiles_do_without_memory_that_others_need(backend):
    """Where the device has no room for the tiles, the solves go by slot (the
    start's bits); the tiles that a context holds are given back when another
    of its buffers needs the room."""
    torch = pytest.importorskip("torch")
    cells = 400_000
    world = workloads.jammed(cells, seed=7)
    p = ContactDynamicsParameters(overlap_tolerance=5e-4)
    system = mixed_system(2, cells, cells, LAWS[0])
    initial = multipliers_for(system, 2)
    expected = backend.evaluate_contact_response(system, initial)

    def step(b, form):
        b.set_relaxation(form)
        stepped = world.copy()
        b.advance_contact_dynamics(stepped, None, 0.002, p)
        return stepped.geometry()

    with B200Backend(0) as b:
        by_slot = step(b, B200Backend.RELAXATION_GRAPH)
        step(b, B200Backend.RELAXATION_GRAPH)  # rows and the last step's rows have their buffers
        held = hold_all_but(64 << 20)
        without = step(b, B200Backend.RELAXATION_AUTOMATIC)
        assert set(b.last_step_solve_forms()) == {"slots"}
        assert np.array_equal(without, by_slot)
        del held
        torch.cuda.empty_cache()
        tiled = step(b, B200Backend.RELAXATION_AUTOMATIC)
        assert any(form.startswith("tiles") for form in b.last_step_solve_forms())
        held = hold_all_but(16 << 20)
        got = b.evaluate_contact_response(system, initial)  # 64 MB of records
        del held
        torch.cuda.empty_cache()
        assert np.array_equal(got.velocities, expected.velocities) and np.array_equal(got.loads, expected.loads)
        assert np.array_equal(step(b, B200Backend.RELAXATION_AUTOMATIC), tiled)


def test_a_copy_that_is_late_ends_the_solve(forms):
    """With no polls allowed the tiles' copies count as late: the solve ends
    with its first pass by tiles, after 4 iterations by slot (not after
    max_iterations of them, on sums that the blocks never wrote), its copies
    drained, and the next call is sound."""
    world = workloads.jammed(170_001, seed=6)
    p = ContactDynamicsParameters(overlap_tolerance=5e-4)
    forms.set_relaxation(B200Backend.RELAXATION_AUTOMATIC)
    expected = world.copy()
    forms.advance_contact_dynamics(expected, None, 0.002, p)
    forms.set_wait_limit(0)
    try:
        with pytest.raises(abi.NativeError, match="wait of the relaxation failed at iteration 5$"):
            forms.advance_contact_dynamics(world.copy(), None, 0.002, p)
    finally:
        forms.set_wait_limit()
    again = world.copy()
    forms.advance_contact_dynamics(again, None, 0.002, p)
    assert np.array_equal(again.geometry(), expected.geometry())


def test_timing_hook_times_the_system_it_reports(forms):
    """Systems loaded after a tiled solve are timed by slot: evaluated or
    bounded ones with more bodies than the tiles, whose last tile is partly
    filled.  A batch leaves no system to time."""
    cells = 170_001
    world = workloads.jammed(cells, seed=6)
    p = ContactDynamicsParameters(overlap_tolerance=5e-4)
    forms.set_relaxation(B200Backend.RELAXATION_AUTOMATIC)
    for k, call in enumerate((forms.evaluate_contact_response, forms.evaluate_contact_gaps,
                              lambda system, _: forms.contact_system_diagonal_bound(system))):
        forms.advance_contact_dynamics(world.copy(), None, 0.002, p)
        assert forms.profile_iterations(1)["bodies"] == cells
        system = mixed_system(k, cells + 255 + k, 5000 + k, LAWS[2])
        call(system, multipliers_for(system, k))
        timed = forms.profile_iterations(1)
        assert (timed["rows"], timed["bodies"]) == (5000 + k, cells + 255 + k)
    sizes = [40, 300]
    batch = ColonyBatch([workloads.sweep_colony(n, seed=n) for n in sizes], np.full(2, 1.0), np.full(2, 1.0e4))
    forms.advance_contact_dynamics_batch(batch.concatenated(), batch.counts(), batch.drag, batch.stiffness, 0.002, p)
    with pytest.raises(ValueError, match="no solved system"):
        forms.profile_iterations(1)
