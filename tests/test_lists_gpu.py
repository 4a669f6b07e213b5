"""Steps over neighbour lists that outlive a step (calls of several mechanics
steps): the same trajectories, bit for bit, as the oracle's, which rebuilds the
mesh and searches neighbours every step. The capacity picks the launch form:
one thread per agent in small or large blocks, or several agents per thread."""
import numpy as np
import pytest

from paraphysicell_b200 import build
from paraphysicell_b200 import workloads as wl
from paraphysicell_b200.abi import PPC_ERR_ARG, PPC_ERR_TIMEOUT, AgentArrays, Mesh, Params, PPCError

from tests.gpu_util import assert_same_bins, assert_same_state, fetch, make_pair

pytestmark = pytest.mark.gpu

FORMS = {"small blocks": 0, "large blocks": 45000, "several agents per thread": 96000}


def _agents(n, dims, half, seed, capacity, fast=0.0, radius=(6.0, 10.0)):
    """Agents uniform in a box; `fast`: previous velocities that carry them
    across voxels and out of the box."""
    rng = np.random.default_rng(seed)
    mesh = Mesh.make(dims, (-half,) * 3, (half,) * 3)
    a = AgentArrays(n, dims, 2, max(capacity, n))
    a.arrays["positions"][: n * dims] = rng.uniform(-half, half, n * dims)
    a.arrays["radius"][:n] = rng.uniform(*radius, n)
    a.arrays["cell_definition_indices"][:n] = rng.integers(0, 2, n)
    a.arrays["cell_adhesion_affinities"][: 2 * n] = rng.uniform(0.2, 1.0, 2 * n)
    a.arrays["is_movable"][:n] = rng.random(n) < 0.9
    if fast:
        a.arrays["previous_velocities"][: n * dims] = rng.normal(0, fast, n * dims)
    return mesh, Params.make(dt=0.1, ndefs=2), a


def _mesh(*sims):
    """The mesh and neighbours a step starts from (the oracle's step, like the
    reference's, begins with the forces)."""
    for x in sims:
        x.update_mechanics_mesh()
        x.update_cell_neighbors()


def _run(o, d, a, calls):
    _mesh(o)
    for k in calls:
        o.step(k, 0, 0.0, 0.0)
        d.step(k)
        assert_same_state(fetch(d, a), fetch(o, a))
    o.update_mechanics_mesh()
    assert_same_bins(d, o)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("dims,n,half", [(1, 33, 200), (2, 31, 60), (2, 700, 250), (3, 1, 60), (3, 997, 120),
                                         (3, 2500, 130)])
def test_steps_over_lists_match_the_oracle(form, dims, n, half):
    """Edges of warps and blocks, sparse and dense tissue, agents that leave
    the box (removal without a rebuild) and cross voxels (terms in the order of
    the current mesh, not the lists')."""
    mesh, params, a = _agents(n, dims, half, 5 + n, FORMS[form], fast=20.0)
    o, d = make_pair(mesh, params, a)
    _run(o, d, a, (5, 12, 1, 4, 30))
    d.close()


@pytest.mark.parametrize("form", FORMS)
def test_springs_walls_and_removals(form):
    mesh, params, a = wl.scaled(wl.config3, 1500, 3)
    params.virtual_wall_at_domain_edges = 1
    b = AgentArrays(a.count, 3, 3, max(FORMS[form], a.count))
    for k, v in a.arrays.items():
        b.arrays[k][: v.size] = v
    b.arrays["flags"][[3, 700, 1499]] = 1  # removed by the first step, with their springs
    o, d = make_pair(mesh, params, b)
    _run(o, d, b, (6, 20))
    d.close()


@pytest.mark.parametrize("form", FORMS)
def test_lists_that_do_not_fit(form):
    """A clump with more agents in reach than a list holds, inside ordinary
    tissue: its agents scan the mesh."""
    mesh, params, a = _agents(900, 3, 150, 8, FORMS[form])
    rng = np.random.default_rng(9)
    a.arrays["positions"][: 3 * 400] = rng.normal(0, 3.0, 3 * 400)
    o, d = make_pair(mesh, params, a)
    _run(o, d, a, (4, 7))
    d.close()


@pytest.mark.parametrize("form", FORMS)
def test_uploads_between_calls(form):
    """Uploaded positions and velocities reach the lists: unchanged ones,
    moved ones (within and past the skin), and new radii."""
    mesh, params, a = _agents(1200, 3, 140, 21, FORMS[form])
    o, d = make_pair(mesh, params, a)
    rng = np.random.default_rng(3)
    _mesh(o)
    for shift in (0.0, 0.3, 9.0):
        o.step(6, 0, 0.0, 0.0)
        d.step(6)
        h = fetch(d, a)
        n = h.count
        h.arrays["positions"][: 3 * n] += shift * rng.uniform(-1, 1, 3 * n)
        np.clip(h.arrays["positions"], -139.0, 139.0, out=h.arrays["positions"])
        h.arrays["velocities"][: 3 * n] = rng.normal(0, shift, 3 * n)
        o.upload(h)
        d.upload_fields(h, ("positions", "previous_velocities", "velocities"))
        _run(o, d, a, (5,))
    h = fetch(d, a)
    h.arrays["radius"][: h.count] *= 1.1
    o.upload(h)
    d.upload_fields(h, ("radius",))
    _run(o, d, a, (5, 9))
    d.close()


@pytest.mark.parametrize("form", FORMS)
def test_reach_that_leaves_no_skin(form):
    """Ingestion grows radii on the device until no skin is left beside the
    voxel edge: the mesh is then rebuilt every step."""
    mesh, params, a = _agents(800, 3, 110, 31, FORMS[form], radius=(9.5, 11.0))
    f = wl.interaction_fields(a, 2, 4, scale=40.0)
    o, d = make_pair(mesh, params, a)
    _run(o, d, a, (5,))
    n = fetch(d, a).count
    for x in (o, d):
        g = f.copy()
        g.count = n
        _mesh(x)
        x.update_cell_cell_interactions(g)
        x.update_cell_container_for_mechanics()
    _run(o, d, a, (6, 5))
    d.close()


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("steps", [7, 12])
def test_reach_that_leaves_no_skin_and_goes_with_its_agents(form, steps):
    """The agents whose ingestions took the skin are removed in the first step
    of a call: the mesh rebuilt after it would leave a skin again, and the rest
    of the call sees every neighbour all the same (odd and even numbers of
    steps are left to the pass without lists)."""
    mesh, params, a = _agents(800, 3, 110, 31, FORMS[form], radius=(9.5, 11.0))
    f = wl.interaction_fields(a, 2, 4, scale=40.0)
    o, d = make_pair(mesh, params, a)
    _mesh(o, d)
    for x in (o, d):
        x.update_cell_cell_interactions(f.copy())
        x.update_cell_container_for_mechanics()
    h = fetch(d, a)
    grown = 2 * 1.25 * h["radius"] > 29.0
    assert 0 < grown.sum() < h.count // 2
    h["flags"][grown] = 1
    o.upload(h)
    d.upload_fields(h, ("flags",))
    _run(o, d, a, (steps, 5))
    assert fetch(d, a).count <= h.count - grown.sum()
    d.close()


@pytest.mark.parametrize("capacities", [(1000, 30000), (30000, 1000), (42000, 90000), (90000, 42000)])
def test_two_live_states_of_different_capacity(capacities):
    """Both states run the same kernel with shared memory by their own
    capacity, in turn."""
    pairs = []
    for k, c in enumerate(capacities):
        mesh, params, a = _agents(600, 3, 110, 41 + k, c)
        pairs.append((*make_pair(mesh, params, a), a))
        _mesh(pairs[-1][0])
    for _ in range(3):
        for o, d, a in pairs:
            o.step(5, 0, 0.0, 0.0)
            d.step(5)
            assert_same_state(fetch(d, a), fetch(o, a))
    for o, d, a in pairs:
        d.close()


@pytest.mark.parametrize("form", FORMS)
def test_agents_too_fast_for_lists(form):
    """Repulsion that throws agents past the skin at every step: the call goes
    on without lists, and the calls after it scan the mesh (many launches
    instead of a few), until calmer tissue gets lists again."""
    mesh, params, a = _agents(700, 3, 130, 61, FORMS[form])
    params.virtual_wall_at_domain_edges = 1
    a.arrays["cell_cell_repulsion_strength"][: a.count] = 2000.0
    o, d = make_pair(mesh, params, a)

    def call(k):
        before = d.launches()
        _run(o, d, a, (k,))
        return d.launches() - before

    assert call(12) < 24  # lists, as far as they go
    assert call(9) > 36
    h = fetch(d, a)
    h.arrays["cell_cell_repulsion_strength"][: h.count] = 1e-3
    h.arrays["cell_cell_adhesion_strength"][: h.count] = 1e-3
    h.arrays["previous_velocities"][: 3 * h.count] = 0.0
    h.arrays["positions"][: 3 * h.count] = np.random.default_rng(1).uniform(-120, 120, 3 * h.count)
    o.upload(h)
    d.upload(h)
    assert min(call(20) for _ in range(4)) < 40
    d.close()


@pytest.mark.parametrize("form", FORMS)
def test_barrier_timeout_is_reported_and_recoverable(form):
    """A one-poll wait limit makes the grid barriers of a call over lists give
    up: PPC_ERR_TIMEOUT at the next synchronising call, steps refused until the
    state is uploaded again, and from then on the oracle's trajectory."""
    mesh, params, a = _agents(3000, 3, 150, 51, FORMS[form], fast=20.0)
    o, d = make_pair(mesh, params, a)
    d.step(5)
    d.set_wait_limit(1)
    d.step(60)
    with pytest.raises(PPCError) as e:
        d.synchronize()
    assert e.value.rc == PPC_ERR_TIMEOUT
    with pytest.raises(PPCError) as e:
        d.step(4)
    assert e.value.rc == PPC_ERR_ARG
    d.set_wait_limit(1 << 25)
    d.upload(a)
    _run(o, d, a, (5, 12, 1, 9))
    d.close()


@pytest.mark.parametrize("shrink", [0.8, 1.0])
@pytest.mark.parametrize("steps", [2, 3, 10])
def test_autotuned_states_step_over_lists(steps, shrink):
    """Whatever shape wins for the fused pass (-2 where agents are dense), long
    calls run over lists; a shape the caller sets runs every step."""
    mesh, params, a = wl.config2(seed=2)
    a.arrays["positions"][:] *= shrink
    _, d = make_pair(mesh, params, a)
    d.update_mechanics_mesh()
    d.step(100)  # past the tissue's first relaxation
    d.autotune(steps)

    def launches():
        before = d.launches()
        d.step(60)
        d.synchronize()
        return d.launches() - before

    assert launches() < 20
    d.set_launch_shape(-3, 128, 0)
    assert launches() >= 240
    d.set_launch_shape(-4, 128, 0)
    assert launches() < 20
    d.close()


def test_first_list_call_while_another_stream_captures():
    """The allocation of the lists leaves the program's own capture valid."""
    import torch

    mesh, params, a = _agents(500, 3, 110, 81, 2000)
    o, d = make_pair(mesh, params, a)
    _mesh(o)
    x = torch.zeros(64, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        x += 1
        d.step(8)
    o.step(8, 0, 0.0, 0.0)
    assert_same_state(fetch(d, a), fetch(o, a))
    graph.replay()
    graph.replay()
    assert (x == 2).all().item()
    d.close()


def test_only_calls_over_lists_take_their_memory():
    """200,000 slots: the lists' arrays (some 220 MB) come with the first call
    that steps over lists, not with the state, its uploads or single steps."""
    import torch

    from paraphysicell_b200.device import Simulation

    mesh, params, a = _agents(2000, 3, 150, 71, 200000)
    build.ensure_built()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    d = Simulation(mesh, params, a.capacity)
    d.upload(a)
    for _ in range(3):
        d.step(1)
    d.step_with_phenotype(5, 0.0, 0.0)
    fetch(d, a)
    taken = free - torch.cuda.mem_get_info()[0]
    assert taken < 300 << 20
    d.step(8)
    d.synchronize()
    assert free - torch.cuda.mem_get_info()[0] > taken + (100 << 20)
    d.close()


def test_fp32_force_lists_match_the_scanning_pass():
    """The FP32-force form over lists adds the same terms in the same order as
    its scanning passes, so the two agree bit for bit."""
    from paraphysicell_b200.abi import PPC_FP32_FORCE
    from paraphysicell_b200.device import Simulation

    mesh, params, a = wl.scaled(wl.config2, 1500, 12)
    out = []
    for shape in (-4, -3):
        d = Simulation(mesh, params, a.capacity)
        d.set_precision(PPC_FP32_FORCE)
        d.set_launch_shape(shape, 128, 0)
        d.upload(a)
        d.step(40)
        out.append(fetch(d, a))
        d.close()
    assert_same_state(out[0], out[1])
