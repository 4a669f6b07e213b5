"""The kernels that make up a step with the phenotype update or with stochastic
springs, the walk lists of the interactions and the downloads of large states,
at the sizes where they change form: edges of warps and blocks, one and several
settlement blocks, removal lists beyond the shared sort, columns beyond the
landing area's threshold. Bit for bit the oracle's."""
import numpy as np
import pytest

from paraphysicell_b200 import abi
from paraphysicell_b200 import workloads as wl
from paraphysicell_b200.abi import AgentArrays, Mesh, Params
from paraphysicell_b200.device import Simulation
from tests import gpu_util as gu
from tests import scenarios as sc

pytestmark = pytest.mark.gpu


def _agents(n, dims, half, seed, capacity):
    rng = np.random.default_rng(seed)
    mesh = Mesh.make(dims, (-half,) * 3, (half,) * 3)
    a = AgentArrays(n, dims, 2, capacity)
    a.arrays["positions"][: n * dims] = rng.uniform(-half, half, n * dims)
    a.arrays["radius"][:n] = rng.uniform(6.0, 10.0, n)
    a.arrays["cell_definition_indices"][:n] = rng.integers(0, 2, n)
    a.arrays["cell_adhesion_affinities"][: 2 * n] = rng.uniform(0.2, 1.0, 2 * n)
    a.arrays["is_movable"][:n] = rng.random(n) < 0.9
    return mesh, a


def _start(o, d):
    for x in (o, d):
        x.update_mechanics_mesh()
        x.update_cell_neighbors()


@pytest.mark.parametrize("phenotype", [False, True])
@pytest.mark.parametrize("dims,n,half,most", [(1, 33, 150, 3), (2, 31, 60, 2), (2, 1025, 260, 5), (3, 1, 40, 3),
                                              (3, 129, 60, 12), (3, 17001, 330, 3)])
def test_steps_with_stochastic_springs(phenotype, dims, n, half, most):
    """17,001 agents settle their attachments with two blocks."""
    mesh, a = _agents(n, dims, half, 11 + n, max(n + n // 10 + 8, 512))
    a.arrays["attachment_rate"][:n] = 1.2
    a.arrays["detachment_rate"][:n] = 0.5
    a.arrays["maximum_number_of_attachments"][:n] = most
    o, d = gu.make_pair(mesh, Params.make(dt=0.1, ndefs=2, walls=True, springs=True), a)
    _start(o, d)
    for k in (1, 4):
        if phenotype:
            o.step(k, 1, 4e-3, 4e-3)
            d.step_with_phenotype(k, 4e-3, 4e-3)
        else:
            o.step(k, 0, 0.0, 0.0)
            d.step(k)
        go, gd = gu.fetch(o, a), gu.fetch(d, a)
        assert gd.spring_lists() == go.spring_lists()
        gu.assert_same_state(gd, go)
    d.close()


@pytest.mark.parametrize("dims,n,half,p_divide,p_death", [(1, 257, 900, 0.1, 0.1), (2, 1, 60, 0.5, 0.0),
                                                          (2, 255, 150, 0.3, 0.3), (3, 3001, 200, 0.02, 0.05),
                                                          (3, 12000, 300, 0.05, 0.6)])
def test_steps_with_divisions_and_removals(dims, n, half, p_divide, p_death):
    """12,000 agents remove more than the 4,096 a block sorts in shared memory;
    daughters take slots that removed agents left in the same step."""
    mesh, a = _agents(n, dims, half, 23 + n, 4 * n + 16)
    o, d = gu.make_pair(mesh, Params.make(dt=0.1, ndefs=2), a)
    _start(o, d)
    for k in (1, 1, 2):
        o.step(k, 1, p_divide, p_death)
        d.step_with_phenotype(k, p_divide, p_death)
        gu.assert_same_state(gu.fetch(d, a), gu.fetch(o, a))
        assert d.event_counts() == o.event_counts()
    o.update_mechanics_mesh()
    gu.assert_same_bins(d, o)
    d.close()


@pytest.mark.parametrize("scale", [0.0, 0.05, 1.0])
def test_interactions_leave_the_next_step_a_current_mesh(scale):
    """Without an ingestion or fusion the mesh stays; with them the agents'
    radii and positions reach the next step's key-ordered copies."""
    mesh, params, a = wl.scaled(wl.config2, 1500, seed=31)
    a.arrays["positions"][: 3 * a.count] *= 0.6
    f = sc.random_interaction_fields(a, params.cell_definitions_count, seed=3, scale=scale)
    o, d = gu.make_pair(mesh, params, a)
    _start(o, d)
    for x in (o, d):
        x.upload_interactions(f.copy())
    for _ in range(4):
        o.update_cell_cell_interactions()
        d.update_cell_cell_interactions()
        o.update_mechanics_mesh()
        o.update_cell_neighbors()
        o.step(1, 0, 0.0, 0.0)
        d.step(1)
        o.update_mechanics_mesh()
        o.update_cell_neighbors()
        gu.assert_same_state(gu.fetch(d, a), gu.fetch(o, a))
    d.close()


def test_interaction_scratch_follows_the_live_agents():
    """A state of 400,000 slots and 300 agents allocates rows for its agents,
    not its slots (109 MB of them), and more once divisions outgrow them."""
    import torch

    mesh, params, a = wl.scaled(wl.config2, 300, seed=7, capacity=400000)
    f = sc.random_interaction_fields(a, params.cell_definitions_count, seed=8, scale=0.02)
    o, d = gu.make_pair(mesh, params, a)
    _start(o, d)
    for x in (o, d):
        x.upload_interactions(f.copy())
    free = torch.cuda.mem_get_info()[0]
    d.update_mechanics_mesh()
    for p_divide in (0.0, 0.9, 0.9, 0.9):
        o.step(1, 1, p_divide, 0.0)
        d.step_with_phenotype(1, p_divide, 0.0)
        for x in (o, d):
            x.update_mechanics_mesh()
            x.update_cell_neighbors()
        o.update_cell_cell_interactions()
        d.update_cell_cell_interactions()
        if p_divide == 0.0:
            assert free - torch.cuda.mem_get_info()[0] < 16 << 20
        gu.assert_same_state(gu.fetch(d, a), gu.fetch(o, a))
        o.update_mechanics_mesh()  # the oracle's step starts from the lists it has
        o.update_cell_neighbors()
    assert d.count() > 300 + 300 // 8 + 1024
    d.close()


@pytest.mark.parametrize("n", [131071, 131072, 300001])
def test_large_downloads_into_pageable_rows(n):
    """Columns at the landing area's threshold and beyond its size, and agents
    appended since the host last knew the count."""
    mesh, params, a = wl.scaled(wl.config5, n, seed=3, capacity=n + n // 20)
    d = Simulation(mesh, params, a.capacity)
    d.upload(a)
    got = AgentArrays(0, a.dims, a.ndefs, a.capacity)
    got.count = got.capacity
    d.download(got)
    assert got.count == n
    for f in ("positions", "orientation", "radius", "total_volume", "agent_ids", "cell_adhesion_affinities", "flags"):
        assert np.array_equal(got[f], a[f]), f
    d.step_with_phenotype(1, 0.02, 0.0)
    again = AgentArrays(0, a.dims, a.ndefs, a.capacity)
    again.count = again.capacity
    d.download(again)
    assert again.count == n + d.event_counts()[0] > n
    assert np.array_equal(again["agent_ids"], np.arange(again.count))
    third = AgentArrays(0, a.dims, a.ndefs, a.capacity)
    third.count = third.capacity
    d.download(third)
    gu.assert_same_state(again, third)
    d.close()


@pytest.mark.parametrize("n", [131071, 131072, 300001])
def test_large_downloads_beside_page_locked_vectors(n):
    """Pageable columns land beside page-locked vectors until the landing area
    is full, the rest takes the driver's copies."""
    from paraphysicell_b200.device import PinnedPool

    mesh, params, a = wl.scaled(wl.config5, n, seed=3, capacity=n + 64)
    d = Simulation(mesh, params, a.capacity)
    d.upload(a)
    pool = PinnedPool()
    got = AgentArrays(0, a.dims, a.ndefs, a.capacity)
    for f in ("positions", "orientation"):
        got.arrays[f] = pool(got.arrays[f].size, np.float64)
    for _ in range(2):
        got.count = got.capacity
        d.download(got, fields=("positions", "orientation", "radius", "total_volume", "agent_ids",
                                "cell_adhesion_affinities", "flags"))
        assert got.count == n
        for f in ("positions", "orientation", "radius", "total_volume", "agent_ids", "cell_adhesion_affinities",
                  "flags"):
            assert np.array_equal(got[f], a[f]), f
            got.arrays[f][:] = 0
    d.close()
    pool.free()
