"""The small-grid forms of the stencil kernels (neighbours preloaded before use,
Launcher::pre) against the loops that large grids take, word for word: members
of an ensemble large enough for every launch over cells, edges and tracers to
take the loops, against the same case as an instance of its own, whose launches
all preload.  One tracer and seven (one past the six that a thread preloads),
columns that end inside a chunk, and the step's options.  A mesh of pentagons to
octagons takes every gather past the slots that a thread preloads (six edges of
a cell, ten neighbours of an edge, ten cells of its advection stencil), against
the oracle too."""

import numpy as np
import pytest

import hexdyn
from fixtures import SIDE, STATE, differing_words
from hexdyn.case import build_case, case_arrays
from hexdyn.config import DycoreConfig
from hexdyn.ensemble import HexEnsemble
from hexdyn import mesh as mesh_module
from hexdyn.mesh import build_mesh
from oracle.dycore import OracleConfig, OracleDycore, State

pytestmark = pytest.mark.gpu

PRELOAD_CHUNKS = 40000  # dycore_step.cuh


@pytest.mark.parametrize("levels, tracers, options", [
    (55, 1, {}),
    (53, 7, {}),
    (55, 2, dict(config_monotonic=False, moist_coefficients="dry", config_time_integration_order=2)),
    (48, 1, dict(config_horiz_mixing="2d_smagorinsky", config_smagorinsky_coef=0.125, config_visc4_2dsmag=0.05)),
    (55, 1, dict(numerics="fast", config_xnutr=0.2)),
])
def test_preloaded_kernels_equal_the_loops(levels, tracers, options):
    case = build_case(build_mesh(2, lloyd=2, seed=0), n_levels=levels, seed=1, n_condensates=tracers - 1,
                      theta_noise=0.1)
    cfg = DycoreConfig(**{**dict(config_dt=900.0, config_number_of_sub_steps=2, moist_coefficients="native"),
                          **options})
    chunks = 162 * ((levels + 8) // 8 * 8) // 4
    members = PRELOAD_CHUNKS // chunks + 1
    assert 3 * chunks * ((tracers + 2) // 3) <= PRELOAD_CHUNKS < chunks * members
    single = hexdyn.from_case(case, cfg, capture_graph=True)
    batch = HexEnsemble.from_cases([case] * members, cfg, capture_graph=True)
    single.step_device(2)
    batch.step_device(2)
    state, saved = single.get_state()
    for m in (0, members - 1):
        st, sd = batch.get_member_state(m)
        for k in STATE:
            assert differing_words(getattr(st, k), getattr(state, k)) == 0, (m, k)
        for k in SIDE:
            assert differing_words(getattr(sd, k), getattr(saved, k)) == 0, (m, k)
    single.close()
    batch.close()


@pytest.fixture(scope="module")
def uneven_mesh():
    """120 cells of 5 to 8 edges: relaxed random generators."""
    points = np.random.default_rng(482).standard_normal((120, 3))
    points /= np.linalg.norm(points, axis=1, keepdims=True)
    for _ in range(12):
        points = mesh_module._lloyd_step(points)
    with pytest.MonkeyPatch.context() as patch:
        patch.setattr(mesh_module, "MAX_EDGES", 8)
        patch.setattr(mesh_module, "MAX_EDGES2", 16)
        mesh = mesh_module.VoronoiMesh(arrays=mesh_module._connectivity(points, mesh_module.EARTH_RADIUS))
    assert sorted(set(mesh.nEdgesOnCell)) == [5, 6, 7, 8]
    # more than ten TRiSK neighbours, odd and even counts of them
    assert set(mesh.nEdgesOnEdge) == {8, 9, 10, 11, 12, 13}
    return mesh


@pytest.mark.parametrize("levels, tracers, options", [
    (14, 2, {}),
    (12, 4, dict(order=2, n_sub_steps=4, monotonic=False, moist="dry")),
    (9, 1, dict(apvm_upwinding=0.0, numerics="fast")),
    (12, 2, dict(numerics="fast", xnutr=0.2)),
])
def test_cells_of_more_than_six_edges(uneven_mesh, levels, tracers, options):
    case = build_case(uneven_mesh, n_levels=levels, seed=2, n_condensates=tracers - 1, theta_noise=0.1)
    assert {10, 11, 12, 13} <= set(case.n_adv_cells_for_edge)
    options = {**dict(n_sub_steps=2, moist="native"), **options}
    numerics = options.pop("numerics", "strict")
    names = dict(n_sub_steps="config_number_of_sub_steps", order="config_time_integration_order",
                 monotonic="config_monotonic", moist="moist_coefficients", xnutr="config_xnutr",
                 apvm_upwinding="config_apvm_upwinding")
    cfg = DycoreConfig(config_dt=900.0, numerics=numerics, **{names[k]: v for k, v in options.items()})
    single = hexdyn.from_case(case, cfg, capture_graph=True)
    members = PRELOAD_CHUNKS // (120 * ((levels + 8) // 8 * 8) // 4) + 1
    batch = HexEnsemble.from_cases([case] * members, cfg, capture_graph=True)
    single.step_device(2)
    batch.step_device(2)
    state, saved = single.get_state()
    for m in (0, members - 1):
        st, sd = batch.get_member_state(m)
        for k in STATE:
            assert differing_words(getattr(st, k), getattr(state, k)) == 0, (m, k)
        for k in SIDE:
            assert differing_words(getattr(sd, k), getattr(saved, k)) == 0, (m, k)
    single.close()
    batch.close()
    if numerics == "strict":
        oracle = OracleDycore(case_arrays(case), OracleConfig(dt=900.0, **options))
        st, sd = State(*(getattr(case, k).copy() for k in STATE)), None
        for _ in range(2):
            st, sd = oracle.step(st, sd)
        for k in STATE:
            assert differing_words(getattr(state, k), getattr(st, k)) == 0, k
        for k in SIDE:
            assert differing_words(getattr(saved, k), getattr(sd, k)) == 0, k
