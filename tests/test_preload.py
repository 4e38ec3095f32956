"""The small-grid forms of the stencil kernels (neighbours preloaded before use,
Launcher::pre) against the loops that large grids take, word for word: members
of an ensemble large enough for every launch over cells, edges and tracers to
take the loops, against the same case as an instance of its own, whose launches
all preload.  One tracer and seven (one past the six that a thread preloads),
columns that end inside a chunk, and the step's options."""

import pytest

import hexdyn
from fixtures import SIDE, STATE, differing_words
from hexdyn.case import build_case
from hexdyn.config import DycoreConfig
from hexdyn.ensemble import HexEnsemble
from hexdyn.mesh import build_mesh

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
