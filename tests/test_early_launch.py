"""Launches whose blocks are set up while their predecessor still runs.

Such a kernel is resident while the fields that it will read are being written,
so it may read them with coherent loads only: the read-only load (``__ldg``, or
a load of a ``const float* __restrict__`` parameter that the compiler turns into
one) is for the mesh's arrays and records, which never change.  On the source:
every read-only load names a mesh array.  On the GPU: a step with early launches
(captured and eager) against ``profile``, whose launches are never early and run
on one stream, word for word, on grids below, between and above the limits that
decide which launches are early.
"""

import re
from pathlib import Path

import pytest

import hexdyn
from fixtures import SIDE, STATE, differing_words
from hexdyn.case import build_case
from hexdyn.config import DycoreConfig
from hexdyn.mesh import build_mesh

CSRC = Path(__file__).resolve().parent.parent / "gpuwm-hex_b200" / "csrc"
SMAG = dict(config_horiz_mixing="2d_smagorinsky", config_smagorinsky_coef=0.125, config_visc4_2dsmag=0.05)


def test_read_only_loads_are_of_the_mesh():
    text = re.sub(r"//.*", "", (CSRC / "dycore_kernels_vec.cuh").read_text())
    # pointers that kernels form into the mesh's records
    records = set(re.findall(r"const \w+\* (\w+) = g\.", text))
    for arg in re.findall(r"\b(?:__ldg|ldg4)\(&?([\w.]+)", text) + re.findall(r"win<\d, \d, true>\((\w+\.)", text):
        # (the definitions of ldg4 and ld<MESH>)
        assert arg.startswith("g.") or arg in records or arg in ("const", "p", "reinterpret_cast"), arg
    for parameters in re.findall(r"__global__[^{;]*?\bkv_\w+\((.*?)\)\s*\{", text, re.S):
        assert not re.search(r"const float\s*\*\s*__restrict__", parameters), parameters
    # the shared device functions: only the mesh load itself
    assert len(re.findall(r"const float\s*\*\s*__restrict__", text)) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("level, levels, tracers, options", [
    (2, 55, 2, {}),  # 2 k chunks of cells, 7 k of edges: all launches early
    (2, 20, 2, dict(numerics="fast")),
    (4, 55, 3, SMAG),  # 36 k (early) and 108 k (not)
    (5, 55, 1, {}),  # 143 k (not) and 430 k (early)
    (5, 72, 2, dict(config_monotonic=False)),  # 205 k (early) and 614 k (not)
])
def test_early_launches_change_no_word(level, levels, tracers, options):
    case = build_case(build_mesh(level, lloyd=2, seed=0), n_levels=levels, seed=3, n_condensates=tracers - 1,
                      theta_noise=0.1)
    cfg = DycoreConfig(**{**dict(config_dt=600.0, config_number_of_sub_steps=2), **options})
    serial = hexdyn.from_case(case, cfg)
    serial.profile(4)
    expect = serial.get_state()
    serial.close()
    for graph in (True, False):
        driver = hexdyn.from_case(case, cfg, capture_graph=graph)
        driver.step_device(4)
        got = driver.get_state()
        for part, names in ((0, STATE), (1, SIDE)):
            for k in names:
                assert differing_words(getattr(got[part], k), getattr(expect[part], k)) == 0, (graph, k)
        driver.close()
