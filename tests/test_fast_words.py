"""Fast numerics keeps its words.  The fast build contracts multiply-adds, and
a sum of two products has two contracted forms, so a kernel rewritten for speed
can change a run's last bits where the strict build cannot (up to 3.4e-4 of the
vertical momentum after two steps).  The digests of two fast steps were recorded
from the kernels that took one index and one coefficient at a time (commit
8b650cb); the stencil records, the preloaded forms and the loops give the same
words, as an instance of its own (every launch preloads) and as a member of an
ensemble whose launches all take the loops."""

import json

import numpy as np
import pytest

import hexdyn
from fixtures import GOLDEN, SIDE, STATE, array_digest, case_from_arrays, golden_config, inputs, load_golden
from hexdyn.config import DycoreConfig
from hexdyn.ensemble import HexEnsemble

pytestmark = pytest.mark.gpu

NAMES = ["l2_L12", "l2_L12_sub4", "l2_L12_nomono", "l2_L12_noapvm", "l2_L12_notracers", "l2_L12_xnutr",
         "l2_L12_rk2_sub4", "l2_L12_smag", "l2_L12_t5", "l2_L12_t6", "l3_L20"]
PRELOAD_CHUNKS = 40000  # dycore_step.cuh


def fast_case(name):
    fx = load_golden(name)
    c = golden_config(fx)
    smag = {}
    if c["smagorinsky"] is not None:
        smag = dict(config_horiz_mixing="2d_smagorinsky", config_smagorinsky_coef=c["smagorinsky"][0],
                    config_visc4_2dsmag=c["smagorinsky"][1], config_del4u_div_factor=c["smagorinsky"][2])
    cfg = DycoreConfig(config_dt=c["dt"], config_number_of_sub_steps=c["n_sub_steps"], config_monotonic=c["monotonic"],
                       config_apvm_upwinding=c["apvm_upwinding"], config_xnutr=c["xnutr"], config_zd=c["zd"],
                       config_time_integration_order=c["order"], moist_coefficients="native", numerics="fast", **smag)
    return case_from_arrays(inputs(fx)), cfg


def digests(state, saved) -> dict:
    pairs = [(k, getattr(state, k)) for k in STATE] + [(k, getattr(saved, k)) for k in SIDE]
    return {k: array_digest(np.asarray(a, dtype=np.float32)) for k, a in pairs}


def single_digests(name) -> dict:
    driver = hexdyn.from_case(*fast_case(name), capture_graph=True)
    driver.step_device(2)
    out = digests(*driver.get_state())
    driver.close()
    return out


@pytest.mark.parametrize("name", NAMES)
def test_fast_words_are_the_recorded_ones(name):
    record = json.loads((GOLDEN / "digests_fast.json").read_text())[name]
    got = single_digests(name)
    assert [k for k in record if got[k] != record[k]] == []


@pytest.mark.parametrize("name", ["l2_L12", "l2_L12_nomono", "l2_L12_smag", "l2_L12_xnutr", "l2_L12_t5"])
def test_fast_words_of_the_loops(name):
    record = json.loads((GOLDEN / "digests_fast.json").read_text())[name]
    case, cfg = fast_case(name)
    members = PRELOAD_CHUNKS // (162 * 16 // 4) + 1
    batch = HexEnsemble.from_cases([case] * members, cfg, capture_graph=True)
    batch.step_device(2)
    for m in (0, members - 1):
        got = digests(*batch.get_member_state(m))
        assert [k for k in record if got[k] != record[k]] == [], m
    batch.close()
