"""The calls that a program using hexdyn makes, at the sizes it makes them.

Sizes are those of this repository's tests, configurations and benchmark: the
icosahedral meshes of 162, 642, 2562, 10242 and 40962 cells, 12 to 72 levels,
1 to 6 tracers, and the corrector's column and edge networks.  A case is one
call sequence through the public entry points: large steps of one instance
(captured as CUDA graphs, or eagerly under a physics callback), of an uneven
batch of ensembles, from host buffers to host buffers, the learned corrector's
step, and its networks' forward and training passes.

The strict step is defined word for word (FP32 in a fixed order), so its
tolerance is "exact"; the other tolerances are measured (see ``tolerance``).
"""

from __future__ import annotations

import dataclasses
import functools
import math
import sys
from pathlib import Path
from types import SimpleNamespace

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "gpuwm-hex_b200"))

import hexdyn  # noqa: E402
from hexdyn import mlp  # noqa: E402
from hexdyn.case import build_case  # noqa: E402
from hexdyn.config import DycoreConfig  # noqa: E402
from hexdyn.corrector import LearnedStepper, StateFeatures, TrainedNet  # noqa: E402
from hexdyn.driver import DeviceAtmosphere  # noqa: E402
from hexdyn.ensemble import HexEnsemble, step_batched  # noqa: E402
from hexdyn.mesh import build_mesh  # noqa: E402

STATE = ("rho", "rho_theta", "rho_u", "rho_w", "scalars")
SIDE = ("theta_m", "exner", "density_perturbation", "rho_theta_perturbation", "pressure_perturbation",
        "normal_velocity", "vertical_velocity")
# large time steps (s) of each mesh, half of what its resolution allows, so
# that a run of thousands of steps stays in the regime of a forecast
DT = {2: 900.0, 3: 900.0, 4: 900.0, 5: 600.0, 6: 360.0}
CELLS = {level: 10 * 4 ** level + 2 for level in DT}


def step_case(name, level, levels, scalars, **options):
    case = dict(name=name, kind="step", level=level, levels=levels, scalars=scalars, substeps=2, order=3, fct=True,
                moist=True, smag=False, xnutr=0.0, numerics="strict")
    case.update(options)
    return case


def listed():
    return [
        # the smallest instance (the size of the parity fixtures): a coupled
        # program's unit runs, where launches and latency are everything
        step_case("step_162x12", 2, 12, 1),
        # the 480 km configuration with vapour, stepped as the reference's
        # caller does: one step and its validation flag at a time
        step_case("step_2562x55", 4, 55, 1, kind="step_device"),
        # ragged columns (41 of 48 stored levels), the order-2 schedule,
        # standard transport, dry coefficients, five tracers
        step_case("step_642x41_rk2", 3, 41, 5, order=2, substeps=4, fct=False, moist=False),
        # 240 km with 2-D Smagorinsky mixing and four acoustic substeps
        step_case("step_10242x55_smag", 5, 55, 3, smag=True, substeps=4),
        # the headline workload: 120 km, vapour and five condensates
        step_case("step_40962x55", 6, 55, 6),
        # contracted arithmetic, deep columns, implicit w damping on
        step_case("fast_10242x72", 5, 72, 2, numerics="fast", xnutr=0.2),
        # an uneven batch: coarse members one long step, fine members two
        # short ones, both groups at once (the largest call)
        dict(name="ensemble_uneven", kind="ensemble", levels=55, scalars=3, coarse_level=5, coarse=4, fine_level=6,
             fine=3),
        # a physics suite in the loop: a host callback before every RK stage
        step_case("physics_2562x55", 4, 55, 2, kind="physics"),
        # a caller that keeps its state on the host: up, one step, down
        step_case("host_10242x55", 5, 55, 3, kind="host"),
        # the corrected step: features, both networks, increments, checks
        step_case("corrected_10242x55", 5, 55, 3, kind="corrected", substeps=3),
        # the column network over every column of the 40962-cell mesh
        dict(name="forward_column", kind="forward", rows=40962, n_in=330, hidden=512, depth=3, n_out=165),
        # one optimizer step of the column network on the training batch
        dict(name="train_column", kind="train", rows=2048, n_in=330, hidden=512, depth=3, n_out=165),
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step_device", "ensemble", "physics", "host", "corrected", "forward",
                       "train"])
    if kind == "forward":
        return dict(kind=kind, rows=int(2 ** rng.uniform(9, 16.9)), n_in=rng.randint(60, 400),
                    hidden=rng.choice([128, 256, 384, 512]), depth=rng.choice([2, 3, 4]), n_out=rng.randint(20, 200))
    if kind == "train":
        return dict(kind=kind, rows=int(2 ** rng.uniform(7, 13)), n_in=rng.randint(60, 400),
                    hidden=rng.choice([128, 256, 384, 512]), depth=rng.choice([2, 3, 4]), n_out=rng.randint(20, 200))
    if kind == "ensemble":
        return dict(kind=kind, levels=rng.randint(12, 60), scalars=rng.randint(1, 4), coarse_level=rng.choice([2, 3]),
                    coarse=rng.randint(1, 8), fine_level=rng.choice([4, 5]), fine=rng.randint(1, 4))
    # the cells of a mesh grow by four from level to level
    level = rng.choice([2, 3, 4, 4, 5, 5, 6] if kind == "step" else [2, 3, 4, 5])
    case = step_case("", level, rng.randint(8, 72 if level < 6 else 55), rng.randint(1, 6 if level < 6 else 4),
                     kind=kind, substeps=rng.choice([2, 2, 4, 6]) if kind != "corrected" else 3)
    del case["name"]
    if kind != "corrected":
        case.update(order=rng.choice([3, 3, 3, 2]), fct=rng.random() < 0.75, moist=rng.random() < 0.75,
                    smag=rng.random() < 0.25 and level < 6, xnutr=rng.choice([0.0, 0.0, 0.2]),
                    numerics=rng.choice(["strict", "strict", "strict", "fast"]))
    return case


# ------------------------------------------------------------------ inputs


@functools.lru_cache(maxsize=None)
def _mesh(level):
    return build_mesh(level, lloyd=2, seed=0)


@functools.lru_cache(maxsize=None)
def _base(level, levels, scalars):
    """The balanced jet over seeded terrain that the states of a mesh start from."""
    geometry = _geometry(level, levels)
    if scalars == 1:
        return geometry
    return build_case(_mesh(level), n_levels=levels, seed=0, n_condensates=scalars - 1, like=geometry)


@functools.lru_cache(maxsize=None)
def _geometry(level, levels):
    return build_case(_mesh(level), n_levels=levels, seed=0, n_condensates=0)


def _state(level, levels, scalars, seed):
    """A state of the mesh: the jet with seeded small-scale noise in every
    field (0.01 K, 0.1 m/s, 1 cm/s of vertical motion, 5 % of the tracers)."""
    base = _base(level, levels, scalars)
    rng = np.random.default_rng([seed, level, levels, scalars])

    def noise(shape):
        return rng.standard_normal(shape, dtype=np.float32)

    c1, c2 = base.mesh.cellsOnEdge[:, 0], base.mesh.cellsOnEdge[:, 1]
    rho_u = base.rho_u + np.float32(0.05) * (base.rho[:, c1] + base.rho[:, c2]) * noise(base.rho_u.shape)
    rho_w = np.zeros_like(base.rho_w)
    rho_w[1:-1] = np.float32(0.01) * base.rho[1:] * noise(base.rho[1:].shape)
    scalars_ = base.scalars * np.maximum(1.0 + np.float32(0.05) * noise(base.scalars.shape), np.float32(0.0))
    return dataclasses.replace(base, rho_theta=base.rho_theta * (1.0 + np.float32(3e-5) * noise(base.rho.shape)),
                               rho_u=rho_u, rho_w=rho_w, scalars=scalars_)


def _config(case, dt):
    return DycoreConfig(config_dt=dt, config_number_of_sub_steps=case["substeps"],
                        config_time_integration_order=case["order"], config_monotonic=case["fct"],
                        moist_coefficients="native" if case["moist"] else "dry", config_xnutr=case["xnutr"],
                        numerics=case["numerics"],
                        **(dict(config_horiz_mixing="2d_smagorinsky", config_smagorinsky_coef=0.125,
                                config_visc4_2dsmag=0.05) if case["smag"] else {}))


def _fields(driver):
    """Every field of the current state: the library's buffers, in place.  Even
    numbers of steps end in the buffers that they started from."""
    atm = DeviceAtmosphere(driver)
    return {n: atm.padded(n) for n in (*STATE, *SIDE)}


def _weights(case, seed):
    """FP32 weights and biases of a network (He initialisation on the real
    block of the padded layers), on the GPU."""
    up = lambda n: -(-n // 128) * 128  # noqa: E731
    real = [case["n_in"]] + [case["hidden"]] * case["depth"] + [case["n_out"]]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    out = []
    for i in range(case["depth"] + 1):
        w = torch.zeros(up(real[i + 1]), up(real[i]), device="cuda")
        w[: real[i + 1], : real[i]] = torch.randn(real[i + 1], real[i], device="cuda", generator=gen) * math.sqrt(
            2.0 / real[i])
        b = torch.zeros(up(real[i + 1]), device="cuda")
        b[: real[i + 1]] = 0.1 * torch.randn(real[i + 1], device="cuda", generator=gen)
        out.append((w, b))
    return out


def _samples(case, seed):
    """Normalised features [rows][n_in] as bf16 and targets, both padded."""
    up = lambda n: -(-n // 128) * 128  # noqa: E731
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    rows = up(case["rows"])
    x = torch.zeros(rows, up(case["n_in"]), device="cuda")
    x[: case["rows"], : case["n_in"]] = torch.randn(case["rows"], case["n_in"], device="cuda", generator=gen)
    t = torch.zeros(rows, up(case["n_out"]), device="cuda")
    t[: case["rows"], : case["n_out"]] = torch.randn(case["rows"], case["n_out"], device="cuda", generator=gen)
    return x.to(torch.bfloat16), t


def _network(case, seed):
    net = mlp.TensorCoreMLP(case["n_in"], case["hidden"], case["depth"], case["n_out"], seed=0)
    for layer, (w, b) in zip(net.layers, _weights(case, seed)):
        layer.w.copy_(w)
        layer.b.copy_(b)
        layer.wb.copy_(w.to(torch.bfloat16))
        layer.wbt.copy_(w.t().to(torch.bfloat16))
    return net


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("forward", "train"):
        net = _network(case, seed)
        x, t = _samples(case, seed)
        return SimpleNamespace(kind=kind, net=net, x=x, xt=x.t().contiguous(), t=t, rows=case["rows"])
    if kind == "ensemble":
        groups = []
        for k, part in enumerate(("coarse", "fine")):
            level = case[part + "_level"]
            dt = 2.0 * DT[case["fine_level"]] if part == "coarse" else DT[level]
            members = [_state(level, case["levels"], case["scalars"], 100 * seed + 50 * k + m)
                       for m in range(case[part])]
            groups.append(HexEnsemble.from_cases(members, DycoreConfig(config_dt=dt), capture_graph=True))
        return SimpleNamespace(kind=kind, groups=groups, out=[_fields(g) for g in groups])
    level, levels, scalars = case["level"], case["levels"], case["scalars"]
    start = _state(level, levels, scalars, seed)
    if kind == "corrected":
        return _prepare_corrected(case, start, seed)
    driver = hexdyn.from_case(start, _config(case, DT[level]), capture_graph=kind != "physics")
    state = SimpleNamespace(kind=kind, driver=driver, out=_fields(driver))
    if kind == "physics":
        # the tendencies of a physics suite: a few K and m/s a day
        gen = torch.Generator(device="cuda").manual_seed(seed)
        def tendency(scale, n):
            return scale * torch.randn(levels, n, device="cuda", generator=gen)
        n_cells, n_edges = CELLS[level], start.rho_u.shape[1]
        given = SimpleNamespace(rho_u=tendency(1e-5, n_edges), rho_theta=tendency(1e-5, n_cells),
                                rho=tendency(1e-9, n_cells), diabatic_theta=tendency(1e-5, n_cells))
        state.callback = lambda **_: given
    if kind == "host":
        st, sd = driver.get_state()

        def pinned(source, names, copy):
            out = {}
            for n in names:
                t = torch.empty(driver.field_shape(n), dtype=torch.float32, pin_memory=True)
                if copy:
                    t.numpy()[...] = getattr(source, n)
                out[n] = t
            return out

        inputs = {**pinned(st, STATE, True), **pinned(sd, SIDE, True)}
        state.out = {**pinned(st, STATE, False), **pinned(sd, SIDE, False)}
        state.buffers = [{n: d[n].numpy() for n in names} for d in (inputs, state.out) for names in (STATE, SIDE)]
        state.inputs = inputs
    return state


def _prepare_corrected(case, start, seed):
    level, L, dt = case["level"], case["levels"], DT[case["level"]]
    full = hexdyn.from_case(start, _config({**case, "substeps": 2}, dt), capture_graph=True)
    reduced = hexdyn.from_case(start, _config(case, 2.0 * dt), capture_graph=True)
    features = StateFeatures(reduced)
    features.compute(reduced)
    rng = np.random.default_rng(seed)
    nets = []
    for raw, hidden, n_out, fields in ((features.col, 512, 3 * L, 3), (features.edge, 256, L, 1)):
        rows = torch.linspace(0, raw.shape[0] - 1, 640, device="cuda").long()
        x = raw.index_select(0, rows).cpu().numpy()
        # increments of the size that a trained network gives late in training
        y = x[:, : fields * L].std(axis=0) * 1e-6 * rng.standard_normal((640, n_out))
        net = TrainedNet(raw.shape[1], hidden, 3, n_out, seed=7)
        net.fit(x, y.astype(np.float32), epochs=1, batch=128, lr=1e-3, seed=1)
        nets.append(net)
    zgrid = np.asarray(start.vertical.zgrid, dtype=np.float64)
    z = torch.zeros(CELLS[level], reduced.level_stride, device="cuda")
    z[:, :L] = torch.from_numpy((0.5 * (zgrid[:-1] + zgrid[1:])).T.astype(np.float32)).cuda()
    stepper = LearnedStepper(full, reduced, *nets, z, energy_tol=1e-2, w_growth_tol=10.0, ratio=2)
    return SimpleNamespace(kind="corrected", stepper=stepper, out=_fields(reduced))


# --------------------------------------------------------------------- run


def run(state):
    kind = state.kind
    if kind == "step":
        state.driver.step_async(2)
    elif kind == "step_device":
        state.driver.step_device(1)
        state.driver.step_device(1)
    elif kind == "physics":
        for _ in range(2):
            state.driver._step_device_v841(physics_stage_callback=state.callback)
    elif kind == "host":
        state.driver.step_host_buffers(*state.buffers)
    elif kind == "ensemble":
        # two periods, so that the coarse members' one step a period ends in
        # the buffers it started from
        for _ in range(2):
            step_batched(state.groups, (1, 2), read_flags=False)
    elif kind == "corrected":
        state.stepper.step()
        state.stepper.step()
    elif kind == "forward":
        return state.net.forward(state.x)
    else:
        net = state.net
        loss = net.gradients(state.x, state.xt, state.t, state.rows)
        net.adam(1e-4)
        return {"loss": loss, "gw": [l.gw for l in net.layers], "gb": [l.gb for l in net.layers],
                "w": [l.w for l in net.layers], "b": [l.b for l in net.layers]}
    return state.out


# -------------------------------------------------------- work, tolerances


def _step_work(cells, levels, scalars, substeps):
    """Bytes and operations of one large step: the state, the saved
    diagnostics and the mesh's fields read once, the new state written once;
    operations of the stencils (9 RK stages, 9 + 3 n/2 substeps, 3 transport
    passes), each field value formed once."""
    edges = 3 * cells
    per_cell, per_edge = cells * levels * 4, edges * levels * 4
    state = (9 + scalars) * per_cell + 2 * per_edge
    fixed = (5 + 2 * 6) * per_cell + per_edge + 4 * (cells * 30 + edges * 52)
    acoustic = 3 * (1 + max(1, substeps // 2) + substeps)
    flops = cells * levels * (9 * (3 * 140 + 220) + acoustic * (100 + 3 * 30) + scalars * (3 * 3 * 20 + 3 * 60 + 250))
    return 2 * state + fixed, flops


def work(case):
    kind = case["kind"]
    if kind in ("forward", "train"):
        dims = [case["n_in"]] + [case["hidden"]] * case["depth"] + [case["n_out"]]
        weights = sum(a * b for a, b in zip(dims[:-1], dims[1:]))
        rows = case["rows"]
        if kind == "forward":
            return {"bytes": 2 * rows * dims[0] + 4 * rows * dims[-1] + 2 * weights, "flops": 2 * rows * weights}
        # forward, both backward products (none for the inputs), Adam on three arrays
        return {"bytes": rows * (2 * dims[0] + 4 * dims[-1]) + 24 * weights,
                "flops": 2 * rows * (3 * weights - dims[0] * dims[1])}
    if kind == "ensemble":
        total = [0, 0]
        for part, steps in (("coarse", 2), ("fine", 4)):
            w = _step_work(case[part] * CELLS[case[part + "_level"]], case["levels"], case["scalars"], 2)
            total = [t + steps * x for t, x in zip(total, w)]
        return {"bytes": total[0], "flops": total[1]}
    nbytes, flops = _step_work(CELLS[case["level"]], case["levels"], case["scalars"], case["substeps"])
    steps = 1 if kind == "host" else 2
    if kind == "corrected":
        L = case["levels"]
        rows = CELLS[case["level"]]
        flops += 2 * rows * (6 * L * 512 + 2 * 512 * 512 + 512 * 3 * L) + 6 * rows * (
            4 * L * 256 + 2 * 256 * 256 + 256 * L)
    return {"bytes": steps * nbytes, "flops": steps * flops}


def tolerance(case):
    """Four times what another correct form was measured to differ by, as the
    largest over the outputs.  bf16 networks: 3.6e-3 from 64 bits (the first
    layer's weight gradient, the predictions).  Fast numerics: 1.9e-4 from the
    strict build (the vertical momentum, the other fields 1e-6 or less).  The
    corrected step: 1.3e-4 with a relative noise of 1e-2 on both networks'
    predictions (the vertical velocity)."""
    if case["kind"] in ("forward", "train"):
        return {"rel": 1.5e-2}
    if case["kind"] == "corrected":
        return {"rel": 5e-4}
    if case.get("numerics") == "fast":
        return {"rel": 8e-4}
    return "exact"


def exact(case, seed):
    """The networks' passes in 64 bits.  The strict step's words are fixed, so
    any change of them shows as a difference; a whole step has no short plain
    form in 64 bits."""
    if case["kind"] not in ("forward", "train"):
        return None
    layers = [(w.to(torch.bfloat16).double(), b.double()) for w, b in _weights(case, seed)]
    x, t = _samples(case, seed)
    zs, acts = [], [x.double()]
    for i, (w, b) in enumerate(layers):
        z = acts[-1] @ w.t() + b
        zs.append(z)
        acts.append(torch.nn.functional.gelu(z, approximate="tanh") if i < case["depth"] else z)
    if case["kind"] == "forward":
        return acts[-1]
    rows, n_out = case["rows"], case["n_out"]
    d = torch.zeros_like(acts[-1])
    diff = acts[-1][:rows, :n_out] - t[:rows, :n_out].double()
    d[:rows, :n_out] = 2.0 * diff / (rows * n_out)
    loss = diff.square().sum().reshape(1)
    gw, gb = [], []
    for i in range(case["depth"], -1, -1):
        gw.insert(0, d.t() @ acts[i])
        gb.insert(0, d.sum(0))
        if i > 0:
            z = zs[i - 1]
            u = math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)
            th = torch.tanh(u)
            slope = 0.5 * (1 + th) + 0.5 * z * (1 - th ** 2) * math.sqrt(2.0 / math.pi) * (1 + 3 * 0.044715 * z ** 2)
            d = (d @ layers[i][0]) * slope

    def stepped(p, g):  # Adam's first step
        return p.double() - 1e-4 * g / (g.abs() + 1e-8)

    start = _weights(case, seed)
    return {"loss": loss, "gw": gw, "gb": gb, "w": [stepped(w, g) for (w, _), g in zip(start, gw)],
            "b": [stepped(b, g) for (_, b), g in zip(start, gb)]}
