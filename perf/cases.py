"""Performance cases of the public entry points: what each call gets, runs and returns.

A case is a dict of plain values; its ``kind`` names the entry point:

* ``points``    ``J2ViscoplasticMaterial.update`` on device tensors (row-major points, with
                tangent, energy and dissipation): a material call of a small macro mesh.
* ``soa``       ``batched.j2vp_update_soa`` / ``launch_j2vp_soa``: the streaming return map on
                device-resident structure-of-arrays state, FP64 or FP32, with the full 6x6
                tangent, the compact tangent (n, f, c) or none.
* ``assembly``  ``assemble_hex8_material_response_cached``: strains, J2 update, internal force
                and CSR tangent of a macro bar.
* ``rve``       ``solve_rve_microequilibrium`` of one two-phase concrete box RVE in FP64 with the
                effective tangent: one step of an RVE path or of mixed-control loading.
* ``ogrid``     the same call on the cylindrical O-grid RVE (the general-mesh path).
* ``batch``     ``solve_batch_step`` on a batch of uneven box RVEs, FP32 element kernels,
                device-controlled inexact Newton: path generation for the surrogate.
* ``material``  ``RVEHomogenizedMaterial.update`` with the effective tangent, FP64: the material
                call of implicit FE^2.
* ``window``    ``RNOSurrogate.load_window`` + ``window_gradients``: forward, backward and weight
                gradients of one truncated-BPTT window.
* ``infer``     ``RNOSurrogate.predict``: one surrogate step at the macro points of a bar.
* ``energy``    ``EnergyDissipationRVERNO.update_batch``, with or without the algorithmic tangent.

Materials and sizes are those of the concrete configurations: mortar (J2 Perzyna, E 25 GPa,
nu 0.2, sigma_y 20 MPa, H 2 GPa, viscosity 1e-3 s, exponent 1) and elastic aggregate (E 50 GPa,
nu 0.2), RVE edges 8 to 24, windows of 50 steps and 512 paths, a 64x16x16 macro bar with
131,072 points.  ``exact`` evaluates the same mathematics in float64 torch.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from concrete_impact_b200 import batched
from concrete_impact_b200.assembly import assemble_hex8_material_response_cached, build_hex8_material_assembly_cache
from concrete_impact_b200.energy_rno import EnergyDissipationRVERNO, RVERNOModelConfig
from concrete_impact_b200.materials import (
    J2ViscoplasticMaterial,
    LinearElasticMaterial,
    MaterialPointRequest,
    MaterialResponseRequirements,
    MaterialState,
    MaterialUpdateSettings,
    encode_phase_state_key,
)
from concrete_impact_b200.rno import RNOConfig, RNOScales, RNOSurrogate
from concrete_impact_b200.rve import (
    RS_SIGMA,
    LinearSolverOptions,
    RVEBatch,
    RVERequest,
    RVEState,
    build_rve_operator_cache,
    build_structured_hex8_box,
    solve_batch_step,
    solve_rve_microequilibrium,
)
from concrete_impact_b200.rve_builders import (
    build_cylindrical_ogrid_hex8,
    build_cylindrical_two_phase_rve,
    build_two_phase_sphere_rve,
    default_newton,
    fp32_newton,
)
from concrete_impact_b200.rve_material import RVEHomogenizedMaterial

SETTINGS = MaterialUpdateSettings(50, 1.0e-10, 1.0e-12, 1.0e-10)
YOUNG, POISSON, YIELD, HARDENING, TAU = 25.0e9, 0.2, 20.0e6, 2.0e9, 1.0e-3
AGGREGATE_YOUNG = 50.0e9
EDGES = (8, 12, 16, 20, 24)
F64 = torch.float64


def _mortar(exponent: float = 1.0) -> J2ViscoplasticMaterial:
    return J2ViscoplasticMaterial("mortar", 2200.0, YOUNG, POISSON, YIELD, HARDENING, TAU, YIELD, exponent)


def _aggregate() -> LinearElasticMaterial:
    return LinearElasticMaterial("aggregate", 2600.0, AGGREGATE_YOUNG, POISSON)


# --------------------------------------------------------------------------------------
# The cases.


def listed() -> list[dict]:
    return [
        # the material call of a 24-element macro mesh: host path, launch and latency
        {"name": "points_192", "kind": "points", "n": 192, "exponent": 1.0, "tangent": True},
        # the isolated return map at its largest, FP64 with the full tangent
        {"name": "soa_f64_16m", "kind": "soa", "n": 16_777_216, "bits": 64, "tangent": "full"},
        # FP32, a point count that is no multiple of a vector load
        {"name": "soa_f32_1m_odd", "kind": "soa", "n": 1_000_003, "bits": 32, "tangent": "full"},
        # force and tangent assembly of a 32x8x8 bar of J2 points
        {"name": "assembly_32x8x8", "kind": "assembly", "nx": 32, "ny": 8, "nz": 8, "tangent": True},
        # one FP64 RVE step with its effective tangent, the RVE of the FE^2 runs
        {"name": "rve_8_f64", "kind": "rve", "nx": 8, "ny": 8, "nz": 8},
        # the general-mesh RVE at the size of the O-grid path run
        {"name": "ogrid_32x8x8", "kind": "ogrid", "circumferential": 32, "radial": 8, "axial": 8},
        # uneven FP32 batch, the path-generation workload
        {"name": "batch_96_f32", "kind": "batch", "rves": 96, "cluster": 8},
        # implicit FE^2: 192 macro points, each an 8^3 RVE with its effective tangent
        {"name": "material_192_f64", "kind": "material", "points": 192, "edge": 8},
        # one training window at the training configuration
        {"name": "window_512x50", "kind": "window", "paths": 512, "steps": 50, "skip": False},
        # surrogate step at every macro point of the 64x16x16 bar
        {"name": "infer_131072", "kind": "infer", "points": 131_072, "skip": True},
        # the energy-based surrogate at the same points
        {"name": "energy_131072", "kind": "energy", "points": 131_072, "tangent": False},
        # its algorithmic tangent at the points of a 16x4x4 bar (implicit dynamics)
        {"name": "energy_tangent_2048", "kind": "energy", "points": 2048, "tangent": True},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(("points", "soa", "soa", "assembly", "rve", "ogrid", "batch", "material", "window", "infer",
                       "energy", "energy"))  # fmt: skip
    if kind == "points":
        return {"kind": kind, "n": _log_int(rng, 48, 65_536), "exponent": rng.choice((1.0, 2.0)),
                "tangent": rng.random() < 0.5}  # fmt: skip
    if kind == "soa":
        return {"kind": kind, "n": _log_int(rng, 4096, 12_000_000), "bits": rng.choice((32, 64)),
                "tangent": rng.choice(("full", "full", "compact", "none"))}  # fmt: skip
    if kind == "assembly":
        return {"kind": kind, "nx": rng.randint(4, 40), "ny": rng.randint(1, 8), "nz": rng.randint(1, 8),
                "tangent": rng.random() < 0.6}  # fmt: skip
    if kind == "rve":
        return {"kind": kind, "nx": rng.randint(4, 12), "ny": rng.randint(4, 12), "nz": rng.randint(4, 12)}
    if kind == "ogrid":
        return {"kind": kind, "circumferential": 4 * rng.randint(2, 8), "radial": rng.randint(2, 8),
                "axial": rng.randint(2, 8)}  # fmt: skip
    if kind == "batch":
        cluster = rng.choice((2, 4, 8))
        return {"kind": kind, "rves": _log_int(rng, 8, 12 * cluster), "cluster": cluster}
    if kind == "material":
        return {"kind": kind, "points": _log_int(rng, 8, 192), "edge": rng.choice((4, 6, 7, 8))}
    if kind == "window":
        return {"kind": kind, "paths": _log_int(rng, 64, 1024), "steps": rng.choice((10, 25, 50)),
                "skip": rng.random() < 0.5}  # fmt: skip
    if kind == "infer":
        return {"kind": kind, "points": _log_int(rng, 500, 131_072), "skip": rng.random() < 0.5}
    tangent = rng.random() < 0.4
    return {"kind": "energy", "points": _log_int(rng, 100, 4096 if tangent else 131_072), "tangent": tangent}


# --------------------------------------------------------------------------------------
# Inputs.


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(g: torch.Generator, *shape: int) -> torch.Tensor:
    return torch.rand(shape, generator=g, device="cuda", dtype=F64)


def _randn(g: torch.Generator, *shape: int) -> torch.Tensor:
    return torch.randn(shape, generator=g, device="cuda", dtype=F64)


def _deviatoric(t: torch.Tensor) -> torch.Tensor:
    t = t.clone()
    t[:3] -= t[:3].mean(0, keepdim=True)
    return t


def _point_state(g: torch.Generator, n: int) -> dict[str, torch.Tensor]:
    """(6, n) points near yield: equivalent plastic strain U[0, 0.01], a deviatoric stress at
    U[0.8, 1] of the yield radius and strain increments N(0, 2e-4^2) per component."""
    q = 0.01 * _rand(g, n)
    s = _deviatoric(_randn(g, 6, n))
    norm = torch.sqrt(1.5 * ((s[:3] ** 2).sum(0) + 2.0 * (s[3:] ** 2).sum(0)))
    s *= (0.8 + 0.2 * _rand(g, n)) * (YIELD + HARDENING * q) / norm
    ep = 1.0e-3 * _deviatoric(_randn(g, 6, n))
    return {"q": q, "stress": s, "ep": ep, "de": 2.0e-4 * _randn(g, 6, n)}


def _moduli(young: float) -> tuple[float, float]:
    return young / (2.0 * (1.0 + POISSON)), young / (3.0 * (1.0 - 2.0 * POISSON))


def _prepare_points(case: dict, seed: int) -> dict:
    n, dt = case["n"], 1.0e-5
    p = _point_state(_generator(seed), n)
    shear, bulk = _moduli(YOUNG)
    tr = p["stress"][:3].sum(0)
    elastic = torch.cat([(p["stress"][:3] - tr / 3.0) / (2.0 * shear) + tr / (9.0 * bulk), p["stress"][3:] / shear])
    strain = (elastic + p["ep"] + p["de"]).T.contiguous()
    state = MaterialState({"plastic_strain": p["ep"].T.contiguous(), "equivalent_plastic_strain": p["q"],
                           "viscoplastic_multiplier": p["q"].clone()})  # fmt: skip
    request = MaterialPointRequest(strain, (p["de"] / dt).T.contiguous(), dt, "three_dimensional", SETTINGS)
    return {"material": _mortar(case["exponent"]), "request": request, "state": state,
            "needs": MaterialResponseRequirements(case["tangent"], True, True)}  # fmt: skip


def _prepare_soa(case: dict, seed: int) -> dict:
    n, dtype = case["n"], F64 if case["bits"] == 64 else torch.float32
    p = _point_state(_generator(seed), n)
    state = {"material": _mortar(), "dt": 1.0e-5, "de": p["de"].to(dtype), "tangent": case["tangent"],
             "state": batched.SoAState(p["stress"].to(dtype), p["ep"].to(dtype), p["q"])}  # fmt: skip
    if case["tangent"] == "compact":  # the asynchronous form: the caller owns the outputs
        dev = p["q"].device
        state["out"] = batched.SoAState.empty(n, dtype, dev)
        state["rows"] = torch.empty((8, n), dtype=dtype, device=dev)
        state["flags"] = torch.tensor([-1, 0], dtype=torch.int64, device=dev)
    return state


@functools.lru_cache(maxsize=8)
def _bar(nx: int, ny: int, nz: int):
    nodes, elements = build_structured_hex8_box((0.01 * nx, 0.01 * ny, 0.01 * nz), (nx, ny, nz))
    return nodes, elements, build_hex8_material_assembly_cache(nodes, elements)


def _prepare_assembly(case: dict, seed: int) -> dict:
    nodes, elements, cache = _bar(case["nx"], case["ny"], case["nz"])
    g = _generator(seed)
    x = torch.as_tensor(nodes, device="cuda")
    gradient = 4.0e-4 * _randn(g, 3, 3)
    before = x @ gradient.T
    after = 2.0 * before + 2.0e-6 * _randn(g, *x.shape)
    n = 8 * elements.shape[0]
    state = MaterialState({"plastic_strain": 1.0e-4 * _deviatoric(_randn(g, 6, n)).T.contiguous(),
                           "equivalent_plastic_strain": 2.0e-3 * _rand(g, n), "viscoplastic_multiplier": _rand(g, n)})
    return {"nodes": nodes, "elements": elements, "cache": cache, "material": _mortar(), "state": state, "dt": 1.0e-5,
            "u": after.reshape(-1), "previous": before.reshape(-1), "tangent": case["tangent"]}  # fmt: skip


@functools.lru_cache(maxsize=256)
def _box_model(divisions: tuple[int, int, int], layout: int, bits: int):
    newton = default_newton() if bits == 64 else fp32_newton()
    return build_two_phase_sphere_rve(divisions, _mortar(), _aggregate(), newton, seed=layout)


@functools.lru_cache(maxsize=8)
def _box_cache(divisions: tuple[int, int, int]):
    return build_rve_operator_cache(_box_model(divisions, 0, 64))


@functools.lru_cache(maxsize=8)
def _ogrid(circumferential: int, radial: int, axial: int):
    mesh = build_cylindrical_ogrid_hex8((1.0, 1.0, 1.0), 0.3, circumferential, radial, axial)
    model = build_cylindrical_two_phase_rve(mesh, _mortar(), _aggregate(), default_newton(), 1.0)
    return model, build_rve_operator_cache(model)


@functools.lru_cache(maxsize=8)
def _homogenized(edge: int):
    return RVEHomogenizedMaterial(_box_model((edge, edge, edge), 0, 64), "concrete")


def _history(g: torch.Generator, *lead: int) -> dict[str, torch.Tensor]:
    """A mild loading history at every micro point: residual plastic strains of 2e-5 and
    equivalent plastic strains up to 1e-3."""
    ep = 2.0e-5 * _randn(g, *lead, 6)
    ep[..., :3] -= ep[..., :3].mean(-1, keepdim=True)
    q = 1.0e-3 * _rand(g, *lead)
    return {"plastic_strain": ep, "equivalent_plastic_strain": q, "viscoplastic_multiplier": q.clone()}


def _macro_step(g: torch.Generator, n: int) -> torch.Tensor:
    """(n, 6) macro strain increments of norm 1e-3 to 3e-3: parts of the mortar yield."""
    v = _randn(g, n, 6)
    return v / v.norm(dim=1, keepdim=True) * (1.0e-3 + 2.0e-3 * _rand(g, n, 1))


def _prepare_single(case: dict, seed: int) -> dict:
    if case["kind"] == "rve":
        divisions = (case["nx"], case["ny"], case["nz"])
        model, cache = _box_model(divisions, 0, 64), _box_cache(divisions)
    else:
        model, cache = _ogrid(case["circumferential"], case["radial"], case["axial"])
    g = _generator(seed)
    n = 8 * int((model.element_phase_ids == 0).sum())
    variables = {encode_phase_state_key(model.phase_names[0], k): v for k, v in _history(g, n).items()}
    dofs = torch.zeros(model.constraint.transformation.shape[1], dtype=F64, device="cuda")
    state = RVEState(MaterialState(variables), torch.zeros(6, dtype=F64, device="cuda"), dofs)
    request = RVERequest(_macro_step(g, 1)[0].cpu().numpy(), 1.0e-4, SETTINGS)
    return {"model": model, "cache": cache, "request": request, "state": state}


def _batch_models(rves: int) -> list:
    edges = np.random.default_rng(1000).choice(EDGES, size=rves)
    edges[: len(EDGES)] = EDGES
    return [_box_model((int(e),) * 3, i, 32) for i, e in enumerate(edges)]


def _prepare_batch(case: dict, seed: int) -> dict:
    models = _batch_models(case["rves"])
    options = LinearSolverOptions(cluster=case["cluster"], forcing="eisenstat_walker")
    batch = RVEBatch(models, precision=32, linear_solver=options, device_control=True)
    macro, dt, history = _batch_inputs(models, seed)
    batch.macro.copy_(macro)
    batch.dt.copy_(dt)
    batch.ep_n.copy_(history["plastic_strain"].T)
    batch.q_n.copy_(history["equivalent_plastic_strain"])
    batch.vpm_n.copy_(history["viscoplastic_multiplier"])
    batch.newton_graph(models[0].newton_settings, SETTINGS)
    volume = torch.as_tensor(batch.volumes, device="cuda")[:, None]
    return {"batch": batch, "newton": models[0].newton_settings, "volume": volume}


def _batch_inputs(models: list, seed: int):
    g = _generator(seed)
    macro = _macro_step(g, len(models))
    rate = torch.exp(math.log(1000.0) * _rand(g, len(models)))  # 1 to 1000 per second
    points = 8 * sum(m.elements.shape[0] for m in models)
    phase = torch.as_tensor(np.concatenate([np.repeat(m.element_phase_ids, 8) for m in models]), device="cuda")
    history = _history(g, points)
    for v in history.values():
        v[phase != 0] = 0.0
    return macro, macro.norm(dim=1) / rate, {k: v.float().double() for k, v in history.items()}


def _prepare_material(case: dict, seed: int) -> dict:
    material = _homogenized(case["edge"])
    model, n, g = material.model, case["points"], _generator(seed)
    points = 8 * int((model.element_phase_ids == 0).sum())
    variables = {f"rve_material__{encode_phase_state_key(model.phase_names[0], k)}": v
                 for k, v in _history(g, n, points).items()}  # fmt: skip
    variables["rve_macro_strain"] = torch.zeros((n, 6), dtype=F64, device="cuda")
    variables["rve_fluctuation_dofs"] = torch.zeros((n, 3 * case["edge"] ** 3 - 3), dtype=F64, device="cuda")
    request = MaterialPointRequest(_macro_step(g, n), None, 5.0e-6, "three_dimensional", SETTINGS)
    return {"material": material, "request": request, "state": MaterialState(variables),
            "needs": MaterialResponseRequirements(True, True, True)}  # fmt: skip


def _elastic_stiffness() -> np.ndarray:
    shear, bulk = _moduli(30.0e9)
    c = np.zeros((6, 6))
    c[:3, :3] = bulk - 2.0 * shear / 3.0
    c[range(3), range(3)] += 2.0 * shear
    c[range(3, 6), range(3, 6)] = shear
    return c


SCALES = RNOScales(1.0e-3, 10.0, 20.0e6)


def _surrogate(case: dict, seed: int) -> RNOSurrogate:
    rno = RNOSurrogate(RNOConfig(seed=seed % 1000), SCALES)
    if case["skip"]:
        rno.set_elastic_skip(_elastic_stiffness())
    return rno


def _prepare_window(case: dict, seed: int) -> dict:
    paths, steps, g = case["paths"], case["steps"], _generator(seed)
    strain = (0.2 * _randn(g, steps, paths, 6)).cumsum(0)
    window = (strain, 0.5 * _randn(g, steps, paths, 6), 0.8 * strain + 0.1 * _randn(g, steps, paths, 6),
              0.01 + 0.05 * _rand(g, steps, paths), 0.1 * _randn(g, paths, 6))  # fmt: skip
    return {"rno": _surrogate(case, seed), "window": [t.float() for t in window], "paths": paths, "steps": steps}


def _prepare_infer(case: dict, seed: int) -> dict:
    n, g = case["points"], _generator(seed)
    return {"rno": _surrogate(case, seed), "strain": 1.0e-3 * _randn(g, n, 6), "rate": 10.0 * _randn(g, n, 6),
            "latent": (0.5 * _randn(g, n, 6)).float(), "coef": torch.full((n,), 1.0e-3, device="cuda"),
            "buffers": None}  # fmt: skip


ENERGY_CONFIG = RVERNOModelConfig("energy_rve_rno", "continuous", "current_state_stress_forward_euler", "direct_rate",
                                  0.02, 6, 128, 4, "silu")  # fmt: skip
ENERGY_NETWORKS = (("equilibrium_energy.network.network", 6, 1), ("nonequilibrium_energy.network.network", 12, 1),
                   ("state_evolution.network", 12, 6))  # fmt: skip


def _energy_weights(seed: int) -> dict[str, torch.Tensor]:
    """Weights with the spread of a trained model: U(-1.5, 1.5) / sqrt(fan in)."""
    g, out = _generator(seed + 17), {}
    for prefix, n_in, n_out in ENERGY_NETWORKS:
        for layer in range(5):
            fan = n_in if layer == 0 else 128
            rows = 128 if layer < 4 else n_out
            out[f"{prefix}.{2 * layer}.weight"] = ((3.0 * _rand(g, rows, fan) - 1.5) / math.sqrt(fan)).float()
            if layer < 4 or n_out > 1:
                out[f"{prefix}.{2 * layer}.bias"] = ((_rand(g, rows) - 0.5) / math.sqrt(fan)).float()
    return out


def _energy_inputs(case: dict, seed: int):
    n, g = case["points"], _generator(seed)
    return [t.float() for t in (5.0e-3 * _randn(g, n, 6), 1.0e-2 * _randn(g, n, 6), 1.0e-3 * _rand(g, n))]


def _prepare_energy(case: dict, seed: int) -> dict:
    model = EnergyDissipationRVERNO(ENERGY_CONFIG)
    model.load_state_dict(_energy_weights(seed))
    strain, latent, dt = _energy_inputs(case, seed)
    return {"model": model, "anchors": model.prepare_energy_anchors(), "strain": strain, "latent": latent, "dt": dt,
            "tangent": case["tangent"]}  # fmt: skip


PREPARE = {"points": _prepare_points, "soa": _prepare_soa, "assembly": _prepare_assembly, "rve": _prepare_single,
           "ogrid": _prepare_single, "batch": _prepare_batch, "material": _prepare_material, "window": _prepare_window,
           "infer": _prepare_infer, "energy": _prepare_energy}  # fmt: skip


def prepare(case: dict, seed: int) -> dict:
    return {"kind": case["kind"], **PREPARE[case["kind"]](case, seed)}


# --------------------------------------------------------------------------------------
# One pass.


def _run_points(s: dict) -> dict:
    r = s["material"].update(s["request"], s["state"], s["needs"])
    return {"stress": r.stresses, "tangent": r.tangents, "free_energy": r.free_energy, "dissipation": r.dissipation,
            "state": r.state.variables}  # fmt: skip


def _run_soa(s: dict) -> dict:
    if s["tangent"] == "compact":
        batched.launch_j2vp_soa(s["material"], SETTINGS, s["dt"], s["de"], s["state"], s["out"], s["rows"], s["flags"])
        out, tangent = s["out"], s["rows"]
    else:
        out, tangent = batched.j2vp_update_soa(s["material"], SETTINGS, s["dt"], s["de"], s["state"],
                                               with_tangent=s["tangent"] == "full")  # fmt: skip
    return {"stress": out.stress, "plastic_strain": out.plastic_strain, "eqps": out.eqps, "tangent": tangent}


def _run_assembly(s: dict) -> dict:
    r = assemble_hex8_material_response_cached(s["nodes"], s["elements"], s["material"], s["state"], s["u"],
                                               s["previous"], s["dt"], SETTINGS, s["cache"], s["tangent"])  # fmt: skip
    return {"force": r.internal_force, "tangent": r.tangent.values() if s["tangent"] else None, "stress": r.stresses,
            "strain": r.strains, "state": r.state.variables}  # fmt: skip


def _run_single(s: dict) -> dict:
    r = solve_rve_microequilibrium(s["model"], s["request"], s["state"], s["cache"])
    return {"macro_stress": r.macro_stress, "effective_tangent": r.effective_tangent,
            "fluctuation": r.state.fluctuation_dofs, "state": r.state.material_state.variables,
            "micro_stress": r.micro_stresses, "displacement": r.displacement}  # fmt: skip


def _run_batch(s: dict) -> dict:
    """Solve and homogenise; the fields leave in the precision of the element kernels, as the
    training data of the surrogate does (the solve's own tolerance is that of FP32)."""
    batch = s["batch"]
    solve_batch_step(batch, s["newton"], SETTINGS, False)
    batch.response(batch.batch_struct(SETTINGS), batch.w, None, None)
    return {"macro_stress": (batch.sums[:, RS_SIGMA : RS_SIGMA + 6] / s["volume"]).float(), "stress": batch.stress,
            "plastic_strain": batch.ep, "eqps": batch.q.float(), "fluctuation": batch.w.float()}  # fmt: skip


def _run_material(s: dict) -> dict:
    r = s["material"].update(s["request"], s["state"], s["needs"])
    return {"stress": r.stresses, "tangent": r.tangents, "free_energy": r.free_energy, "dissipation": r.dissipation,
            "state": r.state.variables}  # fmt: skip


def _run_window(s: dict) -> list:
    s["rno"].load_window(*s["window"])
    s["rno"].window_gradients(s["steps"], s["paths"])
    return s["rno"].gradients()


def _run_infer(s: dict) -> dict:
    stress, latent, s["buffers"] = s["rno"].predict(s["strain"], s["rate"], s["latent"], s["coef"], s["buffers"])
    return {"stress": stress, "latent": latent}


def _run_energy(s: dict) -> dict:
    r = s["model"].update_batch(s["strain"], s["latent"], s["dt"], s["anchors"], s["tangent"])
    return {"stress": r.stress, "latent": r.latent_state, "rate": r.state_rate, "dissipation": r.dissipation,
            "free_energy": r.free_energy, "energy_increment": r.nonequilibrium_energy_increment,
            "tangent": r.tangent}  # fmt: skip


RUN = {"points": _run_points, "soa": _run_soa, "assembly": _run_assembly, "rve": _run_single, "ogrid": _run_single,
       "batch": _run_batch, "material": _run_material, "window": _run_window, "infer": _run_infer,
       "energy": _run_energy}  # fmt: skip


def run(state: dict):
    return RUN[state["kind"]](state)


# --------------------------------------------------------------------------------------
# Work of one pass: inputs read once, outputs written once, the arithmetic of one residual
# pass (an RVE solve's iterations are not counted: how many there are is the solver's choice).

POINT_FLOPS = 220.0  # return map with its tangent
ELEMENT_FLOPS = 8 * (POINT_FLOPS + 2 * 2 * 72)  # strains and nodal forces around it


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "points":
        values = 6 + 6 + 8 + 6 + 8 + 2 + (36 if case["tangent"] else 0)
        return {"bytes": 8.0 * values * case["n"], "flops": POINT_FLOPS * case["n"]}
    if kind == "soa":
        rows = {"full": 36, "compact": 8, "none": 0}[case["tangent"]]
        return {"bytes": (case["bits"] // 8 * (30 + rows) + 16.0) * case["n"], "flops": POINT_FLOPS * case["n"]}
    if kind == "assembly":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        elements, nodes = nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)
        couplings = (3 * nx + 1) * (3 * ny + 1) * (3 * nz + 1)
        bytes_ = 8.0 * (elements * (8 * 24 + 8 + 8 * (8 + 8 + 12)) + 9 * nodes)
        if case["tangent"]:
            bytes_ += 8.0 * 9 * couplings
        return {"bytes": bytes_, "flops": elements * (ELEMENT_FLOPS + (8 * 6 * 24 * 30 if case["tangent"] else 0))}
    if kind in ("rve", "ogrid", "material", "batch"):
        if kind == "rve":
            elements, solves, width = case["nx"] * case["ny"] * case["nz"], 7, 8
        elif kind == "ogrid":
            c = case["circumferential"] // 4
            elements, solves, width = (c * c + 4 * c * case["radial"]) * case["axial"], 7, 8
        elif kind == "material":
            elements, solves, width = case["points"] * case["edge"] ** 3, 7, 8
        else:
            edges = np.random.default_rng(1000).choice(EDGES, size=case["rves"])
            edges[: len(EDGES)] = EDGES
            elements, solves, width = int((edges**3).sum()), 1, 4
        return {"bytes": float(elements) * (8 * (18 * width + 4 * 8) + 6 * 8), "flops": elements * ELEMENT_FLOPS * solves}
    per_step = 2.0 * (18 * 128 + 2 * 128 * 128 + 128 * 12)
    if kind == "window":
        rows = case["paths"] * case["steps"]
        return {"bytes": 4.0 * (19 * rows + 6 * case["paths"] + 2 * 39_000), "flops": 3 * per_step * rows}
    if kind == "infer":
        return {"bytes": 37.0 * 4 * case["points"], "flops": per_step * case["points"]}
    hidden = 3 * 128 * 128
    update = 2.0 * (7 * hidden + 2 * (6 + 3 * 12) * 128)
    flops = update + (35.0 * 2 * hidden if case["tangent"] else 0.0)
    return {"bytes": 4.0 * (13 + 22 + (36 if case["tangent"] else 0)) * case["points"], "flops": flops * case["points"]}


# --------------------------------------------------------------------------------------
# The same mathematics in float64.

SHEAR_WEIGHT = (1.0, 1.0, 1.0, 2.0, 2.0, 2.0)


def _return_map(trial, q_n, dt, shear, bulk, yielding, exponent=1.0):
    """Perzyna return map of (..., 6) trial stresses; ``shear``, ``bulk`` and ``yielding`` are
    scalars or (...) tensors.  Returns stress, flow direction, multiplier, f and c of the
    consistent tangent K 1(x)1 + f P + c n(x)n."""
    weight = torch.tensor(SHEAR_WEIGHT, dtype=F64, device=trial.device)
    dev = trial.clone()
    dev[..., :3] -= trial[..., :3].mean(-1, keepdim=True)
    q = torch.sqrt(1.5 * (weight * dev * dev).sum(-1))
    over = q - (YIELD + HARDENING * q_n)
    active = (over > 1.0e-10 * torch.clamp(q, min=YIELD)) & yielding
    slope = 3.0 * shear + HARDENING
    if exponent == 1.0:
        hv = TAU * YIELD / dt + slope
        dg = over / hv
    else:
        dg = 0.5 * over / slope
        for _ in range(60):
            ratio = torch.clamp((over - slope * dg) / YIELD, min=1.0e-30)
            f = dg - dt / TAU * ratio**exponent
            dg = dg - f / (1.0 + dt / TAU * exponent * slope / YIELD * ratio ** (exponent - 1.0))
        ratio = torch.clamp((over - slope * dg) / YIELD, min=1.0e-30)
        hv = slope + TAU * YIELD / (dt * exponent * ratio ** (exponent - 1.0))
    zero = torch.zeros_like(q)
    dg = torch.where(active, dg, zero)
    n = torch.where(active[..., None], 1.5 * dev / q[..., None], torch.zeros_like(dev))
    two_g = 2.0 * shear + zero
    f = torch.where(active, two_g - 6.0 * shear**2 * dg / q, two_g)
    c = torch.where(active, 4.0 * shear**2 * (dg / q - 1.0 / hv), zero)
    return trial - (2.0 * shear * dg)[..., None] * n, n, dg, f, c


def _elastic(e, shear, bulk):
    tr = e[..., :3].sum(-1)
    out = torch.empty_like(e)
    out[..., :3] = ((bulk - 2.0 * shear / 3.0) * tr)[..., None] + (2.0 * shear * e[..., :3].movedim(-1, 0)).movedim(0, -1)
    out[..., 3:] = (shear * e[..., 3:].movedim(-1, 0)).movedim(0, -1)
    return out


def _tangent_matrix(n, f, c, bulk):
    p = torch.zeros((6, 6), dtype=F64, device=n.device)
    p[:3, :3] = -1.0 / 3.0
    p[range(3), range(3)] = 2.0 / 3.0
    p[range(3, 6), range(3, 6)] = 0.5
    volumetric = torch.zeros((6, 6), dtype=F64, device=n.device)
    volumetric[:3, :3] = 1.0
    bulk = torch.as_tensor(bulk, dtype=F64, device=n.device).expand(f.shape)
    return (bulk[..., None, None] * volumetric + f[..., None, None] * p
            + c[..., None, None] * n[..., :, None] * n[..., None, :])  # fmt: skip


def _plastic_increment(dg, n):
    return dg[..., None] * n * torch.tensor(SHEAR_WEIGHT, dtype=F64, device=n.device)


def _exact_points(case: dict, seed: int) -> dict:
    s = _prepare_points(case, seed)
    shear, bulk = _moduli(YOUNG)
    eps, dt, v = s["request"].strains, s["request"].time_step, s["state"].variables
    ep, q = v["plastic_strain"], v["equivalent_plastic_strain"]
    yes = torch.ones_like(q, dtype=torch.bool)
    stress, n, dg, f, c = _return_map(_elastic(eps - ep, shear, bulk), q, dt, shear, bulk, yes, case["exponent"])
    inc = _plastic_increment(dg, n)
    ee = eps - (ep + inc)
    energy = 0.5 * (_elastic(ee, shear, bulk) * ee).sum(-1) + 0.5 * HARDENING * (q + dg) ** 2
    dissipation = (stress * inc).sum(-1) / dt - HARDENING * (q + dg) * dg / dt
    return {"stress": stress, "tangent": _tangent_matrix(n, f, c, bulk) if case["tangent"] else None,
            "free_energy": energy, "dissipation": dissipation,
            "state": {"plastic_strain": ep + inc, "equivalent_plastic_strain": q + dg,
                      "viscoplastic_multiplier": v["viscoplastic_multiplier"] + dg}}  # fmt: skip


def _exact_soa(case: dict, seed: int) -> dict:
    s = _prepare_soa(case, seed)
    shear, bulk = _moduli(YOUNG)
    parts = {"stress": [], "plastic_strain": [], "eqps": [], "tangent": []}
    for at in range(0, case["n"], 1 << 22):
        cut = slice(at, at + (1 << 22))
        q = s["state"].eqps[cut]
        trial = s["state"].stress[:, cut].double().T + _elastic(s["de"][:, cut].double().T, shear, bulk)
        stress, n, dg, f, c = _return_map(trial, q, s["dt"], shear, bulk, torch.ones_like(q, dtype=torch.bool))
        parts["stress"].append(stress.T)
        parts["plastic_strain"].append(s["state"].plastic_strain[:, cut].double() + _plastic_increment(dg, n).T)
        parts["eqps"].append(q + dg)
        if case["tangent"] == "full":
            parts["tangent"].append(_tangent_matrix(n, f, c, bulk).reshape(-1, 36).T.contiguous())
        elif case["tangent"] == "compact":
            parts["tangent"].append(torch.cat([n.T, f[None], c[None]]))
    return {k: torch.cat(v, -1) if v else None for k, v in parts.items()}


class _Solid:
    """Hex8 operators of meshes side by side, on the periodic classes of each (or its nodes)."""

    def __init__(self, meshes: list[tuple[np.ndarray, np.ndarray, np.ndarray | None]]) -> None:
        a = 1.0 / math.sqrt(3.0)
        points = np.array([(x, y, z) for x in (-a, a) for y in (-a, a) for z in (-a, a)])
        signs = np.array([[2.0 * ((i >> d) & 1) - 1.0 for d in range(3)] for i in range(8)])
        f = 1.0 + points[:, None, :] * signs[None]
        local = 0.125 * np.stack([signs[:, d] * f[..., (d + 1) % 3] * f[..., (d + 2) % 3] for d in range(3)], 2)
        local = torch.as_tensor(local, device="cuda")
        dofs, owner, coords, base = [], [], [], 0
        for r, (nodes, elements, classes) in enumerate(meshes):
            ids = np.arange(nodes.shape[0]) if classes is None else classes
            dofs.append(base + ids[elements])
            owner.append(np.full(elements.shape[0], r))
            coords.append(nodes[elements])
            base += int(ids.max()) + 1
        self.count = base
        self.nodes = torch.as_tensor(np.concatenate(dofs), device="cuda")
        self.owner = torch.as_tensor(np.concatenate(owner), device="cuda")
        jacobian = torch.einsum("eai,qaj->eqij", torch.as_tensor(np.concatenate(coords), device="cuda"), local)
        self.weight = torch.linalg.det(jacobian)
        grad = torch.einsum("qaj,eqji->eqai", local, torch.linalg.inv(jacobian))
        x, y, z = grad.unbind(-1)
        b = torch.zeros((*x.shape[:2], 6, 8, 3), dtype=F64, device="cuda")
        b[:, :, 0, :, 0], b[:, :, 1, :, 1], b[:, :, 2, :, 2] = x, y, z
        b[:, :, 3, :, 1], b[:, :, 3, :, 2] = z, y
        b[:, :, 4, :, 0], b[:, :, 4, :, 2] = z, x
        b[:, :, 5, :, 0], b[:, :, 5, :, 1] = y, x
        self.b = b.reshape(x.shape[0], 48, 24)

    def strain(self, u):
        return torch.bmm(self.b, u[self.nodes].reshape(-1, 24, 1)).reshape(-1, 8, 6)

    def force(self, stress):
        t = (self.weight[..., None] * stress).reshape(-1, 1, 48)
        out = torch.zeros((self.count, 3), dtype=F64, device="cuda")
        return out.index_add_(0, self.nodes.reshape(-1), torch.bmm(t, self.b).reshape(-1, 3))


class _Cells(_Solid):
    """Periodic cells of mortar and aggregate, solved for their fluctuations."""

    def __init__(self, models: list) -> None:
        super().__init__([(m.nodes, m.elements, np.asarray(m.constraint.equivalence_class_ids)) for m in models])
        counts = [int(np.max(m.constraint.equivalence_class_ids)) + 1 for m in models]
        start = np.concatenate([[0], np.cumsum(counts)])
        self.cells = len(models)
        self.cell_of_node = torch.as_tensor(np.repeat(np.arange(len(models)), counts), device="cuda")
        fixed = [s + m.constraint.reference_class for s, m in zip(start, models)]
        self.free = torch.ones((self.count, 1), dtype=F64, device="cuda")
        self.free[torch.as_tensor(fixed, device="cuda")] = 0.0
        phase = np.concatenate([m.element_phase_ids for m in models])
        self.mortar = torch.as_tensor(phase == 0, device="cuda")[:, None].expand(-1, 8)
        mortar = self.mortar.double()
        self.shear, self.bulk = (a * mortar + b * (1.0 - mortar)
                                 for a, b in zip(_moduli(YOUNG), _moduli(AGGREGATE_YOUNG)))  # fmt: skip
        self.volume = torch.zeros(self.cells, dtype=F64, device="cuda").index_add_(0, self.owner, self.weight.sum(1))

    def _sum(self, v):
        return torch.zeros(self.cells, dtype=F64, device="cuda").index_add_(0, self.cell_of_node, v.sum(1))

    def mean(self, v):
        """Volume average of (elements, 8, k) point values per cell."""
        total = torch.zeros((self.cells, v.shape[-1]), dtype=F64, device="cuda")
        return total.index_add_(0, self.owner, (self.weight[..., None] * v).sum(1)) / self.volume[:, None]

    def update(self, macro, w, state, dt):
        eps = macro[self.owner][:, None, :] + self.strain(w)
        trial = _elastic(eps - state["ep"], self.shear, self.bulk)
        return eps, *_return_map(trial, state["q"], dt[self.owner][:, None], self.shear, self.bulk, self.mortar)

    def tangent(self, e, n, f, c):
        tr = e[..., :3].sum(-1)
        out = (0.5 * f)[..., None] * e + (c * (n * e).sum(-1))[..., None] * n
        out[..., :3] += (0.5 * f)[..., None] * e[..., :3] + (self.bulk * tr - f * tr / 3.0)[..., None]
        return out

    def linear(self, rhs, n, f, c, rtol):
        """Conjugate gradients of every cell at once, each to its own tolerance."""
        column = (self.b.reshape(-1, 8, 6, 24) ** 2).sum(2)
        diagonal = torch.zeros((self.count, 3), dtype=F64, device="cuda")
        stiff = (self.weight * (self.bulk + f))[..., None] * column
        diagonal.index_add_(0, self.nodes.reshape(-1), stiff.sum(1).reshape(-1, 3))
        x, r = torch.zeros_like(rhs), rhs * self.free
        z = r / diagonal
        p, rz, goal = z.clone(), self._sum(r * z), rtol * torch.sqrt(self._sum(r * r))
        for k in range(4000):
            ap = self.force(self.tangent(self.strain(p), n, f, c)) * self.free
            live = torch.sqrt(self._sum(r * r)) > goal
            alpha = torch.where(live, rz / self._sum(p * ap), torch.zeros_like(rz))[self.cell_of_node][:, None]
            x, r = x + alpha * p, r - alpha * ap
            z = r / diagonal
            new = self._sum(r * z)
            p, rz = z + torch.where(live, new / rz, torch.zeros_like(rz))[self.cell_of_node][:, None] * p, new
            if k % 16 == 15 and not bool(live.any()):
                break
        return x

    def solve(self, macro, state, dt, tangent=False):
        w, first = torch.zeros((self.count, 3), dtype=F64, device="cuda"), None
        for _ in range(14):
            eps, stress, n, dg, f, c = self.update(macro, w, state, dt)
            r = self.force(stress) * self.free
            norm = float(torch.sqrt(self._sum(r * r)).max())
            first = norm if first is None else first
            if norm <= 1.0e-12 * first:
                break
            w = w - self.linear(r, n, f, c, 1.0e-7)
        out = {"eps": eps, "stress": stress, "n": n, "dg": dg, "w": w, "effective": None}
        if tangent:
            columns = []
            for j in range(6):
                unit = torch.zeros((*f.shape, 6), dtype=F64, device="cuda")
                unit[..., j] = 1.0
                k = self.tangent(unit, n, f, c)
                s = self.linear(self.force(k), n, f, c, 1.0e-13)
                columns.append(self.mean(k - self.tangent(self.strain(s), n, f, c)))
            out["effective"] = torch.stack(columns, 2)
        return out


def _cell_state(cells: _Cells, history: dict) -> dict:
    """Point state over all points of the cells from the mortar points' history."""
    points = cells.mortar.reshape(-1).nonzero()[:, 0]
    total = cells.mortar.numel()
    ep = torch.zeros((total, 6), dtype=F64, device="cuda")
    q = torch.zeros(total, dtype=F64, device="cuda")
    ep[points] = history["plastic_strain"].reshape(-1, 6)
    q[points] = history["equivalent_plastic_strain"].reshape(-1)
    return {"ep": ep.reshape(-1, 8, 6), "q": q.reshape(-1, 8), "points": points}


def _exact_single(case: dict, seed: int) -> dict:
    s = _prepare_single(case, seed)
    model, v = s["model"], s["state"].material_state.variables
    names = {k.split("__", 1)[1]: k for k in v}
    history = {k: v[name] for k, name in names.items()}
    cells = _Cells([model])
    state = _cell_state(cells, history)
    macro = torch.as_tensor(s["request"].macro_strain, device="cuda").reshape(1, 6)
    dt = torch.full((1,), s["request"].time_step, dtype=F64, device="cuda")
    out = cells.solve(macro, state, dt, tangent=True)
    points, dg = state["points"], out["dg"].reshape(-1)
    inc = _plastic_increment(out["dg"], out["n"]).reshape(-1, 6)
    x = torch.as_tensor(model.nodes - model.nodes.min(0), device="cuda")
    e = macro[0]
    sym = torch.stack([e[0], e[5] / 2, e[4] / 2, e[5] / 2, e[1], e[3] / 2, e[4] / 2, e[3] / 2, e[2]]).reshape(3, 3)
    classes = torch.as_tensor(np.asarray(model.constraint.equivalence_class_ids), device="cuda")
    return {"macro_stress": cells.mean(out["stress"])[0], "effective_tangent": out["effective"][0],
            "fluctuation": out["w"][cells.free[:, 0] > 0].reshape(-1),
            "state": {names["plastic_strain"]: history["plastic_strain"] + inc[points],
                      names["equivalent_plastic_strain"]: history["equivalent_plastic_strain"] + dg[points],
                      names["viscoplastic_multiplier"]: history["viscoplastic_multiplier"] + dg[points]},
            "micro_stress": out["stress"].reshape(-1, 6),
            "displacement": (out["w"][classes] + x @ sym).reshape(-1)}  # fmt: skip


def _exact_batch(case: dict, seed: int) -> dict:
    models = _batch_models(case["rves"])
    macro, dt, history = _batch_inputs(models, seed)
    cells = _Cells(models)
    state = {"ep": history["plastic_strain"].reshape(-1, 8, 6), "q": history["equivalent_plastic_strain"].reshape(-1, 8)}
    out = cells.solve(macro, state, dt)
    ep = state["ep"] + _plastic_increment(out["dg"], out["n"])
    return {"macro_stress": cells.mean(out["stress"]), "stress": out["stress"].reshape(-1, 6).T.contiguous(),
            "plastic_strain": ep.reshape(-1, 6).T.contiguous(), "eqps": (state["q"] + out["dg"]).reshape(-1),
            "fluctuation": out["w"].reshape(-1)}  # fmt: skip


def _exact_material(case: dict, seed: int) -> dict:
    s = _prepare_material(case, seed)
    n, v, model = case["points"], s["state"].variables, s["material"].model
    names = {k.split("__")[-1]: k for k in v if k.startswith("rve_material__")}
    history = {k: v[name] for k, name in names.items()}
    cells = _Cells([model] * n)
    state = _cell_state(cells, history)
    dt = torch.full((n,), s["request"].time_step, dtype=F64, device="cuda")
    out = cells.solve(s["request"].strains, state, dt, tangent=True)
    points = state["points"]
    dg = out["dg"].reshape(-1)[points].reshape(n, -1)
    inc = _plastic_increment(out["dg"], out["n"]).reshape(-1, 6)[points].reshape(n, -1, 6)
    q1 = state["q"] + out["dg"]
    ee = out["eps"] - (state["ep"] + _plastic_increment(out["dg"], out["n"]))
    energy = 0.5 * (_elastic(ee, cells.shear, cells.bulk) * ee).sum(-1) + 0.5 * HARDENING * q1**2
    step = s["request"].time_step
    work_ = (out["stress"] * _plastic_increment(out["dg"], out["n"])).sum(-1) / step
    loss = work_ - HARDENING * q1 * out["dg"] / step
    keep = cells.free[:, 0] > 0
    return {"stress": cells.mean(out["stress"]), "tangent": out["effective"], "free_energy": cells.mean(energy[..., None])[:, 0],
            "dissipation": cells.mean(loss[..., None])[:, 0],
            "state": {"rve_macro_strain": s["request"].strains, "rve_fluctuation_dofs": out["w"][keep].reshape(n, -1),
                      names["plastic_strain"]: history["plastic_strain"] + inc,
                      names["equivalent_plastic_strain"]: history["equivalent_plastic_strain"] + dg,
                      names["viscoplastic_multiplier"]: history["viscoplastic_multiplier"] + dg}}  # fmt: skip


def _exact_assembly(case: dict, seed: int) -> dict:
    s = _prepare_assembly(case, seed)
    solid = _Solid([(s["nodes"], s["elements"], None)])
    shear, bulk = _moduli(YOUNG)
    v = {k: t.reshape(-1, 8, *t.shape[1:]) for k, t in s["state"].variables.items()}
    eps = solid.strain(s["u"].reshape(-1, 3))
    ep, q = v["plastic_strain"], v["equivalent_plastic_strain"]
    yes = torch.ones_like(q, dtype=torch.bool)
    stress, n, dg, f, c = _return_map(_elastic(eps - ep, shear, bulk), q, s["dt"], shear, bulk, yes)
    values = None
    if case["tangent"]:
        b = solid.b.reshape(-1, 8, 6, 24)
        ke = torch.einsum("eqia,eq,eqij,eqjb->eab", b, solid.weight, _tangent_matrix(n, f, c, bulk), b)
        dofs = (3 * solid.nodes[..., None] + torch.arange(3, device="cuda")).reshape(-1, 24)
        rows, cols = dofs[:, :, None].expand(-1, -1, 24).reshape(-1), dofs[:, None, :].expand(-1, 24, -1).reshape(-1)
        key, place = torch.unique(rows * (3 * solid.count) + cols, return_inverse=True)
        values = torch.zeros(key.numel(), dtype=F64, device="cuda").index_add_(0, place, ke.reshape(-1))
    state = {"plastic_strain": (ep + _plastic_increment(dg, n)).reshape(-1, 6),
             "equivalent_plastic_strain": (q + dg).reshape(-1),
             "viscoplastic_multiplier": (v["viscoplastic_multiplier"] + dg).reshape(-1)}  # fmt: skip
    return {"force": solid.force(stress).reshape(-1), "tangent": values, "stress": stress.reshape(-1, 6),
            "strain": eps.reshape(-1, 6), "state": state}  # fmt: skip


def _rno_layers(rno: RNOSurrogate) -> list:
    state = rno.state_dict()
    return [[state[f"layers.{i}.{k}"].cuda().double() for k in ("weight", "bias")] for i in range(4)]


def _rno_step(layers, skip, strain, rate, z, coef):
    h = torch.cat([strain, rate, z], 1)
    h = torch.nn.functional.pad(h, (0, layers[0][0].shape[1] - h.shape[1]))
    for w, b in layers[:3]:
        h = torch.nn.functional.gelu(h @ w.T + b)
    y = h @ layers[3][0].T + layers[3][1]
    stress = y[:, :6] if skip is None else y[:, :6] + (strain - z) @ skip.T
    return stress, z + coef[:, None] * y[:, 6:12]


def _exact_window(case: dict, seed: int) -> list:
    s = _prepare_window(case, seed)
    layers = _rno_layers(s["rno"])
    for pair in layers:
        for t in pair:
            t.requires_grad_(True)
    skip = None if s["rno"].skip is None else s["rno"].skip.double()
    strain, rate, target, coef, z = (t.double() for t in s["window"])
    loss = 0.0
    for t in range(case["steps"]):
        stress, z = _rno_step(layers, skip, strain[t], rate[t], z, coef[t])
        loss = loss + ((stress - target[t]) ** 2).sum()
    (loss / (case["paths"] * case["steps"] * 6)).backward()
    return [(w.grad, b.grad) for w, b in layers]


def _exact_infer(case: dict, seed: int) -> dict:
    s = _prepare_infer(case, seed)
    skip = None if s["rno"].skip is None else s["rno"].skip.double()
    stress, z = _rno_step(_rno_layers(s["rno"]), skip, s["strain"] / SCALES.strain, s["rate"] / SCALES.rate,
                          s["latent"].double(), s["coef"].double())  # fmt: skip
    return {"stress": stress * SCALES.stress, "latent": z}


def _exact_energy(case: dict, seed: int) -> dict:
    weights = {k: v.double() for k, v in _energy_weights(seed).items()}
    strain, latent, dt = (t.double() for t in _energy_inputs(case, seed))

    def net(prefix, x):
        for layer in range(4):
            x = torch.nn.functional.silu(x @ weights[f"{prefix}.{2 * layer}.weight"].T + weights[f"{prefix}.{2 * layer}.bias"])
        y = x @ weights[f"{prefix}.8.weight"].T
        return y + weights[f"{prefix}.8.bias"] if f"{prefix}.8.bias" in weights else y

    def potential(prefix, x, graph=False):
        y = net(prefix, x)[:, 0]
        return y, torch.autograd.grad(y.sum(), x, create_graph=graph)[0]

    eq, neq, evo = (name for name, _, _ in ENERGY_NETWORKS)
    tau = ENERGY_CONFIG.reference_time_scale
    rows = {k: [] for k in ("stress", "latent", "rate", "dissipation", "free_energy", "energy_increment", "tangent")}
    zero = torch.zeros((1, 12), dtype=F64, device="cuda", requires_grad=True)
    w0, g0 = potential(eq, zero[:, :6])
    v0, h0 = potential(neq, zero)
    for at in range(0, case["points"], 16_384):
        e = strain[at : at + 16_384].clone().requires_grad_(True)
        z, step = latent[at : at + 16_384], dt[at : at + 16_384, None]
        before = torch.cat([e, z], 1)
        rate = net(evo, before)
        after = z + step / tau * rate
        w, g = potential(eq, e, True)
        _, h1 = potential(neq, before)
        v1 = net(neq, before)[:, 0]
        candidate = torch.cat([e, after], 1)
        v2, h2 = potential(neq, candidate, True)
        stress = (g - g0) + (h2[:, :6] - h0[:, :6])
        if case["tangent"]:
            grads = [torch.autograd.grad(stress[:, i].sum(), e, retain_graph=True)[0] for i in range(6)]
            rows["tangent"].append(torch.stack(grads, 1))
        shift = (e * (g0 + h0[:, :6])).sum(1)
        values = {"stress": stress, "latent": after, "rate": rate / tau, "dissipation": -(h1[:, 6:] * rate / tau).sum(1),
                  "free_energy": w - w0 + v2 - v0 - shift, "energy_increment": v2 - v1}  # fmt: skip
        for k, t in values.items():
            rows[k].append(t.detach())
    return {k: torch.cat(v) if v else None for k, v in rows.items()}


EXACT = {"points": _exact_points, "soa": _exact_soa, "assembly": _exact_assembly, "rve": _exact_single,
         "ogrid": _exact_single, "batch": _exact_batch, "material": _exact_material, "window": _exact_window,
         "infer": _exact_infer, "energy": _exact_energy}  # fmt: skip


def exact(case: dict, seed: int):
    return EXACT[case["kind"]](case, seed)
