"""Performance cases: the work a user of this package has it do, through its public entry points.

Twelve listed cases cover every compute path (Monte-Carlo records of drops and prisms, batched
records, stored CDFs, the learned surrogate in both directions, the wave-stage record, Table-II
diffraction, the deterministic atlas and its composition) from calls of a fraction of a millisecond
to the benchmark's 1e8-ray record; ``draw`` gives more of the same ranges.

  listed() / draw(rng)   cases (dicts of plain values)
  prepare(case, seed)    inputs, plans and handles, made from the seed
  run(state)             one pass, its outputs
  work(case)             bytes and operations the pass cannot do without
  exact(case, seed)      the outputs in plain 64-bit torch / numpy, where they have such a value

Entry points with host outputs (generate_drop_record, generate_hex_record, generate_drop_batch,
Surrogate.gradient) are called as such; the others take device memory, as the command-line programs
and bench.py call them.
"""
from __future__ import annotations

import ctypes as C
import json
import math

import numpy as np
import torch

import ice_crystal_phase_b200 as I
from ice_crystal_phase_b200 import atlas as A
from ice_crystal_phase_b200 import surrogate as S

# The benchmark's oblate shape r/a = 1 - 0.08 cos x - 0.02 cos 2x + 0.005 cos 3x, and the published
# equilibrium shapes of falling drops (Sadeghi et al. 2012, Table I), linear in the radius.
OBLATE = (0.0, -0.08, -0.02, 0.005, 0.0, 0.0, 0.0, 0.0)
TABLE_RADII = (0.4, 1.0, 1.5, 2.0, 2.5, 3.0)
TABLE_SHAPES = ((0, 0, 0, 0, 0, 0, 0, 0),
                (-0.0131, -0.0120, -0.0376, -0.0096, -0.0004, 0.0015, 0.0005, 0),
                (-0.0282, -0.0230, -0.0779, -0.0175, 0.0021, 0.0046, 0.0011, -0.0006),
                (-0.0458, -0.0335, -0.1211, -0.0227, 0.0083, 0.0089, 0.0012, -0.0021),
                (-0.0644, -0.0416, -0.1629, -0.0246, 0.0176, 0.0131, 0.0002, -0.0044),
                (-0.0840, -0.0480, -0.2034, -0.0237, 0.0297, 0.0166, -0.0021, -0.0072))


def listed() -> list[dict]:
    return [
        # the smallest record people make: a preview of a Table-I drop, default chain length; launch
        # latency, the longest chain and the host side of the call count
        {"name": "drop_preview", "kind": "drop", "shape": "table", "radius": 1.5, "nt": 72, "np": 144, "ct": 36,
         "cp": 72, "rays": 100_000, "hits": 1024, "fp64": False, "diffraction": False},
        # the benchmark's record: 1.5 mm oblate drop, 1e8 rays, 900 x 1800 cells, chains of 10
        {"name": "drop_record", "kind": "drop", "shape": "oblate", "radius": 1.5, "nt": 900, "np": 1800, "ct": 900,
         "cp": 1800, "rays": 100_000_000, "hits": 10, "fp64": False, "diffraction": True},
        # a hexagonal column over a plan of eight orientations at the command line's defaults
        {"name": "hex_record", "kind": "hex", "radius": 0.05, "length": 0.2, "nt": 512, "np": 1024, "ct": 512,
         "cp": 1024, "rays": 16_000_000, "nodes": 8, "hits": 1024, "fp64": False},
        # the same command with --precision fp64, a plate over two orientations
        {"name": "hex_record_fp64", "kind": "hex", "radius": 0.1, "length": 0.2, "nt": 180, "np": 360, "ct": 90,
         "cp": 180, "rays": 1_000_000, "nodes": 2, "hits": 1024, "fp64": True},
        # one batch of the dataset orchestrator: 32 drops of every size in one call
        {"name": "drop_batch", "kind": "batch", "records": 32, "nt": 180, "np": 360, "ct": 90, "cp": 180,
         "rays_max": 3_000_000, "hits": 10},
        # a stored CDF of a finished 900 x 1800 histogram (device-resident caller)
        {"name": "cdf_build", "kind": "cdf", "nt": 900, "np": 1800, "ct": 900, "cp": 1800, "density": False},
        # serving: 64 records from the trained network in one call
        {"name": "surrogate_serve", "kind": "serve", "records": 64, "logits": False},
        # training: one gradient of a 16-record step of the trained network's configuration
        {"name": "surrogate_gradient", "kind": "gradient", "records": 16, "nt": 256, "np": 512},
        # one wave-stage record of a 1.0 mm drop at the command line's default lattice and grid
        {"name": "wave_record", "kind": "wave", "radius": 1.0, "lattice": 513, "nt": 360, "np": 720},
        # the Table-II pass on the drop records' 0.1-degree query grid
        {"name": "rainbow_diffraction", "kind": "rainbow", "radius": 0.5, "nt": 1800, "np": 3600},
        # a 28-node atlas of the hexagonal column traced node by node
        {"name": "atlas_nodes", "kind": "atlas_nodes", "it": 6, "ip": 3, "nt": 900, "np": 1800, "subdivisions": 2},
        # one record composed from that atlas: coupling, composition, stored CDF
        {"name": "atlas_record", "kind": "atlas_record", "it": 6, "ip": 3, "nt": 900, "np": 1800, "azimuth": 16,
         "tilt": 8, "spin": 12},
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi) -> dict:
    """Query cells (odd counts among them) and the stored grid that divides them."""
    f = rng.choice((1, 1, 2, 3))
    ct = max(8, _log(rng, lo, hi) // f)
    cp = max(8, int(2 * ct * rng.uniform(0.8, 1.1)))
    return {"nt": ct * f, "np": cp * f, "ct": ct, "cp": cp}


def draw(rng) -> dict:
    kind = rng.choice(("drop", "hex", "drop64", "hex64", "batch", "cdf", "serve", "gradient", "wave", "rainbow",
                       "atlas_nodes", "atlas_record"))
    if kind in ("drop", "drop64"):
        deep = rng.random() < 0.5
        top = 1_000_000 if kind == "drop64" else 30_000_000
        return {"kind": "drop", "shape": rng.choice(("oblate", "table", "table")), "radius": round(rng.uniform(0.1, 3.0), 3),
                **_grid(rng, 48, 900), "rays": _log(rng, 20_000, top), "hits": 1024 if deep else rng.choice((6, 10, 30)),
                "fp64": kind == "drop64", "diffraction": rng.random() < 0.5}
    if kind in ("hex", "hex64"):
        nodes = rng.choice((1, 2, 3, 8, 13))
        top = 1_000_000 if kind == "hex64" else 30_000_000
        return {"kind": "hex", "radius": round(rng.uniform(0.02, 0.2), 4), "length": round(rng.uniform(0.02, 0.6), 4),
                **_grid(rng, 48, 900), "rays": _log(rng, 20_000, top), "nodes": nodes,
                "hits": rng.choice((12, 1024)), "fp64": kind == "hex64"}
    if kind == "batch":
        return {"kind": "batch", "records": rng.randint(2, 64), **_grid(rng, 48, 400), "rays_max": _log(rng, 100_000, 2_000_000),
                "hits": rng.choice((10, 30))}
    if kind == "cdf":
        return {"kind": "cdf", **_grid(rng, 24, 1000), "density": rng.random() < 0.5}
    if kind == "serve":
        return {"kind": "serve", "records": _log(rng, 1, 128), "logits": rng.random() < 0.5}
    if kind == "gradient":
        nt = rng.choice((64, 128, 256))
        return {"kind": "gradient", "records": rng.randint(1, 16), "nt": nt, "np": 2 * nt}
    if kind == "wave":
        nt = rng.randint(60, 400)
        return {"kind": "wave", "radius": round(rng.uniform(0.1, 1.0), 3), "lattice": rng.randint(129, 513), "nt": nt,
                "np": 2 * nt}
    if kind == "rainbow":
        nt = _log(rng, 180, 1800)
        return {"kind": "rainbow", "radius": round(rng.uniform(0.1, 1.0), 3), "nt": nt, "np": 2 * nt - rng.randint(0, 9)}
    it, ip, nt = rng.randint(1, 6), rng.randint(1, 3), _log(rng, 60, 900)
    case = {"kind": kind, "it": it, "ip": ip, "nt": nt, "np": 2 * nt - rng.randint(0, 3)}
    if kind == "atlas_nodes":
        return {**case, "subdivisions": rng.randint(1, 4)}
    return {**case, "azimuth": rng.randint(4, 16), "tilt": rng.randint(2, 8), "spin": rng.randint(2, 12)}


# ------------------------------------------------------------------------------------------ inputs
_context = None
_surrogates: dict = {}


def _ctx() -> I.Context:
    """One context per program, as the command-line programs keep."""
    global _context
    if _context is None:
        torch.cuda.init()
        _context = I.Context(0)
    return _context


def _shape(case: dict, radius: float) -> list[float]:
    if case.get("shape") == "oblate":
        return list(OBLATE)
    return [float(np.interp(radius, TABLE_RADII, [t[k] for t in TABLE_SHAPES])) for k in range(8)]


def _drop_inputs(case: dict, seed: int) -> dict:
    r = np.random.default_rng(seed)
    return {"coefficients": _shape(case, case["radius"]), "radius_mm": case["radius"],
            "interior_index": float(r.uniform(1.330, 1.344)), "inclination_deg": float(r.uniform(5.0, 85.0)),
            "wavelength_nm": float(r.uniform(400.0, 700.0)), "seed": int(r.integers(1, 2 ** 62)), "rays": case["rays"],
            "diffraction": case.get("diffraction", True)}


def _hex_inputs(case: dict, seed: int) -> dict:
    r = np.random.default_rng(seed)
    q = r.normal(size=(case["nodes"], 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    share = r.uniform(0.5, 1.5, case["nodes"])
    samples = np.maximum(1, (share / share.sum() * case["rays"]).astype(np.int64))
    a = math.radians(float(r.uniform(10, 80)))
    return {"quaternions": q, "weights": np.full(case["nodes"], 1.0 / case["nodes"]), "samples": samples,
            "seeds": r.integers(1, 2 ** 62, case["nodes"]), "index": float(r.uniform(1.30, 1.32)),
            "ki": (math.cos(a), -math.sin(a), 0.0)}


def _drop_specs(case: dict, seed: int) -> list[I.DropSpec]:
    """Records of the batched distribution: radius log-uniform in 0.1..3 mm, rays in proportion to
    the drop's area with a floor of a sixtieth."""
    r = np.random.default_rng(seed)
    out = []
    top = case.get("rays_max", 1_000_000)
    for _ in range(case["records"]):
        radius = float(np.exp(r.uniform(math.log(0.1), math.log(3.0))))
        rays = int(min(top, max(top / 60, top * radius * radius / 9.0)))
        out.append(I.DropSpec(_shape({}, radius), radius, float(r.uniform(1.330, 1.344)), rays,
                              seed=int(r.integers(1, 2 ** 62)), inclination_deg=float(r.uniform(-90, 90)),
                              wavelength_nm=float(r.uniform(400, 700)), diffraction=True))
    return out


def _gen(seed: int, salt: int = 0) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 64 + salt)
    return g


def _cdf_values(case: dict, seed: int) -> torch.Tensor:
    """A histogram as a traced record leaves it: a forward-peaked profile with Monte-Carlo noise and
    empty cells."""
    nt, np_ = case["nt"], case["np"]
    g = _gen(seed, 1)
    th = (torch.arange(nt, device="cuda", dtype=torch.float64) + 0.5) * (math.pi / nt)
    profile = (torch.exp(-3 * th) + 0.05)[:, None] * torch.sin(th)[:, None]
    noise = -torch.log(torch.rand(nt, np_, device="cuda", dtype=torch.float64, generator=g) + 1e-12)
    hole = torch.rand(nt, np_, device="cuda", generator=g) < 0.02
    v = torch.where(hole, 0.0, profile * noise) * 1e-3
    return v / torch.sin(th)[:, None] if case["density"] else v


def _parameters() -> np.ndarray:
    return np.load(S.DEFAULT_MODEL, allow_pickle=False)["parameters"]


def _surrogate(records: int, nt: int | None = None) -> I.Surrogate:
    key = (records, nt)
    if key not in _surrogates:
        if nt is None:
            _surrogates[key], _ = S.load(_ctx(), S.DEFAULT_MODEL, max_records=records)
        else:
            fields = json.loads(str(np.load(S.DEFAULT_MODEL, allow_pickle=False)["config"]))
            fields.update(nt=nt, np=2 * nt, max_records=records)
            sur = I.Surrogate(_ctx(), I.surrogate_config(**fields))
            sur.set_parameters(_parameters())
            _surrogates[key] = sur
    return _surrogates[key]


def _targets(case: dict, seed: int) -> torch.Tensor:
    """Cell probabilities of traced records: a smooth pattern with Monte-Carlo noise, FP32."""
    cells = case["nt"] * case["np"]
    g = _gen(seed, 2)
    base = torch.rand(case["records"], 1, case["nt"], 1, device="cuda", generator=g) * 3
    u = torch.rand(case["records"], 1, case["nt"], case["np"], device="cuda", generator=g)
    p = (torch.exp(base) * -torch.log(u + 1e-7)).reshape(case["records"], cells)
    return (p / p.sum(dim=1, keepdim=True)).float().contiguous()


def _focal(case: dict, seed: int) -> torch.Tensor:
    """A focal-stage grid with wobbling primary and secondary bows (144-byte records as 18 doubles)."""
    nt, np_ = case["nt"], case["np"]
    n = nt * np_
    g = _gen(seed, 3)
    deg = (180.0 * (torch.arange(nt, device="cuda", dtype=torch.float64) + 0.5) / nt)[:, None]
    phi = (2 * math.pi * torch.arange(np_, device="cuda", dtype=torch.float64) / np_)[None, :]
    rnd = lambda: torch.rand(nt, np_, device="cuda", dtype=torch.float64, generator=g)  # noqa: E731
    primary = deg > 138.0 + 0.8 * torch.sin(phi) + 0.6 * torch.cos(2 * phi)
    secondary = deg < 129.0 + 0.5 * torch.sin(phi) - 0.4 * torch.cos(3 * phi)
    total = (1 + 8 * primary + 2 * secondary) * (1 + 0.2 * (2 * rnd() - 1))
    split = 0.2 + 0.7 * rnd()
    f = torch.zeros(n, 18, dtype=torch.float64, device="cuda")
    f[:, 4] = (split * total).reshape(-1)
    f[:, 5] = ((1 - split) * total).reshape(-1)
    f[:, 7] = rnd().reshape(-1)
    f[:, 8] = torch.where(primary, 0.5 + 8 * rnd(), 0.0).reshape(-1)
    f[:, 9] = torch.where(secondary, 0.1 + 3 * rnd(), 0.0).reshape(-1)
    words = f.view(torch.int32)
    words[:, 22] = torch.where(primary, (1 + 5 * rnd()).int(), 0).reshape(-1)
    words[:, 23] = torch.where(secondary, (1 + 5 * rnd()).int(), 0).reshape(-1)
    return f


def _rule(case: dict, seed: int) -> dict:
    r = np.random.default_rng(seed)
    f = float(r.uniform(0.6, 0.95))
    return {"quadrature": {"azimuth": case["azimuth"], "tilt": case["tilt"], "spin": case["spin"]},
            "components": [{"kind": "horizontal_gaussian", "sigma_deg": float(r.uniform(4, 15)), "fraction": f},
                           {"kind": "isotropic", "fraction": 1.0 - f}]}


def _atlas_inputs(case: dict, seed: int) -> dict:
    r = np.random.default_rng(seed + 1)
    a = math.radians(float(r.uniform(5, 80)))
    return {"radius": 0.05, "length": float(r.uniform(0.1, 0.3)), "ki": (math.cos(a), -math.sin(a), 0.0),
            "index": float(r.uniform(1.305, 1.32))}


def _atlas_masses(case: dict, seed: int) -> torch.Tensor:
    """Node responses of a prism: a few thousand occupied cells of a node over an empty grid."""
    nodes, cells = (case["it"] + 1) * (case["ip"] + 1), case["nt"] * case["np"]
    g = _gen(seed, 4)
    m = torch.rand(nodes, cells, device="cuda", dtype=torch.float64, generator=g)
    return torch.where(m < 0.9, 0.0, m * 1e-5)


def _hex_area(radius: float, length: float, b) -> float:
    """Projected area of the hexagonal prism along the body direction b."""
    u = np.asarray(b) / np.linalg.norm(b)
    sides = sum(max(0.0, -(math.cos(math.pi * f / 3) * u[0] + math.sin(math.pi * f / 3) * u[2])) for f in range(6))
    return radius * length * sides + 1.5 * math.sqrt(3) * radius * radius * abs(u[1])


def prepare(case: dict, seed: int) -> dict:
    ctx, kind = _ctx(), case["kind"]
    st: dict = {"case": case, "ctx": ctx}
    f64 = lambda n: torch.empty(int(n), dtype=torch.float64, device="cuda")  # noqa: E731
    if kind == "drop":
        st["in"] = _drop_inputs(case, seed)
    elif kind == "hex":
        x = st["in"] = _hex_inputs(case, seed)
        st["plan"] = I.OrientationPlan([I.OrientationNode(tuple(map(float, q)), float(w), int(n), int(s)) for q, w, n, s in
                                        zip(x["quaternions"], x["weights"], x["samples"], x["seeds"])],
                                       int(x["samples"].sum()), 1.0, "")
    elif kind == "batch":
        st["specs"] = _drop_specs(case, seed)
        st["settings"] = I.batch_settings(case["nt"], case["np"], case["ct"], case["cp"], max_internal_hits=case["hits"])
    elif kind == "cdf":
        st.update(values=_cdf_values(case, seed), phi=f64(case["cp"] + 1), theta=f64(case["cp"] * (case["ct"] + 1)),
                  policy=I.CdfPolicy(1e-10, 1e-12, 1.0), report=I.CdfReport())
    elif kind == "serve":
        n = case["records"]
        sur = _surrogate(n)
        st.update(sur=sur, specs=_drop_specs(case, seed), policy=I.CdfPolicy(1e-10, 1e-12, 1.0))
        if case["logits"]:
            st["logits"] = torch.empty(n, sur.cells, dtype=torch.float32, device="cuda")
        else:
            st.update(phi=f64(n * 129), theta=f64(n * 128 * 65))
    elif kind == "gradient":
        st.update(sur=_surrogate(case["records"], case["nt"]), specs=_drop_specs(case, seed), target=_targets(case, seed))
    elif kind == "wave":
        _prepare_wave(st, case, seed)
    elif kind == "rainbow":
        n = case["nt"] * case["np"]
        st.update(focal=_focal(case, seed), edges=torch.empty(n, dtype=torch.int32, device="cuda"),
                  results=torch.empty(n, 5, dtype=torch.float64, device="cuda"), density=f64(n),
                  config=I.diffraction_config(case["radius"]), stats=I.DiffractionStats())
    elif kind == "atlas_nodes":
        x = _atlas_inputs(case, seed)
        nodes = (case["it"] + 1) * (case["ip"] + 1)
        st.update(settings=A.settings(x["radius"], x["length"], x["index"], case["it"], case["ip"], case["nt"],
                                      case["np"], case["subdivisions"]),
                  mass=torch.empty(nodes, case["nt"] * case["np"], dtype=torch.float64, device="cuda"))
    else:
        x = st["in"] = _atlas_inputs(case, seed)
        nodes = (case["it"] + 1) * (case["ip"] + 1)
        rot, w, _ = A.orientation_rule(_rule(case, seed))
        areas = [_hex_area(x["radius"], x["length"], _canonical(i * math.pi / 2 / case["it"], j * math.pi / 6 / case["ip"]))
                 for i in range(case["it"] + 1) for j in range(case["ip"] + 1)]
        st.update(rot=torch.from_numpy(np.ascontiguousarray(rot.reshape(-1, 9))).cuda(), w=torch.from_numpy(w).cuda(),
                  areas=(C.c_double * nodes)(*areas), mass=_atlas_masses(case, seed), coupling=f64(nodes * 2 * case["np"]),
                  out=f64(case["nt"] * case["np"]), phi=f64(case["np"] + 1), theta=f64(case["np"] * (case["nt"] + 1)),
                  policy=I.CdfPolicy(1e-10, 1e-12, 1.0), report=I.CdfReport())
    torch.cuda.synchronize()  # the context has its own stream
    return st


def _prepare_wave(st: dict, case: dict, seed: int) -> None:
    r = np.random.default_rng(seed)
    ctx, w, nt, np_ = st["ctx"], case["lattice"], case["nt"], case["np"]
    a = math.radians(float(r.uniform(10, 40)))
    cfg = I.raindrop_config(case["radius"], float(r.uniform(500, 700)), float(np.float32(r.uniform(1.331, 1.337))),
                            (math.cos(a), -math.sin(a), 0.0), w)
    k = np.array([cfg.incident_direction.x, cfg.incident_direction.y, cfg.incident_direction.z], np.float32)
    e0 = np.array([cfg.incident_basis_x.x, cfg.incident_basis_x.y, cfg.incident_basis_x.z], np.float32)
    nv, n, cells = 4 * w * w, nt * np_, 4 * (w - 1) * (w - 1)
    d = lambda count, dtype=np.float64: I.DeviceArray(ctx, count, dtype)  # noqa: E731
    st.update(cfg=cfg, k=k, e0=e0, kin=(C.c_float * 3)(*map(float, k)), vertices=d(nv, I.VERTEX_DTYPE), second=d(4 * nv, np.float32),
              patches=d(cells, I.PATCH_DTYPE), boxes=d(cells, I.AABB_DTYPE),
              dirs=d(3 * n, np.float32).upload(I.query_directions(nt, np_, k, e0).reshape(-1)), offsets=d(n + 1, np.uint64),
              summaries=d(n, I.SUMMARY_DTYPE), hits=d(4 * n, I.HIT_DTYPE), optical=d(n, I.OPTICAL_DTYPE), focal=d(n, I.FOCAL_DTYPE),
              transitions=d(n, np.uint32), diffraction=d(n, I.DIFFRACTION_DTYPE), indices=d(cells, np.uint32),
              folded=d(max(1024, cells // 64), I.FOLDED_DTYPE), dcfg=I.diffraction_config(case["radius"]),
              density=torch.empty(n, dtype=torch.float64, device="cuda"), phi=torch.empty(np_ + 1, dtype=torch.float64, device="cuda"),
              theta=torch.empty(np_ * (nt + 1), dtype=torch.float64, device="cuda"))


# --------------------------------------------------------------------------------------------- run
def _p(t: torch.Tensor) -> C.c_void_p:
    return C.c_void_p(t.data_ptr())


def run(st: dict):
    case, ctx, kind = st["case"], st["ctx"], st["case"]["kind"]
    if kind == "drop":
        x = st["in"]
        r = I.generate_drop_record(ctx, x["coefficients"], x["radius_mm"], x["interior_index"], case["nt"], case["np"],
                                   x["rays"], seed=x["seed"], inclination_deg=x["inclination_deg"], ct=case["ct"],
                                   cp=case["cp"], max_internal_hits=case["hits"],
                                   precision=I.ICP_FP64 if case["fp64"] else I.ICP_FP32,
                                   wavelength_nm=x["wavelength_nm"], diffraction=x["diffraction"])
        return {"phi": r.phi, "theta": r.theta, "u": r.u_edges, "g": r.report.cdf.g_stored}
    if kind == "hex":
        x = st["in"]
        r = I.generate_hex_record(ctx, case["radius"], case["length"], x["ki"], x["index"], case["nt"], case["np"], st["plan"],
                                  case["ct"], case["cp"], max_internal_hits=case["hits"],
                                  precision=I.ICP_FP64 if case["fp64"] else I.ICP_FP32)
        return {"phi": r.phi, "theta": r.theta, "u": r.u_edges, "g": r.report.cdf.g_stored}
    if kind == "batch":
        r = I.generate_drop_batch(ctx, st["specs"], st["settings"])
        return {"phi": r.phi, "theta": r.theta, "u": r.u_edges}
    if kind == "cdf":
        I.check(I.LIB.icp_phase_cdf_build(ctx.handle, _p(st["values"]), int(case["density"]), case["nt"], case["np"],
                                          0.0, 0.0, case["ct"], case["cp"], C.byref(st["policy"]), _p(st["phi"]),
                                          _p(st["theta"]), C.byref(st["report"])))
        return {"phi": st["phi"], "theta": st["theta"], "g": st["report"].g_stored}
    if kind == "serve":
        if case["logits"]:
            st["sur"].predict(st["specs"], st["logits"].data_ptr())
            return {"logits": st["logits"]}
        st["sur"].generate(st["specs"], 64, 128, st["phi"].data_ptr(), st["theta"].data_ptr(), st["policy"])
        return {"phi": st["phi"], "theta": st["theta"]}
    if kind == "gradient":
        loss, grad = st["sur"].gradient(st["specs"], st["target"].data_ptr())
        return {"loss": loss, "grad": grad}
    if kind == "wave":
        return _run_wave(st)
    if kind == "rainbow":
        I.check(I.LIB.icp_rainbow_diffraction(ctx.handle, _p(st["focal"]), case["nt"], case["np"], C.byref(st["config"]),
                                              _p(st["edges"]), _p(st["results"]), _p(st["density"]), C.byref(st["stats"])))
        return {"edges": st["edges"], "results": st["results"][:, :4], "flags": st["results"].view(torch.int32)[:, 8:],
                "density": st["density"]}
    if kind == "atlas_nodes":
        s, reps = st["settings"], []
        for n in range(st["mass"].shape[0]):
            i, j = divmod(n, s.phi_intervals + 1)
            rep = I.AtlasNodeReport()
            I.check(I.LIB.icp_atlas_trace_node(ctx.handle, C.byref(s), i, j, _p(st["mass"][n]), C.byref(rep)))
            reps.append([rep.projected_area_mm2, rep.escaped_mm2, rep.unresolved_mm2])
        return {"mass": st["mass"], "areas": np.array(reps)[:, :2]}
    x, nodes, expected = st["in"], len(st["areas"]), C.c_double()
    st["coupling"].zero_()
    torch.cuda.current_stream().synchronize()  # the coupling is added to the buffer on the context's stream
    I.check(I.LIB.icp_atlas_coupling(ctx.handle, case["it"], case["ip"], case["np"], x["radius"], x["length"], st["areas"],
                                     _p(st["rot"]), _p(st["w"]), len(st["w"]), (C.c_double * 3)(*x["ki"]), 1.0, 0,
                                     _p(st["coupling"]), C.byref(expected)))
    I.check(I.LIB.icp_atlas_compose(ctx.handle, nodes, case["nt"], case["np"], _p(st["mass"]), _p(st["coupling"]),
                                    _p(st["out"])))
    I.check(I.LIB.icp_phase_cdf_build(ctx.handle, _p(st["out"]), 0, case["nt"], case["np"], 0.0, 0.0, case["nt"],
                                      case["np"], C.byref(st["policy"]), _p(st["phi"]), _p(st["theta"]),
                                      C.byref(st["report"])))
    return {"area": expected.value, "coupling": st["coupling"], "mass": st["out"], "phi": st["phi"], "theta": st["theta"]}


def _run_wave(st: dict) -> dict:
    """rainbow_generate's record path for --stage diffraction --allow-underresolved."""
    case, ctx, cfg, L, ck = st["case"], st["ctx"], st["cfg"], I.LIB, I.check
    w, nt, np_ = case["lattice"], case["nt"], case["np"]
    n, nv = nt * np_, 4 * w * w
    lstats, fstats, dstats = I.LatticeStats(), I.FoldedStats(), I.DiffractionStats()
    npatch, hits, nrec, hist = C.c_uint32(0), C.c_uint64(0), C.c_uint32(0), (C.c_uint64 * 8)()
    ck(L.icp_lattice_trace(ctx.handle, C.byref(cfg), st["vertices"].ptr, st["second"].ptr, C.byref(lstats)))
    ck(L.icp_patch_build(ctx.handle, st["vertices"].ptr, w, w, cfg.grid_half_extent, st["patches"].ptr, st["boxes"].ptr, None,
                         C.byref(npatch), hist))
    for _ in range(2):  # once more with room for all hits when the first guess was short
        rc = L.icp_patch_query(ctx.handle, st["vertices"].ptr, nv, st["patches"].ptr, st["boxes"].ptr, npatch.value,
                               st["dirs"].ptr, n, st["offsets"].ptr, st["summaries"].ptr, st["hits"].ptr,
                               st["hits"].count, C.byref(hits))
        if rc != I.ICP_ERR_CAPACITY:
            break
        st["hits"] = I.DeviceArray(ctx, hits.value, I.HIT_DTYPE)
    ck(rc)
    fc = I.FocalConfig(w, w, cfg.grid_half_extent, 0, (C.c_uint32 * 4)(0, 0, 0, 0))
    for _ in range(2):
        rc = L.icp_folded_prepare(ctx.handle, st["vertices"].ptr, nv, st["patches"].ptr, npatch.value, st["kin"], C.byref(fc), None,
                                  st["indices"].ptr, st["folded"].ptr, st["folded"].count, C.byref(nrec), C.byref(fstats))
        if rc != I.ICP_ERR_CAPACITY:
            break
        st["folded"] = I.DeviceArray(ctx, nrec.value, I.FOLDED_DTYPE)
    ck(rc)
    inp = I.OpticsInput(st["vertices"].ptr, st["patches"].ptr, st["dirs"].ptr, st["offsets"].ptr, st["summaries"].ptr,
                        st["hits"].ptr, st["second"].ptr, hits.value, nv, npatch.value, n, nv, I.Vec3f(*map(float, st["k"])),
                        I.Vec3f(*map(float, st["e0"])), 1, 0)
    view = I.FoldedView(st["indices"].ptr, st["folded"].ptr, npatch.value, nrec.value)
    ck(L.icp_patch_optics_folded(ctx.handle, C.byref(inp), st["optical"].ptr, C.byref(fc), st["focal"].ptr,
                                 C.byref(view) if nrec.value else None))
    ck(L.icp_rainbow_diffraction(ctx.handle, st["focal"].ptr, nt, np_, C.byref(st["dcfg"]), st["transitions"].ptr,
                                 st["diffraction"].ptr, None, C.byref(dstats)))
    drep, crep, pol = I.DensityReport(), I.CdfReport(), I.CdfPolicy(1e-10, 1e-12, 1.0)
    ck(L.icp_stage_density(ctx.handle, I.WAVE_STAGES["diffraction"], st["optical"].ptr, st["focal"].ptr, st["diffraction"].ptr, n,
                           _p(st["density"]), C.byref(drep)))
    out = {"counts": [hits.value, npatch.value, nrec.value, dstats.filtered_directions, drep.incomplete],
           "density": st["density"]}
    if drep.invalid_values or drep.incomplete or not drep.maximum > 0:
        return out  # a lattice too coarse for its grid: rainbow_generate rejects the record here
    ck(L.icp_phase_cdf_build(ctx.handle, _p(st["density"]), 1, nt, np_, 0.0, 0.0, nt, np_, C.byref(pol), _p(st["phi"]),
                             _p(st["theta"]), C.byref(crep)))
    return {**out, "phi": st["phi"], "theta": st["theta"]}


# -------------------------------------------------------------------------------------------- work
def work(case: dict) -> dict:
    """Each input read once and each output written once; operations as the algorithm's own count
    (bench.py: per prism interaction 296, per drop interaction 347 + 2 surface evaluations of 110)."""
    kind = case["kind"]
    if kind in ("drop", "hex", "batch"):
        rays = case.get("rays") or int(case["records"] * case["rays_max"] * 0.2)
        steps = min(case["hits"], 10.6)
        per = 250 + 296 * steps if kind == "hex" else 370 + 570 * steps
        stored = 8.0 * case["cp"] * (case["ct"] + 1) * case.get("records", 1)
        return {"bytes": stored + 8.0 * case["nt"] * case["np"] * case.get("records", 1), "flops": per * rays}
    if kind == "cdf":
        return {"bytes": 8.0 * (case["nt"] * case["np"] + case["cp"] * (case["ct"] + 2)), "flops": 6.0 * case["nt"] * case["np"]}
    if kind == "serve":
        n, cells = case["records"], 256 * 512
        return {"bytes": 4.0 * n * (cells if case["logits"] else 2 * 128 * 65) + 2.0 * cells * 112,
                "flops": 2.0 * n * cells * (128 * 256 + 2 * 256 * 256 + 256)}
    if kind == "gradient":
        cells = case["nt"] * case["np"]
        return {"bytes": 4.0 * case["records"] * cells + 2.0 * cells * 112,
                "flops": 2.0 * case["records"] * cells * (2 * 128 * 256 + 6 * 256 * 256 + 3 * 256)}
    n = case["nt"] * case["np"]
    if kind == "wave":
        v = 4 * case["lattice"] ** 2
        return {"bytes": 84.0 * v + (144 + 144 + 40 + 32 + 16) * n, "flops": 2000.0 * v / 4 + 3000.0 * n}
    if kind == "rainbow":
        return {"bytes": 96.0 * n, "flops": 10.0 * n}
    nodes = (case["it"] + 1) * (case["ip"] + 1)
    if kind == "atlas_nodes":
        rays = 200.0 * case["subdivisions"] ** 2 / 4
        return {"bytes": 8.0 * nodes * n, "flops": nodes * rays * 5000}
    weights = 2 * case["azimuth"] * case["tilt"] * case["spin"] * 4 / 3  # nonzero weights of such a rule, about
    return {"bytes": 8.0 * n * (nodes + 2), "flops": 2.0 * n * weights}


# ------------------------------------------------------------------------------------------- exact
def exact(case: dict, seed: int):
    """The outputs of run() in 64 bits.  None for the wave record and the atlas nodes: a record of a
    lattice of bilinear patches is defined by its binary32 vertices, and the node directions lie on
    the prism's symmetry planes, where exits fall exactly on cell edges and the library's rounding
    rule says which cell takes them."""
    kind = case["kind"]
    if kind == "drop":
        x = _drop_inputs(case, seed)
        if case["fp64"] and case["hits"] > 100 and case["rays"] > 300_000:
            return None  # chains of a thousand bounces: minutes of plain torch at this size
        return _stored(_exact_drop(case, x), case)
    if kind == "hex":
        return _stored(_exact_hex(case, _hex_inputs(case, seed)), case)
    if kind == "batch":
        parts = [_stored(_exact_drop(case, {**vars(sp)}), case) for sp in _drop_specs(case, seed)]
        return {"phi": torch.stack([p["phi"] for p in parts]), "theta": torch.stack([p["theta"] for p in parts]),
                "u": parts[0]["u"]}
    if kind == "cdf":
        v = _cdf_values(case, seed)
        if case["density"]:
            v = v * _edges(case["nt"]).diff()[:, None]
        out = _stored(v, case)
        del out["u"]
        out["theta"] = out["theta"].reshape(-1)
        return out
    if kind == "serve":
        return _exact_serve(case, seed)
    if kind == "gradient":
        return _exact_gradient(case, seed)
    if kind == "rainbow":
        return _exact_rainbow(case, seed)
    if kind == "atlas_record":
        return _exact_atlas_record(case, seed)
    return None


_D = {"dtype": torch.float64, "device": "cuda"}


def _edges(nt: int) -> torch.Tensor:
    e = torch.sin(0.5 * math.pi * torch.arange(nt + 1, **_D) / nt) ** 2
    e[-1] = 1.0
    return e


def _stored(mass: torch.Tensor, case: dict) -> dict:
    """The stored CDF of a cell-mass grid [nt][np]."""
    nt, np_, ct, cp = case["nt"], case["np"], case.get("ct", case["nt"]), case.get("cp", case["np"])
    m = mass.reshape(ct, nt // ct, cp, np_ // cp).sum(dim=(1, 3)).t()
    u = _edges(nt)[:: nt // ct]
    col = m.cumsum(1)
    theta = torch.zeros(cp, ct + 1, **_D)
    theta[:, 1:] = torch.where(col[:, -1:] > 0, col / col[:, -1:], u[1:])
    phi = torch.zeros(cp + 1, **_D)
    phi[1:] = col[:, -1].cumsum(0) / col[:, -1].sum()
    g = (m * (1 - u[:-1] - u[1:])).sum() / m.sum()
    return {"phi": phi, "theta": theta, "u": u, "g": float(g)}


def _mix(x: torch.Tensor) -> torch.Tensor:
    """SplitMix64's finaliser on wrapping int64."""
    s = lambda v, k: (v >> k) & ((1 << (64 - k)) - 1)  # noqa: E731
    x = (x ^ s(x, 30)) * (0xBF58476D1CE4E5B9 - (1 << 64))
    x = (x ^ s(x, 27)) * (0x94D049BB133111EB - (1 << 64))
    return x ^ s(x, 31)


def _uniform(seed: int, ids: torch.Tensor, dim: int) -> torch.Tensor:
    x = (3 * ids + dim + 1) * (0x9E3779B97F4A7C15 - (1 << 64)) + seed
    return (((_mix(x) >> 12) & ((1 << 52) - 1)).double() + 0.5) * 2.0 ** -52


def _dot(a, b):
    return (a * b).sum(0)


def _cross(a, b):
    return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


def _norm(a):
    return a / torch.sqrt(_dot(a, a))


def _interface(d, e, S_, n, ni, nt_):
    """Fresnel split of Stokes vectors [4, rays] at normals n (into the incident medium):
    (frame, reflected direction and Stokes, transmitted direction and Stokes, total reflection)."""
    ci = (-_dot(d, n)).clamp(0, 1)
    s = _cross(d, n)
    sine = torch.sqrt(_dot(s, s))
    s = torch.where(sine > 0, s / sine.clamp_min(1e-300), e)
    c, sg = _dot(e, s), _dot(_cross(d, e), s)
    q = (c * c - sg * sg) * S_[1] + 2 * c * sg * S_[2]
    u = -2 * c * sg * S_[1] + (c * c - sg * sg) * S_[2]
    eta = ni / nt_
    st = eta * sine
    tir = st > 1
    ct = torch.sqrt(((1 - st) * (1 + st)).clamp_min(0)).to(torch.complex128)
    ct = torch.where(tir, 1j * torch.sqrt(((st - 1) * (st + 1)).clamp_min(0)), ct)
    rs = (ni * ci - nt_ * ct) / (ni * ci + nt_ * ct)
    rp = (nt_ * ci - ni * ct) / (nt_ * ci + ni * ct)
    Rs, Rp = rs.abs() ** 2, rp.abs() ** 2
    z = rs * rp.conj()
    hs, hd = 0.5 * (Rs + Rp), 0.5 * (Rs - Rp)
    r = torch.stack([hs * S_[0] + hd * q, hd * S_[0] + hs * q, z.real * u - z.imag * S_[3], z.imag * u + z.real * S_[3]])
    r[0] = torch.where(tir, S_[0], r[0])
    zt = torch.sqrt(((1 - Rs) * (1 - Rp)).clamp_min(0))
    t = torch.stack([S_[0] - r[0], q - r[1], zt * u, zt * S_[3]])
    dr = _norm(d + n * (2 * ci))
    dt = torch.where(tir, d, _norm((d + n * ci) * eta - n * ct.real))
    return s, dr, r, dt, t, tir


def _frame(k):
    k = np.asarray(k, dtype=np.float64) / np.linalg.norm(k)
    a = np.eye(3)[int(np.argmin(np.abs(k)))]
    e0 = a - k * (k @ a)
    e0 /= np.linalg.norm(e0)
    return k, e0, np.cross(k, e0)


class _Bins:
    """Cell masses [nt][np] of directions in the frame (e0, e1, k); near-axial power to the end rows."""

    def __init__(self, case, k, e0, e1):
        self.nt, self.np = case["nt"], case["np"]
        self.m = torch.from_numpy(np.stack([e0, e1, k])).cuda()
        self.mass = torch.zeros(self.nt * self.np, **_D)
        self.edges = _edges(self.nt)

    def add(self, d, power):
        x, y, z = self.m @ d
        s = torch.hypot(x, y)
        u = torch.where(z >= 0, 0.5 * s * s / (1 + z.abs()), 1 - 0.5 * s * s / (1 + z.abs()))
        row = (torch.searchsorted(self.edges, u, right=True) - 1).clamp(0, self.nt - 1)
        col = ((torch.atan2(y, x) / (2 * math.pi) + 0.5) * self.np).long() % self.np
        pole = s <= 2.0 ** -15
        self.mass.index_add_(0, row * self.np + col, torch.where(pole, 0.0, power))
        cap = self.mass.reshape(self.nt, self.np)
        cap[0] += power[pole & (z >= 0)].sum() / self.np
        cap[-1] += power[pole & (z < 0)].sum() / self.np


def _chain(p, d, s, S_, n, n_in, hits, bins, scale, advance, tail=1e-12):
    """The linear reflection chain inside a particle from its entry points (p on the surface with
    outward normals n, external incidence d, frame s): every exit binned."""
    s, dr, r, d, S_, _ = _interface(d, s, S_, n, 1.0, n_in)
    bins.add(dr, r[0] * scale)
    face = None
    for _ in range(hits):
        keep = S_[0] > tail
        if not bool(keep.any()):
            break
        if not bool(keep.all()):
            p, d, s, S_ = p[:, keep], d[:, keep], s[:, keep], S_[:, keep]
        p, n = advance(p, d)
        s, dr, r, dt, t, tir = _interface(d, s, S_, -n, n_in, 1.0)
        bins.add(dt[:, ~tir], (t[0] * scale)[~tir])
        d, S_ = dr, r


def _exact_drop(case: dict, x: dict) -> torch.Tensor:
    a = math.radians(x["inclination_deg"])
    k, e0, e1 = _frame((math.cos(a), -math.sin(a), 0.0))
    c = list(x["coefficients"])
    sphere = not any(c[1:])
    out_r = (1 + c[0] + sum(abs(v) for v in c[1:])) * (1 + 1e-6) + 1e-6
    disk, back = (1 + c[0]) if sphere else out_r, 2 * out_r + 1
    power = np.polynomial.chebyshev.cheb2poly([1 + c[0], *c[1:]])
    power = np.concatenate([power, np.zeros(8 - len(power))])

    def radius(mu):
        r, dr = torch.zeros_like(mu), torch.zeros_like(mu)
        for j in range(7, -1, -1):
            dr = dr * mu + r
            r = r * mu + float(power[j])
        return r, dr

    def gauge(p, d):
        r = torch.sqrt(_dot(p, p))
        rd, mu = _dot(p, d) / r, -p[1] / r
        rm, drm = radius(mu)
        return r / rm - 1, (rd - r / rm * drm * (-d[1] - mu * rd) / r) / rm

    def normal(p):
        r = torch.sqrt(_dot(p, p))
        u = p / r
        mu = -u[1]
        _, drm = radius(mu)
        down = torch.zeros_like(u)
        down[1] = -1
        return _norm(u - (down - u * mu) * (drm / r))

    def root(p, d, sign):  # Newton on the convex gauge from the bounding sphere: monotone
        b, q = _dot(p, d), _dot(p, p) - out_r * out_r
        t = -b + sign * torch.sqrt((b * b - q).clamp_min(0))
        hit = b * b > q
        for _ in range(60):
            h, dh = gauge(p + d * t, d)
            hit = hit & ((sign * dh > 0) | (h <= 1e-12))
            step = torch.where(hit & (h > 0), h / dh, 0.0)
            t = t - step
            if float(step.abs().max()) < 1e-15:
                break
        return p + d * t, hit

    bins = _Bins(case, k, e0, e1)
    kk, ee0, ee1 = (torch.from_numpy(v).cuda()[:, None] for v in (k, e0, e1))
    step, incident = 2_000_000, 0
    for first in range(0, x["rays"], step):
        ids = torch.arange(first, min(first + step, x["rays"]), device="cuda", dtype=torch.int64)
        rad = disk * torch.sqrt(_uniform(x["seed"], ids, 0))
        ang = 2 * math.pi * _uniform(x["seed"], ids, 1)
        o = ee0 * (rad * torch.cos(ang)) + ee1 * (rad * torch.sin(ang)) - kk * back
        d = kk.expand(3, ids.numel())
        p, hit = root(o, d, -1.0)
        p = p[:, hit]
        n = p.shape[1]
        incident += n
        S_ = torch.zeros(4, n, **_D)
        S_[0] = 1
        _chain(p, kk.expand(3, n), ee0.expand(3, n), S_, normal(p), x["interior_index"], case["hits"], bins, 1.0,
               lambda q, w: (lambda y: (y, normal(y)))(root(q, w, 1.0)[0]))
    m = bins.mass.reshape(case["nt"], case["np"])
    if x["diffraction"]:  # Fraunhofer diffraction of the circle of the incident area, with its power
        area = math.pi * (disk * x["radius_mm"]) ** 2 * incident / x["rays"]
        m = m + incident * _airy(case["nt"], area, x["wavelength_nm"])[:, None] / case["np"]
    return m


def _airy(nt: int, area: float, wavelength: float) -> torch.Tensor:
    """Row shares of the Airy pattern over the forward hemisphere."""
    z = 2 * math.pi * math.sqrt(area / math.pi) / (wavelength * 1e-6)
    u = torch.cat([_edges(nt), torch.tensor([0.5], **_D)]).clamp_max(0.5)
    y = z * 2 * torch.sqrt(u * (1 - u))
    enc = 1 - torch.special.bessel_j0(y) ** 2 - torch.special.bessel_j1(y) ** 2
    return enc[:-1].diff() / enc[-1]


def _exact_hex(case: dict, x: dict) -> torch.Tensor:
    k, e0, e1 = _frame(x["ki"])
    half = 0.5 * case["length"] / case["radius"]
    faces = np.array([[math.cos(math.pi * f / 3), 0.0, math.sin(math.pi * f / 3)] for f in range(6)] + [[0, 1, 0], [0, -1, 0]])
    offsets = np.array([math.sqrt(3) / 2] * 6 + [half] * 2)
    corner = np.array([[math.cos(math.pi / 6 + math.pi * f / 3), 0.0, math.sin(math.pi / 6 + math.pi * f / 3)] for f in range(7)])
    N, O, V = (torch.from_numpy(v).cuda() for v in (faces, offsets, corner))
    total = None
    for q, w, samples, seed in zip(x["quaternions"], x["weights"], x["samples"], x["seeds"]):
        R = A_rotation(q)
        kb = R.T @ k
        size = np.maximum(0.0, -(faces @ kb)) * np.array([2 * half] * 6 + [1.5 * math.sqrt(3)] * 2)
        cum, area = np.cumsum(size), size.sum()
        bins = _Bins(case, R.T @ k, R.T @ e0, R.T @ e1)
        fb = torch.from_numpy(_frame(kb)[1]).cuda()[:, None]
        kk = torch.from_numpy(kb).cuda()[:, None]
        for first in range(0, int(samples), 2_000_000):
            ids = torch.arange(first, min(first + 2_000_000, int(samples)), device="cuda", dtype=torch.int64)
            u0, u1, u2 = (_uniform(int(seed), ids, j) for j in range(3))
            f = torch.searchsorted(torch.from_numpy(cum).cuda(), u0 * area, right=True).clamp_max(7)
            n = N[f].t()
            tangent = torch.stack([-n[2], torch.zeros_like(u0), n[0]])
            side = n * (math.sqrt(3) / 2) + tangent * (u1 - 0.5)
            side[1] = (2 * u2 - 1) * half
            j = (6 * u1).long()
            cap = (V[j].t() * (1 - u2) + V[j + 1].t() * u2) * torch.sqrt(6 * u1 - j)
            cap[1] = n[1] * half
            p = torch.where(f < 6, side, cap)
            state = {"face": f}

            def advance(p, d, state=state):
                c = N @ d
                t = (O[:, None] - N @ p) / c
                t = torch.where((c > 1e-14) & (t > 1e-10), t, 1e300)
                t, g = t.min(0)
                return p + d * t, N[g].t()

            S_ = torch.zeros(4, ids.numel(), **_D)
            S_[0] = 1
            _chain(p, kk.expand(3, -1).expand(3, ids.numel()), fb.expand(3, ids.numel()), S_, n, x["index"], case["hits"], bins,
                   float(w * area / samples), advance)
        total = bins.mass if total is None else total + bins.mass
    return total.reshape(case["nt"], case["np"])


def A_rotation(q) -> np.ndarray:
    w, x, y, z = q
    return np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)],
                     [2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
                     [2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]])


def _network_rows(sp, nt: int, np_: int) -> torch.Tensor:
    """The 128 inputs of every cell of one record (16 record, 96 cell and 16 axis features)."""
    unit = lambda v, lo, hi: 2 * (v - lo) / (hi - lo) - 1  # noqa: E731
    a = math.radians(sp.inclination_deg)
    rec = [unit(math.log(sp.radius_mm), math.log(0.1), math.log(3.0)), unit(sp.wavelength_nm, 400.0, 700.0),
           sp.inclination_deg / 90, math.sin(a), math.cos(a),
           unit(math.log(sp.wavelength_nm * 1e-6 / sp.radius_mm), math.log(400e-6 / 3), math.log(700e-6 / 0.1)),
           (sp.interior_index - 1.337) / 0.0065]
    rec += [v * s for v, s in zip(sp.coefficients, (12, 20, 5, 40, 33, 60, 400, 140))] + [0.0]
    i = torch.arange(nt, **_D).repeat_interleave(np_)
    j = torch.arange(np_, **_D).repeat(nt)
    th, ph = math.pi * (i + 0.5) / nt, 2 * math.pi * (j + 0.5) / np_
    cols = [torch.full_like(i, v) for v in rec] + [2 * (i + 0.5) / nt - 1, torch.cos(th), (i == 0).double(), (i == nt - 1).double()]
    for k in range(1, 41):
        cols += [torch.sin(k * th), torch.cos(k * th)]
    cols += [torch.cos(m * (ph - math.pi / 2)) for m in range(1, 13)]
    psi = torch.acos((-math.sin(a) * torch.cos(th) - math.cos(a) * torch.sin(th) * torch.sin(ph - math.pi)).clamp(-1, 1))
    cols += [torch.cos(k * psi) for k in range(1, 17)]
    return torch.stack(cols, 1)


def _network(params) -> list[torch.Tensor]:
    p = torch.as_tensor(params, **_D)
    shapes = ((256, 128), (256,), (256, 256), (256,), (256, 256), (256,), (256,), (1,))
    return [v.reshape(s) for v, s in zip(p.split([int(np.prod(s)) for s in shapes]), shapes)]


def _forward(net, x):
    for w, b in ((net[0], net[1]), (net[2], net[3]), (net[4], net[5])):
        x = torch.nn.functional.silu(x @ w.t() + b)
    return x @ net[6] + net[7]


def _drop_area(sp) -> float:
    """Projected area of an axisymmetric convex drop: half the integral of h (h + h'') over the
    directions of the projection plane, h the support function, which depends on e_y alone."""
    a = math.radians(sp.inclination_deg)
    power = np.polynomial.chebyshev.cheb2poly([1 + sp.coefficients[0], *sp.coefficients[1:]])
    chi = np.linspace(0, math.pi, 4001)
    r = np.polynomial.polynomial.polyval(np.cos(chi), power)
    ang = 2 * math.pi * np.arange(1024) / 1024
    ey = np.cos(a) * np.cos(ang)
    g = r[None, :] * (-np.cos(chi)[None, :] * ey[:, None] + np.sin(chi)[None, :] * np.sqrt(1 - ey ** 2)[:, None])
    at = np.clip(g.argmax(1), 1, 3999)
    rows = np.arange(1024)
    lo, mid, hi = g[rows, at - 1], g[rows, at], g[rows, at + 1]
    h = mid + 0.125 * (hi - lo) ** 2 / np.maximum(2 * mid - hi - lo, 1e-300)
    f = np.fft.rfft(h) / 1024
    return float(math.pi * (f[0].real ** 2 + 2 * np.sum(np.abs(f[1:]) ** 2 * (1 - np.arange(1, 513) ** 2))) * sp.radius_mm ** 2)


def _exact_serve(case: dict, seed: int) -> dict:
    net, out = _network(_parameters()), []
    for sp in _drop_specs(case, seed):
        y = _forward(net, _network_rows(sp, 256, 512))
        if case["logits"]:
            out.append(y)
            continue
        m = torch.softmax(y, 0).reshape(256, 512)
        m = m + _airy(256, _drop_area(sp), sp.wavelength_nm)[:, None] / 512
        out.append(_stored(m, {"nt": 256, "np": 512, "ct": 64, "cp": 128}))
    if case["logits"]:
        return {"logits": torch.stack(out)}
    return {"phi": torch.cat([o["phi"] for o in out]), "theta": torch.cat([o["theta"].reshape(-1) for o in out])}


def _exact_gradient(case: dict, seed: int) -> dict:
    target, n = _targets(case, seed).double(), case["records"]
    params = torch.as_tensor(_parameters(), **_D).requires_grad_()
    loss = 0.0
    for r, sp in enumerate(_drop_specs(case, seed)):
        x = _network_rows(sp, case["nt"], case["np"])
        logq = torch.log_softmax(_forward(_network(params), x), 0)
        p = target[r]
        one = torch.where(p > 0, p * (torch.log(p.clamp_min(1e-300)) - logq), 0.0).sum() / n
        one.backward()
        loss += float(one)
    return {"loss": loss, "grad": params.grad}


def _exact_rainbow(case: dict, seed: int) -> dict:
    nt, np_ = case["nt"], case["np"]
    f = _focal(case, seed)
    sigma = I.diffraction_config(case["radius"]).primary_sigma_rad  # an input: Table II at the radius
    s, p = f[:, 4].reshape(nt, np_), f[:, 5].reshape(nt, np_)
    hits = f.view(torch.int32)[:, 22:24].reshape(nt, np_, 2)
    tot = s + p
    jump = (tot[1:] - tot[:-1]).abs() >= 0.25 * torch.maximum(tot[1:], tot[:-1])
    prim = jump & (hits[:-1, :, 0] == 0) & (hits[1:, :, 0] > 0)
    sec = jump & (hits[:-1, :, 1] > 0) & (hits[1:, :, 1] == 0)
    edges = torch.zeros(nt, np_, dtype=torch.int32, device="cuda")
    edges[:-1] = prim.int() + 2 * sec.int()
    dt, dp, support, inner = math.pi / nt, 2 * math.pi / np_, 4.0, 3.0
    rows = torch.nonzero((edges != 0).any(1)).reshape(-1)
    reach = int(2 * support * sigma / dt) + 3
    lo, hi = max(0, int(rows.min()) - reach), min(nt - 1, int(rows.max()) + reach)
    th = (torch.arange(lo, hi + 1, **_D) + 0.5) * dt
    inf = torch.full((hi - lo + 1, np_), 1e300, **_D)
    near = {1: inf.clone(), 2: inf.clone()}

    def window(radius, fn):
        """fn(row offset, rows, column shift, distance) over the cap around every direction."""
        width = min(np_ // 2, int(math.asin(min(1.0, math.sin(radius) / min(math.sin(float(th[0])), math.sin(float(th[-1]))))) / dp) + 2)
        for off in range(-int(radius / dt) - 2, int(radius / dt) + 3):
            for j in range(-width, width + (1 if 2 * width < np_ else 0)):
                fn(off, j)

    def distance(t, other, j):
        return 2 * torch.asin(torch.sqrt((torch.sin(0.5 * (t - other)) ** 2 + torch.sin(t) * torch.sin(other) * math.sin(0.5 * j * dp) ** 2).clamp(0, 1)))

    at = torch.arange(lo, hi + 1, device="cuda")

    def nearest(off, j):
        r = at + off
        ok = (r >= 0) & (r < nt - 1)
        d = torch.where(ok, distance(th, (r + 1.0) * dt, j), 1e300)[:, None]
        e = edges[r.clamp(0, nt - 1)].roll(-j, 1)
        for kind in (1, 2):
            near[kind] = torch.where(((e & kind) != 0) & (d <= 2 * support * sigma), torch.minimum(near[kind], d / (kind * sigma)), near[kind])

    window(2 * support * sigma, nearest)
    pick2 = near[2] < near[1] - 1e-12
    best = torch.where(pick2, near[2], near[1])
    kind = torch.where(best < support, torch.where(pick2, 2, 1), 0)
    res_s, res_p, sig, blend = (torch.zeros(nt, np_, **_D) for _ in range(4))
    res_s += s
    res_p += p
    flags = torch.zeros(nt, np_, dtype=torch.int32, device="cuda")
    kinds = torch.zeros(nt, np_, dtype=torch.int32, device="cuda")
    x = ((best - inner) / (support - inner)).clamp(0, 1)
    b = 1 - x * x * (3 - 2 * x)
    for q in (1, 2):
        acc = [torch.zeros_like(inf) for _ in range(3)]

        def gather(off, j, q=q, acc=acc):
            r = at + off
            ok = (r >= 0) & (r < nt)
            d = distance(th, (r + 0.5) * dt, j)
            w = torch.where(ok & (d <= support * q * sigma), torch.exp(-0.5 * (d / (q * sigma)) ** 2) * 2 * torch.sin((r + 0.5) * dt) * math.sin(0.5 * dt) * dp, 0.0)[:, None]
            if bool((w > 0).any()):
                rr = r.clamp(0, nt - 1)
                acc[0] += w
                acc[1] += w * s[rr].roll(-j, 1)
                acc[2] += w * p[rr].roll(-j, 1)

        window(support * q * sigma, gather)
        m = kind == q
        cs, cp = s[lo:hi + 1], p[lo:hi + 1]
        res_s[lo:hi + 1] = torch.where(m, cs + b * (acc[1] / acc[0] - cs), res_s[lo:hi + 1])
        res_p[lo:hi + 1] = torch.where(m, cp + b * (acc[2] / acc[0] - cp), res_p[lo:hi + 1])
        sig[lo:hi + 1] = torch.where(m, q * sigma, sig[lo:hi + 1])
        under = (dt > 0.5 * q * sigma) | (torch.sin(th) * dp > 0.5 * q * sigma)
        flags[lo:hi + 1] += torch.where(m, 1 + 2 * under.int()[:, None], 0)
    blend[lo:hi + 1] = torch.where(kind > 0, b, 0.0)
    kinds[lo:hi + 1] = kind.int()
    return {"edges": edges.reshape(-1), "results": torch.stack([v.reshape(-1) for v in (res_s, res_p, sig, blend)], 1),
            "flags": torch.stack([flags.reshape(-1), kinds.reshape(-1)], 1), "density": (res_s + res_p).reshape(-1)}


def _canonical(t: float, p: float) -> np.ndarray:
    return np.array([math.sin(t) * math.cos(p), math.cos(t), math.sin(t) * math.sin(p)])


def _exact_rotations(case: dict, seed: int):
    """The product rule Ry(alpha) Rz(beta) Ry(gamma) at midpoints, per component."""
    rule = _rule(case, seed)
    na, nb, ng = case["azimuth"], case["tilt"], case["spin"]
    mid = (np.arange(nb) + 0.5) / nb
    rots, ws = [], []
    for c in rule["components"]:
        if c["kind"] == "isotropic":
            beta = np.arccos(1 - 2 * mid)
        else:
            sg = math.radians(c["sigma_deg"])
            full = math.erf(math.pi / (2 * math.sqrt(2) * sg))
            beta = math.pi / 2 + math.sqrt(2) * sg * torch.erfinv(torch.from_numpy((2 * mid - 1) * full)).numpy()
        for al in 2 * math.pi * (np.arange(na) + 0.5) / na:
            for be in beta:
                for ga in math.pi / 3 * (np.arange(ng) + 0.5) / ng:
                    ca, sa, cb, sb, cg, sg_ = math.cos(al), math.sin(al), math.cos(be), math.sin(be), math.cos(ga), math.sin(ga)
                    ry = np.array([[ca, 0, sa], [0, 1, 0], [-sa, 0, ca]])
                    rz = np.array([[cb, -sb, 0], [sb, cb, 0], [0, 0, 1]])
                    rots.append(ry @ rz @ np.array([[cg, 0, sg_], [0, 1, 0], [-sg_, 0, cg]]))
                    ws.append(c["fraction"] / (na * nb * ng))
    return np.array(rots), np.array(ws)


def _exact_atlas_record(case: dict, seed: int) -> dict:
    x = _atlas_inputs(case, seed)
    it, ip, np_ = case["it"], case["ip"], case["np"]
    nodes = (it + 1) * (ip + 1)
    k, e0, e1 = _frame(x["ki"])
    rots, ws = _exact_rotations(case, seed)
    wts, expected = np.zeros((nodes, 2, np_)), 0.0
    third = math.pi / 3
    for R, nw in zip(rots, ws):
        b = R.T @ k
        t = math.atan2(math.hypot(b[0], b[2]), abs(b[1]))
        az = math.atan2(b[2], b[0]) % (2 * math.pi)
        sector = min(5, int(az / third))
        p = az - sector * third
        mirror = p > third / 2
        if mirror:
            p, sector = third - p, sector + 1
        sy, sz = (-1.0 if b[1] < 0 else 1.0), (-1.0 if mirror else 1.0)
        c, s = math.cos(sector * third), -math.sin(sector * third)
        ec = np.array([math.cos(t) * math.cos(p), -math.sin(t), math.cos(t) * math.sin(p)])
        ew = R @ np.array([c * ec[0] + s * sz * ec[2], sy * ec[1], -s * ec[0] + c * sz * ec[2]])
        shift = math.atan2(ew @ e1, ew @ e0) / (2 * math.pi) * np_
        low = math.floor(shift)
        frac, q = shift - low, int(sy * sz < 0)
        area = _hex_area(x["radius"], x["length"], b)
        u, v = t / (math.pi / 2) * it, p / (math.pi / 6) * ip
        i0, j0 = min(it - 1, int(u)), min(ip - 1, int(v))
        for i, ai in ((i0, 1 - (u - i0)), (i0 + 1, u - i0)):
            for j, bj in ((j0, 1 - (v - j0)), (j0 + 1, v - j0)):
                row = wts[i * (ip + 1) + j, q]
                row[low % np_] += nw * area * ai * bj * (1 - frac)
                row[(low + 1) % np_] += nw * area * ai * bj * frac
        expected += nw * area
    for n in range(nodes):
        wts[n] /= _hex_area(x["radius"], x["length"], _canonical((n // (ip + 1)) * math.pi / 2 / it, (n % (ip + 1)) * math.pi / 6 / ip))
    mass = _atlas_masses(case, seed).reshape(nodes, case["nt"], np_)
    total = torch.zeros(case["nt"], np_ // 2 + 1, dtype=torch.complex128, device="cuda")
    for n in range(nodes):
        for q in (0, 1):
            cell = mass[n].flip(1) if q else mass[n]
            total += torch.fft.rfft(cell, dim=1) * torch.fft.rfft(torch.from_numpy(wts[n, q]).cuda())
    m = torch.fft.irfft(total, n=np_, dim=1)
    out = _stored(m, case)
    return {"area": expected, "coupling": torch.from_numpy(wts.reshape(-1)), "mass": m.reshape(-1), "phi": out["phi"],
            "theta": out["theta"].reshape(-1)}
