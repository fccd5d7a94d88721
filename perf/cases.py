"""Performance cases: the work users of this package have it do, through its public entry points.

``listed()`` gives fixed cases, ``draw(rng)`` more of the same ranges.  ``prepare(case, seed)`` builds
what a program holds before the call, ``run(state)`` makes one pass, ``work(case)`` states the bytes
and operations a pass cannot do without, and ``exact(case, seed)`` computes the outputs of ``run``
in 64 bits with torch alone.

Kinds of case:

domain   one ``LatticeBoltzmannStep`` (or, call "kernel", the function of ``create_lb_function`` on the
         caller's fields).  call: "sweeps" advances by ``steps`` sweeps and returns the populations;
         "monitor" also takes the FP64 mass, momentum and energy, as a run that watches its
         conservation does; "run" is lbmpy's ``run``: sweeps, then density and velocity into the
         step's host arrays; "restart" first sets the populations from those host arrays.
         walls: "none" (periodic), "channel" (NoSlip on y and z, body force along x), "cavity" (UBB lid
         on y max, NoSlip elsewhere).
batch    a ``LatticeBoltzmannBatch`` of lid-driven cavities of uneven sizes.
sparse   the list-based sweep of a porous medium.
train    one forward and backward pass of the learned closure over a batch of samples.
"""
import math

import numpy as np
import torch

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
LID = 0.05
ITEM = {"float64": 8, "float32": 4, "float16": 2, "bfloat16": 2, "e3m12": 2}
# arithmetic of one cell update, rounded, by method
CELL_FLOPS = {"srt": 250, "trt": 250, "mrt": 600, "cumulant": 1000}
# the closure network 10 -> 32 -> 32 -> 1: weights and biases of three layers, output scale
N_PARAMS = 10 * 32 + 32 + 32 * 32 + 32 + 32 + 1 + 1


def _domain(name, stencil, method, storage, pattern, size, walls, call, steps, sgs="none"):
    c = {"kind": "domain", "stencil": stencil, "method": method, "storage": storage, "pattern": pattern,
         "nx": size[0], "ny": size[1], "nz": size[2], "walls": walls, "call": call, "steps": steps, "sgs": sgs}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a first cavity of a tutorial: double precision, a few steps, density and velocity looked at
        _domain("cavity-24-f64", "D3Q19", "trt", "float64", "pull", (24, 24, 24), "cavity", "run", 10),
        # a validation run: 64^3 Taylor-Green box in FP64 with its conserved sums watched
        _domain("tgv-64-f64", "D3Q19", "trt", "float64", "pull", (64, 64, 64), "none", "monitor", 20),
        # the production channel of the benchmark, in place
        _domain("channel-cumulant-aa", "D3Q27", "cumulant", "float32", "aa", (256, 128, 128), "channel", "sweeps", 10),
        # the same channel from host fields to host fields, as the benchmark's end-to-end figure runs it
        _domain("channel-restart", "D3Q27", "cumulant", "float32", "aa", (256, 128, 128), "channel", "restart", 20),
        # a large eddy simulation on a grid whose sizes come from a geometry, not from a tuner
        _domain("ragged-smagorinsky", "D3Q27", "cumulant", "float32", "pull", (205, 91, 67), "channel", "sweeps", 10,
                "smagorinsky"),
        # mixed precision: 16-bit storage, FP32 collision
        _domain("tgv-256-f16", "D3Q19", "trt", "float16", "pull", (256, 256, 256), "none", "sweeps", 10),
        # the largest box: caller-owned fields, one sweep into the other field
        _domain("box-512-f32", "D3Q19", "trt", "float32", "pull", (512, 512, 512), "none", "kernel", 1),
        # a single large cavity with separate shear and bulk rates
        _domain("cavity-mrt-f32", "D3Q19", "mrt", "float32", "pull", (200, 160, 120), "cavity", "sweeps", 10),
        # a parameter study: many small cavities in one launch per step
        {"name": "batch-64-cavities", "kind": "batch", "cavities": 64, "edge_max": 96, "plan_seed": 0, "steps": 10},
        # flow through a packed bed, stored as a list of fluid cells
        {"name": "sparse-porous-128", "kind": "sparse", "n": 128, "spheres_seed": 0, "steps": 10},
        # decaying turbulence at 128^3 with the learned eddy viscosity in the sweep
        _domain("closure-128", "D3Q27", "cumulant", "float32", "aa", (128, 128, 128), "none", "sweeps", 10, "learned"),
        # training that network: one minibatch
        {"name": "closure-train-65536", "kind": "train", "samples": 65536},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("domain", "batch", "sparse", "train"), (8, 1, 1, 1))[0]
    if kind == "batch":
        return {"kind": "batch", "cavities": _log_int(rng, 4, 48), "edge_max": rng.choice((32, 48, 64, 96)),
                "plan_seed": rng.randrange(1000), "steps": rng.choice((4, 10))}
    if kind == "sparse":
        return {"kind": "sparse", "n": rng.randrange(32, 145), "spheres_seed": rng.randrange(1000),
                "steps": rng.choice((2, 10))}
    if kind == "train":
        return {"kind": "train", "samples": _log_int(rng, 1000, 500000)}
    stencil, method, sgs = rng.choice((
        ("D3Q19", "trt", "none"), ("D3Q19", "trt", "none"), ("D3Q19", "srt", "none"), ("D3Q19", "mrt", "none"),
        ("D3Q27", "trt", "none"), ("D3Q27", "mrt", "none"), ("D3Q27", "cumulant", "none"),
        ("D3Q27", "cumulant", "none"), ("D3Q27", "cumulant", "smagorinsky"), ("D3Q27", "cumulant", "learned")))
    storage = "float32"
    if sgs != "learned":
        storage = rng.choice(("float64", "float32", "float32", "float16", "bfloat16", "e3m12"))
    if (stencil, method) == ("D3Q27", "mrt"):       # built for FP64 / FP32 storage, pull and AA
        storage = "float64" if storage == "float64" else "float32"
    few = sgs == "learned" or (stencil, method) == ("D3Q27", "mrt")
    pattern = rng.choice(("pull", "aa") if few else ("pull", "pull", "aa", "aa", "esotwist"))
    walls = rng.choice(("none", "channel", "cavity") if method != "cumulant" else ("none", "channel"))
    # an e3m12 field is 16-bit codes; a program looks at its density and velocity
    call = rng.choice(("run", "restart") if storage == "e3m12" else ("sweeps", "sweeps", "monitor", "run", "restart"))
    steps = rng.choice((2, 4, 10, 20))
    while True:
        size = tuple(_log_int(rng, 12, 320) for _ in range(3))
        if rng.random() < 0.5:       # many grids are multiples of 8 along x
            size = (max(16, size[0] // 8 * 8),) + size[1:]
        cells = size[0] * size[1] * size[2]
        if 4000 <= cells <= 8_000_000 and 2 * int(stencil[3:]) * ITEM[storage] * cells * steps <= 1.5e10:
            break
    return _domain(None, stencil, method, storage, pattern, size, walls, call, steps, sgs)


# ------------------------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _velocity(case, seed):
    """Initial velocity, [x, y, z, 3] FP32 on the device: Taylor-Green vortex plus seeded noise in
    periodic boxes, seeded noise next to walls."""
    n = (case["nx"], case["ny"], case["nz"])
    noise = torch.rand(n + (3,), generator=_generator(seed), device=DEVICE, dtype=torch.float32) * 2 - 1
    if case["walls"] != "none":
        return noise * (1e-4 if case["walls"] == "channel" else 1e-3)
    if case["sgs"] == "learned":
        return noise * 0.02
    u = noise * 1e-3
    x = torch.arange(n[0], device=DEVICE, dtype=torch.float32) * (2 * math.pi / n[0])
    y = torch.arange(n[1], device=DEVICE, dtype=torch.float32) * (2 * math.pi / n[1])
    u[..., 0] += (0.04 * torch.sin(x)[:, None] * torch.cos(y)[None, :])[:, :, None]
    u[..., 1] -= (0.04 * torch.cos(x)[:, None] * torch.sin(y)[None, :])[:, :, None]
    return u


def _physics(case):
    """(omega, omega_bulk, omega_minus, force, compressible, galilean) of a domain case."""
    force = 1e-7 if case["walls"] == "channel" else 0.0
    if case["method"] == "cumulant":
        return (1.95 if case["walls"] == "channel" else 1.99), 1.0, None, force, True, case["sgs"] == "none"
    if case["method"] == "mrt":
        return 1.8, 1.6, None, force, case["walls"] == "none", False
    minus = 1.8 if case["method"] == "srt" else 1 / (0.1875 / (1 / 1.8 - 0.5) + 0.5)
    return 1.8, None, minus, force, case["walls"] != "cavity", False


def _network_params(seed=0):
    """The closure's parameter vector: W1, b1, W2, b2, W3, b3, output scale."""
    rng = np.random.default_rng(seed)
    p = np.zeros(N_PARAMS, np.float32)
    p[:320] = rng.normal(0, math.sqrt(0.1), 320)
    p[320:352] = rng.normal(0, 0.1, 32)
    p[352:1376] = rng.normal(0, math.sqrt(1 / 32), 1024)
    p[1376:1408] = rng.normal(0, 0.1, 32)
    p[1408:1440] = rng.normal(0, math.sqrt(1 / 32), 32)
    p[1440] = -2.0
    p[1441] = 3e-4
    return torch.from_numpy(p)


def _cavity_sizes(case):
    rng = np.random.default_rng(case["plan_seed"])
    edges = rng.choice(np.arange(16, case["edge_max"] + 1, 8), case["cavities"])
    return [(int(e),) * 3 for e in edges], rng.uniform(1.5, 1.95, (case["cavities"], 2))


def _cavity_velocity(size, seed, k):
    return 1e-3 * (torch.rand(size + (3,), generator=_generator(seed * 1000 + k), device=DEVICE,
                              dtype=torch.float32) * 2 - 1)


def _porous_flags(case):
    """Ghost-layered flags of a periodic box of random spheres: 1 fluid, 2 solid, 0 outside (the
    ghost layers mirror the solid cells of their periodic images)."""
    n = case["n"]
    rng = np.random.default_rng(case["spheres_seed"])
    centres = rng.uniform(0, n, (max(1, int(0.02 * n ** 3 / 27)), 3))
    radii = rng.uniform(3, min(7, n / 4), len(centres))
    solid = np.zeros((n + 2,) * 3, bool)
    ax = np.arange(n)
    for c, r in zip(centres, radii):
        lo = np.maximum(np.floor(c - r).astype(int), 0)
        hi = np.minimum(np.ceil(c + r).astype(int) + 1, n)
        x, y, z = np.meshgrid(*(ax[a:b] for a, b in zip(lo, hi)), indexing="ij")
        solid[lo[0] + 1:hi[0] + 1, lo[1] + 1:hi[1] + 1, lo[2] + 1:hi[2] + 1] |= \
            (x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2 < r * r
    for a in range(3):
        s = np.moveaxis(solid, a, 0)
        s[0], s[n + 1] = s[n], s[1]
    flags = np.zeros((n + 2,) * 3, np.uint8)
    flags[1:-1, 1:-1, 1:-1] = 1
    flags[solid] = 2
    return flags


def _samples(case, seed):
    """Closure features [10, n], target eddy viscosities [n] and weights [n], FP32."""
    g, n = _generator(seed), case["samples"]
    feats = torch.randn(10, n, generator=g, device=DEVICE)
    target = 2e-4 * torch.rand(n, generator=g, device=DEVICE) ** 2
    return feats, target, torch.rand(n, generator=g, device=DEVICE) + 0.1


# ------------------------------------------------------------------------------------- passes
def prepare(case, seed):
    import lbmpy_b200 as L
    if case["kind"] == "train":
        from lbmpy_b200.closure import MLPClosure
        return {"case": case, "closure": MLPClosure(_network_params(), device=DEVICE), "data": _samples(case, seed)}
    if case["kind"] == "batch":
        from lbmpy_b200.batched import lid_driven_cavity_batch
        sizes, rates = _cavity_sizes(case)
        batch = lid_driven_cavity_batch(case["cavities"], seed=case["plan_seed"],
                                        edges=tuple(range(16, case["edge_max"] + 1, 8)), lid_velocity=LID, device=DEVICE)
        assert batch.domain_sizes == sizes
        for k, s in enumerate(sizes):
            batch.set_pdf_fields_from_macroscopic_values(k, 1.0, _cavity_velocity(s, seed, k))
        batch.finalize()
        return {"case": case, "batch": batch}
    if case["kind"] == "sparse":
        from lbmpy_b200 import sparse as S
        rule = L.create_lb_collision_rule(lbm_config=L.LBMConfig(
            stencil=L.Stencil.D3Q19, method=L.Method.TRT, relaxation_rate=1.8, compressible=False, force=(1e-6, 0, 0)))
        mapper = S.SparseLbMapper([tuple(d) for d in rule.method.stencil], _porous_flags(case), 1, 2, 0)
        idx = mapper.create_index_array(1)
        lists = [S.pdf_list(len(mapper), 19, torch.float32, DEVICE) for _ in range(2)]
        u = 1e-3 * (torch.rand(mapper.num_fluid_cells, 3, generator=_generator(seed), device=DEVICE) * 2 - 1).double()
        S.create_macroscopic_value_setter_sparse(rule.method, "f", 1.0, u.cpu().numpy())(lists[0])
        kernel = S.create_lb_function_sparse(S.create_lb_update_rule_sparse(rule, "f", "d", "idx"))
        return {"case": case, "kernel": kernel, "lists": lists, "idx": idx}
    size = (case["nx"], case["ny"], case["nz"])
    omega, bulk, _, force, compressible, galilean = _physics(case)
    kw = {"stencil": L.Stencil[case["stencil"]], "method": L.Method[case["method"].upper()],
          "compressible": compressible, "streaming_pattern": case["pattern"]}
    kw.update({"relaxation_rates": [omega, bulk, 1.0, 1.0]} if case["method"] == "mrt" else {"relaxation_rate": omega})
    if case["stencil"] == "D3Q27" and case["method"] == "mrt":
        kw["relaxation_rates"] = [omega, bulk] + [1.0] * 4
    if force:
        kw["force"] = (force, 0, 0)
    if galilean:
        kw["galilean_correction"] = True
    if case["sgs"] == "smagorinsky":
        kw["subgrid_scale_model"] = (L.SubgridScaleModel.SMAGORINSKY, 0.1)
    elif case["sgs"] == "learned":
        from lbmpy_b200.closure import MLPClosure
        kw["subgrid_scale_model"] = (L.SubgridScaleModel.LEARNED, MLPClosure(_network_params(), device=DEVICE))
    config = L.CreateKernelConfig(data_type="float64" if case["storage"] == "float64" else "float32")
    if case["call"] == "kernel":
        kernel = L.create_lb_function(lbm_config=L.LBMConfig(**kw), config=config,
                                      lbm_optimisation=L.LBMOptimisation(storage_dtype=case["storage"]))
        q = int(case["stencil"][3:])
        fields = [L.create_pdf_array(size, q, dtype=case["storage"], device=DEVICE) for _ in range(2)]
        L.macroscopic_values_setter(kernel.method, 1.0, _velocity(case, seed), fields[0])
        return {"case": case, "kernel": kernel, "fields": fields}
    step = L.LatticeBoltzmannStep(domain_size=size, periodicity=[a not in _walled_axes(case) for a in range(3)],
                                  optimization={"storage_dtype": case["storage"]}, config=config, device=DEVICE, **kw)
    if case["walls"] == "cavity":
        step.boundary_handling.set_boundary(L.UBB((LID, 0, 0)), L.slice_from_direction("N", 3))
    for d in {"none": "", "channel": "NSTB", "cavity": "WESTB"}[case["walls"]]:
        step.boundary_handling.set_boundary(L.NoSlip(), L.slice_from_direction(d, 3))
    step.velocity_array[...] = _velocity(case, seed).cpu().numpy()
    step.set_pdf_fields_from_macroscopic_values()
    return {"case": case, "step": step}


def run(state):
    case = state["case"]
    if case["kind"] == "train":
        loss, grad = state["closure"].loss_and_grad(*state["data"])
        return {"loss": loss.float(), "grad": grad}
    if case["kind"] == "batch":
        state["batch"].run(case["steps"])
        return [state["batch"].pdfs(k) for k in range(state["batch"].n_domains)]
    if case["kind"] == "sparse":
        for _ in range(case["steps"]):
            f, d = state["lists"]
            state["kernel"](f=f, d=d, idx=state["idx"])
            state["lists"] = [d, f]
        return state["lists"][0]
    if case["call"] == "kernel":
        for _ in range(case["steps"]):
            f, d = state["fields"]
            state["kernel"](src=f, dst=d, periodicity=(True, True, True))
            state["fields"] = [d, f]
        return state["fields"][0]
    step = state["step"]
    if case["call"] == "restart":
        step.set_pdf_fields_from_macroscopic_values()
    if case["call"] in ("run", "restart"):
        step.run(case["steps"])
        return {"density": step.density_array, "velocity": step.velocity_array}
    step.run_sweeps(case["steps"])
    if case["call"] == "monitor":
        return {"pdfs": step.current_pdfs, "sums": step.reduce_conserved()}
    return step.current_pdfs


def work(case):
    """Every sweep reads and writes each population of each cell once (a sparse sweep its pull index
    too); the getter reads them once more and the host fields move once."""
    if case["kind"] == "train":
        return {"bytes": 4.0 * case["samples"] * 12, "flops": 6.0 * 1441 * case["samples"]}
    if case["kind"] == "batch":
        cells = sum(a * b * c for a, b, c in _cavity_sizes(case)[0])
        return {"bytes": 2.0 * 19 * 4 * cells * case["steps"], "flops": 600.0 * cells * case["steps"]}
    if case["kind"] == "sparse":
        cells = int((_porous_flags(case) == 1).sum())
        return {"bytes": (2.0 * 19 * 4 + 18 * 4) * cells * case["steps"], "flops": 250.0 * cells * case["steps"]}
    cells, q, item = case["nx"] * case["ny"] * case["nz"], int(case["stencil"][3:]), ITEM[case["storage"]]
    flops = CELL_FLOPS[case["method"]] + (2 * 1441 if case["sgs"] == "learned" else 0)
    total = 2.0 * q * item * cells * case["steps"]
    fields = 4.0 * (8 if item == 8 else 4) * cells          # density and velocity
    if case["call"] in ("monitor", "run", "restart"):
        total += q * item * cells
    if case["call"] in ("run", "restart"):
        total += 2 * fields
    if case["call"] == "restart":
        total += 2 * fields + q * item * cells
    return {"bytes": total, "flops": float(flops) * cells * case["steps"]}


# ------------------------------------------------------------------------------------- 64-bit values
_NAMES = ("C N S W E T B NW NE SW SE TN TS TW TE BN BS BW BE TNE TNW TSE TSW BNE BNW BSE BSW").split()
_UNIT = {"C": (0, 0, 0), "N": (0, 1, 0), "S": (0, -1, 0), "W": (-1, 0, 0), "E": (1, 0, 0), "T": (0, 0, 1),
         "B": (0, 0, -1)}


def _lattice(q):
    c = [tuple(sum(v) for v in zip(*(_UNIT[x] for x in name))) for name in _NAMES[:q]]
    ws = {19: {0: 1 / 3, 1: 1 / 18, 2: 1 / 36}, 27: {0: 8 / 27, 1: 2 / 27, 2: 1 / 54, 3: 1 / 216}}[q]
    return c, [ws[sum(map(abs, v))] for v in c], [c.index(tuple(-x for x in v)) for v in c]


def _walled_axes(case):
    return {"none": (), "channel": (1, 2), "cavity": (0, 1, 2)}[case["walls"]]


def _equilibrium_tables(q):
    """Populations per u_a and per u_a u_b of the second-order continuous Maxwellian equilibrium on
    the stencil's monomial moments."""
    c = _lattice(q)[0]
    mono = [(a, b, d) for a in range(3) for b in range(3) for d in range(3)
            if q == 27 or (a * b * d == 0 and not (a and b and d))]
    assert len(mono) == q
    back = np.linalg.inv(np.array([[np.prod([x ** e for x, e in zip(v, m)]) for v in c] for m in mono], float))
    line = {0: (1, 0, 0), 1: (0, 1, 0), 2: (1 / 3, 0, 1)}        # 1-D moments by power of u

    def part(powers):
        return back @ np.array([np.prod([line[e][p] for e, p in zip(m, powers)]) for m in mono])
    lin = [part([int(k == a) for k in range(3)]) for a in range(3)]
    quad = {(a, b): part([int(k == a) + int(k == b) for k in range(3)]) for a in range(3) for b in range(a, 3)}
    return lin, quad


def _feq(q, rho, u, rho_ref, product):
    """Zero-centred equilibrium populations."""
    c, w, _ = _lattice(q)
    out = []
    if product:
        line = [[0.5 * (1 / 3 + v * v - v), 2 / 3 - v * v, 0.5 * (1 / 3 + v * v + v)] for v in u]
        for v, wi in zip(c, w):
            out.append(rho * line[0][v[0] + 1] * line[1][v[1] + 1] * line[2][v[2] + 1] - wi)
        return torch.stack(out)
    lin, quad = _equilibrium_tables(q)
    for i in range(q):
        e = (rho - 1) * w[i]
        for a in range(3):
            if abs(lin[a][i]) > 1e-14:
                e = e + rho_ref * float(lin[a][i]) * u[a]
        for (a, b), t in quad.items():
            if abs(t[i]) > 1e-14:
                e = e + rho_ref * float(t[i]) * u[a] * u[b]
        out.append(e)
    return torch.stack(out)


def _macro(q, f, force, compressible):
    c = _lattice(q)[0]
    rho = 1 + f.sum(0)
    rho_ref = rho if compressible else torch.ones_like(rho)
    u = []
    for a in range(3):
        j = sum(v[a] * f[i] for i, v in enumerate(c) if v[a])
        u.append((j + (0.5 * force if a == 0 else 0.0)) / rho_ref)
    return rho, u, rho_ref


def _collide_populations(q, f, omega, bulk, minus, force, compressible, method):
    c, w, inv = _lattice(q)
    rho, u, rho_ref = _macro(q, f, force, compressible)
    eq = _feq(q, rho, u, rho_ref, False)
    cf = torch.tensor(c, dtype=torch.float64, device=f.device)
    wf = torch.tensor(w, dtype=torch.float64, device=f.device)
    frc = None
    if force:      # Guo: w_i (3 c.F + 9 (c.F)(c.u) - 3 u.F), relaxed with its moments
        frc = torch.stack([w[i] * force * (3 * v[0] + 9 * v[0] * sum(v[a] * u[a] for a in range(3)) - 3 * u[0])
                           for i, v in enumerate(c)])
    if method in ("srt", "trt"):
        n = eq - f
        out = f + 0.5 * omega * (n + n[inv]) + 0.5 * minus * (n - n[inv])
        if force:
            out = out + 0.5 * (1 - omega / 2) * (frc + frc[inv]) + 0.5 * (1 - minus / 2) * (frc - frc[inv])
        return out
    # weighted-orthogonal MRT, higher moments relaxed with 1: what is left of the non-equilibrium
    # is its shear and its bulk part
    x, y, z = cf.T
    shear = [x * y, x * z, y * z, x * x - y * y, x * x + y * y - 2 * z * z]
    parts = [(p, omega) for p in shear] + [(x * x + y * y + z * z - 1, bulk)]
    out = eq.clone()
    n = f - eq
    if force:      # first moments keep the force, all others (1 - rate / 2) of it
        out += 0.5 * frc
        parts += [(p, 0.0) for p in (x, y, z)]
    for p, r in parts:
        scale = wf * p / (wf * p * p).sum()
        keep = (1 - r) * torch.tensordot(p, n, 1)
        if force:
            keep = keep + (0.5 - r / 2) * torch.tensordot(p, frc, 1)
        for i in range(q):
            if float(scale[i]):
                out[i] += float(scale[i]) * keep
    return out


def _features(p, rho, u):
    """Features of the closure network from the non-equilibrium stress (xx, yy, zz, xy, xz, yz)."""
    pxx, pyy, pzz, pxy, pxz, pyz = p
    off = pxy ** 2 + pxz ** 2 + pyz ** 2
    s2 = pxx ** 2 + pyy ** 2 + pzz ** 2 + 2 * off
    pim = torch.sqrt(2 * s2) / rho
    tr = pxx + pyy + pzz
    dxx, dyy, dzz = (v - tr / 3 for v in (pxx, pyy, pzz))
    d2 = dxx ** 2 + dyy ** 2 + dzz ** 2 + 2 * off
    dn = torch.sqrt(d2)
    tr3 = dxx ** 3 + dyy ** 3 + dzz ** 3 + 3 * (dxx * (pxy ** 2 + pxz ** 2) + dyy * (pxy ** 2 + pyz ** 2) +
                                                 dzz * (pxz ** 2 + pyz ** 2)) + 6 * pxy * pxz * pyz
    u2 = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
    uau = (u[0] * (dxx * u[0] + pxy * u[1] + pxz * u[2]) + u[1] * (pxy * u[0] + dyy * u[1] + pyz * u[2]) +
           u[2] * (pxz * u[0] + pyz * u[1] + dzz * u[2]))
    mx = torch.maximum(torch.maximum(dxx.abs(), dyy.abs()), dzz.abs())
    return torch.stack([torch.log(pim + 1e-9), 100 * pim, tr / (torch.sqrt(s2) + 1e-12),
                        math.sqrt(6) * tr3 / (d2 * dn + 1e-30), 30 * torch.sqrt(u2), 1000 * (rho - 1),
                        uau / ((u2 + 1e-12) * dn + 1e-30), off / (s2 + 1e-30), mx / (dn + 1e-30), 1000 * u2])


def _network(params, x):
    """Eddy viscosity of features x [10, n]."""
    w1, b1 = params[:320].view(10, 32), params[320:352]
    w2, b2 = params[352:1376].view(32, 32), params[1376:1408]
    silu = torch.nn.functional.silu
    h = silu(w1.T @ x + b1[:, None])
    h = silu(w2.T @ h + b2[:, None])
    y = params[1408:1440] @ h + params[1440]
    return params[1441] * torch.nn.functional.softplus(y, threshold=100.0)


def _wick(cov, powers):
    """Moment x^a y^b z^c of a centred Gaussian with covariance cov."""
    axes = [a for a in range(3) for _ in range(powers[a])]
    if not axes:
        return 1.0
    if len(axes) % 2:
        return 0.0
    total = 0.0
    for k in range(1, len(axes)):
        rest = [0, 0, 0]
        for j, a in enumerate(axes):
            if j not in (0, k):
                rest[a] += 1
        total = total + cov[axes[0]][axes[k]] * _wick(cov, rest)
    return total


def _collide_cumulant(f, omega, bulk, force, galilean, sgs):
    """Cumulants of order two relax with omega (shear) and bulk, higher ones with 1: the state after
    the collision is Gaussian in its central moments; the force enters as half before, half after."""
    c, w, _ = _lattice(27)
    rho, u, _ = _macro(27, f, force, True)

    def central(a, b):
        t = 0.0
        for i, v in enumerate(c):
            t = t + (f[i] + w[i]) * (v[a] - u[a]) * (v[b] - u[b])
        return t
    k = {(a, b): central(a, b) for a in range(3) for b in range(a, 3)}
    xx, yy, zz = k[0, 0], k[1, 1], k[2, 2]
    rate = omega
    if sgs is not None:
        neq = [xx - rho / 3 - u[0] * force, yy - rho / 3, zz - rho / 3, k[0, 1] - 0.5 * u[1] * force,
               k[0, 2] - 0.5 * u[2] * force, k[1, 2]]
        if sgs == "smagorinsky":
            s2 = neq[0] ** 2 + neq[1] ** 2 + neq[2] ** 2 + 2 * (neq[3] ** 2 + neq[4] ** 2 + neq[5] ** 2)
            rate = 2 / (1 / omega + torch.sqrt(18 * 0.1 ** 2 * torch.sqrt(2 * s2) / rho + 1 / omega ** 2))
        else:
            x = _features(neq, rho, u)
            nu = _network(_network_params().double().to(f.device), x.reshape(10, -1)).reshape(rho.shape)
            rate = 1 / (1 / omega + 3 * nu)
    d1, d2, tr = (xx - yy) * (1 - rate), (xx - zz) * (1 - rate), xx + yy + zz
    s = tr + bulk * (rho - tr)
    if galilean:
        dx = -omega / (2 * rho) * (2 * xx - yy - zz) - bulk / (2 * rho) * (tr - rho)
        dy = dx + 1.5 * omega / rho * (xx - yy)
        dz = dx + 1.5 * omega / rho * (xx - zz)
        qx, qy, qz = u[0] ** 2 * dx, u[1] ** 2 * dy, u[2] ** 2 * dz
        d1 = d1 - 3 * rho * (1 - omega / 2) * (qx - qy)
        d2 = d2 - 3 * rho * (1 - omega / 2) * (qx - qz)
        s = s - 3 * rho * (1 - bulk / 2) * (qx + qy + qz)
    nxx = (s + d1 + d2) / 3
    off = {ab: k[ab] * (1 - rate) / rho for ab in ((0, 1), (0, 2), (1, 2))}
    cov = [[nxx / rho, off[0, 1], off[0, 2]], [off[0, 1], (nxx - d1) / rho, off[1, 2]],
           [off[0, 2], off[1, 2], (nxx - d2) / rho]]
    zero = torch.zeros_like(rho)
    m = [[[zero + rho * _wick(cov, (a, b, e)) for e in range(3)] for b in range(3)] for a in range(3)]
    m[1][0][0] = m[1][0][0] + 0.5 * force
    m = torch.stack([torch.stack([torch.stack(r) for r in p]) for p in m])        # central moments [a, b, e]
    for axis in range(3):          # moments about u -> populations, one axis at a time
        v = u[axis]
        k0, k1, k2 = m.unbind(axis)
        m1, m2 = k1 + v * k0, k2 + 2 * v * k1 + v * v * k0
        m = torch.stack([0.5 * (m2 - m1), k0 - m2, 0.5 * (m2 + m1)], axis)
    return torch.stack([m[v[0] + 1, v[1] + 1, v[2] + 1] - w[i] for i, v in enumerate(c)])


def _access(q, pattern, odd):
    """(slot, offset) that a step reads and writes per direction."""
    c, _, inv = _lattice(q)
    neg = [tuple(-x for x in v) for v in c]
    if pattern == "pull":
        return [(i, neg[i]) for i in range(q)], [(i, (0, 0, 0)) for i in range(q)]
    if pattern == "aa" and not odd:
        return [(i, (0, 0, 0)) for i in range(q)], [(inv[i], (0, 0, 0)) for i in range(q)]
    if pattern == "aa":
        return [(inv[i], neg[i]) for i in range(q)], [(i, c[i]) for i in range(q)]
    up = [tuple(max(x, 0) for x in v) for v in c]
    down = [tuple(max(-x, 0) for x in v) for v in c]
    if not odd:
        return [(i, down[i]) for i in range(q)], [(inv[i], up[i]) for i in range(q)]
    return [(inv[i], down[i]) for i in range(q)], [(i, up[i]) for i in range(q)]


def _gather(field, off, periodic):
    """Values at x + off of a ghost-layered field, per interior cell x."""
    sl = tuple(slice(1, -1) if periodic[a] else slice(1 + off[a], field.shape[a] - 1 + off[a]) for a in range(3))
    dims = [a for a in range(3) if periodic[a] and off[a]]
    v = field[sl]
    return torch.roll(v, [-off[a] for a in dims], dims) if dims else v


def _scatter(field, off, periodic, values):
    sl = tuple(slice(1, -1) if periodic[a] else slice(1 + off[a], field.shape[a] - 1 + off[a]) for a in range(3))
    dims = [a for a in range(3) if periodic[a] and off[a]]
    field[sl] = torch.roll(values, [off[a] for a in dims], dims) if dims else values


def _simulate(q, pattern, periodic, types, rho, u, steps, collide, product, force, compressible):
    """`steps` steps from the equilibrium at (rho, u); types: ghost-layered cell types (0 fluid, 1
    NoSlip, 2 lid) or None.  Returns the ghost-layered field [q, x, y, z] and the interior values
    that the last step wrote."""
    c, w, inv = _lattice(q)
    inplace = pattern != "pull"
    size = rho.shape
    field = torch.zeros((q,) + tuple(n + 2 for n in size), dtype=torch.float64, device=rho.device)
    shift = 0.5 * force / (rho if compressible else torch.ones_like(rho))
    start = _feq(q, rho, [u[0] - shift, u[1], u[2]], rho if compressible else torch.ones_like(rho), product)
    odd = True
    for i, (slot, off) in enumerate(_access(q, pattern, odd)[1]):
        _scatter(field[slot], off, periodic, start[i])
    post = start
    inner = None if types is None else types[1:-1, 1:-1, 1:-1]
    fluid = inner == 0 if inner is not None and bool(inner.any()) else None
    for _ in range(steps):
        before = _access(q, pattern, odd)[1]
        odd = not odd
        reads, writes = _access(q, pattern, odd)
        f = torch.empty_like(start)
        for i, (slot, off) in enumerate(reads):
            v = _gather(field[slot], off, periodic)
            if types is not None and i:
                kind = _gather(types, tuple(-x for x in c[i]), periodic)
                js, jo = before[inv[i]]
                back = _gather(field[js], jo, periodic)
                v = torch.where(kind == 0, v, back + (kind == 2).double() * (6 * w[i] * c[i][0] * LID))
            f[i] = v
        post = collide(f)
        nxt = field if inplace else torch.zeros_like(field)
        for i, (slot, off) in enumerate(writes):
            v = post[i]
            if fluid is not None:
                v = torch.where(fluid, v, _gather(nxt[slot], off, periodic))
            _scatter(nxt[slot], off, periodic, v)
        field = nxt
    return field, post


def _cavity_types(size):
    types = torch.ones(tuple(n + 2 for n in size), dtype=torch.int32, device=DEVICE)
    types[1:-1, 1:-1, 1:-1] = 0
    types[1:-1, -1, 1:-1] = 2
    return types


def exact(case, seed):
    if case["kind"] == "train":
        feats, target, weight = (t.double() for t in _samples(case, seed))
        params = _network_params().double().to(DEVICE).requires_grad_(True)
        loss = (weight * (_network(params, feats) - target) ** 2).sum() / weight.sum()
        grad = torch.autograd.grad(loss, params)[0]
        grad[1441] = 0          # the output scale is not trained
        return {"loss": loss.detach().reshape(1), "grad": grad}
    if case["kind"] == "batch":
        sizes, rates = _cavity_sizes(case)
        out = []
        for k, (s, r) in enumerate(zip(sizes, rates)):
            u = _cavity_velocity(s, seed, k).double()
            field, _ = _simulate(
                19, "pull", (False,) * 3, _cavity_types(s), torch.ones(s, dtype=torch.float64, device=DEVICE),
                list(u.unbind(-1)), case["steps"],
                lambda f, r=r: _collide_populations(19, f, float(r[0]), float(r[1]), None, 0.0, False, "mrt"),
                False, 0.0, False)
            out.append(field.permute(1, 2, 3, 0))
        return out
    if case["kind"] == "sparse":
        flags = torch.from_numpy(_porous_flags(case)).to(DEVICE)
        inner = flags[1:-1, 1:-1, 1:-1] == 1
        cells = torch.nonzero(inner)
        vel = 1e-3 * (torch.rand(len(cells), 3, generator=_generator(seed), device=DEVICE) * 2 - 1).double()
        u = torch.zeros(tuple(inner.shape) + (3,), dtype=torch.float64, device=DEVICE)
        u[inner] = vel
        u[..., 0] += 0.5e-6     # the list's setter takes the velocity as it is, without the force shift
        types = (flags == 2).to(torch.int32)
        minus = 1 / (0.1875 / (1 / 1.8 - 0.5) + 0.5)
        _, post = _simulate(19, "pull", (True,) * 3, types, torch.ones(inner.shape, dtype=torch.float64, device=DEVICE),
                            list(u.unbind(-1)), case["steps"],
                            lambda f: _collide_populations(19, f, 1.8, None, minus, 1e-6, False, "trt"),
                            False, 1e-6, False)
        return post[:, inner].T
    n = (case["nx"], case["ny"], case["nz"])
    q = int(case["stencil"][3:])
    if n[0] * n[1] * n[2] * case["steps"] > (2e8 if q == 19 else 1e8):
        return None
    omega, bulk, minus, force, compressible, galilean = _physics(case)
    cumulant = case["method"] == "cumulant"
    if cumulant:
        sgs = None if case["sgs"] == "none" else case["sgs"]

        def collide(f):
            return _collide_cumulant(f, omega, bulk, force, galilean, sgs)
    else:
        def collide(f):
            return _collide_populations(q, f, omega, bulk, minus, force, compressible, case["method"])
    walled = _walled_axes(case)
    types = None
    if walled:
        types = _cavity_types(n) if case["walls"] == "cavity" else torch.zeros(
            tuple(v + 2 for v in n), dtype=torch.int32, device=DEVICE)
        if case["walls"] == "channel":
            types[:, 0], types[:, -1], types[:, :, 0], types[:, :, -1] = 1, 1, 1, 1
    u = _velocity(case, seed).double()
    field, post = _simulate(q, case["pattern"], [a not in walled for a in range(3)], types,
                            torch.ones(n, dtype=torch.float64, device=DEVICE), list(u.unbind(-1)), case["steps"],
                            collide, cumulant, force, compressible)
    if case["call"] == "sweeps" or case["call"] == "kernel":
        return field.permute(1, 2, 3, 0)
    rho, vel, rho_ref = _macro(q, post, force, compressible)
    if case["call"] == "monitor":
        kinetic = 0.5 * rho * (vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2)
        sums = torch.stack([rho.sum()] + [(rho_ref * v).sum() for v in vel] + [kinetic.sum()])
        return {"pdfs": field.permute(1, 2, 3, 0), "sums": sums}
    return {"density": rho, "velocity": torch.stack(vel, -1)}
