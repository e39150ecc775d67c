"""The performance cases of the hot path: what a user of the library has it do, through its public
entry points, from the smallest scenes to the largest.

Kinds of case
  step     el_step: one whole sub-step (extrapolation, both advections, gravity and masks, the
           ghost-fluid build, the pressure solve, the velocity update)
  batch    el_batch_step: independent scenes advanced by one graph launch
  solve    el_solve_pressure alone, on the caller's velocity
  advect   the stateless advection operators on the caller's device memory
  conv     one layer of the warm-start network: forward, backward data, backward weight

The caller of step, batch and solve hands its fields over on the device (el_field_device_ptr) before
each call, as a program does that reinitialises the level set or drives several solvers on one
state; so a pass starts from the same fields every time.
"""

import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    name = "eulerian_liquid_gb300"
    if name not in sys.modules:
        folder = os.path.join(ROOT, "eulerian-liquid_gb300")
        spec = importlib.util.spec_from_file_location(name, os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


# ---- the cases ----------------------------------------------------------------------------------

def _step(name, ni, nj, nk, dtype, scene, weno, rk3, solver):
    return {"name": name, "kind": "step", "ni": ni, "nj": nj, "nk": nk, "dtype": dtype, "scene": scene,
            "weno": weno, "rk3": rk3, "solver": solver}


def listed():
    return [
        # the headline configuration: spheres over a pool with a solid box, WENO6 level set, RK3
        # velocity, FP32 fields, mixed-precision solve to 1e-6
        _step("step_pool_256", 256, 256, 256, "f32", "pool", True, True, "mixed"),
        # a stand-alone scene of uneven odd sizes, as in the batched configuration's {48..160} range
        _step("step_ragged_151", 151, 97, 133, "f32", "drop", True, True, "mixed"),
        # the reference application's own schemes (trilinear, RK2) on a small scene: latency
        _step("step_drop_48", 48, 48, 48, "f32", "drop", False, False, "mixed"),
        # the plain FP64 configurations: 64^3 trilinear, and 128^3 with WENO6 and RK3
        _step("step_dam_64_f64", 64, 64, 64, "f64", "dam", False, False, "jacobi"),
        _step("step_dam_128_f64", 128, 128, 128, "f64", "dam", True, True, "jacobi"),
        # batched scenes of seeded uneven sizes
        {"name": "batch_12", "kind": "batch", "scenes": 12, "lo": 48, "hi": 160, "sizes": 7},
        # the FP64 multigrid solve on its own (FP64 users; the tight reference solve of the
        # benchmark), and the mixed solve on a small uneven grid
        {"name": "solve_mg_f64", "kind": "solve", "ni": 112, "nj": 128, "nk": 96, "dtype": "f64", "scene": "pool",
         "solver": "mg"},
        {"name": "solve_mixed_75", "kind": "solve", "ni": 75, "nj": 62, "nk": 53, "dtype": "f32", "scene": "pool",
         "solver": "mixed"},
        # the reference's free functions: advect_collocated_grid (WENO6) and advect_staggered_grid
        {"name": "advect_phi_weno", "kind": "advect", "what": "phi", "ni": 203, "nj": 149, "nk": 181, "dtype": "f32",
         "weno": True, "rk3": False},
        {"name": "advect_vel_tri", "kind": "advect", "what": "vel", "ni": 256, "nj": 128, "nk": 192, "dtype": "f32",
         "weno": False, "rk3": True},
        # the warm-start network's layers at the 128^3 training size: the finest level's 16 -> 16
        # layer, and the decoder's 96 -> 32 layer at level 1 (upsampled input and skip)
        {"name": "conv_e0_128", "kind": "conv", "n0": 128, "n1": 128, "n2": 128, "ca": 16, "up": False, "cb": 0,
         "cout": 16},
        {"name": "conv_d1a_64", "kind": "conv", "n0": 64, "n1": 64, "n2": 64, "ca": 64, "up": True, "cb": 32,
         "cout": 32},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["step32", "step32", "step64", "batch", "solve", "solve", "advect", "advect", "conv", "conv"])
    if kind == "step32":
        ni, nj, nk = (_log_int(rng, 40, 240) for _ in range(3))
        if rng.random() < 0.5:
            ni -= ni % 8
        return {"kind": "step", "ni": ni, "nj": nj, "nk": nk, "dtype": "f32",
                "scene": rng.choice(["pool", "drop", "dam"]), "weno": rng.random() < 0.6, "rk3": rng.random() < 0.5,
                "solver": "mixed"}
    if kind == "step64":
        ni, nj, nk = (_log_int(rng, 32, 120) for _ in range(3))
        return {"kind": "step", "ni": ni, "nj": nj, "nk": nk, "dtype": "f64",
                "scene": rng.choice(["pool", "drop", "dam"]), "weno": rng.random() < 0.5, "rk3": rng.random() < 0.5,
                "solver": rng.choice(["jacobi", "mixed"])}
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.randint(3, 12), "lo": 48, "hi": rng.randint(96, 160),
                "sizes": rng.randint(0, 1 << 20)}
    if kind == "solve":
        ni, nj, nk = (_log_int(rng, 40, 160) for _ in range(3))
        dtype = rng.choice(["f32", "f64"])
        return {"kind": "solve", "ni": ni, "nj": nj, "nk": nk, "dtype": dtype, "scene": rng.choice(["pool", "drop"]),
                "solver": "mixed" if dtype == "f32" else rng.choice(["mg", "jacobi"])}
    if kind == "advect":
        ni, nj, nk = (_log_int(rng, 48, 240) for _ in range(3))
        what = rng.choice(["phi", "vel"])
        dtype = rng.choice(["f32", "f32", "f64"])
        if dtype == "f64":
            ni, nj, nk = min(ni, 112), min(nj, 112), min(nk, 112)
        return {"kind": "advect", "what": what, "ni": ni, "nj": nj, "nk": nk, "dtype": dtype,
                "weno": what == "phi" and rng.random() < 0.6, "rk3": rng.random() < 0.5}
    ca, up, cb, cout, level = rng.choice([(16, False, 0, 16, 0), (16, False, 0, 32, 1), (32, False, 0, 32, 1),
                                          (32, False, 0, 64, 2), (64, False, 0, 64, 2), (64, True, 64, 64, 2),
                                          (64, True, 32, 32, 1), (32, True, 16, 16, 0)])
    n0, n1, n2 = (max(1, _log_int(rng, 4, 16)) * 8 >> level for _ in range(3))
    return {"kind": "conv", "n0": n0, "n1": n1, "n2": n2, "ca": ca, "up": up, "cb": cb, "cout": cout}


# ---- inputs -------------------------------------------------------------------------------------

FACES = ("u", "v", "w")


def _dtype(case):
    return torch.float64 if case.get("dtype") == "f64" else torch.float32


def _dx(case):
    ni = case["ni"]
    return 1.0 / ni if case["dtype"] == "f64" else float(np.float32(1.0) / np.float32(ni))


def _dt(case):
    """CFL 1 for the inputs' velocity (at most 1 on each axis), in the field type."""
    dx = _dx(case)
    return dx if case["dtype"] == "f64" else float(np.float32(dx))


def _coords(ni, nj, nk, dx, shift):
    """x, y, z of the samples of a grid whose first sample lies at (0.5 - shift) dx on each axis."""
    dims = (ni, nj, nk)
    return [((torch.arange(n, device="cuda", dtype=torch.float64) + 0.5 - s) * dx).view(
        *[(-1 if a == 2 - q else 1) for a in range(3)]) for q, (n, s) in enumerate(zip(dims, shift))]


def _grids(case):
    ni, nj, nk = case["ni"], case["nj"], case["nk"]
    return [((ni + 1, nj, nk), (0.5, 0, 0)), ((ni, nj + 1, nk), (0, 0.5, 0)), ((ni, nj, nk + 1), (0, 0, 0.5))]


def _sphere(x, y, z, c, r):
    return torch.sqrt((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) - r


def _box(x, y, z, lo, hi):
    q = [torch.maximum(a - v, v - b) for v, a, b in zip((x, y, z), lo, hi)]
    outside = torch.sqrt(sum(t.clamp(min=0) ** 2 for t in q))
    return outside + torch.maximum(torch.maximum(q[0], q[1]), q[2]).clamp(max=0)


def _scene(case, seed):
    """Level set, velocity, face weights and valid masks of a seeded scene, in the field type: the
    emitters of the package's scenes, walls one cell thick and (pool) a solid box, a smooth
    velocity of at most 1 on each axis, zero off the faces a step leaves valid."""
    rng = np.random.default_rng([seed, case["ni"], case["nj"], case["nk"]])
    ni, nj, nk = case["ni"], case["nj"], case["nk"]
    dx, dt = _dx(case), _dtype(case)
    ext = np.array([ni, nj, nk]) * dx  # the domain, 1 wide
    x, y, z = _coords(ni, nj, nk, dx, (0, 0, 0))
    if case["scene"] == "dam":
        lim = (0.4 + 0.05 * rng.uniform(-1, 1)) * ext[0], (0.5 + 0.05 * rng.uniform(-1, 1)) * ext[1]
        phi = torch.maximum(x - lim[0], y - lim[1]) + 0 * z
        phi = torch.minimum(phi, _sphere(x, y, z, (0.7 * ext[0], 0.75 * ext[1], 0.5 * ext[2]), 0.12 * ext.min()))
    else:
        phi = y - rng.uniform(0.25, 0.35) * ext[1] + 0 * x + 0 * z
        for _ in range(3 if case["scene"] == "pool" else 1):
            r = rng.uniform(0.08, 0.2) * ext.min()
            c = [rng.uniform(0.1 * e + r, 0.9 * e - r) for e in ext]
            c[1] = rng.uniform(min(0.4 * ext[1] + r, 0.85 * ext[1] - r), 0.9 * ext[1] - r)
            phi = torch.minimum(phi, _sphere(x, y, z, c, r))
    out = {"phi": phi.to(dt).contiguous()}
    box = None
    if case["scene"] == "pool":
        size = rng.uniform(0.25, 0.45, 3) * ext
        lo = [rng.uniform(0.08 * e, 0.92 * e - s) for e, s in zip(ext, size)]
        box = (lo, [a + s for a, s in zip(lo, size)])

    def solid(px, py, pz):  # signed distance to the solid, positive in the open
        s = None
        for q, e in zip((px, py, pz), ext):
            t = torch.minimum(q, e - q) - dx
            s = t if s is None else torch.minimum(s, t)
        return torch.minimum(s, _box(px, py, pz, *box)) if box else s

    out["valid_phi"] = (solid(x, y, z) >= 0).to(torch.uint8)
    wet = out["phi"] < 0
    for axis, ((dims, shift), f) in enumerate(zip(_grids(case), FACES)):
        fx, fy, fz = _coords(*dims, dx, shift)
        wt = (0.5 + solid(fx, fy, fz) / dx).clamp(0, 1)
        modes = rng.integers(1, 4, (3, 3)), rng.uniform(0, 2 * math.pi, (3, 3)), np.array([0.5, 0.3, 0.2])
        vel = torch.zeros((), device="cuda", dtype=torch.float64)
        for m, ph, a in zip(*modes):
            vel = vel + a * torch.sin(2 * math.pi * m[0] * fx / ext[0] + ph[0]) * torch.cos(
                2 * math.pi * m[1] * fy / ext[1] + ph[1]) * torch.cos(2 * math.pi * m[2] * fz / ext[2] + ph[2])
        d = 2 - axis  # the face's normal axis in (k, j, i) order
        pad = torch.zeros_like(wet.narrow(d, 0, 1))
        near = torch.cat([pad, wet], d) | torch.cat([wet, pad], d)
        valid = (near & (wt > 0)).contiguous()
        out["weight_" + f] = wt.to(dt).contiguous()
        out[f] = torch.where(valid, vel, torch.zeros((), device="cuda", dtype=torch.float64)).to(dt).contiguous()
        out["valid_" + f] = valid.to(torch.uint8)
    return out


class _DevicePtr:
    def __init__(self, owner, ptr, shape, dtype):
        self.owner = owner  # the scene's memory lives as long as any tensor on it
        self.__cuda_array_interface__ = {"shape": tuple(int(s) for s in shape), "typestr": np.dtype(dtype).str,
                                         "data": (int(ptr), False), "version": 3}


class _Views:
    """Torch views of a Simulator's fields (advection moves a field between two buffers).  A view
    keeps `owner`, which frees the fields, alive; `owner` must not hold the views."""

    def __init__(self, sim, owner):
        self.sim = sim
        self.owner = owner
        self.seen = {}

    def __call__(self, field):
        ptr, _ = self.sim.device_ptr(field)
        v = self.seen.get((field, ptr))
        if v is None:
            v = torch.as_tensor(_DevicePtr(self.owner, ptr, self.sim.shape(field), self.sim.field_dtype(field)),
                                device="cuda")
            self.seen[field, ptr] = v
        return v


_stream = None


def _work_stream():
    """The one stream the program enqueues its scenes' work on."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _sim(case, fields, stream=None, owner=None):
    el = _package()
    sim = el.Simulator(case["ni"], case["nj"], case["nk"], dx=_dx(case),
                       dtype=el.EL_F64 if case["dtype"] == "f64" else el.EL_F32)
    if stream is not None:
        sim.set_stream(stream.cuda_stream)
    torch.cuda.synchronize()
    views = _Views(sim, owner or sim)
    for f, a in fields.items():
        views(f).copy_(a)
    return sim, views


def _params(case):
    el = _package()
    solver = {"jacobi": el.SOLVER_JACOBI_FP64, "mg": el.SOLVER_MG_FP64, "mixed": el.SOLVER_MIXED}[case["solver"]]
    return dict(solver=solver, tol=1e-6, max_iter=20000, check_every=16 if case["solver"] == "jacobi" else 4)


def _step_params(case):
    el = _package()
    return el.step_params(trace_phi=el.TRACE_RK2, sample_phi=el.SAMPLE_WENO6 if case["weno"] else el.SAMPLE_TRILINEAR,
                          trace_vel=el.TRACE_RK3 if case["rk3"] else el.TRACE_RK2, sample_vel=el.SAMPLE_TRILINEAR,
                          gravity=9.8, extrapolation_layers=10, **_params(case))


class _Scenes:
    """The scenes of a batch and the batch, which goes before them."""

    def __init__(self):
        self.sims, self.batch = [], None

    def __del__(self):
        if self.batch is not None:
            self.batch.close()
        for s in self.sims:
            s.close()


def _prepare_batch(case, seed):
    el = _package()
    own, views, fields = _Scenes(), [], []
    for q, spec in enumerate(el.scenes.batch_scenes(case["scenes"], case["sizes"], case["lo"], case["hi"])):
        ni, nj, nk = spec["shape"]
        c = {"ni": ni, "nj": nj, "nk": nk, "dtype": "f32", "scene": "drop" if q % 2 else "dam"}
        f = _scene(c, seed + 1000 * q)
        sim, v = _sim(c, f, owner=own)
        own.sims.append(sim)
        views.append(v)
        fields.append({name: f[name] for name in CARRIED})
    torch.cuda.synchronize()
    # a long frame: every sub-step has its scene's own CFL time step
    own.batch = el.Batch(own.sims, trace_phi=el.TRACE_RK2, sample_phi=el.SAMPLE_WENO6, trace_vel=el.TRACE_RK3,
                         sample_vel=el.SAMPLE_TRILINEAR, gravity=9.8, cfl=1.0, dt_frame=1000.0,
                         solver=el.SOLVER_MIXED, tol=1e-6, max_iter=2000)
    return {"case": case, "own": own, "views": views, "fields": fields,
            "stream": torch.cuda.ExternalStream(own.batch.stream)}


CARRIED = ("phi", "u", "v", "w", "valid_u", "valid_v", "valid_w")  # what a step changes of its inputs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    if kind in ("step", "solve"):
        stream = _work_stream()
        fields = _scene(case, seed)
        with torch.cuda.stream(stream):
            sim, views = _sim(case, fields, stream)
        carried = CARRIED if kind == "step" else FACES
        params = _step_params(case) if kind == "step" else _params(case)
        return {"case": case, "sim": sim, "views": views, "fields": {f: fields[f] for f in carried}, "stream": stream,
                "params": params, "dt": _dt(case)}
    if kind == "advect":
        f = _scene(dict(case, scene="pool"), seed)
        vel = [_smooth_velocity(case, seed, c) for c in range(3)]
        src = [f["phi"]] if case["what"] == "phi" else vel
        return {"case": case, "src": src, "vel": vel, "out": [torch.empty_like(a) for a in src], "dt": _dt(case)}
    return _prepare_conv(case, seed)


def _smooth_velocity(case, seed, comp):
    """A velocity component over the whole domain (as the extrapolation leaves it), at most 1."""
    rng = np.random.default_rng([seed, 77, comp])
    dims, shift = _grids(case)[comp]
    dx = _dx(case)
    ext = np.array([case["ni"], case["nj"], case["nk"]]) * dx
    x, y, z = _coords(*dims, dx, shift)
    vel = torch.zeros((), device="cuda", dtype=torch.float64)
    for a in (0.5, 0.3, 0.2):
        m, ph = rng.integers(1, 5, 3), rng.uniform(0, 2 * math.pi, 3)
        vel = vel + a * torch.sin(2 * math.pi * m[0] * x / ext[0] + ph[0]) * torch.cos(
            2 * math.pi * m[1] * y / ext[1] + ph[1]) * torch.cos(2 * math.pi * m[2] * z / ext[2] + ph[2])
    return vel.to(_dtype(case)).contiguous()


def _conv_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n0, n1, n2, ca, cb, cout = (case[k] for k in ("n0", "n1", "n2", "ca", "cb", "cout"))
    cin = ca + cb

    def act(*shape):  # what a ReLU layer hands on: half of it zero
        return torch.randn(*shape, generator=g, device="cuda").relu().to(torch.bfloat16)

    s = 2 if case["up"] else 1
    a = act(n2 // s, n1 // s, n0 // s, ca)
    b = act(n2, n1, n0, cb) if cb else None
    w = torch.randn(cout, 27, cin, generator=g, device="cuda") * math.sqrt(2.0 / (27 * cin))
    bias = 0.1 * torch.randn(cout, generator=g, device="cuda")
    grad = (1e-2 * torch.randn(n2, n1, n0, cout, generator=g, device="cuda")).to(torch.bfloat16)
    saved = act(n2, n1, n0, cout)  # the output that the training step saved for the backward passes
    return a, b, w, bias, grad, saved


def _prepare_conv(case, seed):
    W = _package().warmstart
    L = W.lib()
    a, b, w, bias, grad, saved = _conv_inputs(case, seed)
    n0, n1, n2, ca, cb, cout = (case[k] for k in ("n0", "n1", "n2", "ca", "cb", "cout"))
    cin = ca + cb

    def buf(*shape, dtype=torch.bfloat16):
        return torch.empty(shape, dtype=dtype, device="cuda")

    size = L.el_nn_packed_weight_bytes(cin, cout) // 2
    packed, packed_tc = [buf(size), buf(size)], [None, None]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert L.el_nn_pack_weights(cin, cout, w.data_ptr(), packed[0].data_ptr(), packed[1].data_ptr(), stream) == 0
    prefers = L.el_nn_tc_preferred(cin, cout), L.el_nn_tc_preferred(cout, cin)
    if any(prefers):  # the network's own choice of kernel, layer by layer
        tc = [buf(size), buf(size)]
        assert L.el_nn_pack_weights_tc(cin, cout, w.data_ptr(), tc[0].data_ptr(), tc[1].data_ptr(), stream) == 0
        packed_tc = [t if p else None for t, p in zip(tc, prefers)]
    st = {"case": case, "a": a, "b": b, "w": w, "bias": bias, "grad": grad, "saved": saved, "packed": packed,
          "packed_tc": packed_tc, "y": buf(n2, n1, n0, cout), "ga": buf(*a.shape), "gb": buf(*b.shape) if cb else None,
          "gup": buf(n2, n1, n0, ca) if case["up"] else None, "dw": buf(cout, 27, cin, dtype=torch.float32),
          "db": buf(cout, dtype=torch.float32)}
    need = L.el_nn_conv3_backward_weight_workspace(n0, n1, n2, cin, cout)
    st["ws"] = buf(need // 4 + 1, dtype=torch.float32)
    f = W.ConvArgs()
    f.nx, f.ny, f.nz, f.cin, f.cout = n0, n1, n2, cin, cout
    f.in_a, f.ca, f.upsample_a = a.data_ptr(), ca, int(case["up"])
    f.in_b, f.cb = (b.data_ptr(), cb) if cb else (None, 0)
    f.weights, f.bias, f.relu = packed[0].data_ptr(), bias.data_ptr(), 1
    f.weights_tc = packed_tc[0].data_ptr() if packed_tc[0] is not None else None
    f.out_a, f.out_a_channels, f.out_b = st["y"].data_ptr(), cout, None
    d = W.ConvArgs()
    d.nx, d.ny, d.nz, d.cin, d.cout = n0, n1, n2, cout, cin
    d.in_a, d.ca, d.upsample_a, d.in_b, d.cb = grad.data_ptr(), cout, 0, None, 0
    d.mask, d.weights, d.bias, d.relu = saved.data_ptr(), packed[1].data_ptr(), None, 0
    d.weights_tc = packed_tc[1].data_ptr() if packed_tc[1] is not None else None
    d.out_a = (st["gup"] if case["up"] else st["ga"]).data_ptr()
    d.out_a_channels, d.out_b = ca, (st["gb"].data_ptr() if cb else None)
    wg = W.ConvArgs.from_buffer_copy(f)
    wg.out_a = saved.data_ptr()
    st["fwd"], st["bwd"], st["wgrad"] = f, d, wg
    return st


# ---- one pass -----------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        sim, views = state["sim"], state["views"]
        with torch.cuda.stream(state["stream"]):
            for f, a in state["fields"].items():
                views(f).copy_(a)
            sim.step(state["dt"], state["params"])
        return {f: views(f) for f in ("phi", "u", "v", "w", "pressure")}
    if kind == "solve":
        sim, views = state["sim"], state["views"]
        with torch.cuda.stream(state["stream"]):
            for f, a in state["fields"].items():
                views(f).copy_(a)
            sim.solve_pressure(state["dt"], **state["params"])
        return {f: views(f) for f in ("pressure", "u", "v", "w")}
    if kind == "batch":
        with torch.cuda.stream(state["stream"]):
            for fields, views in zip(state["fields"], state["views"]):
                for f, a in fields.items():
                    views(f).copy_(a)
        state["own"].batch.step(1)
        return [{f: views(f) for f in ("phi", "u", "v", "w", "pressure")} for views in state["views"]]
    if kind == "advect":
        return _run_advect(state)
    return _run_conv(state)


def _run_advect(state):
    el = _package()
    case = state["case"]
    dt = el.EL_F64 if case["dtype"] == "f64" else el.EL_F32
    trace = el.TRACE_RK3 if case["rk3"] else el.TRACE_RK2
    sample = el.SAMPLE_WENO6 if case["weno"] else el.SAMPLE_TRILINEAR
    vel = [a.data_ptr() for a in state["vel"]]
    dims = case["ni"], case["nj"], case["nk"], _dx(case), dt
    stream = torch.cuda.current_stream().cuda_stream
    if case["what"] == "phi":
        el.advect_collocated_grid(*dims, state["out"][0].data_ptr(), state["src"][0].data_ptr(), *vel, state["dt"],
                                  trace, sample, stream)
    else:
        el.advect_staggered_grid(*dims, [a.data_ptr() for a in state["out"]], [a.data_ptr() for a in state["src"]],
                                 vel, state["dt"], trace, sample, stream)
    return list(state["out"])


def _run_conv(st):
    L = _package().warmstart.lib()
    case = st["case"]
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    status = L.el_nn_conv3_forward(ctypes.byref(st["fwd"]), s)
    status |= L.el_nn_conv3_forward(ctypes.byref(st["bwd"]), s)
    if case["up"]:
        status |= L.el_nn_gather8(case["n0"], case["n1"], case["n2"], case["ca"], st["gup"].data_ptr(),
                                  st["ga"].data_ptr(), s)
    st["dw"].zero_()
    st["db"].zero_()
    status |= L.el_nn_conv3_backward_weight(ctypes.byref(st["wgrad"]), st["grad"].data_ptr(), st["dw"].data_ptr(),
                                            st["db"].data_ptr(), st["ws"].data_ptr(), st["ws"].numel() * 4, s)
    if status:
        raise RuntimeError("convolution")
    out = {"y": st["y"], "ga": st["ga"], "dw": st["dw"], "db": st["db"]}
    if st["gb"] is not None:
        out["gb"] = st["gb"]
    return out


# ---- what a pass cannot do without --------------------------------------------------------------

def _step_work(ni, nj, nk, e, weno, rk3):
    n = ni * nj * nk
    faces = (ni + 1) * nj * nk + ni * (nj + 1) * nk + ni * nj * (nk + 1)
    # phi, u, v, w, the weights and masks in; phi, u, v, w, the pressure and the masks out
    moved = e * (3 * n + 3 * faces) + 2 * faces + n
    # a trilinear read is 21 operations, a WENO6 read 43 six-point passes of about 70; one
    # application of the operator and the ghost-fluid row
    flops = n * (2 * 63 + (43 * 70 if weno else 21)) + faces * ((3 if rk3 else 2) * 63 + 21) + 40 * n
    return moved, flops


def work(case):
    kind = case["kind"]
    if kind == "batch":
        el = _package()
        moved = flops = 0
        for spec in el.scenes.batch_scenes(case["scenes"], case["sizes"], case["lo"], case["hi"]):
            b, f = _step_work(*spec["shape"], 4, True, True)
            moved, flops = moved + b, flops + f
        return {"bytes": moved, "flops": flops}
    if kind == "conv":
        vox = case["n0"] * case["n1"] * case["n2"]
        cin = case["ca"] + case["cb"]
        a = vox * case["ca"] // (8 if case["up"] else 1)
        b = vox * case["cb"]
        # the inputs, their gradients, the output and its gradient
        return {"bytes": 2 * (2 * (a + b) + 2 * vox * case["cout"]) + 8 * 27 * cin * case["cout"],
                "flops": 3 * 2 * 27 * cin * case["cout"] * vox}
    ni, nj, nk = case["ni"], case["nj"], case["nk"]
    e = 8 if case["dtype"] == "f64" else 4
    n = ni * nj * nk
    faces = (ni + 1) * nj * nk + ni * (nj + 1) * nk + ni * nj * (nk + 1)
    if kind == "step":
        moved, flops = _step_work(ni, nj, nk, e, case["weno"], case["rk3"])
    elif kind == "solve":  # phi, weights and velocity in; pressure and velocity out
        moved, flops = e * (2 * n + 3 * faces), 40 * n
    else:
        src = n if case["what"] == "phi" else faces
        moved = e * (faces + n * 2 if case["what"] == "phi" else 2 * faces)
        flops = src * ((3 if case["rk3"] else 2) * 63 + (43 * 70 if case["weno"] else 21))
    return {"bytes": moved, "flops": flops}


# ---- the same in 64 bits ------------------------------------------------------------------------

def _gather(g, i, j, k):
    n2, n1, n0 = g.shape
    return g.reshape(-1)[i.clamp(0, n0 - 1) + n0 * (j.clamp(0, n1 - 1) + n1 * k.clamp(0, n2 - 1))]


def _locate(p, shift, dx):
    """Cell indices and fractions of positions on a grid."""
    idx, frac = [], []
    for q, s in zip(p, shift):
        t = q / dx - 0.5 + s
        fl = torch.floor(t)
        idx.append(fl.long())
        frac.append(t - fl)
    return idx, frac


def _trilinear(g, shift, p, dx):
    (i, j, k), (fx, fy, fz) = _locate(p, shift, dx)
    planes = []
    for c in (0, 1):
        rows = [_gather(g, i, j + b, k + c) * (1 - fx) + _gather(g, i + 1, j + b, k + c) * fx for b in (0, 1)]
        planes.append(rows[0] * (1 - fy) + rows[1] * fy)
    return planes[0] * (1 - fz) + planes[1] * fz


def _weno_line(v, f):
    """Six-point WENO interpolation at f in [0, 1) on nodes -2..3 (the published indicators)."""
    x = f
    cand, weight = [], []
    gam = ((2 - x) * (3 - x) / 20, (3 - x) * (x + 2) / 10, (x + 2) * (x + 1) / 20)
    for s in range(3):
        a, b, c, d = v[s:s + 4]
        e0, e1, e2 = x + 2 - s, x + 1 - s, x - s
        cand.append(a + (b - a) * e0 + (c - 2 * b + a) * e0 * e1 / 2 + (d - 3 * c + 3 * b - a) * e0 * e1 * e2 / 6)
    d1, d2, d3, d4, d5 = (v[m + 1] - v[m] for m in range(5))
    ind = ((244 * d1 * d1 - 1171 * d1 * d2 + 683 * d1 * d3 + 1561 * d2 * d2 - 1951 * d2 * d3 + 814 * d3 * d3) / 180,
           (244 * d2 * d2 - 781 * d2 * d3 + 293 * d2 * d4 + 961 * d3 * d3 - 781 * d3 * d4 + 244 * d4 * d4) / 180,
           (814 * d3 * d3 - 1951 * d3 * d4 + 683 * d3 * d5 + 1561 * d4 * d4 - 1171 * d4 * d5 + 244 * d5 * d5) / 180)
    weight = [g / (1e-6 + b) ** 2 for g, b in zip(gam, ind)]
    return sum(w * c for w, c in zip(weight, cand)) / (weight[0] + weight[1] + weight[2])


def _weno6(g, shift, p, dx):
    (i, j, k), (fx, fy, fz) = _locate(p, shift, dx)
    zl = []
    for c in range(-2, 4):
        yl = [_weno_line([_gather(g, i + a, j + b, k + c) for a in range(-2, 4)], fx) for b in range(-2, 4)]
        zl.append(_weno_line(yl, fy))
    return _weno_line(zl, fz)


def _advected(src, src_shift, dims, vel, shifts, dx, dt, rk3, weno):
    """src at the backtraced positions of its own samples, in 64 bits, a few planes at a time."""
    n0, n1, n2 = dims
    out = torch.empty((n2, n1, n0), device="cuda", dtype=torch.float64)

    def field(p):
        return [_trilinear(g, s, p, dx) for g, s in zip(vel, shifts)]

    def moved(p, *terms):
        return [q + sum(h * k[a] for h, k in terms) for a, q in enumerate(p)]

    planes = max(1, (1 << 20) // (n0 * n1))
    x, y, z = _coords(n0, n1, n2, dx, src_shift)
    for k0 in range(0, n2, planes):
        zz = z[k0:k0 + planes]
        p = [q.expand(zz.shape[0], n1, n0).reshape(-1) for q in (x, y, zz)]
        k1 = field(p)
        k2 = field(moved(p, (-0.5 * dt, k1)))
        if rk3:
            k3 = field(moved(p, (-0.75 * dt, k2)))
            foot = moved(p, (-dt * 2 / 9, k1), (-dt / 3, k2), (-dt * 4 / 9, k3))
        else:
            foot = moved(p, (-dt, k2))
        out[k0:k0 + planes] = (_weno6 if weno else _trilinear)(src, src_shift, foot, dx).reshape(-1, n1, n0)
    return out


def _box_sum(a):
    a = torch.nn.functional.pad(a, (1, 1, 1, 1, 1, 1))
    a = a[:, :, :-2] + a[:, :, 1:-1] + a[:, :, 2:]
    a = a[:, :-2] + a[:, 1:-1] + a[:, 2:]
    return a[:-2] + a[1:-1] + a[2:]


def _extrapolated(g, valid, layers=10):
    """Layers of invalid cells take the mean of their valid 26-neighbours."""
    valid = valid.bool()
    for _ in range(layers):
        count = _box_sum(valid.double())
        total = _box_sum(torch.where(valid, g, torch.zeros_like(g)))
        new = ~valid & (count > 0.5)
        g = torch.where(new, total / count.clamp(min=1), g)
        valid = valid | new
    return g


def _inside(a, b):
    """Fraction of the segment between two level-set values that is inside."""
    one = torch.where(a < 0, a / (a - b), b / (b - a))
    return torch.where((a < 0) & (b < 0), torch.ones_like(a), torch.where((a < 0) | (b < 0), one,
                                                                          torch.zeros_like(a)))


def _projected(case, f, dt):
    """Pressure and velocity of the ghost-fluid projection of fields f, solved to 1e-13."""
    dx = _dx(case)
    phi = f["phi"].double()
    vel = [f[c].double() for c in FACES]
    wts = [f["weight_" + c].double() for c in FACES]
    low = [w.narrow(2 - a, 0, phi.shape[2 - a]) for a, w in enumerate(wts)]
    high = [w.narrow(2 - a, 1, phi.shape[2 - a]) for a, w in enumerate(wts)]
    open_ = sum(((lo > 0) | (hi > 0)).int() for lo, hi in zip(low, high)) > 0
    fluid = open_ & (phi < 0)
    zero = torch.zeros_like(phi)
    diag, rhs, couple = zero.clone(), zero.clone(), []
    for a in range(3):
        d = 2 - a
        n = phi.shape[d]
        rhs += low[a] * vel[a].narrow(d, 0, n) - high[a] * vel[a].narrow(d, 1, n)
        up = lambda t: torch.cat([t.narrow(d, 1, n - 1), torch.zeros_like(t.narrow(d, 0, 1))], d)  # noqa: E731
        dn = lambda t: torch.cat([torch.zeros_like(t.narrow(d, 0, 1)), t.narrow(d, 0, n - 1)], d)  # noqa: E731
        for shift, w in ((dn, low[a]), (up, high[a])):
            nb_open, nb_phi = shift(open_.double()) > 0.5, shift(phi)
            theta = _inside(phi, nb_phi).clamp(min=0.01)
            diag += torch.where(nb_open, torch.where(nb_phi < 0, w, w / theta), zero)
        couple.append(torch.where(fluid & (up(fluid.double()) > 0.5), high[a], zero))
    rhs = torch.where(fluid, rhs * (dx / dt), zero)
    diag = torch.where(fluid, diag, torch.ones_like(diag))
    live = fluid & (diag > 0)

    def apply(p):
        q = diag * p
        for a, c in enumerate(couple):
            d = 2 - a
            n = p.shape[d]
            lo, hi = p.narrow(d, 0, n - 1), p.narrow(d, 1, n - 1)
            cc = c.narrow(d, 0, n - 1)
            q.narrow(d, 0, n - 1).sub_(cc * hi)
            q.narrow(d, 1, n - 1).sub_(cc * lo)
        return q

    inv = torch.where(live, 1.0 / diag, zero)
    p, r = zero.clone(), torch.where(live, rhs, zero)
    s = inv * r
    rho, stop = (r * s).sum(), 1e-26 * (r * r).sum()
    for it in range(6000):
        q = apply(s)
        alpha = rho / (s * q).sum()
        p += alpha * s
        r -= alpha * q
        if it % 16 == 15 and bool((r * r).sum() < stop):
            break
        t = inv * r
        new = (r * t).sum()
        s = t + (new / rho) * s
        rho = new
    out = {"pressure": p}
    n2, n1, n0 = phi.shape
    for a, c in enumerate(FACES):
        d = 2 - a
        n = phi.shape[d]
        pa, pb = phi.narrow(d, 0, n - 1), phi.narrow(d, 1, n - 1)
        theta = torch.where((pa < 0) & (pb < 0), torch.ones_like(pa), _inside(pa, pb)).clamp(min=0.01)
        grad = torch.where((pa < 0) | (pb < 0), dt * (p.narrow(d, 1, n - 1) - p.narrow(d, 0, n - 1)) / (dx * theta),
                           torch.zeros_like(pa))
        for t in range(3):  # interior on the tangential axes
            if t != d:
                edge = torch.zeros(phi.shape[t], device="cuda", dtype=torch.float64)
                edge[1:-1] = 1
                grad = grad * edge.view(*[(-1 if q == t else 1) for q in range(3)])
        v = vel[a].clone()
        v.narrow(d, 1, n - 1).sub_(grad)
        out[c] = v
    return out


def _conv_exact(case, seed):
    a, b, w, bias, grad, saved = _conv_inputs(case, seed)
    n = a.shape[:3]
    x = a.double()
    if case["up"]:
        for q in range(3):
            x = x.repeat_interleave(2, q)
    if b is not None:
        x = torch.cat([x, b.double()], 3)
    cout, _, cin = w.shape
    # the layer's own weights are their bf16 roundings
    wt = w.to(torch.bfloat16).double().reshape(cout, 3, 3, 3, cin)
    shape = x.shape[:3]
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    y = bias.double().expand(*shape, cout).clone()
    taps = [(c, d, e) for c in range(3) for d in range(3) for e in range(3)]

    def window(t, c, d, e):
        return t[c:c + shape[0], d:d + shape[1], e:e + shape[2]].reshape(-1, t.shape[3])

    for c, d, e in taps:
        y += (window(xp, c, d, e) @ wt[:, c, d, e].t()).reshape(y.shape)
    y = y.relu()
    gm = grad.double() * (saved > 0)
    flat = gm.reshape(-1, cout)
    dw = torch.stack([flat.t() @ window(xp, c, d, e) for c, d, e in taps], 1)
    gp = torch.nn.functional.pad(gm, (0, 0, 1, 1, 1, 1, 1, 1))
    gx = torch.zeros_like(x)
    for c, d, e in taps:
        gx += (window(gp, 2 - c, 2 - d, 2 - e) @ wt[:, c, d, e]).reshape(x.shape)
    ca = case["ca"]
    ga = gx[..., :ca]
    if case["up"]:
        ga = ga.reshape(n[0], 2, n[1], 2, n[2], 2, ca).sum(dim=(1, 3, 5))
    out = {"y": y, "ga": ga.contiguous(), "dw": dw, "db": flat.sum(0)}
    if b is not None:
        out["gb"] = gx[..., ca:].contiguous()
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "conv":
        return _conv_exact(case, seed)
    if kind == "advect":
        f = _scene(dict(case, scene="pool"), seed)
        vel = [_smooth_velocity(case, seed, c).double() for c in range(3)]
        grids = _grids(case)
        shifts = [s for _, s in grids]
        dx, dt = _dx(case), _dt(case)
        if case["what"] == "phi":
            todo = [(f["phi"].double(), (0, 0, 0), (case["ni"], case["nj"], case["nk"]))]
        else:
            todo = [(v, s, d) for v, (d, s) in zip(vel, grids)]
        return [_advected(g, s, d, vel, shifts, dx, dt, case["rk3"], case["weno"]) for g, s, d in todo]
    if kind == "solve":
        return _projected(case, _scene(case, seed), _dt(case))
    if kind == "step":
        # the level set; what follows it hangs on its sign, cell by cell
        f = _scene(case, seed)
        vel = [_extrapolated(f[c].double(), f["valid_" + c]) for c in FACES]
        phi = _extrapolated(f["phi"].double(), f["valid_phi"])
        new = _advected(phi, (0, 0, 0), (case["ni"], case["nj"], case["nk"]), vel, [s for _, s in _grids(case)],
                        _dx(case), _dt(case), False, case["weno"])
        return {"phi": new, "u": None, "v": None, "w": None, "pressure": None}
    return None
