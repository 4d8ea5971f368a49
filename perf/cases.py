"""The work that a user of svirl_gb300 has it do, as cases to be timed.

Kinds:
  td       glgpu_td on one handle: the state is set from device memory, advanced by
           `steps` time steps and read back into device memory (the C ABI's set / get
           calls take host or device pointers).
  batch_td HandleBatch.td_raw: many instances of uneven sizes in one device loop.
  batch_cg HandleBatch.cg_device: the batched device CG, a fixed number of iterations.
  session  the GLSolver drop-in on host arrays: set psi, solve.td, solve.cg, observables.
  conv     learned.Conv3x3 of one layer, forward and both gradients.
  predict  learned.WarmStartNet.predict, the whole network.

`exact` restates each kind in 64 bits with plain torch and numpy."""
import ctypes
import math

import numpy as np
import torch
import torch.nn.functional as F

from svirl_gb300 import GLSolver, _lib, learned
from svirl_gb300.batch import HandleBatch

DX = 0.5
DT = 0.1
SIGMA = 200.0
CIN, NOUT = 8, 4


def listed():
    return [
        # the smallest call: one serving-size instance advanced by a few steps
        {"name": "td_65_f32", "kind": "td", "nx": 65, "ny": 65, "bits": 32, "kappa": 0.0, "H": 0.1, "holes": 0.0,
         "steps": 5, "noise": 0.0, "eps": False},
        # the plain small configuration (129^2, kappa = 5, FP64, full domain)
        {"name": "td_129_f64_k5", "kind": "td", "nx": 129, "ny": 129, "bits": 64, "kappa": 5.0, "H": 0.1, "holes": 0.0,
         "steps": 20, "noise": 0.0, "eps": False},
        # an ordinary oblong film with holes and Langevin noise
        {"name": "td_385x321_f32_k4_noise", "kind": "td", "nx": 385, "ny": 321, "bits": 32, "kappa": 4.0, "H": 0.2,
         "holes": 0.03, "steps": 20, "noise": 0.01, "eps": False},
        # the large single domain of the benchmark
        {"name": "td_2049_f32", "kind": "td", "nx": 2049, "ny": 2049, "bits": 32, "kappa": 0.0, "H": 0.05,
         "holes": 0.05, "steps": 20, "noise": 0.0, "eps": False},
        # the same domain with the vector-potential equation
        {"name": "td_2049_f32_k4", "kind": "td", "nx": 2049, "ny": 2049, "bits": 32, "kappa": 4.0, "H": 0.05,
         "holes": 0.05, "steps": 10, "noise": 0.0, "eps": False},
        # a large FP64 film with a spatial linear coefficient
        {"name": "td_1025x769_f64_eps", "kind": "td", "nx": 1025, "ny": 769, "bits": 64, "kappa": 0.0, "H": 0.1,
         "holes": 0.02, "steps": 5, "noise": 0.0, "eps": True},
        # what the serving loop runs: requests of uneven sizes, kappa finite or infinite
        {"name": "batch_td_f32", "kind": "batch_td", "count": 32, "nmin": 64, "nmax": 512, "bits": 32, "steps": 20},
        # the field sweep of relaxed states (129 .. 513), FP32
        {"name": "batch_cg_f32", "kind": "batch_cg", "count": 48, "nmin": 129, "nmax": 513, "bits": 32, "kinf": 0.0,
         "iters": 8},
        # FP64 relaxation of small states (reference energies, the strict criterion)
        {"name": "batch_cg_f64", "kind": "batch_cg", "count": 8, "nmin": 97, "nmax": 193, "bits": 64, "kinf": 0.25,
         "iters": 20},
        # the drop-in API on host arrays
        {"name": "session_129_f64", "kind": "session", "n": 129, "holes": 0.03, "H": 0.2, "steps": 20, "iters": 10},
        # the first decoder convolution at full resolution: upsampled 64 channels and the 32-channel skip
        {"name": "conv_skip_32x128x128", "kind": "conv", "batch": 32, "h": 128, "w": 128, "c1": 64, "c2": 32, "cout": 32,
         "relu": True},
        # a batch of warm starts
        {"name": "predict_64x128x128", "kind": "predict", "batch": 64, "h": 128, "w": 128},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["td", "td", "td", "batch_td", "batch_cg", "batch_cg", "session", "conv", "conv", "predict"])
    if kind == "td":
        bits = rng.choice([32, 32, 64])
        top = 2049 if bits == 32 else 900
        nx, ny = _log_int(rng, 48, top), _log_int(rng, 48, top)
        return {"kind": "td", "nx": nx, "ny": ny, "bits": bits,
                "kappa": rng.choice([0.0, round(rng.uniform(2.0, 8.0), 2)]), "H": round(rng.uniform(0.02, 0.4), 3),
                "holes": rng.choice([0.0, round(rng.uniform(0.005, 0.05), 3)]),
                "steps": rng.randint(3, 20) if nx * ny < 600000 else rng.randint(3, 10 if bits == 32 else 4),
                "noise": rng.choice([0.0, 0.0, 0.01]), "eps": rng.random() < 0.2}
    if kind == "batch_td":
        bits = 32 if rng.random() < 0.7 else 64
        return {"kind": kind, "count": rng.randint(2, 32), "nmin": _log_int(rng, 48, 96), "nmax": _log_int(rng, 129, 512),
                "bits": bits, "steps": rng.randint(2, 8 if bits == 32 else 4)}
    if kind == "batch_cg":
        if rng.random() < 0.6:
            return {"kind": kind, "count": _log_int(rng, 1, 48), "nmin": _log_int(rng, 65, 129),
                    "nmax": _log_int(rng, 193, 513), "bits": 32, "kinf": rng.choice([0.0, 0.5]),
                    "iters": rng.randint(4, 8)}
        return {"kind": kind, "count": _log_int(rng, 1, 8), "nmin": _log_int(rng, 65, 97), "nmax": _log_int(rng, 129, 257),
                "bits": 64, "kinf": rng.choice([0.0, 0.5]), "iters": rng.randint(8, 20)}
    if kind == "session":
        return {"kind": kind, "n": _log_int(rng, 49, 257), "holes": round(rng.uniform(0.0, 0.05), 3),
                "H": round(rng.uniform(0.05, 0.4), 3), "steps": rng.randint(3, 20), "iters": rng.randint(3, 12)}
    level = rng.randint(0, 3)  # of the network: full resolution and 32 channels, down to an eighth and 128
    if kind == "conv":
        c = {"kind": kind, "batch": rng.randint(1, 32), "h": (8 * rng.randint(8, 16)) >> level,
             "w": (8 * rng.randint(8, 16)) >> level, "relu": True}
        c.update(rng.choice([[{"c1": 8, "c2": 0, "cout": 32}, {"c1": 32, "c2": 0, "cout": 32}, {"c1": 64, "c2": 32, "cout": 32}],
                             [{"c1": 32, "c2": 0, "cout": 64}, {"c1": 64, "c2": 0, "cout": 64}, {"c1": 128, "c2": 64, "cout": 64}],
                             [{"c1": 64, "c2": 0, "cout": 128}, {"c1": 128, "c2": 0, "cout": 128},
                              {"c1": 128, "c2": 128, "cout": 128}],
                             [{"c1": 128, "c2": 0, "cout": 128}]][level]))
        return c
    n = 8 * rng.randint(8, 16)
    return {"kind": kind, "batch": _log_int(rng, 1, 64), "h": n, "w": n}


# --- inputs --------------------------------------------------------------------

def _instances(case, seed):
    """Sizes and kappas of a batch (from the case), its fields and masks (from the seed)."""
    sizes, rng = np.random.default_rng(case["count"] + case["nmax"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        n = int(sizes.integers(case["nmin"], case["nmax"] + 1))
        if case["kind"] == "batch_cg":
            kinf = sizes.random() < case["kinf"]
            kappa = 0.0 if kinf else 4.0
        else:
            kappa = 0.0 if sizes.random() < 0.5 else 2.0 + 6.0 * sizes.random()
        H = 0.02 + 0.38 * rng.random()
        out.append({"nx": n, "ny": n, "kappa": kappa, "H": H, "noise": 0.0,
                    "mt": learned.holes_mask(n, DX, 0.05 * rng.random(), 2.0, 6.0, rng).T.copy()})
    return out


def _holes(nx, ny, frac, rng):
    """Cells [j, i] outside circular holes of radius 4 that cover `frac` of the film."""
    mt = np.ones((ny - 1, nx - 1), dtype=np.uint8)
    r = 4.0 / DX
    k = int(math.ceil(frac * mt.size / (math.pi * r * r)))
    for cx, cy in zip(rng.random(k) * nx, rng.random(k) * ny):
        i0, i1 = max(0, int(cx - r) - 1), min(nx - 1, int(cx + r) + 2)
        j0, j1 = max(0, int(cy - r) - 1), min(ny - 1, int(cy + r) + 2)
        jj, ii = np.mgrid[j0:j1, i0:i1]
        mt[j0:j1, i0:i1][(ii + 0.5 - cx) ** 2 + (jj + 0.5 - cy) ** 2 < r * r] = 0
    return mt


def _td_instance(case, seed):
    rng = np.random.default_rng(seed)
    return {"nx": case["nx"], "ny": case["ny"], "kappa": case["kappa"], "H": case["H"], "noise": case["noise"],
            "rand_t": 1 + seed % 100000,
            "mt": _holes(case["nx"], case["ny"], case["holes"], rng) if case["holes"] > 0 else None}


def _psi0(n, gen, bits):
    """Amplitude U(0, 1], phase U(-pi, pi]: the reference's random start."""
    u = torch.rand((2, n), generator=gen, device="cuda", dtype=torch.float64)
    p = torch.polar(1.0 - u[0], math.pi * (2.0 * u[1] - 1.0))
    return p.to(torch.complex64 if bits == 32 else torch.complex128)


def _landau(nx, ny, H, bits):
    """A = (-H y, 0), flat [a | b]."""
    a = (-H * DX * torch.arange(ny, device="cuda", dtype=torch.float64))[:, None].expand(ny, nx - 1).reshape(-1)
    ab = torch.cat([a, torch.zeros(nx * (ny - 1), device="cuda", dtype=torch.float64)])
    return ab.to(torch.float32 if bits == 32 else torch.float64)


def _eps_field(nx, ny, gen, bits):
    e = 1.0 - 0.3 * torch.rand(nx * ny, generator=gen, device="cuda", dtype=torch.float64)
    return e.to(torch.float32 if bits == 32 else torch.float64)


def _np_dtype(bits):
    return np.float32 if bits == 32 else np.float64


def _handle(inst, bits, eps=None):
    h = _lib.Handle(inst["nx"], inst["ny"], DX, DX, _np_dtype(bits))
    h.set_params(kappa=inst["kappa"] if inst["kappa"] > 0 else float("inf"), H=inst["H"], sigma=SIGMA, epsilon=1.0,
                 langevin_psi=inst["noise"], langevin_A=0.01 * inst["noise"], rand_t=inst.get("rand_t", 1))
    if inst["mt"] is not None:
        h.set_mask(inst["mt"].reshape(-1).astype(np.uint8))
    if eps is not None:
        h.set_eps_field(eps.cpu().numpy())
    return h


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _conv_inputs(case, seed):
    g = _gen(seed)
    n, h, w = case["batch"], case["h"], case["w"]
    cin = case["c1"] + case["c2"]

    def act(c):  # what a ReLU layer passes on
        return torch.randn((n, h, w, c), generator=g, device="cuda").clamp_min(0).to(torch.bfloat16) if c else None

    x1, x2 = act(case["c1"]), act(case["c2"])
    wt = torch.randn((case["cout"], 3, 3, cin), generator=g, device="cuda") * math.sqrt(2.0 / (9 * cin))
    wt = wt.to(torch.bfloat16).float()  # the ReLU's sign is then the exact one
    b = 0.1 * torch.randn((case["cout"],), generator=g, device="cuda")
    dy = 1e-3 * torch.randn((n, h, w, case["cout"]), generator=g, device="cuda")
    return x1, x2, wt, b, dy.to(torch.bfloat16)


def _features(case, seed):
    """[node mask, H, 1/kappa, Re psi0, Im psi0, 0, 0, 0]."""
    g = _gen(seed)
    n, h, w = case["batch"], case["h"], case["w"]
    x = torch.zeros((n, h, w, CIN), device="cuda")
    coarse = torch.rand((n, 1, h // 8, w // 8), generator=g, device="cuda")
    x[..., 0] = (F.interpolate(coarse, size=(h, w), mode="bilinear")[:, 0] > 0.2).float()
    x[..., 1] = (0.02 + 0.48 * torch.rand((n, 1, 1), generator=g, device="cuda"))
    x[..., 2] = 1.0 / (2.0 + 8.0 * torch.rand((n, 1, 1), generator=g, device="cuda"))
    p = _psi0(n * h * w, g, 32).reshape(n, h, w)
    x[..., 3], x[..., 4] = p.real, p.imag
    return x.to(torch.bfloat16)


# --- the passes ------------------------------------------------------------------

def _p(t, offset=0):
    return ctypes.c_void_p(t.data_ptr() + offset)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "td":
        inst, gen = _td_instance(case, seed), _gen(seed)
        s["psi0"] = _psi0(inst["nx"] * inst["ny"], gen, case["bits"])
        s["ab0"] = _landau(inst["nx"], inst["ny"], inst["H"], case["bits"])
        s["h"] = _handle(inst, case["bits"], _eps_field(inst["nx"], inst["ny"], gen, case["bits"]) if case["eps"] else None)
        s["psi"], s["ab"] = torch.empty_like(s["psi0"]), torch.empty_like(s["ab0"])
    elif kind in ("batch_td", "batch_cg"):
        insts, gen, bits = _instances(case, seed), _gen(seed), case["bits"]
        s["hs"] = [_handle(it, bits) for it in insts]
        s["batch"] = HandleBatch(s["hs"])
        s["psi0"] = torch.cat([_psi0(h.N, gen, bits) for h in s["hs"]])
        s["ab0"] = torch.cat([_landau(it["nx"], it["ny"], it["H"], bits) for it in insts])
        s["psi"], s["ab"] = torch.empty_like(s["psi0"]), torch.empty_like(s["ab0"])
    elif kind == "session":
        rng = np.random.default_rng(seed)
        n = case["n"]
        mt = _holes(n, n, case["holes"], rng).astype(bool).T if case["holes"] > 0 else None
        s["gl"] = GLSolver(Nx=n, Ny=n, dx=DX, dy=DX, order_parameter=1.0, gl_parameter=np.inf, material_tiling=mt,
                           homogeneous_external_field=case["H"], convergence_rtol=1e-30)
        s["psi0"] = _psi0(n * n, _gen(seed), 64).cpu().numpy().reshape(n, n).T.copy()  # [i, j]
        s["ab0"] = s["gl"].vars.vector_potential
    elif kind == "conv":
        x1, x2, w, b, dy = _conv_inputs(case, seed)
        s["dy"] = dy
        s["in"] = [None if t is None else t.requires_grad_() for t in (x1, x2, w, b)]
    else:
        net = learned.WarmStartNet(seed=seed % 1000)
        s["net"], s["x"] = net, _features(case, seed)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "td":
        h = s["h"]
        _lib.check(h.lib.glgpu_set_order_parameter(h.h, _p(s["psi0"])), h.h, "set_order_parameter")
        _lib.check(h.lib.glgpu_set_vector_potential(h.h, _p(s["ab0"])), h.h, "set_vector_potential")
        h.td(DT, case["steps"])
        _lib.check(h.lib.glgpu_get_order_parameter(h.h, _p(s["psi"])), h.h, "get_order_parameter")
        if case["kappa"] > 0:
            _lib.check(h.lib.glgpu_get_vector_potential(h.h, _p(s["ab"])), h.h, "get_vector_potential")
            return {"psi": s["psi"], "ab": s["ab"]}
        return {"psi": s["psi"]}
    if kind in ("batch_td", "batch_cg"):
        return _run_batch(s)
    if kind == "session":
        gl = s["gl"]
        gl.vars.order_parameter = s["psi0"]
        gl.solve.td(dt=DT, Nt=case["steps"])
        vx, vy, vv = gl.vortex_detector.vortices
        gl.solve.cg(n_iter=case["iters"])
        o = gl.observables
        found = np.zeros((3, gl.cfg.Nc))  # as many columns as there can be vortices
        found[:, :len(vx)] = vx, vy, vv
        return {"vortices": found, "psi": gl.vars.order_parameter, "energy": o.free_energy,
                "energies": np.array(gl.solve._cg.cg_energies), "js": o.supercurrent_density, "B": o.magnetic_field}
    if kind == "conv":
        x1, x2, w, b = s["in"]
        y = learned.Conv3x3.apply(x1, x2, w, b, case["relu"])
        g = torch.autograd.grad(y, [t for t in s["in"] if t is not None], s["dy"])
        return {"y": y.detach(), "grads": list(g)}
    return s["net"].predict(s["x"])


def _run_batch(s):
    case, lib = s["case"], s["hs"][0].lib
    cs, rs = s["psi0"].element_size(), s["ab0"].element_size()
    at, al = 0, 0
    for h in s["hs"]:
        _lib.check(lib.glgpu_set_order_parameter(h.h, _p(s["psi0"], at * cs)), h.h, "set_order_parameter")
        _lib.check(lib.glgpu_set_vector_potential(h.h, _p(s["ab0"], al * rs)), h.h, "set_vector_potential")
        at, al = at + h.N, al + h.Nab
    out = {}
    if case["kind"] == "batch_td":
        s["batch"].td_raw(DT, case["steps"])
    else:
        r = s["batch"].cg_device(n_iter=case["iters"], rtol=0.0, gtol=0.0, exact_boundary=True)
        # (the energy of an FP32 state has FP32's precision)
        out = {"energy": r["energy"].astype(_np_dtype(case["bits"])), "iters": r["iters"], "status": r["status"]}
    at, al = 0, 0
    for h in s["hs"]:
        _lib.check(lib.glgpu_get_order_parameter(h.h, _p(s["psi"], at * cs)), h.h, "get_order_parameter")
        _lib.check(lib.glgpu_get_vector_potential(h.h, _p(s["ab"], al * rs)), h.h, "get_vector_potential")
        at, al = at + h.N, al + h.Nab
    out.update(psi=s["psi"], ab=s["ab"])
    return out


# --- what a pass cannot do without -------------------------------------------------

PSI_SWEEPS, A_SWEEPS = 20, 3       # Jacobi sweeps of a usual step
PSI_FLOPS, A_FLOPS = 40, 60        # per node and sweep
CG_FLOPS = 400                     # per node and iteration: gradient, line-search sums, step and energy


def _td_work(nx, ny, kappa, bits, steps, mask):
    n, rs = nx * ny, bits // 8
    reals = 2 * n * 2 + (2 * n * 2 if kappa > 0 else 2 * n)  # psi in and out, A in (and out)
    return n * mask + reals * rs, steps * n * (PSI_SWEEPS * PSI_FLOPS + (A_SWEEPS * A_FLOPS if kappa > 0 else 0))


def work(case):
    kind = case["kind"]
    if kind == "td":
        b, f = _td_work(case["nx"], case["ny"], case["kappa"], case["bits"], case["steps"], 1 if case["holes"] > 0 else 0)
    elif kind in ("batch_td", "batch_cg"):
        b = f = 0
        for it in _instances(case, 0):
            if kind == "batch_td":
                x, y = _td_work(it["nx"], it["ny"], it["kappa"], case["bits"], case["steps"], 1)
            else:
                n = it["nx"] * it["ny"]
                x, y = n * (8 * case["bits"] // 8 + 1), n * case["iters"] * CG_FLOPS
            b, f = b + x, f + y
    elif kind == "session":
        n = case["n"] ** 2
        b = n * 16 * 2 + n * 8 * 5 + n
        f = case["steps"] * n * PSI_SWEEPS * PSI_FLOPS + case["iters"] * n * CG_FLOPS
    elif kind == "conv":
        p, cin, co = case["batch"] * case["h"] * case["w"], case["c1"] + case["c2"], case["cout"]
        b = 2 * p * (2 * cin + 2 * co) + 4 * 9 * cin * co * 2  # x, dx; y, dy; w, dw
        f = 3 * 2 * p * 9 * cin * co
    else:
        p = case["batch"] * case["h"] * case["w"]
        c = learned.LEVELS
        per = 9 * (CIN * c[0] + c[0] * c[0] + (c[1] + c[0]) * c[0] + c[0] * c[0] + c[0] * 8)
        per += 9 * (c[0] * c[1] + c[1] * c[1] + (c[2] + c[1]) * c[1] + c[1] * c[1]) / 4
        per += 9 * (c[1] * c[2] + c[2] * c[2] + (c[3] + c[2]) * c[2] + c[2] * c[2]) / 16
        per += 9 * (c[2] * c[3] + c[3] * c[3]) / 64
        b, f = 2 * p * (CIN + 8), 2 * p * per
    return {"bytes": float(b), "flops": float(f)}


# --- the same in 64 bits -------------------------------------------------------------

def _cells(mt, nx, ny):
    """Material of the four cells around each node [j, i]: (mm, mp, pm, pp); first
    sign the cell's x side, second its y side."""
    m = torch.ones((ny - 1, nx - 1), dtype=torch.bool) if mt is None else torch.from_numpy(np.ascontiguousarray(mt) != 0)
    q = F.pad(m.cuda().to(torch.uint8), (1, 1, 1, 1)).bool()
    return q[:-1, :-1], q[1:, :-1], q[:-1, 1:], q[1:, 1:]


def _noise(numbers, t, k0, k1, k2):
    """The hash noise U[0, 1) - 1/2 of the Langevin terms."""
    m = 0xFFFFFFFF
    s = (numbers * k0 + k1 * t + k2) & m
    s = ((s ^ 61) ^ (s >> 16)) & m
    s = (s * 9) & m
    s = s ^ (s >> 4)
    s = (s * 0x27D4EB2D) & m
    s = s ^ (s >> 15)
    return s.double() * 2.0 ** -32 - 0.5


def _split(ab, nx, ny):
    na = (nx - 1) * ny
    return ab[:na].reshape(ny, nx - 1), ab[na:].reshape(ny - 1, nx)


def _exact_td(inst, psi, ab, eps, steps, stop=1e-6):
    """Backward-Euler TDGL: Jacobi iteration of the psi step, then of the A step."""
    nx, ny, H = inst["nx"], inst["ny"], inst["H"]
    mm, mp, pm, pp = _cells(inst["mt"], nx, ny)
    left, right, down, up = mm | mp, pm | pp, mm | pm, mp | pp
    psi, ab = psi.to(torch.complex128).reshape(ny, nx), ab.double()
    a, b = (t.clone() for t in _split(ab, nx, ny))
    i2 = 1.0 / (DX * DX)
    eps = 1.0 if eps is None else eps.double().reshape(ny, nx)
    cnt = left.double() + right.double() + down.double() + up.double()
    own = (left | right).double()
    solve_a = inst["kappa"] > 0
    rho, k2 = 1.0 / SIGMA, inst["kappa"] ** 2
    t = inst.get("rand_t", 1)
    nodes = torch.arange(nx * ny, device="cuda", dtype=torch.int64).reshape(ny, nx)
    nla = torch.arange(a.numel(), device="cuda", dtype=torch.int64).reshape(a.shape)
    nlb = a.numel() + torch.arange(b.numel(), device="cuda", dtype=torch.int64).reshape(b.shape)
    lp = float(np.float32(inst["noise"])) if inst.get("bits") == 32 else inst["noise"]
    la = 0.01 * inst["noise"]
    wx, wy = right[:, :-1].double(), up[:-1].double()
    for _ in range(steps):
        ux, uy = DT * i2 * wx * torch.exp(-1j * DX * a), DT * i2 * wy * torch.exp(-1j * DX * b)
        rq = psi
        if lp > 0:
            rq = psi + lp * torch.complex(_noise(nodes, t, 71, 9887, 0), _noise(nodes, t, 73, 9901, 1))
        inv = own / (1.0 + DT * (rq.real ** 2 + rq.imag ** 2 - eps + i2 * cnt))
        for _ in range(1024):
            new = rq.clone()
            new[:, 1:] += ux.conj() * psi[:, :-1]
            new[:, :-1] += ux * psi[:, 1:]
            new[1:] += uy.conj() * psi[:-1]
            new[:-1] += uy * psi[1:]
            new *= inv
            r = torch.view_as_real(new - psi).abs().max().item()
            psi = new
            if not r >= stop:
                break
        t += 1
        if not solve_a:
            continue
        ra, rb = a, b
        if la > 0:
            ra, rb = a + la * _noise(nla, t, 71, 9887, 0), b + la * _noise(nlb, t, 73, 9901, 1)
        ha, hb = torch.zeros_like(a), torch.zeros_like(b)
        ha[0], ha[-1] = 2 * k2 * H / DX, -2 * k2 * H / DX
        hb[:, 0], hb[:, -1] = -2 * k2 * H / DX, 2 * k2 * H / DX
        da, db = torch.ones_like(a), torch.ones_like(b)
        da[0] = da[-1] = 2.0
        db[:, 0] = db[:, -1] = 2.0
        c = DT * rho * k2
        for k in range(1024):
            if k % 2 == 0:  # the supercurrent of A^(2 floor(k / 2))
                ja = wx * torch.imag(psi[:, :-1].conj() * torch.exp(-1j * DX * a) * psi[:, 1:]) / DX
                jb = wy * torch.imag(psi[:-1].conj() * torch.exp(-1j * DX * b) * psi[1:]) / DX
            na, nb = torch.zeros_like(a), torch.zeros_like(b)
            cb, ca = b[:, 1:] - b[:, :-1], a[1:] - a[:-1]
            na[1:] += i2 * (a[:-1] + cb)
            na[:-1] += i2 * (a[1:] - cb)
            nb[:, 1:] += i2 * (b[:, :-1] + ca)
            nb[:, :-1] += i2 * (b[:, 1:] - ca)
            va = (ra + DT * rho * (ja + ha) + c * da * na) / (1 + 2 * c * i2)
            vb = (rb + DT * rho * (jb + hb) + c * db * nb) / (1 + 2 * c * i2)
            r = max((va - a).abs().max().item(), (vb - b).abs().max().item())
            a, b = va, vb
            if not r >= stop:
                break
        t += 1
    return psi.reshape(-1), torch.cat([a.reshape(-1), b.reshape(-1)])


class _Film:
    """Free energy, its gradient (autograd) and its line-search polynomial, 64 bits."""

    def __init__(self, mt, nx, ny, kappa, H):
        mm, mp, pm, pp = (q.double() for q in _cells(mt, nx, ny))
        self.nx, self.ny, self.k2, self.H = nx, ny, kappa ** 2, H
        self.wg = 0.25 * (mm + mp + pm + pp)
        self.wx, self.wy = 0.5 * (pm + pp)[:, :-1], 0.5 * (mp + pp)[:-1]
        self.i2 = 1.0 / (DX * DX)

    def curl(self, a, b):
        return (b[:, 1:] - b[:, :-1]) / DX - (a[1:] - a[:-1]) / DX

    def energy(self, p, a, b):
        p2 = p.real ** 2 + p.imag ** 2
        gx = p[:, 1:] * torch.exp(-1j * DX * a) - p[:, :-1]
        gy = p[1:] * torch.exp(-1j * DX * b) - p[:-1]
        e = (self.wg * (0.5 * p2 - 1.0) * p2).sum()
        e = e + self.i2 * ((self.wx * (gx.real ** 2 + gx.imag ** 2)).sum() + (self.wy * (gy.real ** 2 + gy.imag ** 2)).sum())
        if self.k2 > 0:
            e = e + self.k2 * ((self.curl(a, b) - self.H) ** 2).sum()
        return e * DX * DX

    def grad(self, p, a, b):
        pr = torch.view_as_real(p).clone().requires_grad_()
        a, b = a.clone().requires_grad_(), b.clone().requires_grad_()
        g = torch.autograd.grad(self.energy(torch.view_as_complex(pr), a, b), [pr, a, b])
        return torch.view_as_complex(g[0].contiguous()), g[1], g[2]

    def poly(self, p, a, b, d, da, db):
        """c[i, j] of F(psi + x d, A + y dA), to the fourth order in y."""
        c = np.zeros((5, 5))
        p2, d2 = p.real ** 2 + p.imag ** 2, d.real ** 2 + d.imag ** 2
        tw = 2.0 * (p.real * d.real + p.imag * d.imag)
        ks = [(0.5 * p2 - 1) * p2, tw * (p2 - 1), -d2 + 0.5 * tw * tw + p2 * d2, tw * d2, 0.5 * d2 * d2]
        for i, k in enumerate(ks):
            c[i, 0] += (self.wg * k).sum().item()
        for w, A, dA, p0, p1, d0, d1 in ((self.wx, a, da, p[:, :-1], p[:, 1:], d[:, :-1], d[:, 1:]),
                                         (self.wy, b, db, p[:-1], p[1:], d[:-1], d[1:])):
            w = w * self.i2
            U = torch.exp(-1j * DX * A)
            gp, gd = p1 * U - p0, d1 * U - d0
            c[0, 0] += (w * (gp.real ** 2 + gp.imag ** 2)).sum().item()
            c[1, 0] += 2 * (w * (gp.real * gd.real + gp.imag * gd.imag)).sum().item()
            c[2, 0] += (w * (gd.real ** 2 + gd.imag ** 2)).sum().item()
            if self.k2 > 0:
                f = DX * dA
                um = U.conj()
                for i, z in enumerate((p0 * um * p1.conj(), p0 * um * d1.conj() + d0 * um * p1.conj(), d0 * um * d1.conj())):
                    c[i, 1] += 2 * (w * z.imag * f).sum().item()
                    c[i, 2] += (w * z.real * f ** 2).sum().item()
                    c[i, 3] -= (w * z.imag * f ** 3).sum().item() / 3
                    c[i, 4] -= (w * z.real * f ** 4).sum().item() / 12
        if self.k2 > 0:
            BH, dB = self.curl(a, b) - self.H, self.curl(da, db)
            c[0, 0] += self.k2 * (BH ** 2).sum().item()
            c[0, 1] += 2 * self.k2 * (BH * dB).sum().item()
            c[0, 2] += self.k2 * (dB ** 2).sum().item()
        return c


def _cubic_step(c):
    r = np.polynomial.polynomial.polyroots([c[1, 0], 2 * c[2, 0], 3 * c[3, 0], 4 * c[4, 0]])
    r = r[np.isclose(r.imag, 0)].real
    return r[r >= 0].min()


def _joint_step(c):
    """The local minimum that a damped Newton descent from (0, 0) reaches."""
    P = np.polynomial.polynomial
    c = c / np.abs(c.reshape(-1)[1:]).max()
    c[0, 0] = 0.0
    der = lambda *ax: P.polyder(der(*ax[1:]), axis=ax[0]) if ax else c  # noqa: E731
    x = np.zeros(2)
    for _ in range(60):
        val = lambda *ax: P.polyval2d(x[0], x[1], der(*ax))  # noqa: E731
        g = np.array([val(0), val(1)])
        h = np.array([[val(0, 0), val(0, 1)], [val(0, 1), val(1, 1)]])
        if h[0, 0] > 0 and np.linalg.det(h) > 0:
            s = -np.linalg.solve(h, g)
        else:
            s = -g / (abs(h[0, 0]) + abs(h[1, 1]) + 1e-30)
        f0, t = val(), 1.0
        while t > 1e-12 and P.polyval2d(x[0] + t * s[0], x[1] + t * s[1], c) > f0 + 1e-4 * t * g.dot(s):
            t *= 0.5
        if t <= 1e-12:
            break
        x = x + t * s
        if np.abs(t * s).sum() < 1e-15:
            break
    return x


def _exact_cg(film, p, a, b, iters):
    """Polak-Ribiere+ CG from a zero direction; psi and A with a beta each."""
    d, da, db = torch.zeros_like(p), torch.zeros_like(a), torch.zeros_like(b)
    old, energies = None, []
    dot = lambda u, v: (u.real * v.real + u.imag * v.imag).sum().item()  # noqa: E731
    for _ in range(iters):
        g, ga, gb = film.grad(p, a, b)
        bp = bA = 0.0
        if old is not None:
            bp = max(dot(g, g - old[0]) / dot(old[0], old[0]), 0.0)
            if film.k2 > 0:
                num = (ga * (ga - old[1])).sum() + (gb * (gb - old[2])).sum()
                bA = max((num / ((old[1] ** 2).sum() + (old[2] ** 2).sum())).item(), 0.0)
        old = (g, ga, gb)
        d, da, db = bp * d - g, bA * da - ga, bA * db - gb
        c = film.poly(p, a, b, d, da, db)
        x, y = _joint_step(c) if film.k2 > 0 else (_cubic_step(c), 0.0)
        p = p + x * d
        if film.k2 > 0:
            a, b = a + y * da, b + y * db
        energies.append(film.energy(p, a, b).item())
    return p, a, b, energies


def _exact_session(case, seed):
    n, H = case["n"], case["H"]
    rng = np.random.default_rng(seed)
    mt = _holes(n, n, case["holes"], rng) if case["holes"] > 0 else None
    y = DX * torch.arange(n, device="cuda", dtype=torch.float64) - 0.5 * DX * (n - 1)
    a = (-0.5 * H * y)[:, None].expand(n, n - 1)
    b = (0.5 * H * y)[None, :].expand(n - 1, n)
    inst = {"nx": n, "ny": n, "kappa": 0.0, "H": H, "noise": 0.0, "mt": mt}
    mm, mp, pm, pp = _cells(mt, n, n)
    psi = _psi0(n * n, _gen(seed), 64).reshape(n, n) * (mm | mp | pm | pp)
    psi, _ = _exact_td(inst, psi.reshape(-1), torch.cat([a.reshape(-1), b.reshape(-1)]), None, case["steps"])
    film = _Film(mt, n, n, 0.0, H)
    p, _, _, es = _exact_cg(film, psi.reshape(n, n), a, b, case["iters"])
    jx = film.wx * torch.imag(p[:, :-1].conj() * torch.exp(-1j * DX * a) * p[:, 1:]) / DX
    jy = film.wy * torch.imag(p[:-1].conj() * torch.exp(-1j * DX * b) * p[1:]) / DX
    return {"vortices": None, "psi": p.T.contiguous().cpu().numpy(), "energy": es[-1], "energies": np.array(es),
            "js": (jx.T.contiguous().cpu().numpy(), jy.T.contiguous().cpu().numpy()),
            "B": film.curl(a, b).T.contiguous().cpu().numpy()}


def _exact_net(case, seed):
    net = learned.WarmStartNet(seed=seed % 1000)  # its initial weights, for their values alone
    w = {k: v.detach().double().permute(0, 3, 1, 2) for k, v in net.w.items()}
    bias = {k: v.detach().double() for k, v in net.b.items()}

    def c(name, *xs):
        y = F.conv2d(torch.cat(xs, 1), w[name], bias[name], padding=1)
        return y if name == "out" else y.clamp_min(0)

    def up(x):
        return x.repeat_interleave(2, 2).repeat_interleave(2, 3)

    out = []
    for x in _features(case, seed).double().permute(0, 3, 1, 2).split(8):
        e0 = c("e0b", c("e0a", x))
        e1 = c("e1b", c("e1a", F.avg_pool2d(e0, 2)))
        e2 = c("e2b", c("e2a", F.avg_pool2d(e1, 2)))
        m = c("m_b", c("m_a", F.avg_pool2d(e2, 2)))
        d2 = c("d2b", c("d2a", up(m), e2))
        d1 = c("d1b", c("d1a", up(d2), e1))
        out.append(c("out", c("d0b", c("d0a", up(d1), e0))).permute(0, 2, 3, 1))
    return torch.cat(out).contiguous()


def exact(case, seed):
    kind = case["kind"]
    if kind == "td":
        inst, gen = dict(_td_instance(case, seed), bits=case["bits"]), _gen(seed)
        psi0 = _psi0(inst["nx"] * inst["ny"], gen, case["bits"])
        eps = _eps_field(inst["nx"], inst["ny"], gen, case["bits"]) if case["eps"] else None
        psi, ab = _exact_td(inst, psi0, _landau(inst["nx"], inst["ny"], inst["H"], case["bits"]), eps, case["steps"])
        return {"psi": psi, "ab": ab} if case["kappa"] > 0 else {"psi": psi}
    if kind in ("batch_td", "batch_cg"):
        insts, gen = _instances(case, seed), _gen(seed)
        starts = [_psi0(it["nx"] * it["ny"], gen, case["bits"]) for it in insts]
        psis, abs_, es = [], [], []
        for it, p in zip(insts, starts):
            nx, ny = it["nx"], it["ny"]
            ab = _landau(nx, ny, it["H"], case["bits"])
            if kind == "batch_td":
                p, ab = _exact_td(it, p, ab, None, case["steps"])
            else:
                a, b = _split(ab.double(), nx, ny)
                p, a, b, e = _exact_cg(_Film(it["mt"], nx, ny, it["kappa"], it["H"]), p.to(torch.complex128).reshape(ny, nx),
                                       a, b, case["iters"])
                p, ab = p.reshape(-1), torch.cat([a.reshape(-1), b.reshape(-1)])
                es.append(e[-1])
            psis.append(p)
            abs_.append(ab)
        out = {"psi": torch.cat(psis), "ab": torch.cat(abs_)}
        if kind == "batch_cg":
            out.update(energy=np.array(es), iters=None, status=None)
        return out
    if kind == "session":
        return _exact_session(case, seed)
    if kind == "conv":
        x1, x2, w, b, dy = _conv_inputs(case, seed)
        leaves = [t.double().requires_grad_() for t in (x1, x2, w, b) if t is not None]
        x = torch.cat(leaves[:-2], 3).permute(0, 3, 1, 2)
        y = F.conv2d(x, leaves[-2].permute(0, 3, 1, 2), leaves[-1], padding=1)
        y = (y.clamp_min(0) if case["relu"] else y).permute(0, 2, 3, 1)
        g = torch.autograd.grad(y, leaves, dy.double())
        return {"y": y.detach().contiguous(), "grads": [t.contiguous() for t in g]}
    return _exact_net(case, seed)
