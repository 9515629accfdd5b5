"""The work that a user of this library has it do, as timed cases.

One case is one pass through the public entry points (Solver, step_noalloc,
Batch, Amr2D, Amr3D, Server): some steps of a flow and the readback of its
result, as a program that draws frames, logs drag or collects finished
solves does them. The families, and the sizes they are used at:

  call    one step between the caller's own device buffers (step_noalloc)
  dense3  a 3D session: n steps, the drag logged every few of them into pinned
          memory, the field into a device tensor
  dense2  a 2D session (the pinned-cylinder page): the same, the field to the host
  free    a 3D session whose rigid body the device integrates
  batch   many small 2D domains advanced together
  amr2    the two-level 2D cylinder with its refine rounds
  amr3    a two-level 3D hierarchy around a body
  serve   a stream of 3D requests through the request loop

`work` counts, for every step, each population read once and written once
(the usual lattice-Boltzmann traffic: 2 Q values per cell and step), plus
the field that is read back. Populations that stay in the L2 cache between
steps are counted the same way.
"""
from __future__ import annotations

import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
U0 = 0.05
EVERY = 5  # steps between two entries of a dense session's drag log


def package():
    """The library's package (its folder's name is no Python identifier)."""
    if "getting_air_b200" in sys.modules:
        return sys.modules["getting_air_b200"]
    pkg = ROOT / "getting-air_b200"
    spec = importlib.util.spec_from_file_location("getting_air_b200", pkg / "__init__.py",
                                                  submodule_search_locations=[str(pkg)])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["getting_air_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


# ---- the cases ---------------------------------------------------------------

def listed():
    return [
        # The smallest call: one step of the smoke-test domain between buffers
        # an engine owns, field and force written on the device. Latency.
        {"name": "call-q19-48", "family": "call", "q": 19, "nx": 48, "ny": 32, "nz": 32, "shape": "sphere",
         "storage": "fp32", "trt": False},
        # An ordinary solve of the serving range (32^3 .. 192^3), its rows no
        # multiple of a warp: D3Q27 around a rounded box, populations near L2 size.
        {"name": "q27-box-100", "family": "dense3", "q": 27, "nx": 100, "ny": 100, "nz": 100, "shape": "roundbox",
         "storage": "fp32", "trt": False, "steps": 50},
        # The benchmark's sphere, 32-bit storage: the headline workload.
        {"name": "q19-sphere-256-fp32", "family": "dense3", "q": 19, "nx": 256, "ny": 128, "nz": 128,
         "shape": "sphere", "storage": "fp32", "trt": False, "steps": 50},
        # The same sphere in half-precision storage.
        {"name": "q19-sphere-256-fp16", "family": "dense3", "q": 19, "nx": 256, "ny": 128, "nz": 128,
         "shape": "sphere", "storage": "fp16", "trt": False, "steps": 50},
        # Odd sizes, bfloat16 storage and the two-relaxation-time collision.
        {"name": "q27-sphere-151-bf16-trt", "family": "dense3", "q": 27, "nx": 151, "ny": 110, "nz": 121,
         "shape": "sphere", "storage": "bf16", "trt": True, "steps": 50},
        # The dense 2D cylinder page at its resolution 9: a short step many times.
        {"name": "cylinder2d-512", "family": "dense2", "nx": 512, "ny": 512, "storage": "fp32", "steps": 200},
        # A free body tumbling in the flow: force pass, 6-DOF update, step.
        {"name": "free-spheroid-96", "family": "free", "q": 19, "nx": 96, "ny": 64, "nz": 64, "steps": 50},
        # A batch of vortices and channels, 64^2 .. 512^2, tuned once as the
        # benchmark tunes its own.
        {"name": "batch-64", "family": "batch", "domains": 64, "nmin": 64, "nmax": 512, "storage": "fp32",
         "steps": 200},
        # The 2D AMR cylinder of the benchmark, 16 refine rounds.
        {"name": "amr2d-cylinder-1024", "family": "amr2", "nx": 1024, "ny": 256, "r": 20.0, "steps": 256},
        # The reference's sphere hierarchy (Re 20, D = 16), 160 tiles.
        {"name": "amr3d-sphere-192", "family": "amr3", "q": 19, "nx": 192, "ny": 128, "nz": 128, "r": 8.0,
         "shape": "sphere", "steps": 32},
        # A large hierarchy: the biggest two-level request of the served
        # stream, a rounded box with thousands of tiles.
        {"name": "amr3d-box-180", "family": "amr3", "q": 19, "nx": 180, "ny": 180, "nz": 180, "r": 22.5,
         "shape": "roundbox", "steps": 16},
        # A short request stream through the server, small and middle sizes,
        # two lattices, a quarter two-level hierarchies, results read to the host.
        {"name": "serve-10", "family": "serve", "requests": 10, "nmin": 32, "nmax": 128, "steps": 200, "pick": 3},
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    fam = rng.choice(("call", "dense3", "dense3", "dense3", "dense2", "free", "batch", "amr2", "amr3", "serve"))
    if fam == "dense2":
        return {"family": fam, "nx": int(_log(rng, 96, 1100)), "ny": int(_log(rng, 96, 700)),
                "storage": rng.choice(("fp32", "fp32", "fp16", "bf16")), "steps": rng.randrange(20, 200)}
    if fam == "batch":
        return {"family": fam, "domains": rng.randrange(8, 65), "nmin": 64, "nmax": rng.randrange(128, 512),
                "storage": rng.choice(("fp32", "fp32", "fp16")), "steps": rng.randrange(40, 200)}
    if fam == "amr2":
        h = 16 * rng.randrange(10, 20)
        return {"family": fam, "nx": 16 * rng.randrange(24, 65), "ny": h, "r": round(rng.uniform(0.05, 0.09) * h, 2),
                "steps": rng.randrange(32, 256)}
    if fam == "serve":
        return {"family": fam, "requests": rng.randrange(3, 11), "nmin": 32, "nmax": rng.randrange(48, 128),
                "steps": rng.randrange(60, 200), "pick": rng.randrange(1000)}
    if fam == "amr3":
        ax = [4 * int(_log(rng, 14, 45)) for _ in range(3)]
        return {"family": fam, "q": rng.choice((19, 27)), "nx": ax[0], "ny": ax[1], "nz": ax[2],
                "r": round(rng.uniform(0.08, 0.125) * min(ax), 2), "shape": rng.choice(("sphere", "roundbox")),
                "steps": rng.randrange(2, 17)}
    if fam == "free":
        return {"family": fam, "q": rng.choice((19, 27)), "nx": int(_log(rng, 48, 160)), "ny": int(_log(rng, 40, 96)),
                "nz": int(_log(rng, 40, 96)), "steps": rng.randrange(10, 50)}
    ax = [int(_log(rng, 32, hi)) for hi in (256, 160, 128)] if fam == "dense3" else \
        [int(_log(rng, 24, 96)) for _ in range(3)]
    c = {"family": fam, "q": rng.choice((19, 27)), "nx": ax[0], "ny": ax[1], "nz": ax[2],
         "shape": rng.choice(("sphere", "roundbox", "none")), "storage": rng.choice(("fp32", "fp16", "bf16")),
         "trt": rng.random() < 0.25}
    if fam == "dense3":
        c["steps"] = min(rng.randrange(4, 50), int(4e9 / (ax[0] * ax[1] * ax[2] * c["q"])))
    return c


# ---- configurations and inputs --------------------------------------------------

def _cells(c):
    return c["nx"] * c["ny"] * c.get("nz", 1)


def _f32(v):
    return float(np.float32(v))


def _body3(c):
    """A third of the way along x, in the middle of y and z."""
    centre = (float(round(c["nx"] / 3)), c["ny"] / 2.0, c["nz"] / 2.0)
    r = _f32(c.get("r", min(c["ny"], c["nz"]) / 8.0))
    if c["shape"] == "roundbox":
        return dict(shape="roundbox", centre=centre, a=r, b=r, c=r, r=r / 4)
    return dict(shape="sphere", centre=centre, a=r)


def _config3(c):
    """Bounce-back body in a stream along x with the sponge round the domain
    and the benchmark's body force, or without a body a periodic box."""
    kw = dict(tau=_f32(0.56), force=(1e-6, 0.0, 0.0), storage=c.get("storage", "fp32"),
              sponge_u=(U0, 0.0, 0.0))
    if c.get("shape", "sphere") != "none":
        kw.update(has_body=1, use_bounceback=1, body=_body3(c), sponge_w=float(max(6, min(c["ny"], c["nz"]) // 16)))
    if c.get("trt"):
        kw.update(trt=1, trt_lambda=0.1875)
    return kw


def _config2(c):
    """main-cylinder.js: a circle of 1/24 of the height's diameter, Re 100."""
    r = c["ny"] / 48.0
    return dict(tau=_f32(0.5 + 3 * 0.04 * 2 * r / 100.0), has_body=1, use_bounceback=1, solid_eq=1, sponge_w=4.0,
                sponge_u=(0.04, 0.0, 0.0), storage=c["storage"],
                body=dict(shape="ellipse", centre=(24 * r, c["ny"] / 2.0, 0.0), a=r, b=r))


def _stream(n, u, seed, planar=False):
    """[rho, ux, uy, uz] per cell: the free stream with a 2 % perturbation."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    m = torch.empty((n, 4), device="cuda")
    m[:, 1:] = (2 * torch.rand((n, 3), generator=g, device="cuda") - 1) * (0.02 * u)
    m[:, 1] += u
    if planar:
        m[:, 3] = 0
    m[:, 0] = 1 - 1.5 * u * u
    return m


def _domains(c, seed):
    """Alternating Taylor-Green vortices and forced channels (batched_domains)."""
    r = np.random.RandomState(seed % (1 << 31))
    sizes = np.random.RandomState(12345)
    out = []
    for k in range(c["domains"]):
        n = int(round(c["nmin"] * (c["nmax"] / c["nmin"]) ** sizes.rand()))
        tau = _f32(0.55 + 0.35 * sizes.rand())
        x = (2 * math.pi / n) * np.arange(n)
        amp = 0.04 * (0.8 + 0.2 * r.rand())
        mac = np.zeros((n, n, 4), np.float32)
        mac[..., 0] = 1
        if k % 2 == 0:
            mac[..., 1] = -amp * np.cos(x)[None, :] * np.sin(x)[:, None]
            mac[..., 2] = amp * np.sin(x)[None, :] * np.cos(x)[:, None]
            kw = dict(tau=tau, sponge_w=0.0)
        else:
            mac[..., 1] = amp * np.sin(0.5 * x)[:, None]
            kw = dict(tau=tau, sponge_w=0.0, wall=(0, 1, 0),
                      force=(_f32(8 * (tau - 0.5) / 3 * 0.04 / (n * n)), 0.0, 0.0))
        out.append((n, dict(kw, storage=c["storage"]), mac.reshape(-1, 4)))
    return out


def _requests(c, seed):
    """Requests as serving_stream makes them; sizes from `pick` alone."""
    s = np.random.RandomState(c["pick"])
    out = []
    for k in range(c["requests"]):
        n = int(round(c["nmin"] * (c["nmax"] / c["nmin"]) ** s.rand()))
        amr = k % 4 == 1
        n = max(16, 4 * (n // 4)) if amr else n
        d = {"q": 19 if s.rand() < 0.5 else 27, "nx": n, "ny": n, "nz": n, "r": n / 8.0,
             "shape": "roundbox" if s.rand() < 0.5 else "sphere", "amr": amr,
             "steps": int(c["steps"] * (0.5 + 0.5 * s.rand())), "tau": _f32(0.55 + 0.15 * s.rand())}
        out.append(d)
    return out


def _log_buffer(c):
    return torch.zeros((-(-c["steps"] // EVERY), 6), dtype=torch.float64).pin_memory()


def _amr3_config(lbm, c):
    kw = dict(_config3(c), tau=c.get("tau", _f32(0.62)), force=(0.0, 0.0, 0.0))
    return lbm.amr3d_config(c["q"], (c["nx"], c["ny"], c["nz"]), refine="body", rb=4, margin=2.0, **kw)


def prepare(case, seed):
    lbm = package()
    fam = case["family"]
    st = torch.cuda.Stream()
    s = {"case": case, "stream": st}
    n = _cells(case) if "nx" in case else 0
    if fam in ("dense3", "free"):
        dims = (case["nx"], case["ny"], case["nz"])
        kw = _config3(dict(case, shape="sphere")) if fam == "free" else _config3(case)
        if fam == "free":
            r = min(dims[1:]) / 10.0
            kw.update(trt=1, trt_lambda=0.1875,
                      body=dict(shape="spheroid", centre=(dims[0] / 3.0, dims[1] / 2.0, dims[2] / 2.0), a=1.2 * r,
                                c=0.6 * r, quat=(math.cos(0.3), math.sin(0.3), 0.0, 0.0)))
        v = lbm.Solver(lbm.config_from(case["q"], dims, **kw))
        v.set_stream(st.cuda_stream)
        v.init_macro(_stream(n, U0, seed).cpu().numpy())
        if fam == "free":
            v.set_free_body(lbm.body_state(v.cfg.body, 2.0), lbm.body_opts(gravity=(0.0, 0.0, -1e-5)))
        s.update(solver=v, mac=torch.empty((dims[2], dims[1], dims[0], 4), device="cuda"), log=_log_buffer(case))
    elif fam == "dense2":
        v = lbm.Solver(lbm.config_from(9, (case["nx"], case["ny"]), **_config2(case)))
        v.init_macro(_stream(n, 0.04, seed, planar=True).cpu().numpy())
        s.update(solver=v, mac=torch.empty((n, 4)).pin_memory(), log=_log_buffer(case))
    elif fam == "call":
        cfg = lbm.config_from(case["q"], (case["nx"], case["ny"], case["nz"]), **_config3(case))
        v = lbm.Solver(cfg)
        v.init_macro(_stream(n, U0, seed).cpu().numpy())
        raw = v.read_f_raw()
        v.close()
        raw = torch.from_numpy(raw.view(np.int16) if raw.dtype == np.uint16 else raw).cuda()
        raw = raw.view({"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}[case["storage"]])
        s.update(cfg=cfg, f=raw, out=torch.empty_like(raw), mac=torch.empty((n, 4), device="cuda"),
                 force=torch.zeros(8, dtype=torch.float64, device="cuda"))
    elif fam == "batch":
        doms = _domains(case, seed)
        b = lbm.Batch([lbm.config_from(9, (d[0], d[0]), **d[1]) for d in doms])
        for k, d in enumerate(doms):
            b.init_macro(k, d[2])
        b.autotune(3)
        s["batch"] = b
    elif fam == "amr2":
        nu = 0.08 * 2 * case["r"] / 100.0
        cfg = lbm.amr2d_config(case["nx"], case["ny"], tau=_f32(0.5 + 3 * nu), use_bounceback=0, sponge_w=4.0,
                               sponge_u=(0.08, 0.0), max_slots=4 * _quads(case) + 64,
                               body=dict(shape="ellipse", centre=(case["nx"] / 4.0, case["ny"] / 2.0, 0.0),
                                         a=case["r"], b=case["r"]))
        m = _stream(n, 0.08, seed, planar=True).double()
        m[:, 0] = 1
        m[:, 1] = 0.08
        lat = _Lattice(9)
        a = lbm.Amr2D(cfg)
        a.write_root(lat.equilibrium(m[:, 0], m[:, 1:].t()).float().cpu().numpy(), m[:, 1:3].float().cpu().numpy())
        a.set_stream(st.cuda_stream)
        s["amr"] = a
    elif fam == "amr3":
        a = lbm.Amr3D(_amr3_config(lbm, case))
        a.set_stream(st.cuda_stream)
        a.init_macro(_stream(n, U0, seed).cpu().numpy())
        s.update(amr=a, mac=torch.empty((case["nz"], case["ny"], case["nx"], 4), device="cuda"))
    else:
        sv = lbm.Server(6 << 30)
        sv.set_policy("sjf", 16 << 20)
        reqs = []
        for k, r in enumerate(_requests(case, seed)):
            kw = dict(_config3(r), tau=r["tau"], force=(0.0, 0.0, 0.0))
            cfg = _amr3_config(lbm, r) if r["amr"] else lbm.config_from(r["q"], (r["nx"],) * 3, **kw)
            reqs.append((k, r, cfg, _stream(r["nx"] ** 3, U0, seed * 64 + k).cpu().numpy()))
        s.update(server=sv, requests=reqs)
    torch.cuda.synchronize()
    return s


def _advance(v, steps, log):
    """The steps of a dense session, its drag logged every EVERY of them."""
    for k in range(len(log)):
        v.step(min(EVERY, steps - k * EVERY))
        v.forces_async(log[k].data_ptr())


def _advance_amr(a, steps, chunk):
    log = []
    for k in range(0, steps, chunk):
        a.step(min(chunk, steps - k))
        log.append(a.forces())
    return np.array(log)


def run(state):
    c = state["case"]
    fam = c["family"]
    if fam == "call":
        # an engine's own loop: one step on the current stream
        lbm = package()
        lbm.step_noalloc(state["cfg"], state["f"].data_ptr(), state["out"].data_ptr(), state["mac"].data_ptr(),
                         state["force"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"f": state["out"], "mac": state["mac"], "force": state["force"]}
    if fam in ("dense3", "free"):
        v = state["solver"]
        _advance(v, c["steps"], state["log"])
        v.resample(out=state["mac"])
        out = {"mac": state["mac"], "force": state["log"]}
        if fam == "free":
            b = v.body_state().as_dict()
            out["body"] = np.concatenate([b[k] for k in ("x", "q", "v", "L")])
        v.sync()
        return out
    if fam == "dense2":
        v = state["solver"]
        _advance(v, c["steps"], state["log"])
        v.read_mac(out=state["mac"].numpy())
        return {"mac": state["mac"], "force": state["log"]}
    if fam == "batch":
        b = state["batch"]
        b.step(c["steps"])
        return {"mac": np.concatenate([b.read_mac(k) for k in range(c["domains"])])}
    if fam == "amr2":
        a = state["amr"]
        log = _advance_amr(a, c["steps"], 32)
        f, vel = a.read_root()
        return {"f": f, "vel": vel, "force": log}
    if fam == "amr3":
        a = state["amr"]
        log = _advance_amr(a, c["steps"], 8)
        a.resample(out=state["mac"])
        return {"mac": state["mac"], "force": log}
    sv, out = state["server"], {}
    for k, r, cfg, mac in state["requests"]:
        if r["amr"]:
            sv.submit_amr3d(k, cfg, r["steps"], mac)
        else:
            sv.submit(k, cfg, r["steps"], mac)
    while len(out) < len(state["requests"]):
        for d in sv.poll(64):
            _, r, cfg, _ = state["requests"][d["id"]]
            mac = sv.read(d["id"], cfg, f=False)[1]
            out[d["id"]] = {"mac": mac, "force": np.array(d["forces"])}
            sv.release(d["id"])
    return [out[k] for k in sorted(out)]


# ---- work and tolerance ---------------------------------------------------------

def _quads(c):
    """Root blocks of 16 x 16 cells that a circle with its margin covers."""
    return math.ceil(2 * (c["r"] + 8) / 16) ** 2


def _tiles(c):
    """Refined blocks (4^3 cells) within 2 cells of the body, roughly."""
    r = c["r"] + 2 + 2
    vol = (2 * r) ** 3 if c["shape"] == "roundbox" else 4.19 * r ** 3
    return vol / 64


def work(case):
    c = case
    fam = c["family"]
    q = c.get("q", 9)
    size = 4 if c.get("storage", "fp32") == "fp32" else 2
    flops = {9: 110, 19: 260, 27: 370}
    if fam == "serve":
        upd = {19: 0.0, 27: 0.0}
        cells = 0
        for r in _requests(c, 0):
            cells += r["nx"] ** 3
            upd[r["q"]] += r["steps"] * (r["nx"] ** 3 + (_tiles(r) * (2 * 512 - 64) if r["amr"] else 0))
        return {"bytes": sum(u * 8 * k for k, u in upd.items()) + 32 * cells,
                "flops": sum(u * flops[k] for k, u in upd.items())}
    if fam == "batch":
        n = sum(d[0] ** 2 for d in _domains(c, 0))
    else:
        n = _cells(c)
    upd, back = n * c.get("steps", 1), 16 * n
    if fam == "amr2":
        upd += c["steps"] * 4 * _quads(c) * 2 * 256
        back = 9 * 4 * n + 8 * n
    elif fam == "amr3":
        upd += c["steps"] * _tiles(c) * (2 * 512 - 64)
        back = 32 * n
    elif fam in ("dense3", "free"):
        back = 32 * n
    return {"bytes": float(upd * 2 * q * size + back), "flops": float(upd * flops[q])}


def tolerance(case):
    # Measured against 64 bits (the field is closer than the drag log, a
    # difference of large momentum sums): 32-bit dense sessions 1.1e-5, 16-bit
    # storage 2e-3 (half) and 1.7e-2 (bfloat16), its rounding of the deviation
    # from the far field. About four times that; the hierarchies, whose
    # transfers amplify a rounding at the seams, four times more.
    s = case.get("storage", "fp32")
    if s == "bf16":
        return {"rel": 3e-2, "max": 0.3}
    if s == "fp16":
        return {"rel": 8e-3, "max": 0.1}
    if case["family"] in ("amr2", "amr3", "serve", "free"):
        return {"rel": 2e-4, "max": 0.01}
    return {"rel": 5e-5, "max": 2e-3}


# ---- the same flows in 64 bits ----------------------------------------------------

class _Lattice:
    """D2Q9 / D3Q19 / D3Q27 in this library's direction order."""

    def __init__(self, q):
        t = package().lattice_tables(q)
        self.q = q
        self.e = np.stack([t["ex"], t["ey"], t["ez"]], 1).astype(np.int64)
        self.opp = t["opp"].astype(np.int64)
        exact = {9: {0: 4 / 9, 1: 1 / 9, 2: 1 / 36}, 19: {0: 1 / 3, 1: 1 / 18, 2: 1 / 36},
                 27: {0: 8 / 27, 1: 2 / 27, 2: 1 / 54, 3: 1 / 216}}[q]
        self.w = torch.tensor([exact[int(abs(v).sum())] for v in self.e], dtype=torch.float64, device="cuda")
        self.E = torch.from_numpy(self.e).double().cuda()

    def equilibrium(self, rho, u):
        eu = self.E @ u
        return self.w[:, None] * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * (u * u).sum(0))


def _phi(body, dims, device="cuda"):
    """The body's distance at every cell, (z, y, x), in 32 bits: which links
    it cuts is part of the input."""
    x, y, z = (torch.arange(m, dtype=torch.float32, device=device) for m in dims)
    cx, cy, cz = (np.float32(v) for v in body["centre"])
    if body["shape"] == "ellipse":
        dx, dy = x - float(cx), y - float(cy)
        dx = dx - dims[0] * torch.round(dx / dims[0])
        dy = dy - dims[1] * torch.round(dy / dims[1])
        return (torch.sqrt((dx * dx)[None, None, :] + (dy * dy)[None, :, None]) - float(np.float32(body["a"])))
    d = (z - float(cz))[:, None, None], (y - float(cy))[None, :, None], (x - float(cx))[None, None, :]
    a = float(np.float32(body["a"]))
    if body["shape"] == "sphere":
        return torch.sqrt(((d[2] * d[2]) + (d[1] * d[1])) + (d[0] * d[0])) - a
    r = float(np.float32(body["r"]))
    h = float(np.float32(a) - np.float32(r))
    qz, qy, qx = (v.abs() - h for v in d)
    m = torch.sqrt((qx.clamp(min=0) ** 2 + qy.clamp(min=0) ** 2) + qz.clamp(min=0) ** 2)
    return m + torch.maximum(qx, torch.maximum(qy, qz)).clamp(max=0) - r


def _flow64(q, dims, kw, mac, steps):
    """`steps` of stream, collide and force in 64 bits from the equilibrium of
    mac: (f, mac of the last step, force and torque of every EVERY-th and the
    last step). Streaming, walls and the resting body's bounce-back are one
    gather."""
    lat = _Lattice(q)
    nx, ny, nz = dims
    n = nx * ny * nz
    dev = "cuda"
    idx = torch.arange(n, device=dev).view(nz, ny, nx)
    body = kw.get("body")
    phi = _phi(body, dims).expand(nz, ny, nx) if body else None
    solid = phi < 0 if body else None
    src = torch.empty((q, n), dtype=torch.int64, device=dev)
    links = []
    for i in range(q):
        ex, ey, ez = (int(v) for v in lat.e[i])
        sh = (ez, ey, ex)
        s = i * n + torch.roll(idx, sh, (0, 1, 2))
        own = int(lat.opp[i]) * n + idx
        if kw.get("wall", (0, 0, 0))[1] and ey:
            s[:, 0 if ey > 0 else ny - 1, :] = own[:, 0 if ey > 0 else ny - 1, :]
        if body and i:
            cut = torch.roll(solid, sh, (0, 1, 2))
            s = torch.where(cut, own, s)
            links.append((i, (cut & ~solid).view(-1).nonzero().squeeze(1)))
        src[i] = s.view(-1)
    tau = float(np.float32(kw["tau"]))
    om = 1 / tau
    dw = 0.0
    if kw.get("trt"):
        dw = 1 / (0.5 + float(np.float32(kw["trt_lambda"])) / (tau - 0.5)) - om
    F = torch.tensor([_f32(v) for v in kw.get("force", (0, 0, 0))], dtype=torch.float64, device=dev)
    sw = kw.get("sponge_w", 4.0 if q == 9 else 0.0)
    spw = None
    uf = torch.tensor([_f32(v) for v in kw.get("sponge_u", (0, 0, 0))], dtype=torch.float64, device=dev)
    far = lat.equilibrium(torch.ones(1, dtype=torch.float64, device=dev), uf[:, None])
    if sw > 0:
        ax = [torch.arange(m, dtype=torch.float64, device=dev) for m in dims]
        d = [torch.minimum(a, m - 1 - a) for a, m in zip(ax, dims)]
        dist = torch.minimum(d[1][:, None], d[0][None, :])[None].expand(nz, ny, nx)
        if q != 9:
            dist = torch.minimum(dist, d[2][:, None, None])
        t = (1 - dist / sw).clamp(0, 1)
        spw = (t * t * (3 - 2 * t)).reshape(-1)
    ks = 1.0 if spw is None else 1 - spw
    w = lat.w[:, None]
    eF = (lat.E @ F)[:, None]
    opp = torch.from_numpy(lat.opp).to(dev)
    m0 = torch.as_tensor(mac, device=dev).double().t()
    f = lat.equilibrium(m0[0], m0[1:])
    inside = solid.reshape(-1) if body else None
    rest = lat.equilibrium(torch.ones(1, dtype=torch.float64, device=dev), torch.zeros((3, 1), dtype=torch.float64,
                                                                                       device=dev))
    log = []
    out = None
    for k in range(steps):
        last = k == steps - 1
        if last or k % EVERY == EVERY - 1:
            force = np.zeros(6)
            log.append(force)
            for i, cells in links:
                m = 2 * f[int(lat.opp[i])][cells]
                fb = -lat.E[i][:, None] * m
                z, y, x = cells // (nx * ny), (cells // nx) % ny, cells % nx
                r = torch.stack([x, y, z]).double() - torch.tensor([_f32(v) for v in body["centre"]],
                                                                   dtype=torch.float64, device=dev)[:, None]
                if q == 9:
                    for a, m_ in ((0, nx), (1, ny)):
                        r[a] -= m_ * torch.round(r[a] / m_)
                    r[2] = 0
                t = torch.linalg.cross(r, fb, dim=0)
                force += torch.cat([fb.sum(1), t.sum(1)]).cpu().numpy()
        g = f.reshape(-1)[src]
        rho = g.sum(0)
        u = (lat.E.t() @ g) / rho + F[:, None] / (2 * rho)
        usq = (u * u).sum(0)
        eu = lat.E @ u
        uF = (u * F[:, None]).sum(0)
        S = (1 - om / 2) * w * (3 * eF - 3 * uF + 9 * eu * eF)
        col = (1 - om) * g + om * w * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * usq) + S
        if dw:
            col -= dw * (0.5 * (g - g[opp]) - 3 * w * rho * eu) + 0.5 * dw * 3 * w * eF
        f = col if spw is None else ks * col + spw * far
        if body:
            f[:, inside] = rest
        if last:
            out = torch.cat([rho[None], u]).t().contiguous()
            if body and q != 9:
                out[inside] = torch.tensor([1.0, 0, 0, 0], dtype=torch.float64, device=dev)
            if q == 9:
                out[:, 3] = 0
    return f, out, np.array(log)


def exact(case, seed):
    c = case
    fam = c["family"]
    if fam == "batch":
        return {"mac": np.concatenate([_flow64(9, (n, n, 1), kw, mac, c["steps"])[1].cpu().numpy()
                                       for n, kw, mac in _domains(c, seed)])}
    if fam == "dense2":
        _, mac, force = _flow64(9, (c["nx"], c["ny"], 1), _config2(c), _stream(_cells(c), 0.04, seed, planar=True),
                                c["steps"])
        return {"mac": mac, "force": force}
    if fam not in ("call", "dense3"):
        return None  # hierarchies and free bodies: no plain restatement of this length
    dims = (c["nx"], c["ny"], c["nz"])
    f, mac, force = _flow64(c["q"], dims, _config3(c), _stream(_cells(c), U0, seed), c.get("steps", 1))
    if fam == "call":
        # 16-bit buffers hold offsets from the far field, not populations
        return {"f": f if c["storage"] == "fp32" else None, "mac": mac, "force": np.concatenate([force[0], [0.0, 0.0]])}
    # the volume's voxels are (ux, uy, uz, rho)
    return {"mac": torch.roll(mac, -1, 1).view(c["nz"], c["ny"], c["nx"], 4), "force": force}
