"""The performance cases: what a program using this library has it do, with sizes.

Kinds of case (the key "kind"):

* "box"        the device-resident solver of one periodic box: set the fields,
               advance nstep SSP-RK3 steps, read the state (sdg_solver_*);
* "run"        the same with the min/max output of the reference's time loop;
* "loop"       the time loop on the reference's own device arrays in one call
               (sdg_advect3d_eq_step_dev);
* "stages"     one step through the per-stage device entry points, as the
               reference's driver calls them (update_halo, cal_tend, RK stage);
* "tend_host"  advect3d_eq_cal_tend on host arrays, the Fortran drop-in call;
* "operators"  the batched element operators divlike, gradlike and Lift;
* "ensemble"   many boxes of different sizes and orders advanced together;
* "server"     a burst of solve requests served by continuous batching.

Fields follow the workloads of the benchmark: a Gaussian tracer in a smooth
velocity of four Fourier modes (the solvers), in a constant velocity (ensemble
and server), or the reference's sine initial condition in a constant velocity.
Operators are the reference's operator_data/p*.dat.
"""
import math
import os
import random
import sys

import numpy as np
import torch

U0 = (1.0, 0.5, 0.25)
CFL = 0.1
PREC = {"fp64": 0, "fp32": 1, "emu": 2}
OPT = {"general": 1, "opt1": 2, "evenodd": 3}

# The largest work a drawn case may have, in DOF-updates through one RK stage
# at FP64 speed, so that it costs no more than the largest listed case.
MAX_UPDATES = {"box": 2.2e8, "run": 1.5e8, "loop": 1.5e8, "stages": 5.0e7}


def listed():
    return [
        # the reference's own configuration (8^3 elements, p = 3, sine field,
        # 100 steps), in the default order: latency and launches
        {"name": "box_p3_fp64_opt1_small", "kind": "box", "nx": 8, "ny": 8, "nz": 8, "p": 3,
         "opt": "opt1", "prec": "fp64", "nstep": 100, "ic": "sine"},
        # the benchmark's headline box: 16.8M DOF, FP64, even-odd stage
        {"name": "box_p7_fp64_evenodd_large", "kind": "box", "nx": 32, "ny": 32, "nz": 32, "p": 7,
         "opt": "evenodd", "prec": "fp64", "nstep": 5, "ic": "blob"},
        # a plain FP64 solve in the default order at a high order, odd sizes
        {"name": "box_p10_fp64_opt1", "kind": "box", "nx": 17, "ny": 13, "nz": 19, "p": 10,
         "opt": "opt1", "prec": "fp64", "nstep": 4, "ic": "blob"},
        # the FP32-compute form of the order sweep, about 16.8M DOF
        {"name": "box_p5_fp32_large", "kind": "box", "nx": 43, "ny": 41, "nz": 44, "p": 5,
         "opt": "evenodd", "prec": "fp32", "nstep": 10, "ic": "blob"},
        # the emulated-FP64 form on an ordinary box
        {"name": "box_p6_emu", "kind": "box", "nx": 21, "ny": 23, "nz": 19, "p": 6,
         "opt": "evenodd", "prec": "emu", "nstep": 6, "ic": "blob"},
        # a low-order run that prints min/max every few steps
        {"name": "run_p2_fp64_minmax", "kind": "run", "nx": 29, "ny": 31, "nz": 27, "p": 2,
         "opt": "evenodd", "prec": "fp64", "nstep": 20, "ic": "blob", "interval": 5},
        # the reference's loop on the caller's arrays, one call
        {"name": "loop_p7_evenodd", "kind": "loop", "nx": 24, "ny": 24, "nz": 24, "p": 7,
         "opt": "evenodd", "nstep": 4},
        # the reference's loop as its driver writes it, per-stage calls
        {"name": "stages_p4_opt1", "kind": "stages", "nx": 25, "ny": 23, "nz": 27, "p": 4,
         "opt": "opt1", "nstep": 1},
        # one tendency on host arrays, as a Fortran caller makes it
        {"name": "tend_host_p3", "kind": "tend_host", "nx": 12, "ny": 10, "nz": 9, "p": 3,
         "opt": "opt1"},
        # the element operators on a batch of elements
        {"name": "operators_p8_opt1", "kind": "operators", "p": 8, "nelem": 6001, "opt": "opt1"},
        # an ensemble of uneven boxes, FP32 compute, orders 3, 5, 7
        {"name": "ensemble_12", "kind": "ensemble", "n": 12, "ne_min": 4, "ne_max": 24,
         "p_set": "3,5,7", "nstep": 100, "pick": 1},
        # a burst of served solves of different orders, sizes and lengths
        {"name": "server_burst_16", "kind": "server", "n": 16, "ne_min": 4, "ne_max": 20,
         "p_min": 2, "p_max": 11, "nstep_min": 10, "nstep_max": 120, "pick": 1},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw_box(rng, p, lo, hi):
    """Element counts of a box of about lo..hi DOF with uneven axes."""
    side = (_log_uniform(rng, lo, hi) / (p + 1) ** 3) ** (1.0 / 3.0)
    return [max(1, int(round(side * rng.uniform(0.7, 1.35)))) for _ in range(3)]


def draw(rng):
    kind = rng.choices(["box", "run", "loop", "stages", "tend_host", "operators", "ensemble",
                        "server"], [8, 1, 2, 2, 1, 2, 1, 1])[0]
    if kind in ("box", "run", "loop", "stages"):
        p = rng.randint(1, 15)
        nx, ny, nz = _draw_box(rng, p, 3e4, 1.2e7)
        dof = (p + 1) ** 3 * nx * ny * nz
        most = max(1, int(MAX_UPDATES[kind] / (3 * dof)))
        c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "p": p,
             "nstep": 1 if kind == "stages" else min(most, int(_log_uniform(rng, 1, 100)))}
        if kind == "box":
            c["prec"], c["opt"] = rng.choice([("fp64", "evenodd"), ("fp64", "opt1"),
                                              ("fp64", "general"), ("fp32", "evenodd"),
                                              ("emu", "evenodd")])
            c["ic"] = rng.choice(["blob", "blob", "sine"])
        elif kind == "run":
            c["prec"], c["opt"], c["ic"] = "fp64", rng.choice(["evenodd", "opt1"]), "blob"
            c["interval"] = rng.randint(1, 10)
        else:
            c["opt"] = rng.choice(["evenodd", "opt1"])
        return c
    if kind == "tend_host":
        p = rng.randint(1, 15)
        nx, ny, nz = _draw_box(rng, p, 4e3, 4e5)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "p": p,
                "opt": rng.choice(["evenodd", "opt1"])}
    if kind == "operators":
        p = rng.randint(1, 15)
        nelem = max(1, int(_log_uniform(rng, 4e3, 1e7) / (p + 1) ** 3))
        return {"kind": kind, "p": p, "nelem": nelem, "opt": rng.choice(["opt1", "general"])}
    if kind == "ensemble":
        return {"kind": kind, "n": rng.randint(2, 12), "ne_min": rng.randint(2, 6),
                "ne_max": rng.randint(7, 20), "p_set": rng.choice(["3,5,7", "1,2,4", "6,8,9,10,11"]),
                "nstep": rng.randint(10, 100), "pick": rng.randint(1, 10 ** 6)}
    return {"kind": kind, "n": rng.randint(1, 16), "ne_min": rng.randint(2, 6),
            "ne_max": rng.randint(7, 18), "p_min": 2, "p_max": 11, "nstep_min": 10,
            "nstep_max": rng.randint(20, 100), "pick": rng.randint(1, 10 ** 6)}


# ---- inputs --------------------------------------------------------------------


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _operators(p):
    """(x1D, D1D, D1D_tr, Lift_mat) of operator_data/p<p>.dat, flat and column-major."""
    path = os.path.join(os.getcwd(), "tests", "golden", "operator_data.npz")
    with np.load(path) as z:
        return tuple(np.ascontiguousarray(z["%s_p%d" % (k, p)], dtype=np.float64)
                     for k in ("x1D", "D1D", "D1D_tr", "Lift"))


def _nodes(c, x1D):
    """Node coordinates broadcastable to (ez, ey, ex, k, j, i) on the unit box."""
    dev = _device()
    x1 = torch.from_numpy(x1D).to(dev)

    def axis(n, shape_e, shape_n):
        d = 1.0 / n
        e = (torch.arange(n, dtype=torch.float64, device=dev) + 0.5) * d
        return e.reshape(shape_e) + (0.5 * d * x1).reshape(shape_n)

    N = len(x1D)
    return (axis(c["nx"], (1, 1, -1, 1, 1, 1), (1, 1, 1, 1, 1, N)),
            axis(c["ny"], (1, -1, 1, 1, 1, 1), (1, 1, 1, 1, N, 1)),
            axis(c["nz"], (-1, 1, 1, 1, 1, 1), (1, 1, 1, N, 1, 1)))


def _shape(c):
    N = c["p"] + 1
    return (c["nz"], c["ny"], c["nx"], N, N, N)


def _gauss(X, Y, Z, centre, sigma):
    d2 = 0.0
    for x, m in zip((X, Y, Z), centre):
        d = x - m
        d = d - torch.round(d)
        d2 = d2 + d * d
    return torch.exp(-d2 / (2.0 * sigma * sigma))


def _fields(c, seed):
    """q, u, v, w as (ez, ey, ex, k, j, i) tensors, and the time step at CFL 0.1."""
    r = random.Random(int(seed) * 7919 + 17)
    X, Y, Z = _nodes(c, _operators(c["p"])[0])
    shape, dev = _shape(c), _device()
    tau = 2.0 * math.pi
    if c.get("ic") == "sine":
        q = torch.ones(shape, dtype=torch.float64, device=dev)
        for x in (X, Y, Z):
            q = q * torch.sin(tau * x + r.uniform(0.0, tau))
        vel = [torch.full(shape, s, dtype=torch.float64, device=dev) for s in U0]
        vmax = sum(U0)
    else:
        q = _gauss(X, Y, Z, [r.random() for _ in range(3)], 0.1).expand(shape).contiguous()
        vel = [torch.full(shape, s, dtype=torch.float64, device=dev) for s in U0]
        for _ in range(4):
            k = (0, 0, 0)
            while not 1 <= sum(m * m for m in k) <= 9:
                k = [r.randint(-3, 3) for _ in range(3)]
            a = [r.gauss(0.0, 1.0) for _ in range(3)]
            norm = math.sqrt(sum(t * t for t in a))
            s = torch.sin(tau * (k[0] * X + k[1] * Y + k[2] * Z) + r.uniform(0.0, tau))
            for t, f in zip(a, vel):
                f += (0.2 * t / norm) * s
        vmax = float((vel[0].abs() + vel[1].abs() + vel[2].abs()).max())
    h = 1.0 / max(c["nx"], c["ny"], c["nz"])
    return (q, *vel), CFL * h / ((2 * c["p"] + 1) * vmax)


def _members(c, seed):
    """Boxes of an ensemble or a server burst: the shapes from the case, the
    tracer and the velocity from the seed."""
    shapes, r = random.Random(c["pick"]), random.Random(int(seed) * 104729 + 5)
    out = []
    for _ in range(c["n"]):
        ne = [shapes.randint(c["ne_min"], c["ne_max"]) for _ in range(3)]
        if c["kind"] == "ensemble":
            p, nstep = int(shapes.choice(c["p_set"].split(","))), c["nstep"]
        else:
            p = shapes.randint(c["p_min"], c["p_max"])
            nstep = shapes.randint(c["nstep_min"], c["nstep_max"])
        vel = [r.uniform(-1.0, 1.0) for _ in range(3)]
        speed = sum(abs(t) for t in vel)
        vel = [t / max(1.0, speed) for t in vel]
        dt = CFL / (max(ne) * (2 * p + 1) * max(0.1, sum(abs(t) for t in vel)))
        out.append({"nx": ne[0], "ny": ne[1], "nz": ne[2], "p": p, "nstep": nstep, "dt": dt,
                    "centre": [r.random() for _ in range(3)], "sigma": r.uniform(0.05, 0.2),
                    "vel": vel})
    return out


# ---- the library ---------------------------------------------------------------


def _sdg():
    path = os.path.join(os.getcwd(), "scale-dg-kernel-extraction_gb300")
    if path not in sys.path:
        sys.path.insert(0, path)
    import sdg
    return sdg


class _Gpu:
    """A device buffer of the library, for torch.as_tensor; the tensor holds
    this object, and with it the buffer's owner."""

    def __init__(self, ptr, n, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False),
                                         "version": 2}


def _mesh(sdg, c):
    """The reference's mesh arrays (mesh_setup) on the device."""
    N, ne = c["p"] + 1, c["nx"] * c["ny"] * c["nz"]
    nft, nhalo = 6 * N * N, 2 * (c["nx"] * c["ny"] + c["ny"] * c["nz"] + c["nz"] * c["nx"])

    def new(n, t=torch.float64):
        return torch.empty(n, dtype=t, device="cuda")

    m = {"Nq": N, "Np": N ** 3, "NfpTot": nft, "Ne": ne, "NeA": ne + nhalo,
         "NhaloNode": N * N * nhalo, "vm": new(nft * ne, torch.int32),
         "vp": new(nft * ne, torch.int32), "normal": new(3 * nft * ne), "es": new(3 * N ** 3 * ne),
         "fs": new(nft * ne), "halo": new(N * N * nhalo, torch.int32)}
    sdg._check(sdg.lib.sdg_mesh_setup_dev(
        c["nx"], c["ny"], c["nz"], c["p"], 1.0, 1.0, 1.0, None, m["vm"].data_ptr(),
        m["vp"].data_ptr(), m["normal"].data_ptr(), m["es"].data_ptr(), m["fs"].data_ptr(), None,
        m["halo"].data_ptr(), None), "sdg_mesh_setup_dev")
    return m


def _with_halo(m, f):
    """The field with its halo slots filled, (Np, NeA) flat."""
    f = f.reshape(-1)
    out = torch.zeros(m["Np"] * m["NeA"], dtype=f.dtype, device=f.device)
    out[: f.numel()] = f
    out[f.numel(): f.numel() + m["NhaloNode"]] = f[m["halo"].long() - 1]
    return out


def prepare(case, seed):
    c, kind = case, case["kind"]
    sdg = _sdg()
    if kind in ("box", "run"):
        f, dt = _fields(c, seed)
        D, L = _operators(c["p"])[1::2]
        s = sdg.Solver(c["nx"], c["ny"], c["nz"], c["p"], D, L, opt=OPT[c["opt"]],
                       precision=PREC[c["prec"]])
        return {"case": c, "sdg": sdg, "s": s, "f": [x.reshape(-1) for x in f], "dt": dt}
    if kind in ("loop", "stages", "tend_host"):
        f, dt = _fields(c, seed)
        m = _mesh(sdg, c)
        f = [_with_halo(m, x) for x in f]
        x1, D, Dt, L = _operators(c["p"])
        if kind == "tend_host":
            host = {k: m[k].cpu().numpy() for k in ("vm", "vp", "normal", "es", "fs")}
            return {"case": c, "sdg": sdg, "m": m, "h": host, "D": D, "Dt": Dt, "L": L,
                    "f": [x.cpu().numpy() for x in f], "dqdt": np.zeros(m["Np"] * m["NeA"])}
        ops = [torch.from_numpy(a).cuda() for a in (D, Dt, L)]
        st = {"case": c, "sdg": sdg, "m": m, "f": f, "dt": dt, "ops": ops, "q": f[0].clone(),
              "err": torch.zeros(1, dtype=torch.int32, device="cuda")}
        if kind == "loop":
            n = int(sdg.lib.sdg_advect3d_eq_step_scratch_bytes(m["Nq"], m["Ne"]))
            st["scratch"] = torch.empty(n, dtype=torch.uint8, device="cuda")
        else:
            st["dqdt"] = torch.zeros(m["Np"] * m["NeA"], dtype=torch.float64, device="cuda")
            st["q0"] = torch.empty(m["Np"] * m["Ne"], dtype=torch.float64, device="cuda")
            st["flux"] = torch.empty(m["NfpTot"] * m["Ne"], dtype=torch.float64, device="cuda")
        return st
    if kind == "operators":
        vec, face = _operator_inputs(c, seed)
        x1, D, Dt, L = _operators(c["p"])
        ops = [torch.from_numpy(a).cuda() for a in (D, Dt, L)]
        out = [torch.empty_like(vec[0]) for _ in range(7)]
        return {"case": c, "sdg": sdg, "vec": vec, "face": face, "ops": ops, "out": out}
    mem = _members(c, seed)
    table = {p: _operators(p) for p in sorted({m["p"] for m in mem})}
    if kind == "ensemble":
        e = sdg.Ensemble([(m["nx"], m["ny"], m["nz"]) for m in mem], [m["p"] for m in mem],
                         [m["dt"] for m in mem], table)
        return {"case": c, "sdg": sdg, "e": e, "mem": mem}
    return {"case": c, "sdg": sdg, "mem": mem,
            "server": sdg.Server(table, hbm_budget_bytes=16 << 30, max_active=64)}


def run(state):
    c, sdg = state["case"], state["sdg"]
    kind, lib = c["kind"], sdg.lib
    if kind in ("box", "run"):
        s = state["s"]
        sdg._check(lib.sdg_solver_upload_dev(s.handle, *[x.data_ptr() for x in state["f"]]),
                   "sdg_solver_upload_dev")
        rec = None
        if kind == "run":
            rec = s.run(state["dt"], c["nstep"], c["interval"])
        else:
            s.step(state["dt"], c["nstep"])
        q = torch.as_tensor(_Gpu(lib.sdg_solver_state_dev(s.handle), s.ndof, s), device="cuda")
        return (q, rec) if rec is not None and rec.size else q
    if kind == "loop":
        m, (q0, u, v, w) = state["m"], state["f"]
        q = state["q"]
        q.copy_(q0)
        sdg._check(lib.sdg_advect3d_eq_step_dev(
            q.data_ptr(), u.data_ptr(), v.data_ptr(), w.data_ptr(),
            *[a.data_ptr() for a in state["ops"]], m["vm"].data_ptr(), m["vp"].data_ptr(),
            m["normal"].data_ptr(), m["es"].data_ptr(), m["fs"].data_ptr(), m["halo"].data_ptr(),
            m["Nq"], m["Np"], m["NfpTot"], m["Ne"], m["NeA"], m["NhaloNode"], state["dt"],
            c["nstep"], OPT[c["opt"]], state["scratch"].data_ptr(), state["scratch"].numel(),
            state["err"].data_ptr(), None), "sdg_advect3d_eq_step_dev")
        return q, state["err"]
    if kind == "stages":
        m, (qi, u, v, w) = state["m"], state["f"]
        q, q0, dq = state["q"], state["q0"], state["dqdt"]
        q.copy_(qi)
        nown = m["Np"] * m["Ne"]
        for _ in range(c["nstep"]):
            sdg._check(lib.sdg_memcpy_d2d_async(q0.data_ptr(), q.data_ptr(), 8 * nown, None),
                       "sdg_memcpy_d2d_async")
            for stage in (1, 2, 3):
                sdg._check(lib.sdg_update_halo_dev(q.data_ptr(), m["halo"].data_ptr(), m["Np"],
                                                   m["Ne"], m["NhaloNode"], None),
                           "sdg_update_halo_dev")
                sdg._check(lib.sdg_advect3d_eq_cal_tend_dev(
                    dq.data_ptr(), q.data_ptr(), u.data_ptr(), v.data_ptr(), w.data_ptr(),
                    *[a.data_ptr() for a in state["ops"]], m["vm"].data_ptr(), m["vp"].data_ptr(),
                    m["normal"].data_ptr(), m["es"].data_ptr(), m["fs"].data_ptr(), m["Nq"],
                    m["Np"], m["NfpTot"], m["Ne"], m["NeA"], OPT[c["opt"]],
                    state["flux"].data_ptr(), state["err"].data_ptr(), None),
                    "sdg_advect3d_eq_cal_tend_dev")
                sdg._check(lib.sdg_rk_stage_dev(q.data_ptr(), q0.data_ptr(), dq.data_ptr(),
                                                m["Np"], m["Ne"], stage, state["dt"], None),
                           "sdg_rk_stage_dev")
        return q[:nown], dq[:nown], state["err"]
    if kind == "tend_host":
        m, h = state["m"], state["h"]
        sdg.dg_optr_kernel_setup(c["opt"].upper())
        sdg.advect3d_eq_cal_tend(state["dqdt"], *state["f"], state["D"], state["Dt"], state["L"],
                                 h["vm"], h["vp"], h["normal"], h["es"], h["fs"], m["Nq"], m["Np"],
                                 m["NfpTot"], m["Ne"], m["NeA"])
        return state["dqdt"][: m["Np"] * m["Ne"]]
    if kind == "operators":
        D, Dt, L = [a.data_ptr() for a in state["ops"]]
        x, y, z = [a.data_ptr() for a in state["vec"]]
        o = [a.data_ptr() for a in state["out"]]
        N, n = c["p"] + 1, c["nelem"]
        sdg._check(lib.sdg_tensorprod_divlike_dirXYZ_dev(o[0], o[1], o[2], D, Dt, x, y, z, N, n,
                                                         OPT[c["opt"]], None), "divlike")
        sdg._check(lib.sdg_tensorprod_gradlike_dirXYZ_dev(o[3], o[4], o[5], D, Dt, x, N, n, None),
                   "gradlike")
        sdg._check(lib.sdg_tensorprod_Lift_hexahedral_dev(o[6], L, state["face"].data_ptr(), N, n,
                                                          None), "Lift")
        return state["out"]
    if kind == "ensemble":
        e = state["e"]
        for i, m in enumerate(state["mem"]):
            e.init_blob(i, m["centre"], m["sigma"], m["vel"])
        e.step(c["nstep"])
        return [e.download(i) for i in range(c["n"])]
    srv = state["server"]
    tickets = [srv.submit(m["nx"], m["ny"], m["nz"], m["p"], m["nstep"], m["dt"], m["centre"],
                          m["sigma"], m["vel"], want_state=True) for m in state["mem"]]
    got = [srv.wait(t, 60.0) for t in tickets]
    for r, _ in got:
        if r["status"] != 0:
            raise RuntimeError("a served request ended with status %d" % r["status"])
    return [q for _, q in got]


def _operator_inputs(c, seed):
    """Three smooth-plus-noise vector components and the six faces' values."""
    g = torch.Generator(device="cpu").manual_seed(int(seed) * 31 + 7)
    N, n = c["p"] + 1, c["nelem"]
    amp = torch.rand(4, generator=g).tolist()
    t = torch.arange(n * N ** 3, dtype=torch.float64, device=_device())
    vec = [torch.sin(t * (0.37 + 0.11 * k) + 6.0 * amp[k]) + 0.5 * amp[3] for k in range(3)]
    s = torch.arange(n * 6 * N * N, dtype=torch.float64, device=_device())
    return vec, torch.cos(s * 0.29 + 6.0 * amp[3])


# ---- work -----------------------------------------------------------------------


def work(case):
    c, kind = case, case["kind"]

    def updates(dof, p, nstep, vel_bytes):
        # a DOF through one RK stage: q, u, v, w in and q out, q0 in the second
        # and third stage; flux, divergence, lift and RK update
        n = 3.0 * nstep * dof
        return n * (8 + 3 * vel_bytes + 8 + 16.0 / 3), n * (25 + 6 * (p + 1) + 126.0 / (p + 1))

    if kind in ("ensemble", "server"):
        b = f = 0.0
        for m in _members(c, 1):
            x, y = updates((m["p"] + 1) ** 3 * m["nx"] * m["ny"] * m["nz"], m["p"], m["nstep"], 4)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    p, N = c["p"], c["p"] + 1
    if kind == "operators":
        n = float(c["nelem"])
        return {"bytes": 8 * n * (10 * N ** 3 + 6 * N * N),
                "flops": n * N ** 3 * (12 * N + 12)}
    dof = float(N ** 3 * c["nx"] * c["ny"] * c["nz"])
    face = 6.0 * dof / N
    if kind in ("box", "run"):
        b, f = updates(dof, p, c["nstep"], 4 if c["prec"] == "fp32" else 8)
    elif kind == "loop":
        b, f = updates(dof, p, c["nstep"], 8)
        b += 24 * dof + 40 * face
    else:
        # a tendency call: q, u, v, w, Escale in, dqdt out; VMapM, VMapP,
        # normals and Fscale of the face nodes
        calls = 1 if kind == "tend_host" else 3 * c["nstep"]
        b = calls * ((32 + 24 + 8) * dof + 40 * face)
        f = calls * dof * (25 + 6 * N + 126.0 / N)
        if kind == "stages":
            b += calls * (24 + 16.0 / 3) * dof
    return {"bytes": b, "flops": f}


# ---- exact results --------------------------------------------------------------


class _Exact:
    """The tendency and the SSP-RK3 step on a periodic box in plain torch, 64 bits."""

    def __init__(self, c):
        self.N = c["p"] + 1
        dev = _device()
        _, D, _, L = _operators(c["p"])
        self.D = torch.from_numpy(D.reshape(self.N, self.N).T.copy()).to(dev)
        self.L = torch.from_numpy(L.reshape((6,) + (self.N,) * 3)).to(dev)
        self.S = [2.0 * c["nx"], 2.0 * c["ny"], 2.0 * c["nz"]]

    def flux(self, q, vel, axis, side):
        """Upwind flux of the faces of one axis (0 x, 1 y, 2 z) and side (+1, -1)."""
        node, elem = 5 - axis, 2 - axis
        last = self.N - 1
        own, other = (last, 0) if side > 0 else (0, last)
        qm, um = q.select(node, own), vel.select(node, own) * side
        qp = q.select(node, other).roll(-side, elem)
        up = vel.select(node, other).roll(-side, elem) * side
        alpha = 0.5 * (up + um).abs()
        return (0.5 * self.S[axis]) * ((qp * up - qm * um) - alpha * (qp - qm))

    def tendency(self, q, u, v, w):
        N = self.N
        out = self.S[0] * torch.matmul(q * u, self.D.T)
        out += self.S[1] * torch.matmul(self.D, q * v)
        fz = (q * w).reshape(q.shape[:3] + (N, N * N))
        out += self.S[2] * torch.matmul(self.D, fz).reshape(q.shape)
        # faces -y, +x, +y, -x, -z, +z
        for f, (axis, side) in enumerate(((1, -1), (0, 1), (1, 1), (0, -1), (2, -1), (2, 1))):
            g = self.flux(q, (u, v, w)[axis], axis, side)
            out += self.L[f] * g.unsqueeze(5 - axis)
        return -out

    def advance(self, f, dt, nstep, interval=0):
        q, u, v, w = f
        rec = []
        for it in range(nstep):
            q0 = q
            for a, b in ((0.0, 1.0), (0.75, 0.25), (1.0 / 3.0, 2.0 / 3.0)):
                self.dqdt = self.tendency(q, u, v, w)
                q = a * q0 + b * (q + dt * self.dqdt)
            if interval and (it + 1) % interval == 0:
                rec.append([float(q.min()), float(q.max())])
        return q, rec


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "operators":
        if c["nelem"] * (c["p"] + 1) ** 3 > 2e7:
            return None
        N, (vec, face) = c["p"] + 1, _operator_inputs(c, seed)
        _, D, _, L = _operators(c["p"])
        D = torch.from_numpy(D.reshape(N, N).T.copy()).to(_device())
        L = torch.from_numpy(L.reshape(6, N, N, N)).to(_device())
        x, y, z = [a.reshape(-1, N, N, N) for a in vec]

        def along(a, axis):
            if axis == 0:
                return torch.matmul(a, D.T).reshape(-1)
            if axis == 1:
                return torch.matmul(D, a).reshape(-1)
            return torch.matmul(D, a.reshape(-1, N, N * N)).reshape(-1)

        lift = 0.0
        g = face.reshape(-1, 6, N, N)
        for f, node in enumerate((2, 3, 2, 3, 1, 1)):
            lift = lift + L[f] * g[:, f].unsqueeze(node)
        return [along(x, 0), along(y, 1), along(z, 2), along(x, 0), along(x, 1), along(x, 2),
                lift.reshape(-1)]
    if kind in ("ensemble", "server"):
        if sum(m["nstep"] for m in _members(c, seed)) > 3000:
            return None
        out = []
        for m in _members(c, seed):
            X, Y, Z = _nodes(m, _operators(m["p"])[0])
            q = _gauss(X, Y, Z, m["centre"], m["sigma"]).expand(_shape(m)).contiguous()
            vel = [torch.full_like(q, t) for t in m["vel"]]
            out.append(_Exact(m).advance((q, *vel), m["dt"], m["nstep"])[0].reshape(-1))
        return out
    f, dt = _fields(c, seed)
    x = _Exact(c)
    if kind == "tend_host":
        return x.tendency(*f).reshape(-1)
    q, rec = x.advance(f, dt, c["nstep"], c.get("interval", 0))
    if kind == "box":
        return q.reshape(-1)
    if kind == "run":
        return (q.reshape(-1), np.array(rec).reshape(-1, 2)) if rec else q.reshape(-1)
    if kind == "stages":
        return q.reshape(-1), x.dqdt.reshape(-1), None
    nx, ny, nz, N = c["nx"], c["ny"], c["nz"], c["p"] + 1
    flat = q.reshape(-1)
    halo = flat[_halo_sources(nx, ny, nz, N)]
    out = flat.new_zeros(N ** 3 * (nx * ny * nz + 2 * (nx * ny + ny * nz + nz * nx)))
    out[: flat.numel()] = flat
    out[flat.numel(): flat.numel() + halo.numel()] = halo
    return out, None


def _halo_sources(nx, ny, nz, N):
    """The owned node each halo slot copies, in mesh_setup's order: elements in
    turn, their faces -y, +x, +y, -x, -z, +z that lie on the box's boundary."""
    e = np.arange(nx * ny * nz)
    ex, ey, ez = e % nx, (e // nx) % ny, e // (nx * ny)
    a, b = np.meshgrid(np.arange(N), np.arange(N))  # first tangential index fastest
    a, b = a.reshape(-1), b.reshape(-1)
    last = N - 1
    faces = [(ey == 0, ex, ey * 0 + ny - 1, ez, a + last * N + b * N * N),
             (ex == nx - 1, ex * 0, ey, ez, a * N + b * N * N),
             (ey == ny - 1, ex, ey * 0, ez, a + b * N * N),
             (ex == 0, ex * 0 + nx - 1, ey, ez, last + a * N + b * N * N),
             (ez == 0, ex, ey, ez * 0 + nz - 1, a + b * N + last * N * N),
             (ez == nz - 1, ex, ey, ez * 0, a + b * N)]
    keep = np.stack([f[0] for f in faces], 1)
    src = np.stack([(f[1] + nx * (f[2] + ny * f[3]))[:, None] * N ** 3 + f[4][None, :]
                    for f in faces], 1)
    return torch.from_numpy(src[keep].reshape(-1).astype(np.int64)).to(_device())
