"""What the framework is timed on: stretches of a simulation as its users run them.

A lattice is created and initialised once; a pass then advances it by the steps
between two outputs and takes the output (rho and u on the host, with lift and
drag on the way where an obstacle is watched).  The simulation goes on from
pass to pass.  The cases cover the single-lattice path in its three storage
forms and both collision operators on the geometries of the framework's own
workloads (lid-driven cavity, cylinder and disc channels, porous media,
partially saturated obstacles), from calls of a few steps on lattices that fit
one SM to 4096 x 4096, and the batch of uneven lattices, whose engine is also
what the solve server runs.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "latticeboltzmannmethod-fonnesu-grassi-guffanti_b200", "python"))
import llalbm_cuda as L  # noqa: E402
import llb_workloads as W  # noqa: E402

STORAGE = {"f64": L.STORE_F64, "f32": L.STORE_F32S, "f16": L.STORE_F16S}
BYTES = {"f64": 8, "f32": 4, "f16": 2}
BATCH_SIZES = np.arange(64, 513, 32)  # columns of a batch's lattices


def listed():
    return [
        # the smallest call: a few steps of a small cavity, then a look at the fields
        dict(name="cavity48x64_f64_10", kind="cavity", rows=48, cols=64, storage="f64", coll="bgk", steps=10),
        # the reference's own test lattice (129 x 129) between two saves
        dict(name="cavity129_f64", kind="cavity", rows=129, cols=129, storage="f64", coll="bgk", steps=1000),
        # small parameter studies in the compact form, ragged channel with discs and an open outlet
        dict(name="channel181x333_f32", kind="channel", rows=181, cols=333, storage="f32", coll="trt", steps=1000),
        # the cylinder street: drag and lift every 100 steps, fields at the end
        dict(name="cylinder256x1024_f64", kind="cylinder", rows=256, cols=1024, storage="f64", coll="trt", steps=1000),
        # partially saturated obstacles in a mid-size channel
        dict(name="partial300x500_f64", kind="partial", rows=300, cols=500, storage="f64", coll="bgk", steps=200),
        # mid-size cavity, FP64
        dict(name="cavity1000_f64", kind="cavity", rows=1000, cols=1000, storage="f64", coll="trt", steps=500),
        # a large ragged channel with discs, FP32
        dict(name="channel1001x3005_f32", kind="channel", rows=1001, cols=3005, storage="f32", coll="bgk", steps=500),
        # a large cavity in FP16 storage
        dict(name="cavity2048_f16", kind="cavity", rows=2048, cols=2048, storage="f16", coll="bgk", steps=500),
        # the largest open flow, FP64 (the default form)
        dict(name="cavity4096_f64", kind="cavity", rows=4096, cols=4096, storage="f64", coll="bgk", steps=1000),
        # porous media: the framework's headline lattice in its default form ...
        dict(name="porous4096_f64", kind="porous", rows=4096, cols=4096, storage="f64", coll="bgk", steps=1000),
        # ... and a mid-size one in FP32
        dict(name="porous1500x2000_f32", kind="porous", rows=1500, cols=2000, storage="f32", coll="trt", steps=500),
        # many uneven lattices advanced together
        dict(name="batch24_f32", kind="batch", rows=24, cols=512, storage="f32", coll="mixed", steps=400),
    ]


def draw(rng):
    """One more case: size log-uniform (odd sizes among them), any form and operator."""
    kind = rng.choice(["cavity", "cavity", "cylinder", "channel", "channel", "porous", "porous", "partial", "batch"])
    if kind == "batch":
        return dict(kind=kind, rows=rng.randint(8, 28), cols=int(rng.choice([256, 384, 512])),
                    storage=rng.choice(["f32", "f32", "f64"]), coll="mixed", steps=rng.randint(50, 400))
    lo, hi = {"cavity": (32, 4000), "cylinder": (64, 800), "channel": (48, 2400), "porous": (128, 3600),
              "partial": (64, 1000)}[kind]
    rows = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    aspect = {"cavity": rng.uniform(0.8, 1.0), "porous": rng.uniform(0.7, 1.15),
              "cylinder": rng.uniform(2.0, 4.5)}.get(kind, rng.uniform(1.0, 3.0))
    cols = max(32, int(round(rows * aspect)))
    storage = "f64" if kind == "partial" else rng.choice(["f64", "f64", "f32", "f32", "f16"])
    steps = int(round(math.exp(rng.uniform(math.log(10), math.log(1000)))))
    return dict(kind=kind, rows=rows, cols=cols, storage=storage, coll=rng.choice(["bgk", "trt"]), steps=steps)


# ---- inputs ---------------------------------------------------------------------
def _porous(R, C, rng):
    """Channel filled with discs of radius 3..12 on a jittered grid of 26 x 26
    cells, 30 % solid (llb_workloads.porous_types places the same discs by
    rejection, which takes seconds at 4096^2)."""
    t = W.channel_types(R, C)
    cell = 26
    ni, nj = (R - 8) // cell, (C - 8) // cell
    ci, cj = np.meshgrid(4 + cell * np.arange(ni), 4 + cell * np.arange(nj), indexing="ij")
    ci, cj = ci.ravel(), cj.ravel()
    r = rng.integers(3, 13, size=ci.size)
    room = cell - 1 - 2 * r - 1  # one node clear of the next cell's disc
    ci = ci + r + np.floor(rng.random(ci.size) * np.maximum(room, 1)).astype(np.int64)
    cj = cj + r + np.floor(rng.random(cj.size) * np.maximum(room, 1)).astype(np.int64)
    for rad in range(3, 13):
        a = np.arange(-rad, rad + 1)
        di, dj = np.meshgrid(a, a, indexing="ij")
        keep = di * di + dj * dj <= rad * rad
        sel = r == rad
        t[(ci[sel][:, None] + di[keep][None, :]).ravel(), (cj[sel][:, None] + dj[keep][None, :]).ravel()] = W.OBSTACLE
    return t


def _discs(R, C, rng):
    """Channel with three discs in its first half."""
    r = max(3, R // 12)
    out = []
    for q in range(3):
        ci = int(rng.integers(r + 3, R - r - 3))
        cj = int(C * (0.12 + 0.16 * q)) + int(rng.integers(0, max(1, C // 40)))
        out.append((ci, min(max(cj, r + 4), C - r - 5), r))
    return W.channel_types(R, C, out)


def problem(case, seed):
    """The lattice of a case: node types, parameters, boundary values (one row, constant in time)."""
    rng = np.random.Generator(np.random.PCG64([int(seed), case["rows"], case["cols"]]))
    R, C, kind = case["rows"], case["cols"], case["kind"]
    trt = case["coll"] == "trt"
    p = dict(R=R, C=C, kind=kind, trt=trt, outlet="velocity", partial=False)
    if kind == "cavity":
        t = np.zeros((R, C), dtype=np.uint8)
        t[0, :] = t[-1, :] = t[:, 0] = t[:, -1] = W.BOUNDARY
        t[0, 1:-1] = W.INLET
        p.update(types=t, tau=float(rng.uniform(0.7, 0.95)), u=float(rng.uniform(0.05, 0.1)))
    elif kind == "cylinder":
        r = max(3, int(round(20.0 * R / 256.0)))
        y0 = int(round(131.0 * R / 256.0)) + int(rng.integers(-2, 3))
        t = W.cylinder_types(R, C, int(round(200.0 * C / 1024.0)), y0, r)
        p.update(types=t, tau=float(rng.uniform(0.53, 0.6)), u=float(rng.uniform(0.04, 0.05)), outlet="pressure")
    elif kind == "channel":
        p.update(types=_discs(R, C, rng), tau=float(rng.uniform(0.6, 0.9)), u=float(rng.uniform(0.03, 0.06)),
                 outlet="open" if trt else "pressure")
    elif kind == "partial":
        p.update(types=_discs(R, C, rng), tau=float(rng.uniform(0.6, 0.9)), u=float(rng.uniform(0.03, 0.06)),
                 outlet="pressure", partial=True)
    else:
        p.update(types=_porous(R, C, rng), tau=0.8, u=float(rng.uniform(0.01, 0.02)), outlet="pressure")
    p["tau_odd"] = 0.25 / (p["tau"] - 0.5) + 0.5
    return p


def batch_problems(case, seed):
    """Uneven problems as llb_workloads.batch_problems makes them: half cavities,
    half channels with discs, BGK or TRT, own relaxation time each; rows times
    columns from 64 x 64 to 4 cols x cols."""
    rng = np.random.Generator(np.random.PCG64([int(seed), case["rows"], case["cols"], 7]))
    sizes = BATCH_SIZES[BATCH_SIZES <= case["cols"]]
    # the sizes belong to the case, not to the seed: every seed is the same amount of work
    srng = np.random.Generator(np.random.PCG64([case["rows"], case["cols"]]))
    out = []
    for q in range(case["rows"]):
        C = int(srng.choice(sizes))
        R = int(round(C * float(srng.uniform(1.0, 4.0))))
        sub = dict(kind="cavity" if q % 2 == 0 else "channel", rows=R, cols=C,
                   coll="trt" if srng.integers(0, 2) else "bgk")
        p = problem(sub, int(rng.integers(0, 2**31)))
        if sub["kind"] == "channel":
            p["outlet"] = "pressure"
        out.append(p)
    return out


def _open_values(p, lists):
    ni, no = len(lists["inlet"]), len(lists["outlet"])
    v = np.zeros((1, ni + no, 2))
    if p["kind"] in ("cavity", "porous"):
        v[0, :ni, 0] = p["u"]
    else:  # Poiseuille profile across the inlet
        H = float(p["R"] - 2)
        y = lists["inlet"][:, 0] - 0.5
        v[0, :ni, 0] = 4.0 * p["u"] * y * (H - y) / (H * H)
    if p["outlet"] == "pressure":
        v[0, ni:, 0] = 1.0
    else:  # an open outlet keeps the velocity it is given
        v[0, ni:, 0] = p["u"] * 2.0 / 3.0
    return v


def _params(p):
    bc = {"velocity": L.BC_ZH_VELOCITY, "pressure": L.BC_ZH_PRESSURE, "open": L.BC_OPEN}[p["outlet"]]
    kw = dict(collision=L.TRT if p["trt"] else L.BGK, tau=p["tau"], tau_even=p["tau"], tau_odd=p["tau_odd"],
              outlet_bc=bc)
    if p["partial"]:
        kw.update(obstacle_bc=L.OBSTACLE_PARTIAL, ps_tau=p["tau"])
    return kw


def _lists_args(p, n):
    return (p["R"], p["C"], n["fluid"], n["wall"], n["inlet"], n["inlet_side"], n["outlet"], n["outlet_side"],
            n["obstacle"], n["obstacle_dirs"])


def prepare(case, seed):
    storage = STORAGE[case["storage"]]
    if case["kind"] == "batch":
        b = L.CudaBatch(storage=storage)
        b.set_config(2, 1)
        slots = []
        for p in batch_problems(case, seed):
            n = L.classify(p["types"])
            slots.append(b.add(*_lists_args(p, n), open_values=_open_values(p, n), **_params(p)))
        b.synchronize()
        return dict(case=case, batch=b, slots=slots)
    p = problem(case, seed)
    n = L.classify(p["types"])
    lat = L.CudaLattice(*_lists_args(p, n), storage=storage, **_params(p))
    lat.set_open_values(_open_values(p, n))
    lat.init()
    if case["kind"] == "cylinder":
        lat.set_force_points(n["obstacle"], n["obstacle_dirs"])
    lat.synchronize()
    return dict(case=case, lattice=lat)


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.step(case["steps"])
        out = []
        for s in state["slots"]:
            rho, u = b.lattice(s).compute_macro()
            out.append({"rho": rho, "u": u})
        return out
    lat = state["lattice"]
    left, forces = case["steps"], []
    if case["kind"] == "cylinder":  # drag and lift every 100 steps
        while left > 100:
            lat.step(100)
            forces.append(lat.flow_forces())
            left -= 100
    lat.step(left, macro=True)
    rho, u = lat.macro()
    out = {"rho": rho, "u": u}
    if case["kind"] == "cylinder":
        forces.append(lat.flow_forces())
        out["lift_drag"] = np.array(forces)
    return out


def _nodes(case):
    if case["kind"] == "batch":
        srng = np.random.Generator(np.random.PCG64([case["rows"], case["cols"]]))
        sizes, n = BATCH_SIZES[BATCH_SIZES <= case["cols"]], 0
        for _ in range(case["rows"]):
            C = int(srng.choice(sizes))
            n += C * int(round(C * float(srng.uniform(1.0, 4.0))))
            srng.integers(0, 2)
        return n, n
    n = case["rows"] * case["cols"]
    return n, int(n * 0.70) if case["kind"] == "porous" else n


def work(case):
    """The state read and written once and the fields written once; about 130
    operations per active node and step (nine-term moments, nine equilibria,
    the relaxation)."""
    n, active = _nodes(case)
    return {"bytes": 18.0 * BYTES[case["storage"]] * active + 24.0 * n, "flops": 130.0 * active * case["steps"]}


# ---- the same simulation in plain torch, 64 bits ---------------------------------
_DI = (0, 0, -1, 0, 1, -1, -1, 1, 1)
_DJ = (0, 1, 0, -1, 0, 1, -1, -1, 1)
_OPP = (0, 3, 4, 1, 2, 7, 8, 5, 6)
_WGT = (4 / 9,) + (1 / 9,) * 4 + (1 / 36,) * 4
# per side of an open node: the populations known there, doubled or not, the
# directions to complete (straight one first) and the signs of the closure
_SIDES = {
    "top": dict(same=(0, 1, 3), twice=(2, 5, 6), sign=1.0, normal="y"),
    "bottom": dict(same=(0, 1, 3), twice=(4, 7, 8), sign=-1.0, normal="y"),
    "left": dict(same=(0, 2, 4), twice=(3, 7, 6), sign=-1.0, normal="x"),
    "right": dict(same=(0, 2, 4), twice=(1, 5, 8), sign=1.0, normal="x"),
}


def _exact_lattice(p, steps, forces_every, dev):
    f64 = torch.float64
    R, C = p["R"], p["C"]
    types = torch.from_numpy(p["types"].astype(np.int64)).to(dev)
    lists = _open_and_wet_nodes(p["types"])
    inlet, outlet = types == W.INLET, types == W.OUTLET
    fluid = types == W.FLUID
    active = fluid | inlet | outlet
    solid = (types == W.BOUNDARY) | (types == W.OBSTACLE)
    pad = lambda m, v: torch.nn.functional.pad(m.to(torch.uint8), (1, 1, 1, 1), value=v).bool()
    act_p, sol_p = pad(active, 0), pad(solid, 0)
    near = lambda mp, k: mp[1 - _DI[k]:1 - _DI[k] + R, 1 - _DJ[k]:1 - _DJ[k] + C]  # at x - c_k
    from_fluid = [near(act_p, k) for k in range(9)]
    bounce = [near(sol_p, k) & active for k in range(9)]
    vals = torch.from_numpy(_open_values(p, lists)[0]).to(dev)
    ux0 = torch.zeros((R, C), dtype=f64, device=dev)
    rho0 = torch.ones((R, C), dtype=f64, device=dev)
    ii, jj = (torch.from_numpy(np.concatenate([lists["inlet"][:, d], lists["outlet"][:, d]])).to(dev) for d in (0, 1))
    is_out = torch.zeros(len(ii), dtype=torch.bool, device=dev)
    is_out[len(lists["inlet"]):] = True
    pres = is_out & (p["outlet"] == "pressure")
    closed = ~(is_out & (p["outlet"] == "open"))
    groups = []
    for side, sel in (("top", (ii == 0) & (jj > 0) & (jj < C - 1)), ("bottom", (ii == R - 1) & (jj > 0) & (jj < C - 1)),
                      ("left", (jj == 0) & (ii > 0) & (ii < R - 1)), ("right", (jj == C - 1) & (ii > 0) & (ii < R - 1))):
        for pr in (False, True):
            q = torch.nonzero(sel & closed & (pres == pr)).flatten()
            if len(q):
                groups.append((_SIDES[side], pr, ii[q], jj[q], vals[q]))
    prescribed = ~pres
    pi, pj, pv = ii[prescribed], jj[prescribed], vals[prescribed]

    def equilibrium(rho, ux, uy):
        u2 = 1.5 * (ux * ux + uy * uy)
        for k in range(9):
            cu = 3.0 * (_DJ[k] * ux - _DI[k] * uy)
            yield _WGT[k] * rho * (1.0 + cu + 0.5 * cu * cu - u2)

    def stream_and_close(f):
        """S_t from the post-collision populations, closures of the open nodes; velocities that pressure closures imply."""
        s = [f[0]]
        for k in range(1, 9):
            moved = torch.roll(f[k], (_DI[k], _DJ[k]), (0, 1))
            s.append(torch.where(bounce[k], f[_OPP[k]], torch.where(from_fluid[k], moved, _WGT[k])))
        implied = []
        for g, pr, i, j, v in groups:
            at = [x[i, j] for x in s]
            known = sum(at[k] for k in g["same"]) + 2.0 * sum(at[k] for k in g["twice"])
            if pr:
                rho, tang = v[:, 0], v[:, 1]
                out = known / rho - 1.0  # velocity out of the domain
            else:
                un = v[:, 1] if g["normal"] == "y" else v[:, 0]
                tang = v[:, 0] if g["normal"] == "y" else v[:, 1]
                out = g["sign"] * un
                rho = known / (1.0 + out)
            straight = g["twice"][0]
            a, b = g["same"][1], g["same"][2]
            for k in g["twice"]:
                o = _OPP[k]
                if k == straight:
                    new = at[k] - (2.0 / 3.0) * rho * out
                else:
                    # tangential component of the unknown direction o: +1 along direction a, -1 along b
                    tc = _DJ[o] if g["normal"] == "y" else -_DI[o]
                    new = at[k] - rho * out / 6.0 + tc * (0.5 * rho * tang - 0.5 * (at[a] - at[b]))
                s[o][i, j] = new
            if pr:
                un = g["sign"] * out
                implied.append((i, j, un, tang) if g["normal"] == "x" else (i, j, tang, un))
        return s, implied

    te, to = 1.0 / p["tau"], 1.0 / p["tau_odd"]

    def moments(s, implied, first):
        rho = sum(s)
        ux = (s[1] + s[5] + s[8] - s[3] - s[6] - s[7]) / rho
        uy = (s[2] + s[5] + s[6] - s[4] - s[7] - s[8]) / rho
        rho = torch.where(fluid, rho, 1.0)
        ux, uy = torch.where(fluid, ux, 0.0), torch.where(fluid, uy, 0.0)
        ux[pi, pj], uy[pi, pj] = pv[:, 0], pv[:, 1]
        for i, j, x, y in implied:
            ux[i, j], uy[i, j] = x, y
        return rho, ux, uy

    def collide(s, rho, ux, uy):
        e = list(equilibrium(rho, ux, uy))
        if not p["trt"]:
            out = [s[k] + te * (e[k] - s[k]) for k in range(9)]
        else:
            out = []
            for k in range(9):
                b = _OPP[k]
                out.append(s[k] - 0.5 * te * (s[k] + s[b] - e[k] - e[b]) - 0.5 * to * (s[k] - s[b] - e[k] + e[b]))
        return [torch.where(active, out[k], _WGT[k]) for k in range(9)]

    f = [torch.full((R, C), _WGT[k], dtype=f64, device=dev) for k in range(9)]
    zero = torch.zeros((R, C), dtype=f64, device=dev)
    rho, ux, uy = moments([x.clone() for x in f], [], True)
    f = collide([x.clone() for x in f], rho, ux, uy)
    forces = []
    obst = torch.from_numpy(lists["obstacle"]).to(dev)
    for t in range(1, steps + 1):
        s, implied = stream_and_close(f)
        rho, ux, uy = moments(s, implied, False)
        f = collide(s, rho, ux, uy)
        if forces_every and (t == steps or (t % forces_every == 0 and steps - t >= 1)):
            lift = drag = 0.0
            for k in range(1, 9):
                ni, nj = obst[:, 0] + _DI[k], obst[:, 1] + _DJ[k]
                ok = active[ni, nj]
                total = float(f[_OPP[k]][ni[ok], nj[ok]].sum()) * (1.0 if k <= 4 else math.sqrt(2.0) / 2.0)
                drag -= _DJ[k] * total
                lift += _DI[k] * total
            forces.append((lift, drag))
    out = {"rho": rho.T.contiguous().cpu().numpy(), "u": torch.stack([ux.T, uy.T]).contiguous().cpu().numpy()}
    if forces_every:
        out["lift_drag"] = np.array(forces)
    return out


def _open_and_wet_nodes(types):
    """Inlet, outlet and obstacle nodes in row-major order, in numpy."""
    at = lambda code: np.argwhere(types == code).astype(np.int64)
    R, C = types.shape
    obst = at(W.OBSTACLE)
    act = np.isin(types, (W.FLUID, W.INLET, W.OUTLET))
    wet = np.zeros(len(obst), dtype=bool)
    for k in range(1, 9):
        i, j = obst[:, 0] + _DI[k], obst[:, 1] + _DJ[k]
        ok = (i >= 0) & (j >= 0) & (i < R) & (j < C)
        wet[ok] |= act[i[ok], j[ok]]
    return {"inlet": at(W.INLET), "outlet": at(W.OUTLET), "obstacle": obst[wet]}


def exact(case, seed):
    n, _ = _nodes(case)
    if case["kind"] == "partial" or n * case["steps"] > 3e9 or (case["kind"] == "batch" and case["rows"] * case["steps"] > 12000):
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "batch":
        out = []
        for p in batch_problems(case, seed):
            r = _exact_lattice(p, case["steps"] + 1, 0, dev)  # compute_macro: the fields the next step sees
            out.append({"rho": r["rho"], "u": r["u"]})
        return out
    return _exact_lattice(problem(case, seed), case["steps"], 100 if case["kind"] == "cylinder" else 0, dev)
