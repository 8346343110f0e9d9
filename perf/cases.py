"""Workloads of the framework, for timing and for checking its results.

``listed()`` names the workloads, ``draw(rng)`` gives further ones of the same
ranges, ``prepare`` builds what a program holds before the call, ``run`` is one
pass through the public entry points, ``work`` the bytes and operations the
pass cannot do without, and ``exact`` its results in plain 64-bit torch.

Five kinds of work:

* ``torus``   one RK2 step of the Kerr torus (``bhgpu.fixed.FxGrid``) on a
  uniform grid or on blocks of several refinement levels, from a state held
  packed on the device (``unpack_state`` + ``step`` or ``replay``): the time
  loop of the solver, each pass restarted so that every pass does the same work.
* ``box``     one step of the reference-faithful scheme (``bhgpu.StepGraph``
  over ``RK2Integrator.step``) on the periodic magnetised box.
* ``ctop``    con2prim of a batch of independent Kerr cells (``Conserved.ctop``).
* ``learned`` the same started by the network (``C2PGuess.ctop_learned``).
* ``train``   loss and weight gradients of one training batch of that network.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "black-hole-simulator_b200"))
import bhgpu  # noqa: E402
from bhgpu import c2p_guess, configs  # noqa: E402
from bhgpu import fixed as fx  # noqa: E402
from bhgpu.mesh import Quilt  # noqa: E402
from bhgrid.blocks import torus_levels  # noqa: E402

GAMMA = 4.0 / 3.0
SPIN = 0.9375
LO, HI = -40.0, 40.0
F64 = torch.float64


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _torus(name, n, block, precision, limiter="mc", how="step"):
    return {"name": name, "kind": "torus", "n": n, "block": block, "precision": precision, "limiter": limiter,
            "how": how}


def _levels(name, n0, radii, seed, precision, limiter="mc", how="graph"):
    radii = list(radii) + [0.0] * (3 - len(radii))
    return {"name": name, "kind": "levels", "n0": n0, "r1": radii[0], "r2": radii[1], "r3": radii[2],
            "map_seed": seed, "precision": precision, "limiter": limiter, "how": how}


def listed():
    return [
        # the headline configuration: 128^3 torus in one block, FP32 face work,
        # launch bounds tuned and the step captured once, as a long run does
        _torus("torus128_mixed_tuned", 128, 128, "mixed", how="tuned"),
        # the production resolution (256^3), the library's own launch choices
        _torus("torus256_mixed", 256, 256, "mixed"),
        # the plain FP64 form on a grid cut into blocks (ghost exchange between
        # blocks), a run of middling resolution
        _torus("torus96_fp64_blocks", 96, 32, "fp64"),
        # PPM reconstruction, FP64 with contraction, a size that no tile divides
        _torus("torus104_fma_ppm", 104, 104, "fp64-fma", "ppm", "graph"),
        # the smallest torus that is stepped anywhere (the smoke test's):
        # launches and latency are all there is
        _torus("torus16_mixed", 16, 8, "mixed"),
        # blocks of three and of four levels: the block-AMR configurations
        _levels("levels3_mixed", 8, (14.0, 26.0), 3, "mixed"),
        _levels("levels4_fp64", 4, (10.0, 18.0, 28.0), 5, "fp64"),
        # the reference-faithful scheme on the 64^3 box that it is checked on
        {"name": "box64_fp64", "kind": "box", "patches": 4, "limiter": "minmod", "precision": "fp64"},
        # con2prim stress batch: many cells (an odd count), and few
        {"name": "ctop_2M", "kind": "ctop", "n": 2000003},
        {"name": "ctop_4k", "kind": "ctop", "n": 4001},
        # the learned start on a batch, and one training batch of its network
        {"name": "learned_1M", "kind": "learned", "n": 1000000},
        {"name": "train_8k", "kind": "train", "n": 8192},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["torus"] * 5 + ["levels"] * 3 + ["box", "ctop", "ctop", "learned", "train"])
    if kind == "torus":
        m = round(_log(rng, 2, 20))                     # n = 8 m: 16 .. 160
        cuts = [c for c in range(1, m + 1) if m % c == 0 and (m // c) ** 3 <= 512]
        c = _torus("", 8 * m, 8 * rng.choice(cuts), rng.choice(["mixed", "mixed", "fp64", "fp64-fma"]),
                   rng.choice(["mc", "mc", "mc", "ppm", "vanleer", "minmod"]), rng.choice(["step", "graph"]))
    elif kind == "levels":
        r1 = round(rng.uniform(8.0, 16.0), 2)
        radii = [r1, round(r1 + rng.uniform(8.0, 12.0), 2)]
        c = _levels("", rng.choice([4, 8]), radii, rng.randrange(1 << 20),
                    rng.choice(["mixed", "mixed", "fp64", "fp64-fma"]), rng.choice(["mc", "mc", "ppm"]),
                    rng.choice(["step", "graph"]))
    elif kind == "box":
        c = {"kind": "box", "patches": rng.choice([1, 2, 3, 4, 5]), "limiter": rng.choice(["minmod", "vanleer"]),
             "precision": rng.choice(["fp64", "fp64", "fp64-fma", "mixed"])}
    elif kind == "train":
        c = {"kind": "train", "n": round(_log(rng, 256, 16384))}
    else:
        c = {"kind": kind, "n": round(_log(rng, 1000, 2e6)) | 1}
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# what a program has in hand before the call
# ---------------------------------------------------------------------------
def _torus_state(case, seed):
    prm = fx.FxParams(precision=case["precision"], limiter=case["limiter"])
    if case["kind"] == "torus":
        g = fx.FxGrid.uniform(LO, HI, case["n"], case["block"], prm)
    else:
        radii = tuple(case[k] for k in ("r1", "r2", "r3") if case[k] > 0)
        lv = torus_levels(nb=8, r_fine=radii, seed=case["map_seed"])
        g = fx.FxGrid.leveled(LO, HI, lv, case["n0"], prm, persistent=True)
    g.torus_init(seed=1 + seed % (1 << 31))
    # the previous primitives differ from the state's own by about a step's change
    gen = torch.Generator(device="cuda").manual_seed(seed)
    noise = torch.randn(g.W[:5].shape, generator=gen, device="cuda", dtype=torch.float32)
    g.W[:5] *= (1.0 + 0.01 * noise).to(g.W.dtype).clamp_(0.9, 1.1)
    return g


def _batch(n, seed, a=SPIN):
    """Conserved states of n Kerr cells over the stress batch's ranges."""
    W, r, th = configs.con2prim_batch(n, seed=seed, gamma=GAMMA, a=a)
    cn = bhgpu.Conserved(bhgpu.Metric(1.0, a), bhgpu.State(GAMMA))
    rd, thd = torch.as_tensor(r, device="cuda"), torch.as_tensor(th, device="cuda")
    U, _ = cn.ptoc(torch.as_tensor(W, device="cuda"), rd, thd, check_domain=False)
    return cn, U, rd, thd, torch.as_tensor(W, device="cuda")


def _fit(g, pre, r, xi, lor):
    """Weights of the guess network from random features: the feature
    normalisation and hidden layers as they are, the output layer by least
    squares on (log xi / D, log W) -- what a trained network predicts."""
    x = g.features(pre, r)
    tgt = torch.stack([torch.log(xi / pre[0]), torch.log(lor)])
    ok = torch.isfinite(x).all(0) & torch.isfinite(tgt).all(0)
    x, tgt = x[:, ok].double(), tgt[:, ok]
    P, NI, NH = c2p_guess.NPARAM, c2p_guess.NI, c2p_guess.NH
    w = g.w.double()
    w[P:P + NI], w[P + NI:] = x.mean(1), 1.0 / (x.std(1) + 1e-12)
    xn = (x - w[P:P + NI, None]) * w[P + NI:, None]
    wb = w[:P].bfloat16().double()
    o = NH * NI
    h = torch.tanh(wb[:o].view(NH, NI) @ xn + wb[o:o + NH, None])
    o += NH
    h = torch.tanh(wb[o:o + NH * NH].view(NH, NH) @ h + wb[o + NH * NH:o + NH * NH + NH, None])
    o += NH * NH + NH
    A = torch.cat([h, torch.ones_like(h[:1])])
    sol = torch.linalg.solve(A @ A.T + 1e-6 * A.shape[1] * torch.eye(NH + 1, device="cuda", dtype=F64), A @ tgt.T)
    w[o:o + 2 * NH] = sol[:NH].T.reshape(-1)
    w[o + 2 * NH:P] = sol[NH]
    g.w.copy_(w.float())
    g.wb.copy_(g.w[:P].bfloat16())


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("torus", "levels"):
        g = _torus_state(case, seed)
        state = torch.empty(g.state_nbytes(), dtype=torch.uint8, device="cuda")
        g.pack_state(state)
        if case["how"] == "tuned":
            # the choice is process-wide; the captured graph keeps its own
            # kernels, so what other grids had is put back afterwards
            before = {k: fx.tune_get(g.precision, k) for k in fx.TUNE_KNOBS}
            fx.autotune(g)
            g.capture()
            for k, v in before.items():
                fx.tune_set(g.precision, k, v)
        elif case["how"] == "graph":
            g.capture()
        return {"kind": kind, "how": case["how"], "g": g, "state": state}
    if kind == "box":
        n = case["patches"]
        q = Quilt([10.0] * 3, [12.0] * 3, n, periodic=True)
        tree = bhgpu.AmrTree(q.dom_l, q.dom_h, n, M=0.0, a=0.0, Q=0.0, gm=GAMMA, periodic=True,
                             limiter=case["limiter"], quilt=q, init_floor=False, precision=case["precision"])
        W, Bf = configs.magnetised_box(q, seed=seed, gamma=GAMMA)
        tree.load(W=W, Bf=Bf)
        tree.prim_to_cons()
        start = [t.clone() for t in (tree.U, tree.W, tree.Bf)]

        def restart():
            for t, s in zip((tree.U, tree.W, tree.Bf), start):
                t.copy_(s)
        return {"kind": kind, "tree": tree, "graph": bhgpu.StepGraph(tree, bhgpu.RK2Integrator(0.4), before=restart)}
    cn, U, r, th, W = _batch(case["n"], seed)
    if kind == "ctop":
        return {"kind": kind, "cn": cn, "U": U, "r": r, "th": th}
    g = bhgpu.C2PGuess(cn, seed=0)
    pre = g.preamble(U, r, th)
    # targets near the truth: rho h W^2 and W of the primitives the cells came from
    v = W[2:5]
    gam = _kerr_spatial(r, th)
    lor = 1.0 / torch.sqrt(1.0 - torch.einsum("ijn,in,jn->n", gam, v, v))
    xi = W[0] * (1.0 + GAMMA * W[1]) * lor * lor
    _fit(g, pre, r, xi, lor)
    if kind == "learned":
        return {"kind": kind, "g": g, "U": U, "r": r, "th": th,
                "err": torch.zeros(1, dtype=torch.int32, device="cuda")}
    # training: the output layer is not yet fitted
    w = g.w.clone()
    w[c2p_guess.NPARAM - 130:c2p_guess.NPARAM - 2] *= 0.5
    g.w.copy_(w)
    g.wb.copy_(g.w[:c2p_guess.NPARAM].bfloat16())
    target = torch.stack([torch.log(xi / pre[0]), torch.log(lor)]).float()
    return {"kind": kind, "g": g, "pre": pre, "r": r, "target": target}


def _kerr_spatial(r, th):
    c, s = torch.cos(th), torch.sin(th)
    Sig = r * r + SPIN * SPIN * c * c
    H = 2.0 * r / Sig
    gam = torch.zeros((3, 3, r.numel()), dtype=F64, device="cuda")
    gam[0, 0] = 1.0 + H
    gam[0, 2] = gam[2, 0] = -H * SPIN * s * s
    gam[1, 1] = Sig
    gam[2, 2] = (r * r + SPIN * SPIN + H * SPIN * SPIN * s * s) * s * s
    return gam


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind in ("torus", "levels"):
        g = state["g"]
        g.unpack_state(state["state"])
        if state["how"] == "step":
            g.step()
        else:
            g.replay()
        return {"U": g.U, "W": g.W, "Bf": g.Bf, "dt": g.dt}
    if kind == "box":
        dt = state["graph"].replay()
        t = state["tree"]
        return {"U": t.U, "W": t.W, "Bf": t.Bf, "dt": dt}
    if kind == "ctop":
        W, Wd, status, iters, path = state["cn"].ctop(state["U"], state["r"], state["th"], check_domain=False)
        return {"status": status, "iters": iters, "path": path, **_recovered(W, Wd, status)}
    if kind == "learned":
        W, Wd, status, iters, path, xi0 = state["g"].ctop_learned(state["U"], state["r"], state["th"],
                                                                  want_xi0=True, err=state["err"])
        return {"status": status, "iters": iters, "path": path, "xi0": xi0, **_recovered(W, Wd, status)}
    loss, grad = state["g"].gradient(state["pre"], state["r"], state["target"])
    return {"loss": loss, "grad": grad.astype(np.float32)}   # FP32 values (handed over as float64)


def _recovered(W, Wd, status):
    # (the primitives of a cell that was not recovered are not written)
    return {"W": torch.where(status == 1, W, 0.0), "Wd": torch.where(status == 1, Wd, 0.0)}


# ---------------------------------------------------------------------------
# bytes and operations of one pass
# ---------------------------------------------------------------------------
def _blocks_n(case):
    if case["kind"] == "torus":
        return [case["block"]] * (case["n"] // case["block"]) ** 3
    radii = tuple(case[k] for k in ("r1", "r2", "r3") if case[k] > 0)
    lv = torus_levels(nb=8, r_fine=radii, seed=case["map_seed"])
    return [case["n0"] << int(v) for v in lv.ravel()]


def work(case):
    kind = case["kind"]
    if kind in ("torus", "levels"):
        zones = sum(n ** 3 for n in _blocks_n(case))
        wb = 4 if case["precision"] == "mixed" else 8
        # in: the packed state (5 U, 5 W, 3 faces); out: 8 U, 8 W, 3 faces
        byte = zones * ((5 * 8 + 5 * wb + 24) + (64 + 8 * wb + 24))
        # two stages of con2prim (~400), three faces (~700 each), source, EMF and update (~400)
        return {"bytes": byte, "flops": zones * 2 * (400 + 3 * (900 if case["limiter"] == "ppm" else 700) + 400)}
    if kind == "box":
        zones = (16 * case["patches"]) ** 3
        return {"bytes": zones * 2 * (8 + 8 + 3) * 8, "flops": zones * 2 * (1500 + 3 * 1200 + 1000)}
    if kind == "ctop":   # 8 U, r, theta in; 8 W, 5 derived, 3 words out
        return {"bytes": case["n"] * (10 * 8 + 13 * 8 + 12), "flops": case["n"] * 1500}
    if kind == "learned":
        return {"bytes": case["n"] * (10 * 8 + 14 * 8 + 12), "flops": case["n"] * (1500 + 2 * (6 * 64 + 64 * 64 + 128))}
    return {"bytes": case["n"] * (6 * 8 + 2 * 4) + 4738 * (2 + 4),
            "flops": case["n"] * 3 * 2 * (6 * 64 + 64 * 64 + 128)}


# ---------------------------------------------------------------------------
# the results in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] in ("torus", "levels"):
        g = _torus_state(case, seed)
        return _Step(g.blocks_np, g.nbr_np, g.params, g.ghost_depth, g.maxlevel).step(g.U, g.W, g.Bf)
    if case["kind"] == "train":
        return _exact_gradient(prepare(case, seed))
    # the reference-faithful scheme's values are those of the reference's own
    # iterations (a root it stops short of, a fallback that fails): there is
    # no 64-bit value of them beside its own arithmetic
    return None


def _exact_gradient(s):
    g = s["g"]
    NI, NH, NO, P = c2p_guess.NI, c2p_guess.NH, c2p_guess.NO, c2p_guess.NPARAM
    D, tau, S2, B2, SB = s["pre"]
    x = torch.stack([torch.log(D), torch.asinh(tau / D), torch.log1p(S2 / (D * D)), torch.log1p(B2 / D),
                     torch.asinh(SB / (D * torch.sqrt(D))), torch.log(s["r"])])
    norm = g.w[P:].double()
    xn = (x - norm[:NI, None]) * norm[NI:, None]
    w = g.w[:P].bfloat16().double().requires_grad_(True)   # the weights that inference sees
    parts, o = [], 0
    for shape in ((NH, NI), (NH, 1), (NH, NH), (NH, 1), (NO, NH), (NO, 1)):
        k = shape[0] * shape[1]
        parts.append(w[o:o + k].view(shape))
        o += k
    w1, b1, w2, b2, w3, b3 = parts
    y = w3 @ torch.tanh(w2 @ torch.tanh(w1 @ xn + b1) + b2) + b3
    loss = ((y - s["target"].double()) ** 2).sum()
    (loss / x.shape[1]).backward()
    return {"loss": float(loss), "grad": w.grad}


CHUNK = 1 << 21   # positions at once


class _Step:
    """One RK2 step of the torus scheme: Valencia GRMHD in Cartesian
    Kerr-Schild coordinates on a list of cubic blocks with three ghost layers,
    every array a flat [..., ncell] with block b's (n+7)^3 box at off[b]."""

    def __init__(self, blocks, nbr, prm, depth, maxlevel):
        t = lambda a, d: torch.as_tensor(np.ascontiguousarray(a), device="cuda").to(d)  # noqa: E731
        self.n, self.level, self.off = (t(blocks[k], torch.int64) for k in ("n", "level", "off"))
        self.x0, self.dx, self.nbr = t(blocks["x0"], F64), t(blocks["dx"], F64), t(nbr, torch.int64)
        self.blocks, self.prm, self.depth, self.maxlevel = blocks, prm, depth, maxlevel
        self.M, self.a, self.gm = prm.M, prm.a, prm.gamma
        self.gg = prm.gamma / (prm.gamma - 1.0)
        self.r_exc = 1.2 * (prm.M + math.sqrt(prm.M ** 2 - prm.a ** 2)) if prm.r_exc is None else prm.r_exc
        self.cells = self._grid(0, 0)
        self.pos = self._grid(1, 1)

    # ---- index space ---------------------------------------------------
    def _grid(self, below, above):
        """(block, i, j, k) of every position in [-below, n + above)^3."""
        out = []
        for n in np.unique(self.blocks["n"]):
            b = torch.as_tensor(np.nonzero(self.blocks["n"] == n)[0], device="cuda")
            ax = torch.arange(-below, int(n) + above, device="cuda")
            out.append(torch.stack([m.reshape(-1) for m in torch.meshgrid(b, ax, ax, ax, indexing="ij")]))
        return torch.cat(out, 1)

    def at(self, b, i, j, k):
        S = self.n[b] + 7
        return self.off[b] + ((i + 3) * S + (j + 3)) * S + (k + 3)

    def strides(self, b):
        S = self.n[b] + 7
        return S * S, S, torch.ones_like(S)

    def where(self, p, shift=(0.5, 0.5, 0.5)):
        return [self.x0[p[0], d] + (p[1 + d] + shift[d]) * self.dx[p[0]] for d in range(3)]

    # ---- metric ---------------------------------------------------------
    def metric(self, x, y, z):
        a2 = self.a * self.a
        d = x * x + y * y + z * z - a2
        r2 = 0.5 * (d + torch.sqrt(d * d + 4.0 * a2 * z * z))
        r = torch.sqrt(r2)
        q = r2 * r2 + a2 * z * z                     # 0 on the disc inside the ring: flat there
        H = torch.where(q > 0.0, self.M * r * r2 / q, 0.0)
        l = [(r * x + self.a * y) / (r2 + a2), (r * y - self.a * x) / (r2 + a2), torch.where(r > 0.0, z / r, 0.0)]
        f = 1.0 + 2.0 * H
        return {"r": r, "H": H, "l": l, "sg": torch.sqrt(f), "al": 1.0 / torch.sqrt(f),
                "be": [2.0 * H / f * c for c in l], "hf": 2.0 * H / f}

    @staticmethod
    def low(m, v):
        lv = 2.0 * m["H"] * (m["l"][0] * v[0] + m["l"][1] * v[1] + m["l"][2] * v[2])
        return [v[i] + lv * m["l"][i] for i in range(3)]

    @staticmethod
    def up(m, v):
        lv = m["hf"] * (m["l"][0] * v[0] + m["l"][1] * v[1] + m["l"][2] * v[2])
        return [v[i] - lv * m["l"][i] for i in range(3)]

    def derive(self, m, w):
        ut, B = w[2:5], w[5:8]
        ul, Bl = self.low(m, ut), self.low(m, B)
        W = torch.sqrt(1.0 + sum(ul[i] * ut[i] for i in range(3)))
        v, vl = [c / W for c in ut], [c / W for c in ul]
        B2, Bv = sum(Bl[i] * B[i] for i in range(3)), sum(Bl[i] * v[i] for i in range(3))
        b2 = B2 / (W * W) + Bv * Bv
        rhoh = w[0] + self.gg * w[1]
        return {"W": W, "v": v, "vl": vl, "Bl": Bl, "B2": B2, "Bv": Bv, "b2": b2, "rhoh": rhoh, "pt": w[1] + 0.5 * b2}

    @staticmethod
    def cons(m, w, d):
        W2, v2 = d["W"] ** 2, 1.0 - 1.0 / d["W"] ** 2
        D = w[0] * d["W"]
        S = [(d["rhoh"] * W2 + d["B2"]) * d["vl"][i] - d["Bv"] * d["Bl"][i] for i in range(3)]
        # E - D from rho W (W - 1) and the rest
        tau = D * (d["W"] - 1.0) + (d["rhoh"] - w[0]) * W2 - w[1] + 0.5 * d["B2"] * (1.0 + v2) - 0.5 * d["Bv"] ** 2
        return [m["sg"] * q for q in (D, S[0], S[1], S[2], tau, w[5], w[6], w[7])]

    def speeds(self, m, w, d, q):
        c2 = ((self.gm * w[1] + d["b2"]) / (d["rhoh"] + d["b2"])).clamp(0.0, 1.0)
        v2, vd = 1.0 - 1.0 / d["W"] ** 2, d["v"][q]
        gdd = 1.0 - m["hf"] * m["l"][q] ** 2
        den = 1.0 - v2 * c2
        rt = torch.sqrt((c2 * (1.0 - v2) * (gdd * den - vd * vd * (1.0 - c2))).clamp(min=0.0))
        return [m["al"] * (vd * (1.0 - c2) + s * rt) / den - m["be"][q] for s in (-1.0, 1.0)]

    # ---- con2prim, floors, excision and the CFL limit --------------------
    def prims(self, U, W, Bf, want_dt):
        best = math.inf
        for p in self.cells.split(CHUNK, 1):
            c, s = self.at(*p), self.strides(p[0])
            m = self.metric(*self.where(p))
            Bt = [0.5 * (Bf[d, c] + Bf[d, c + s[d]]) for d in range(3)]
            B = [q / m["sg"] for q in Bt]
            w, _ = self.solve(m, [U[v, c] / m["sg"] for v in range(5)], B, [W[v, c] for v in range(5)])
            changed = self.floors(m, w)
            d = self.derive(m, w)
            u = self.cons(m, w, d)
            for v in range(5):
                U[v, c] = torch.where(changed, u[v], U[v, c])
            for q in range(3):
                U[5 + q, c] = Bt[q]
            for v in range(8):
                W[v, c] = w[v]
            if want_dt:
                for q in range(3):
                    lm, lp = self.speeds(m, w, d, q)
                    best = min(best, float((self.dx[p[0]] / torch.maximum(lm.abs(), lp.abs())).min()))
        return best

    def solve(self, m, u, B, wo):
        D, S, tau = u[0], u[1:4], u[4]
        Su, Bl = self.up(m, S), self.low(m, B)
        S2, B2 = sum(Su[i] * S[i] for i in range(3)), sum(Bl[i] * B[i] for i in range(3))
        SB, E, gf = sum(S[i] * B[i] for i in range(3)), tau + D, 1.0 / self.gg
        ul = self.low(m, wo[2:5])
        Z = (wo[0] + self.gg * wo[1]) * (1.0 + sum(ul[i] * wo[2 + i] for i in range(3)))
        v2max = 1.0 - 1.0 / self.prm.W_max ** 2

        def residual(Z):
            ZB = Z + B2
            v2 = (S2 * Z * Z + SB * SB * (B2 + 2.0 * Z)) / (Z * Z * ZB * ZB)
            dv2 = -2.0 / ZB ** 3 * (S2 + SB * SB * (3.0 * Z * (Z + B2) + B2 * B2) / Z ** 3)
            v2, dv2 = v2.clamp(max=v2max), torch.where(v2 > v2max, 0.0, dv2)
            wi = torch.sqrt(1.0 - v2)
            f = Z - gf * (Z * wi * wi - D * wi) + 0.5 * (1.0 + v2) * B2 - 0.5 * SB * SB / Z ** 2 - E
            return f, 1.0 - gf * (wi * wi - Z * dv2 + 0.5 * D * dv2 / wi) + 0.5 * B2 * dv2 + SB * SB / Z ** 3

        # Newton from above, kept inside a bracket [0, Z] with f(Z) > 0
        lo, hi = torch.zeros_like(Z), torch.maximum(Z, E).clamp(min=1e-300)
        for _ in range(40):
            hi = torch.where(residual(hi)[0] > 0.0, hi, 2.0 * hi)
        Z = hi
        for _ in range(60):
            f, df = residual(Z)
            hi, lo = torch.where(f > 0.0, Z, hi), torch.where(f > 0.0, lo, Z)
            nxt = Z - f / df
            Z = torch.where((df > 0.0) & (nxt > lo) & (nxt < hi), nxt, torch.where(f == 0.0, Z, 0.5 * (lo + hi)))
        ZB = Z + B2
        v2 = ((S2 * Z * Z + SB * SB * (B2 + 2.0 * Z)) / (Z * Z * ZB * ZB)).clamp(max=v2max)
        wi = torch.sqrt(1.0 - v2)
        rho = D * wi
        vu = self.up(m, [(S[i] + SB / Z * Bl[i]) / ZB for i in range(3)])
        return [rho, gf * (Z * wi * wi - rho), *[q / wi for q in vu], *B], Z

    def floors(self, m, w):
        prm = self.prm
        re = m["r"].clamp(min=1.0)
        rf, pf = prm.rho_floor * re ** -1.5, (self.gm - 1.0) * prm.u_floor * re ** -2.5
        out = m["r"] < self.r_exc
        ul = self.low(m, w[2:5])
        u2 = sum(ul[i] * w[2 + i] for i in range(3))
        top = prm.W_max ** 2 - 1.0
        fast = u2 > top
        sc = torch.where(fast, torch.sqrt(top / u2.clamp(min=1e-300)), 1.0)
        ut = [w[2 + i] * sc for i in range(3)]
        Bl = self.low(m, w[5:8])
        B2, Bu = sum(Bl[i] * w[5 + i] for i in range(3)), sum(Bl[i] * ut[i] for i in range(3))
        b2 = (B2 + Bu * Bu) / (1.0 + torch.where(fast, top, u2))
        rs = torch.maximum(rf, b2 / prm.sigma_max)
        thin, cold = w[0] < rs, w[1] < pf
        w[0] = torch.where(out, rf, torch.maximum(w[0], rs))
        w[1] = torch.where(out, pf, torch.maximum(w[1], pf))
        for i in range(3):
            w[2 + i] = torch.where(out, 0.0, ut[i])
        return out | fast | thin | cold

    # ---- ghost cells and faces -------------------------------------------
    def source(self, p, d):
        """Block and position that position p (cell, or face of normal d)
        outside its block images; outflow at the outer boundary."""
        b, c, o = p[0], [p[1], p[2], p[3]], []
        n = self.n[b]
        for q in range(3):
            hi = n if q == d else n - 1
            s = (c[q] > hi).long() - (c[q] < 0).long()
            face = [13, 13, 13]
            step = (9, 3, 1)[q]
            none = (self.nbr[b, face[q] + s * step] < 0) & (s != 0)
            c[q] = torch.where(none, torch.where(s < 0, torch.zeros_like(hi), hi), c[q])
            o.append(torch.where(none, 0, s))
        src = self.nbr[b, 13 + 9 * o[0] + 3 * o[1] + o[2]]
        src = torch.where(src < 0, b, src)
        return src, [c[q] - o[q] * n for q in range(3)]

    def ghosts(self, W, Bf):
        if not hasattr(self, "shell"):
            g = self._grid(self.depth, self.depth)
            n = self.n[g[0]]
            inside = torch.stack([(g[q] >= 0) & (g[q] < n) for q in (1, 2, 3)]).all(0)
            self.shell = g[:, ~inside]
        p = self.shell
        n = self.n[p[0]]
        for ps in range(self.maxlevel + 1):
            s, c = self.source(p, -1)
            kind = torch.sign(self.n[s] - n)                     # 0 copy, 1 restrict, -1 prolong
            dst = self.at(*p)
            if ps == 0:
                e = kind == 0
                W[:, dst[e]] = W[:, self.at(s[e], *[q[e] for q in c])]
                e = kind > 0
                W[:, dst[e]] = sum(W[:, self.at(s[e], 2 * c[0][e] + i, 2 * c[1][e] + j, 2 * c[2][e] + k)]
                                   for i in (0, 1) for j in (0, 1) for k in (0, 1)) / 8.0
            else:
                e = (kind < 0) & (self.level[p[0]] == ps)
                h = [torch.div(q[e], 2, rounding_mode="floor") for q in c]
                k0 = self.at(s[e], *h)
                w0, st = W[:, k0], self.strides(s[e])
                val = w0.clone()
                for q in range(3):
                    l, r = w0 - W[:, k0 - st[q]], W[:, k0 + st[q]] - w0
                    sl = torch.where(l * r <= 0.0, 0.0, torch.where(l.abs() < r.abs(), l, r))
                    val += torch.where(c[q][e] % 2 == 1, 0.25, -0.25) * sl
                W[:, dst[e]] = val
            for d in range(3):
                need = (p[1 + d] >= 0) & (p[1 + d] <= n)
                for q in range(3):
                    if q != d:
                        need &= (p[1 + q] >= -1) & (p[1 + q] <= n)
                f = p[:, need]
                s, t = self.source(f, d)
                kind, dst, B = torch.sign(self.n[s] - self.n[f[0]]), self.at(*f), Bf[d]
                if ps == 0:
                    e = kind == 0
                    same = B[self.at(s[e], *[q[e] for q in t])]
                    g = kind > 0
                    fine = 0.0
                    for i in (0, 1):
                        for j in (0, 1):
                            x = [2 * q[g] for q in t]
                            x[(d + 1) % 3] = x[(d + 1) % 3] + i
                            x[(d + 2) % 3] = x[(d + 2) % 3] + j
                            fine = fine + 0.25 * B[self.at(s[g], *x)]
                    B[dst[e]] = same
                    B[dst[g]] = fine
                else:
                    e = (kind < 0) & (self.level[f[0]] == ps)
                    x = [torch.div(q[e], 2, rounding_mode="floor") for q in t]
                    y = list(x)
                    y[d] = y[d] + t[d][e] % 2
                    B[dst[e]] = 0.5 * (B[self.at(s[e], *x)] + B[self.at(s[e], *y)])

    # ---- reconstruction and HLL fluxes -------------------------------------
    def face(self, a):
        """Left and right value of a face from its cells a = [-3 .. 2] (PPM)
        or [-2 .. 1]."""
        lim = self.prm.limiter
        if lim == "ppm":
            dm = []
            for q in range(4):
                l, r = a[q + 1] - a[q], a[q + 2] - a[q + 1]
                c = 0.5 * (a[q + 2] - a[q])
                s = torch.minimum(c.abs(), 2.0 * torch.minimum(l.abs(), r.abs()))
                dm.append(torch.where(l * r <= 0.0, 0.0, torch.sign(c) * s))
            f = [a[q + 1] + 0.5 * (a[q + 2] - a[q + 1]) - (dm[q + 1] - dm[q]) / 6.0 for q in range(3)]

            def parabola(c, l, r):
                d, e = r - l, (r - l) * (c - 0.5 * (l + r))
                flat = (r - c) * (c - l) <= 0.0
                low, high = e > d * d / 6.0, e < -d * d / 6.0
                return (torch.where(flat, c, torch.where(low, 3.0 * c - 2.0 * r, l)),
                        torch.where(flat, c, torch.where(high & ~low, 3.0 * c - 2.0 * l, r)))
            return parabola(a[2], f[0], f[1])[1], parabola(a[3], f[1], f[2])[0]

        def value(wf, w0, wn):
            x, y = w0 - wf, wn - w0
            if lim == "vanleer":
                h = x * y / torch.where(x * y > 0.0, x + y, 1.0)
            elif lim == "mc":
                h = torch.sign(y) * torch.minimum(0.25 * (x.abs() + y.abs()), torch.minimum(x.abs(), y.abs()))
            else:
                h = torch.sign(y) * 0.5 * torch.minimum(x.abs(), y.abs())
            return torch.where(x * y <= 0.0, w0, w0 + h)
        return value(a[0], a[1], a[2]), value(a[3], a[2], a[1])

    def fluxes(self, W, Bf):
        F = torch.zeros((3, 8, W.shape[1]), dtype=F64, device="cuda")
        reach = range(-3, 3) if self.prm.limiter == "ppm" else range(-2, 2)
        for d in range(3):
            shift = [0.5, 0.5, 0.5]
            shift[d] = 0.0
            for p in self.pos[:, self.pos[1 + d] >= 0].split(CHUNK, 1):
                c, st = self.at(*p), self.strides(p[0])[d]
                m = self.metric(*self.where(p, shift))
                wl, wr = [None] * 8, [None] * 8
                for v in range(8):
                    if v == 5 + d:
                        wl[v] = wr[v] = Bf[d, c] / m["sg"]
                    else:
                        wl[v], wr[v] = self.face([W[v, c + o * st] for o in reach])
                side = []
                for w in (wl, wr):
                    q = self.derive(m, w)
                    u = self.cons(m, w, q)
                    ag = m["al"] * m["sg"]
                    vt = [m["al"] * q["v"][i] - m["be"][i] for i in range(3)]
                    Bd = w[5 + d]
                    f = [u[0] * vt[d]]
                    for j in range(3):
                        bj = (q["Bl"][j] / q["W"] ** 2 + q["Bv"] * q["vl"][j]) * Bd
                        f.append(u[1 + j] * vt[d] + ag * ((q["pt"] if j == d else 0.0) - bj))
                    f.append(u[4] * vt[d] + ag * (q["pt"] * q["v"][d] - q["Bv"] * Bd))
                    for k in range(3):
                        f.append(torch.zeros_like(Bd) if k == d else m["sg"] * (w[5 + k] * vt[d] - Bd * vt[k]))
                    side.append((u, f, *self.speeds(m, w, q, d)))
                (uL, fL, aL, bL), (uR, fR, aR, bR) = side
                sl, sr = torch.minimum(aL, aR).clamp(max=0.0), torch.maximum(bL, bR).clamp(min=0.0)
                for v in range(8):
                    if v != 5 + d:
                        F[d, v, c] = (sr * fL[v] - sl * fR[v] + sl * sr * (uR[v] - uL[v])) / (sr - sl)
        return F

    # ---- geometric source ----------------------------------------------------
    def gravity(self, p, w):
        x, y, z = self.where(p)
        m = self.metric(x, y, z)
        a, a2, r, H, l = self.a, self.a ** 2, m["r"], m["H"], m["l"]
        r2 = r * r
        q = r2 * r2 + a2 * z * z
        dr = [x * r2 * r / q, y * r2 * r / q, z * r * (r2 + a2) / q]
        d = self.derive(m, w)
        one = torch.ones_like(r)
        L = [one, *l]
        dH, dL = [], []
        for k in range(3):
            dq = 4.0 * r2 * r * dr[k] + (2.0 * a2 * z if k == 2 else 0.0)
            dH.append(self.M * (3.0 * r2 * dr[k] / q - r2 * r * dq / q ** 2))
            e = [float(k == i) for i in range(3)]
            t = 2.0 * r * dr[k]
            dL.append([torch.zeros_like(r), (dr[k] * x + e[0] * r + a * e[1] - l[0] * t) / (r2 + a2),
                       (dr[k] * y + e[1] * r - a * e[0] - l[1] * t) / (r2 + a2), (e[2] - l[2] * dr[k]) / r])
        u = [d["W"] / m["al"]]
        u += [w[2 + i] - u[0] * m["be"][i] for i in range(3)]
        b = [d["W"] * d["Bv"] / m["al"]]
        b += [(w[5 + i] + m["al"] * b[0] * u[1 + i]) / d["W"] for i in range(3)]
        lu = [-one, *l]
        eta = [-1.0, 1.0, 1.0, 1.0]
        inv = lambda i, j: (eta[i] if i == j else 0.0) - 2.0 * H * lu[i] * lu[j]  # noqa: E731
        T = [[(d["rhoh"] + d["b2"]) * u[i] * u[j] + d["pt"] * inv(i, j) - b[i] * b[j] for j in range(4)]
             for i in range(4)]
        # dg[k][i][j] = d_k g_ij with g = eta + 2 H l l
        dg = [[[2.0 * (dH[k] * L[i] * L[j] + H * (dL[k][i] * L[j] + L[i] * dL[k][j])) for j in range(4)]
               for i in range(4)] for k in range(3)]
        half = [0.5 * sum(T[i][j] * dg[k][i][j] for i in range(4) for j in range(4)) for k in range(3)]
        TG = 0.0
        for v in range(4):
            K = sum(T[1 + k][j] * dg[k][j][v] for k in range(3) for j in range(4))
            TG = TG + inv(0, v) * (K - (half[v - 1] if v else 0.0))
        dlna = [-m["al"] ** 2 * dH[k] for k in range(3)]
        tau = m["al"] * (sum(T[1 + k][0] * dlna[k] for k in range(3)) - TG)
        ag = m["al"] * m["sg"]
        return [torch.zeros_like(r), *[ag * h for h in half], ag * tau]

    # ---- edge EMFs and the update ---------------------------------------------
    def emf(self, F, c, st):
        """E at the lower edges of cells c, from the face fluxes of B."""
        f = lambda d, v, q: F[d, 5 + v, q]  # noqa: E731
        return [0.25 * (f((d + 2) % 3, (d + 1) % 3, c) + f((d + 2) % 3, (d + 1) % 3, c - st[(d + 1) % 3])
                        - f((d + 1) % 3, (d + 2) % 3, c) - f((d + 1) % 3, (d + 2) % 3, c - st[(d + 2) % 3]))
                for d in range(3)]

    def edges(self, F):
        E = torch.zeros((3, F.shape[2]), dtype=F64, device="cuda")
        for p in self.pos[:, (self.pos[1:] >= 0).all(0)].split(CHUNK, 1):
            c = self.at(*p)
            for d, v in enumerate(self.emf(F, c, self.strides(p[0]))):
                E[d, c] = v
        if self.maxlevel > 0:
            raw = E.clone()
            q = self.pos[:, (self.pos[1:] >= 0).all(0)]
            n = self.n[q[0]]
            for d in range(3):
                t1, t2 = (d + 1) % 3, (d + 2) % 3
                side = lambda t, p, m: (p[1 + t] == m).long() - (p[1 + t] == 0).long()  # noqa: E731
                e = (q[1 + d] < n) & ((side(t1, q, n) != 0) | (side(t2, q, n) != 0))
                p, m = q[:, e], n[e]
                done = torch.zeros_like(m, dtype=torch.bool)
                for a1, a2 in ((0, 1), (1, 0), (1, 1)):
                    o = [torch.zeros_like(m)] * 3
                    o[t1], o[t2] = a1 * side(t1, p, m), a2 * side(t2, p, m)
                    ok = ~done
                    if a1:
                        ok &= o[t1] != 0
                    if a2:
                        ok &= o[t2] != 0
                    s = self.nbr[p[0], 13 + 9 * o[0] + 3 * o[1] + o[2]]
                    ok &= (s >= 0) & (self.n[s.clamp(min=0)] == 2 * m)
                    x = [2 * (p[1 + k] - o[k] * m)[ok] for k in range(3)]
                    y = list(x)
                    y[d] = y[d] + 1
                    E[d, self.at(*p[:, ok])] = 0.5 * (raw[d, self.at(s[ok], *x)] + raw[d, self.at(s[ok], *y)])
                    done |= ok
        return E

    def update(self, U, W, Bf, dt):
        """U + dt L(U) in the rows 0-4 of the interior cells and Bf - dt curl E
        on the blocks' own faces, as [(rows, indices, values)]."""
        F = self.fluxes(W, Bf)
        E, out = self.edges(F), []
        for p in self.cells.split(CHUNK, 1):
            c, st, h = self.at(*p), self.strides(p[0]), self.dx[p[0]]
            S = self.gravity(p, [W[v, c] for v in range(8)])
            L = torch.stack([S[v] - sum(F[d, v, c + st[d]] - F[d, v, c] for d in range(3)) / h for v in range(5)])
            out.append(("U", slice(0, 5), c, U[:5, c] + dt * L))
        q = self.pos[:, (self.pos[1:] >= 0).all(0)]
        for d in range(3):
            n = self.n[q[0]]
            own = (q[1 + (d + 1) % 3] < n) & (q[1 + (d + 2) % 3] < n)
            for p in q[:, own].split(CHUNK, 1):
                c, st, h = self.at(*p), self.strides(p[0]), self.dx[p[0]]
                t1, t2 = (d + 1) % 3, (d + 2) % 3
                curl = (E[t2, c + st[t1]] - E[t2, c] - E[t1, c + st[t2]] + E[t1, c]) / h
                out.append(("B", d, c, Bf[d, c] - dt * curl))
        return out

    def step(self, U, W, Bf):
        U, W, Bf = U.double().clone(), W.double().clone(), Bf.double().clone()
        U[5:] = 0.0
        limit = self.prims(U, W, Bf, True)
        dt = self.prm.cfl * limit
        self.ghosts(W, Bf)
        U1, B1 = torch.zeros_like(U), torch.zeros_like(Bf)
        for k, v, c, x in self.update(U, W, Bf, dt):
            (U1 if k == "U" else B1)[v, c] = x
        self.prims(U1, W, B1, False)
        self.ghosts(W, B1)
        for k, v, c, x in self.update(U1, W, B1, dt):
            t = U if k == "U" else Bf
            t[v, c] = 0.5 * (t[v, c] + x)
        return {"U": U, "W": W, "Bf": Bf, "dt": torch.tensor([limit, dt], dtype=F64)}
