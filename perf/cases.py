"""Performance cases of the framework: what a user's program has it do.

A case is a plain dict; its "kind" is the call it makes:
  step     one pseudo-time step on a host-resident solution (GpuSolver.step_host), as the reference's stepSolution works
  march    a solution set, a number of steps marched, the solution read back (GpuSolver.set / march / get)
  batch    the same for several flow conditions on meshes of different sizes in one handle (GpuSolver.batch)
  tridag4  the two line solves of an ADI sweep over an ni x nj block of cells, by the function-level solver: ni open
           lines of nj rows, nj periodic lines of ni rows (native.block_tridag4)
  tridag5  the 5-variable line solver of the strand form, open or periodic (native.block_tridag5)
  roe      Roe fluxes and Jacobians of a list of faces (native.flux_roe2d, native.jacobian_roe2d)
  recon    reconstruction along lines and its linearisation (native.reconstruct)
  forward  the warm-start network's guess for a number of cells (native.Mlp.forward)
  train    optimiser steps of the warm-start network and its parameters (native.Mlp.train_step, get_params)

Meshes are the NACA 0012 O-grids of the benchmark and the tests; initial states are seeded, developed-looking fields
(flow along the wall, smooth modes, cell noise), and the flow condition of a solver case comes from the seed too.
`exact` gives the outputs in 64-bit torch arithmetic, written here from the scheme's formulas.
"""
import math
import tempfile

import numpy as np
import torch

from hamstr_oop_gb300 import meshgen, native

GAMMA = 1.4
DEV = "cuda" if torch.cuda.is_available() else "cpu"
BATCH_MESHES = ((128, 32), (256, 64), (384, 96), (512, 128))
SCHEMES = {  # order, limiter, CFL
    "first": (1, 0, 10.0), "muscl": (3, 0, 10.0), "minmod": (3, 1, 10.0), "vanalbada": (3, 2, 10.0), "weno": (5, 0, 20.0)}


def _cfl(case):
    """WENO marches from such states with the benchmark's ramp: CFL 5 before 20."""
    return 5.0 if case["scheme"] == "weno" and case["kind"] == "march" else SCHEMES[case["scheme"]][2]


def listed():
    return [
        # the smallest mesh in use (128 x 32 quads, MUSCL with minmod): a step is the latency of its periodic lines
        {"name": "step_fp64_128x32", "kind": "step", "ni": 128, "nj": 32, "split": 0.0, "scheme": "minmod", "fp32op": False},
        # the benchmark's default: every second quad split into triangles, WENO, CFL 20
        {"name": "step_fp64_512x128_split", "kind": "step", "ni": 512, "nj": 128, "split": 0.5, "scheme": "weno", "fp32op": False},
        # the FP32-operator form on a transonic mixed mesh with van Albada's limiter
        {"name": "step_fp32op_512x128_split", "kind": "step", "ni": 512, "nj": 128, "split": 0.3, "scheme": "vanalbada", "fp32op": True},
        # the plain drop-in on the warm start's mesh, some steps at a time
        {"name": "march_fp64_256x64", "kind": "march", "ni": 256, "nj": 64, "split": 0.0, "scheme": "first", "fp32op": False, "steps": 8},
        # quads with long periodic lines, FP32 operator, WENO
        {"name": "march_fp32op_512x128", "kind": "march", "ni": 512, "nj": 128, "split": 0.0, "scheme": "weno", "fp32op": True, "steps": 8},
        # many flow conditions in one handle, meshes round-robin: the batched form
        {"name": "batch32_fp32op", "kind": "batch", "n": 32, "scheme": "first", "fp32op": True, "steps": 4},
        # function-level line solves of one sweep over a 384 x 96 mesh
        {"name": "tridag4_384x96", "kind": "tridag4", "ni": 384, "nj": 96},
        # strands: many short open lines of 5 x 5 blocks
        {"name": "tridag5_4099x33", "kind": "tridag5", "lines": 4099, "rows": 33, "periodic": False},
        # every face of the default mesh through the per-face functions
        {"name": "roe_164399", "kind": "roe", "n": 164399},
        # every wrap-around line of a 512 x 128 mesh with its ghosts, WENO and its linearisation
        {"name": "weno_128x518", "kind": "recon", "scheme": "weno", "lines": 128, "imax": 518, "nq": 4},
        # the guess for four conditions on the 256 x 64 mesh, less a few cells; capacity as trained
        {"name": "mlp_forward_65500", "kind": "forward", "n": 65500, "capacity": 16384},
        # training as warmstart.train does it: minibatches of 16,384 cells out of 64 conditions on 128 x 32
        {"name": "mlp_train_16384", "kind": "train", "n": 262144, "batch": 16384, "steps": 4},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "march", "march", "batch", "tridag4", "tridag5", "roe", "recon", "forward", "train"])
    if kind in ("step", "march"):
        c = {"kind": kind, "ni": 2 * size(32, 256), "nj": size(16, 128), "split": rng.choice([0.0, 0.0, 0.3, 0.5]),
             "scheme": rng.choice(sorted(SCHEMES)), "fp32op": rng.random() < 0.5}
        if kind == "march":
            c["steps"] = rng.randint(2, 8)
        return c
    if kind == "batch":
        return {"kind": "batch", "n": rng.randint(2, 31), "scheme": "first", "fp32op": rng.random() < 0.8, "steps": rng.randint(2, 4)}
    if kind == "tridag4":
        return {"kind": "tridag4", "ni": size(3, 512), "nj": size(3, 96)}
    if kind == "tridag5":
        return {"kind": "tridag5", "lines": size(1, 4099), "rows": size(3, 33), "periodic": rng.random() < 0.5}
    if kind == "roe":
        return {"kind": "roe", "n": size(500, 164399)}
    if kind == "recon":
        return {"kind": "recon", "scheme": rng.choice(["weno", "muscl"]), "lines": size(1, 128), "imax": size(9, 518), "nq": rng.choice([4, 4, 5])}
    if kind == "forward":
        return {"kind": "forward", "n": size(100, 65500), "capacity": 16384}
    return {"kind": "train", "n": size(4096, 262144), "batch": 128 * size(4, 128), "steps": rng.randint(1, 4)}


# ---------------------------------------------------------------- meshes and states
_cases, _inputs = {}, {}


def _mesh(ni, nj, split):
    """The mesh read as a case of the framework: a user's program has it on disk and reads it once."""
    key = (ni, nj, split)
    if key not in _cases:
        with tempfile.TemporaryDirectory() as d:
            meshgen.make_case(d, ni, nj, order=3, CFL=10.0, msweep=2, nsteps=1, split=split, seed=0)
            c = native.Case(d)
        x = c.get("x").reshape(-1, 2)
        f = c.get_int("faces").reshape(-1, 6)
        _cases[key] = c
        m = {"x": x, "faces": f, "start": c.get_int("faceStartPerChain"), "conn": c.get_int("chainConn"), "nc": c.sizes["nCell"]}
        m["centres"] = _centres(m)
        m["wall"] = _wall(m)
        _inputs[key] = m
    return _cases[key], _inputs[key]


def _centres(m):
    f, mid = m["faces"], 0.5 * (m["x"][m["faces"][:, 0]] + m["x"][m["faces"][:, 1]])
    acc, cnt = np.zeros((m["nc"], 2)), np.zeros(m["nc"])
    for cells in (f[:, 2], f[:, 4]):
        ok = cells >= 0
        for k in (0, 1):
            acc[:, k] += np.bincount(cells[ok], mid[ok, k], minlength=m["nc"])
        cnt += np.bincount(cells[ok], minlength=m["nc"])
    return acc / cnt[:, None]


def _wall(m):
    """Each cell's distance to the nearest wall face, and that face's unit normal."""
    f = m["faces"][m["faces"][:, 4] == -2]
    a, b = m["x"][f[:, 0]], m["x"][f[:, 1]]
    n = np.stack([b[:, 1] - a[:, 1], a[:, 0] - b[:, 0]], 1)
    n /= np.hypot(n[:, 0], n[:, 1])[:, None]
    mid, d, k = 0.5 * (a + b), [], []
    for part in np.array_split(m["centres"], 1 + m["nc"] // 8192):
        r = np.hypot(part[:, :1] - mid[None, :, 0], part[:, 1:] - mid[None, :, 1])
        k.append(r.argmin(1))
        d.append(r.min(1))
    return np.concatenate(d), n[np.concatenate(k)]


def _flow(case, rng):
    """Mach and angle of attack (degrees) around the benchmark's."""
    mach = 0.8 if case["scheme"] == "vanalbada" and case["fp32op"] else 0.5
    return mach + rng.uniform(-0.02, 0.02), 1.25 + rng.uniform(-0.25, 0.25)


def _state(m, mach, alpha, rng):
    """A developed-looking conserved state: the freestream turned along the wall near it, smooth modes that decay outwards,
    cell noise."""
    c, (d, n) = m["centres"], m["wall"]
    near = np.exp(-d)

    def modes():
        s = np.zeros(m["nc"])
        for _ in range(4):
            k = rng.uniform(-3.0, 3.0, 2)
            s += np.sin(c @ k + rng.uniform(0, 2 * np.pi))
        return 0.25 * s * near + 2e-5 * rng.standard_normal(m["nc"])
    a = math.radians(alpha)
    turn = np.exp(-d / 0.2) * (math.cos(a) * n[:, 0] + math.sin(a) * n[:, 1])
    rho = 1.0 + 0.01 * modes()
    u = mach * (math.cos(a) - turn * n[:, 0]) + 0.01 * modes()
    v = mach * (math.sin(a) - turn * n[:, 1]) + 0.01 * modes()
    p = (1.0 + 0.01 * modes()) / GAMMA
    return np.ascontiguousarray(np.stack([rho, rho * u, rho * v, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)], axis=1))


def _solver_inputs(case, seed):
    """[(mesh key, Mach, alpha, q)] of a solver case."""
    rng = np.random.default_rng(seed)
    if case["kind"] != "batch":
        m = (case["ni"], case["nj"], case["split"])
        mach, alpha = _flow(case, rng)
        return [(m, mach, alpha, _state(_mesh(*m)[1], mach, alpha, rng))]
    got = []
    for k in range(case["n"]):
        m = BATCH_MESHES[k % 4] + (0.0,)
        mach, alpha = rng.uniform(0.3, 0.85), rng.uniform(-2.0, 4.0)
        got.append((m, mach, alpha, _state(_mesh(*m)[1], mach, alpha, rng)))
    return got


def _configured(m, case, mach, alpha):
    order, limiter, _ = SCHEMES[case["scheme"]]
    c = _mesh(*m)[0].clone()
    c.set_run(order, 2, _cfl(case))
    c.set_option("limiter", limiter)
    c.set_option("chain_end_rule", native.END_RULE_EXTENDED if m[2] > 0 else native.END_RULE_REFERENCE)
    c.set_flow(mach, alpha)
    return c


def _pinned(a):
    t = torch.empty(a.size, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    n = t.numpy()
    n[:] = a.ravel()
    return n


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(shape, generator=g, device=DEV, dtype=torch.float64)


def _blocks(g, lines, rows, nq):
    """Rows of an implicit step at a moderate CFL number: I + dt * (couplings), the couplings of flux-Jacobian size."""
    def r(scale):
        return scale * torch.randn((lines, rows, nq, nq), generator=g, device=DEV, dtype=torch.float64)
    eye = torch.eye(nq, device=DEV, dtype=torch.float64)
    return r(0.6), r(0.6) + 6.0 * eye, r(0.6), torch.randn((lines, rows, nq), generator=g, device=DEV, dtype=torch.float64)


def _faces(case, seed):
    g, n = _gen(seed), case["n"]
    ang, mag = _uniform(g, 0, 2 * math.pi, n), 10.0 ** _uniform(g, -3, 0, n)
    nxy = torch.stack([mag * torch.cos(ang), mag * torch.sin(ang)], 1).contiguous()

    def state():
        rho, u, v, p = _uniform(g, 0.4, 1.6, n), _uniform(g, -0.9, 0.9, n), _uniform(g, -0.9, 0.9, n), _uniform(g, 0.3, 1.3, n)
        return torch.stack([rho, rho * u, rho * v, p / (GAMMA - 1) + 0.5 * rho * (u * u + v * v)], 1).contiguous()
    return nxy, state(), state()


def _lines(case, seed):
    g, s = _gen(seed), (case["lines"], case["imax"], case["nq"])
    x = torch.linspace(0, 1, s[1], device=DEV, dtype=torch.float64)[None, :, None]
    f = 1.0 + 0.3 * torch.sin(6.0 * x + _uniform(g, 0, 6, s[0], 1, s[2])) + 0.2 * (x > _uniform(g, 0.2, 0.8, s[0], 1, s[2]))
    f = f + 1e-3 * torch.randn(s, generator=g, device=DEV, dtype=torch.float64)
    return f.contiguous(), 1e-3 * torch.randn(s, generator=g, device=DEV, dtype=torch.float64)


def _net_inputs(case, seed):
    """Parameters (the framework's order), features and targets shaped like those warmstart makes."""
    g = _gen(seed)
    p = []
    for rows, fan in ((256, 5), (256, 256), (256, 256), (4, 256)):
        p += [_uniform(g, -1, 1, rows * fan) / math.sqrt(fan), 0.1 * _uniform(g, -1, 1, rows)]
    params = torch.cat(p).float()
    n = case["n"]
    feat = torch.stack([_uniform(g, -1.7, 1.7, n), _uniform(g, -1.7, 1.7, n), _uniform(g, -1, 1, n), _uniform(g, -1, 1, n),
                        _uniform(g, -1, 1.7, n)], 1).float().contiguous()
    f = feat.double()
    targ = torch.stack([torch.tanh(f[:, 0] + f[:, 4]), torch.sin(2 * f[:, 2]) * f[:, 1], f[:, 3] * torch.exp(-f[:, 4]), f[:, 0] * f[:, 2]], 1)
    return params.cpu().numpy(), feat, targ.float().contiguous()


# ---------------------------------------------------------------- what a program has in hand, and its call
def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("step", "march", "batch"):
        ins = _solver_inputs(case, seed)
        cs = [_configured(m, case, mach, alpha) for m, mach, alpha, _ in ins]
        g = native.GpuSolver.batch(cs) if kind == "batch" else native.GpuSolver(cs[0])
        g.set_precision(case["fp32op"])
        q = np.concatenate([i[3].ravel() for i in ins])
        s.update(solver=g, q=_pinned(q), q_out=_pinned(q))
    elif kind == "tridag4":
        g = _gen(seed)
        s.update(open=_blocks(g, case["ni"], case["nj"], 4), closed=_blocks(g, case["nj"], case["ni"], 4))
    elif kind == "tridag5":
        s.update(blocks=_blocks(_gen(seed), case["lines"], case["rows"], 5))
    elif kind == "roe":
        s.update(faces=_faces(case, seed))
    elif kind == "recon":
        f, dq = _lines(case, seed)
        s.update(f=f, dq=dq, out=[torch.zeros_like(f) for _ in range(6)])
    else:
        params, feat, targ = _net_inputs(case, seed)
        net = native.Mlp(batch_capacity=case["capacity"] if kind == "forward" else case["batch"], seed=1)
        net.set_params(params)
        s.update(net=net, feat=feat, targ=targ, seed=seed + 1, at=0)
        torch.cuda.synchronize()   # the network works on a stream of its own
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        # the norms that a march stops on; the plain form's linear norms are exact as well
        norms = s["solver"].step_host(s["q"], s["q_out"])
        return [s["q_out"], norms[:2] if case["fp32op"] else norms]
    if kind in ("march", "batch"):
        g = s["solver"]
        g.set("q", s["q"])
        hist, _ = g.march(case["steps"], 0.0)
        g.get("q", s["q_out"])
        return [s["q_out"], hist[..., :2] if case["fp32op"] else hist]
    if kind == "tridag4":
        out = []
        for (A, B, C, F), periodic in ((s["open"], False), (s["closed"], True)):
            x = F.clone()
            native.block_tridag4(A, B, C, x, periodic)
            out.append(x)
        return out
    if kind == "tridag5":
        A, B, C, F = (t.clone() for t in s["blocks"])   # solved in place, the blocks become scratch
        native.block_tridag5(A, B, C, F, case["periodic"])
        return [F, A, B, C]
    if kind == "roe":
        return [*native.flux_roe2d(*s["faces"], gamma=GAMMA), *native.jacobian_roe2d(*s["faces"], gamma=GAMMA)]
    if kind == "recon":
        ql, qr, f2, dql, dqr, df2 = s["out"]
        n = case["imax"]
        if case["scheme"] == "weno":
            native.reconstruct("weno", s["f"], ql, qr, 2, n - 1, eps=1e-10)
            native.reconstruct("weno_deriv", s["f"], dql, dqr, 2, n - 1, dq=s["dq"], eps=1e-10)
            return [ql, qr, dql, dqr]
        native.reconstruct("muscl", s["f"], ql, qr, 1, n - 2, f2=f2)
        native.reconstruct("muscl_deriv", s["f"], dql, dqr, 1, n - 2, dq=s["dq"], f2=df2)
        return [ql, qr, f2, dql, dqr, df2]
    if kind == "forward":
        return s["net"].forward(s["feat"])
    losses = []
    for _ in range(case["steps"]):
        losses.append(s["net"].train_step(s["feat"], s["targ"], batch=case["batch"], seed=s["seed"], step=s["at"], lr=2e-3))
        s["at"] += 1
    # the network computes in FP32: so is its loss
    return [np.array(losses, dtype=np.float32), s["net"].get_params()]


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind in ("step", "march", "batch"):
        if kind == "batch":
            nc = sum(BATCH_MESHES[k % 4][0] * BATCH_MESHES[k % 4][1] for k in range(case["n"]))
            nf = 2 * nc
        else:
            quads = case["ni"] * case["nj"]
            nc, nf = quads * (1 + case["split"]), quads * (2 + case["split"])
        steps = case.get("steps", 1)
        # per face: reconstruction, Roe flux, Jacobians, two linearised residuals; per cell: two line solves (block LU
        # and substitutions of two chains on quads), the sums and updates
        recon = {"first": 0, "weno": 8 * 62}.get(case["scheme"], 8 * 14)
        lin = {"first": 0, "weno": 8 * 110}.get(case["scheme"], 8 * 30)
        flops = steps * (nf * (recon + 140 + 420 + 2 * (lin + 64)) + 2 * nc * (2 * 290 + 2 * 128) + 40 * nc)
        # in: q, each face's normal, cells and place in its chain; out: q
        return {"bytes": steps * (64 * nc + 40 * nf), "flops": flops}
    if kind == "tridag4":
        rows = case["ni"] * case["nj"]
        return {"bytes": 2 * rows * (48 + 8) * 8, "flops": rows * (290 + 128 + 290 + 360 + 128)}
    if kind == "tridag5":
        rows = case["lines"] * case["rows"]
        return {"bytes": rows * 2 * (75 + 5) * 8, "flops": rows * (1000 if case["periodic"] else 560)}
    if kind == "roe":
        return {"bytes": case["n"] * (10 * 8 + 5 * 8 + 32 * 8), "flops": case["n"] * 560}
    if kind == "recon":
        v = case["lines"] * case["imax"] * case["nq"]
        return {"bytes": v * 8 * (6 if case["scheme"] == "weno" else 8), "flops": v * (2 * 62 + 2 * 170 if case["scheme"] == "weno" else 2 * 14 + 2 * 30)}
    macs = 5 * 256 + 2 * 256 * 256 + 256 * 4
    if kind == "forward":
        return {"bytes": case["n"] * 36 + 2 * macs, "flops": 2 * macs * case["n"]}
    return {"bytes": case["steps"] * (case["batch"] * 36 + macs * 28), "flops": case["steps"] * 6 * macs * case["batch"]}


# ---------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "march", "batch"):
        ins = _solver_inputs(case, seed)
        if case.get("steps", 1) * sum(len(i[3]) for i in ins) > 600000:
            return None
        qs, hists = zip(*(_march64(case, *i) for i in ins))
        hist = np.stack(hists, 1) if kind == "batch" else hists[0]
        if case["fp32op"]:
            hist = hist[..., :2]
        return [np.concatenate([q.ravel() for q in qs]), hist[0] if kind == "step" else hist]
    if kind == "tridag4":
        g = _gen(seed)
        a, b = _blocks(g, case["ni"], case["nj"], 4), _blocks(g, case["nj"], case["ni"], 4)
        return [_tridag64(*a, False), _tridag64(*b, True)]
    if kind == "tridag5":
        return [_tridag64(*_blocks(_gen(seed), case["lines"], case["rows"], 5), case["periodic"]), None, None, None]
    if kind == "roe":
        nxy, l, r = _faces(case, seed)
        flux, spec, lm, rm = _roe64(nxy, l, r)
        return [flux, spec, lm, rm]
    if kind == "recon":
        f, dq = _lines(case, seed)
        n, z = case["imax"], torch.zeros_like(f)
        if case["scheme"] == "weno":
            outs = [z.clone() for _ in range(4)]
            v, dv = [f[:, k:n - 4 + k] for k in range(5)], [dq[:, k:n - 4 + k] for k in range(5)]
            for o, x in zip(outs, (_weno(v, 1e-15), _weno(v[::-1], 1e-15), _weno_d(v, dv, 1e-10), _weno_d(v[::-1], dv[::-1], 1e-10))):
                o[:, 2:n - 2] = x
            return outs
        outs = [z.clone() for _ in range(6)]
        a, b, da, db = f[:, 1:-1] - f[:, :-2], f[:, 2:] - f[:, 1:-1], dq[:, 1:-1] - dq[:, :-2], dq[:, 2:] - dq[:, 1:-1]
        (outs[0][:, 1:-1], outs[1][:, 1:-1]), (outs[3][:, 1:-1], outs[4][:, 1:-1]) = _muscl(0, f[:, 1:-1], a, b), _muscl_d(0, dq[:, 1:-1], a, b, da, db)
        outs[2][:, :-1] = outs[5][:, :-1] = f[:, 1:] - f[:, :-1]
        return outs
    return _net64(case, seed)


# --- reconstructions (values, and derivatives in the direction d*)
def _muscl(lim, f, a, b):
    """Left- and right-face values of a cell from its value and differences to both sides: the kappa = 1/3 scheme."""
    th, eps = 1.0 / 3.0, 1e-10
    if lim == 0:
        s = 3 * (a * b + eps) / (2 * (b - a) ** 2 + 3 * (a * b + eps))
        return f + 0.25 * s * ((1 - th) * a + (1 + th) * b), f - 0.25 * s * ((1 + th) * a + (1 - th) * b)
    if lim == 1:
        p, q = _minmod(a, 4 * b, a, 4 * b), _minmod(b, 4 * a, b, 4 * a)
        return f + 0.25 * ((1 - th) * p + (1 + th) * q), f - 0.25 * ((1 + th) * p + (1 - th) * q)
    s = (2 * a * b + eps) / (a * a + b * b + eps)
    return (f + 0.25 * s * ((1 - th * s) * a + (1 + th * s) * b), f - 0.25 * s * ((1 + th * s) * a + (1 - th * s) * b))


def _minmod(x, y, u, v):
    """u where minmod(x, y) is x, v where it is y, else 0."""
    return torch.where(x * y > 0, torch.where(x.abs() <= y.abs(), u, v), torch.zeros_like(x))


def _muscl_d(lim, df, a, b, da, db):
    th, eps = 1.0 / 3.0, 1e-10
    if lim == 1:
        p, q = _minmod(a, 4 * b, da, 4 * db), _minmod(b, 4 * a, db, 4 * da)
        return df + 0.25 * ((1 - th) * p + (1 + th) * q), df - 0.25 * ((1 + th) * p + (1 - th) * q)
    if lim == 0:
        num, dnum = 3 * (a * b + eps), 3 * (da * b + a * db)
        den, dden = 2 * (b - a) ** 2 + num, 4 * (b - a) * (db - da) + dnum
        s, ds, k, dk = num / den, dnum / den - num * dden / den ** 2, th, 0.0
    else:
        num, dnum = 2 * a * b + eps, 2 * (da * b + a * db)
        den, dden = a * a + b * b + eps, 2 * (a * da + b * db)
        s, ds = num / den, dnum / den - num * dden / den ** 2
        k, dk = th * s, th * ds
    up, dup = (1 - k) * a + (1 + k) * b, (1 - k) * da + (1 + k) * db + dk * (b - a)
    dn, ddn = (1 + k) * a + (1 - k) * b, (1 + k) * da + (1 - k) * db + dk * (a - b)
    return df + 0.25 * (ds * up + s * dup), df - 0.25 * (ds * dn + s * ddn)


def _weno_parts(v, eps):
    a, b, c, d, e = v
    t = ((a - 2 * b + c, a - 4 * b + 3 * c), (b - 2 * c + d, b - d), (c - 2 * d + e, 3 * c - 4 * d + e))
    beta = [13 / 12 * x * x + 0.25 * y * y + eps for x, y in t]
    q = ((2 * a - 7 * b + 11 * c) / 6, (-b + 5 * c + 2 * d) / 6, (2 * c + 5 * d - e) / 6)
    up = (beta[1] * beta[2], 6 * beta[0] * beta[2], 3 * beta[0] * beta[1])
    return t, beta, q, up


def _weno(v, eps):
    _, _, q, up = _weno_parts(v, eps)
    return (up[0] * q[0] + up[1] * q[1] + up[2] * q[2]) / (up[0] + up[1] + up[2])


def _weno_d(v, dv, eps):
    t, beta, q, up = _weno_parts(v, eps)
    dt, _, dq, _ = _weno_parts(dv, 0.0)
    db = [13 / 6 * x * dx + 0.5 * y * dy for (x, y), (dx, dy) in zip(t, dt)]
    dup = (db[1] * beta[2] + beta[1] * db[2], 6 * (db[0] * beta[2] + beta[0] * db[2]), 3 * (db[0] * beta[1] + beta[0] * db[1]))
    down, ddown = up[0] + up[1] + up[2], dup[0] + dup[1] + dup[2]
    return sum(u / down * y + (du * down - u * ddown) / down ** 2 * x for u, du, x, y in zip(up, dup, q, dq))


# --- Roe flux and its Jacobians with frozen eigenvalues and averages
def _roe64(nxy, ql, qr):
    gm1 = GAMMA - 1
    area = nxy.norm(dim=1)
    nx, ny = nxy[:, 0] / area, nxy[:, 1] / area

    def prim(q):
        r, u, v = q[:, 0], q[:, 1] / q[:, 0], q[:, 2] / q[:, 0]
        p = gm1 * (q[:, 3] - 0.5 * r * (u * u + v * v))
        return r, u, v, p, (q[:, 3] + p) / r, u * nx + v * ny
    (rl, ul, vl, pl, hl, cl), (rr, ur, vr, pr, hr, cr) = prim(ql), prim(qr)
    w = torch.sqrt(rr / rl)
    rb, u, v, h = rl * w, (ul + w * ur) / (1 + w), (vl + w * vr) / (1 + w), (hl + w * hr) / (1 + w)
    c, un = torch.sqrt(gm1 * (h - 0.5 * (u * u + v * v))), u * nx + v * ny
    e1, e2, e3 = un.abs(), (un + c).abs(), (un - c).abs()
    t1, t2 = -e1 + 0.5 * (e2 + e3), 0.5 * (e2 - e3)
    zero, one = torch.zeros_like(c), torch.ones_like(c)
    k1, k2 = torch.stack([one, u, v, h], 1), torch.stack([zero, nx, ny, un], 1)
    d1 = t1 * (pr - pl) / c ** 2 + t2 * rb * (cr - cl) / c
    d2 = t1 * rb * (cr - cl) + t2 * (pr - pl) / c

    def native_flux(q, r, uu, vv, p, hh, cc):
        return torch.stack([r * cc, r * cc * uu + nx * p, r * cc * vv + ny * p, r * cc * hh], 1)
    diss = e1[:, None] * (qr - ql) + d1[:, None] * k1 + d2[:, None] * k2
    flux = 0.5 * (native_flux(ql, rl, ul, vl, pl, hl, cl) + native_flux(qr, rr, ur, vr, pr, hr, cr) - diss) * area[:, None]

    def side(r, uu, vv, p, hh, cc, sign):
        dc = torch.stack([-cc / r, nx / r, ny / r, zero], 1)
        dp = torch.stack([0.5 * gm1 * (uu * uu + vv * vv), -gm1 * uu, -gm1 * vv, gm1 * one], 1)
        w4 = torch.stack([one, uu, vv, hh], 1)
        A = torch.einsum("n,nc,nr->nrc", r, dc, w4) + torch.einsum("nr,nc->nrc", torch.stack([zero, nx, ny, cc], 1), dp)
        A = A + cc[:, None, None] * torch.eye(4, device=r.device, dtype=r.dtype)
        # the mass flux's own derivative moves the velocities: row k gains -U w_k on the density, and the energy row its E
        A[:, 0, 0] = cc + r * dc[:, 0]
        A[:, 1, 0] = cc * uu + r * dc[:, 0] * uu - cc * uu + nx * dp[:, 0]
        A[:, 2, 0] = cc * vv + r * dc[:, 0] * vv - cc * vv + ny * dp[:, 0]
        D1 = (t1 / c ** 2)[:, None] * dp + (t2 * rb / c)[:, None] * dc
        D2 = (t1 * rb)[:, None] * dc + (t2 / c)[:, None] * dp
        M = e1[:, None, None] * torch.eye(4, device=r.device, dtype=r.dtype) + torch.einsum("nr,nc->nrc", k1, D1) + torch.einsum("nr,nc->nrc", k2, D2)
        return 0.5 * (A - sign * M) * area[:, None, None]
    return flux, (e1 + c) * area, side(rl, ul, vl, pl, hl, cl, -1.0), side(rr, ur, vr, pr, hr, cr, 1.0)


# --- block-tridiagonal lines [lines][rows]
def _tridag64(A, B, C, F, periodic):
    n, nq = F.shape[1], F.shape[2]
    if not periodic:
        return _open64(A, B, C, F[..., None])[..., 0]
    # the last row's unknown by itself: the others respond to it through the two couplings around the loop
    rhs = torch.zeros(F.shape[0], n - 1, nq, nq + 1, device=F.device, dtype=F.dtype)
    rhs[..., 0] = F[:, :-1]
    rhs[:, 0, :, 1:] -= A[:, 0]
    rhs[:, -1, :, 1:] -= C[:, n - 2]
    y = _open64(A[:, :-1], B[:, :-1], C[:, :-1], rhs)
    S = B[:, -1] + C[:, -1] @ y[:, 0, :, 1:] + A[:, -1] @ y[:, -1, :, 1:]
    f = F[:, -1, :, None] - C[:, -1] @ y[:, 0, :, :1] - A[:, -1] @ y[:, -1, :, :1]
    last = torch.linalg.solve(S, f)
    x = y[..., :1] + y[..., 1:] @ last[:, None]
    return torch.cat([x, last[:, None]], 1)[..., 0]


def _open64(A, B, C, F):
    n, m = F.shape[1], F.shape[3]
    g, y, D, f = [], [], B[:, 0], F[:, 0]
    for i in range(n):
        if i:
            D, f = B[:, i] - A[:, i] @ g[-1], F[:, i] - A[:, i] @ y[-1]
        s = torch.linalg.solve(D, torch.cat([C[:, i], f], -1))
        g.append(s[..., :-m])
        y.append(s[..., -m:])
    for i in range(n - 2, -1, -1):
        y[i] = y[i] - g[i] @ y[i + 1]
    return torch.stack(y, 1)


# --- the implicit step
class _Step64:
    """Indices of a mesh for the step: per processed face its stencil of six entries (entry 2 and 3 at the face) and the
    sides, per chain its rows."""

    def __init__(self, m):
        f, start, conn = m["faces"], m["start"], m["conn"]
        left, right = f[:, 2], f[:, 4]
        sten, at, face, swap, nsten, self.order = [], [], [], [], 0, []
        first, last_end = np.full(m["nc"], -1), []
        for k in range(len(start) - 1):
            fs = conn[start[k]:start[k + 1]]
            closed = fs[0] == fs[-1]
            cells = left[fs[:-1]]
            if closed:
                idx = np.concatenate([cells[-3:], cells, cells[:3]])
                wall = np.full(idx.size, -1)
                fs = fs[:-1]
            else:
                n = cells.size
                def ghost(face_, inner):
                    r = right[face_]
                    return (np.full(3, r), np.full(3, -1)) if r >= 0 else (inner, np.full(3, face_)) if r == -2 else (np.full(3, -1), np.full(3, -1))
                g0, w0 = ghost(fs[0], cells[np.minimum(np.arange(3), n - 1)][::-1])
                g1, w1 = ghost(fs[-1], cells[n - 1 - np.minimum(np.arange(3), n - 1)])
                idx, wall = np.concatenate([g0, cells, g1]), np.concatenate([w0, np.full(n, -1), w1])
                last_end += [fs[0], fs[-1]]
            sten.append(np.stack([idx, wall], 1))
            at.append(nsten + np.arange(fs.size))
            nsten += idx.size
            face.append(fs)
            sw = np.zeros(fs.size, bool)
            sw[-1] = not closed
            swap.append(sw)
            new = cells[first[cells] < 0]
            first[new] = k
            self.order.append((bool(closed), cells, fs))
        t = lambda a: torch.from_numpy(np.ascontiguousarray(np.concatenate(a) if isinstance(a, list) else a)).to(DEV)  # noqa: E731
        self.sten, self.at, self.face, self.swap = t(sten).long(), t(at).long(), t(face).long(), t(swap)
        nx = m["x"][f[:, 1]] - m["x"][f[:, 0]]
        n = np.stack([nx[:, 1], -nx[:, 0]], 1)
        u = n / np.hypot(n[:, 0], n[:, 1])[:, None]
        self.normal, self.unit = t(n), t(u)
        self.left, self.right = t(left).long(), t(right).long()
        self.nc = m["nc"]
        # faces that end an open chain inside the mesh: their diagonal term goes to the first chain through the cell beyond
        ends = np.unique([e for e in last_end if right[e] >= 0]).astype(np.int64)
        extra = {}
        for e in ends:
            extra.setdefault(int(right[e]), []).append(int(e))
        # waves of chains that share no cell, in file order
        wave, self.waves = np.full(m["nc"], -1), {}
        for k, (closed, cells, fs) in enumerate(self.order):
            w = wave[cells].max() + 1
            wave[cells] = w
            self.waves.setdefault(w, {}).setdefault((closed, cells.size), []).append(k)
        self.plan = []
        for w in sorted(self.waves):
            for (closed, n), ks in self.waves[w].items():
                cells = np.stack([self.order[k][1] for k in ks])
                fs = np.stack([self.order[k][2] for k in ks])
                ex = [(i, r, e) for i, k in enumerate(ks) for r, c in enumerate(self.order[k][1]) if first[c] == k for e in extra.get(int(c), ())]
                ex = np.array(ex, dtype=np.int64).reshape(-1, 3)
                self.plan.append((closed, t(cells).long(), t(fs).long(), t(ex)))

    def gather(self, q, fs):
        """[stencil entries][4], ghosts by the end's kind: a mirror image at walls, `fs` at the far field."""
        c, w = self.sten[:, 0], self.sten[:, 1]
        v = q[c.clamp(min=0)]
        mir = w >= 0
        u = self.unit[w.clamp(min=0)]
        vn = v[:, 1] * u[:, 0] + v[:, 2] * u[:, 1]
        v[:, 1] -= torch.where(mir, 2 * vn * u[:, 0], torch.zeros_like(vn))
        v[:, 2] -= torch.where(mir, 2 * vn * u[:, 1], torch.zeros_like(vn))
        return torch.where((c < 0)[:, None], fs[None, :], v)

    def sides(self, scheme, v, d=None):
        """States (or, with d, their derivatives) left and right of each face."""
        order, lim, _ = SCHEMES[scheme]
        s = [v[self.at + k] for k in range(6)]
        ds = None if d is None else [d[self.at + k] for k in range(6)]
        if order == 1:
            lo, hi = (s if d is None else ds)[2:4]
        elif order == 3:
            a = (s[2], s[2] - s[1], s[3] - s[2])
            b = (s[3], s[3] - s[2], s[4] - s[3])
            if d is None:
                lo, hi = _muscl(lim, *a)[0], _muscl(lim, *b)[1]
            else:
                lo = _muscl_d(lim, ds[2], *a[1:], ds[2] - ds[1], ds[3] - ds[2])[0]
                hi = _muscl_d(lim, ds[3], *b[1:], ds[3] - ds[2], ds[4] - ds[3])[1]
        elif d is None:
            lo, hi = _weno(s[:5], 1e-15), _weno(s[5:0:-1], 1e-15)
        else:
            lo, hi = _weno_d(s[:5], ds[:5], 1e-10), _weno_d(s[5:0:-1], ds[5:0:-1], 1e-10)
        return torch.where(self.swap[:, None], lo, hi), torch.where(self.swap[:, None], hi, lo)

    def scatter(self, flux, scale=None):
        """Sum over each cell's faces of -flux (left cell) and +flux (right cell), with the cell's scale."""
        l, r = self.left[self.face], self.right[self.face]
        out = torch.zeros((self.nc, flux.shape[1]), device=flux.device, dtype=flux.dtype)
        out.index_add_(0, l, -flux)
        ok = r >= 0
        out.index_add_(0, r[ok], flux[ok])
        return out if scale is None else out * scale[:, None]

    def step(self, scheme, cfl, q, fs, msweep=2):
        v = self.gather(q, fs)
        L, R = self.sides(scheme, v)
        flux, spec, lm, rm = _roe64(self.normal[self.face], L, R)
        r = self.scatter(flux)
        l, rt = self.left[self.face], self.right[self.face]
        sig = torch.zeros(self.nc, device=q.device, dtype=q.dtype).index_add_(0, l, spec)
        sig.index_add_(0, rt[rt >= 0], spec[rt >= 0])
        norms = [r[:, 0].norm() / self.nc, r[:, 0].abs().max()]
        dt = cfl / sig
        LM = torch.zeros((self.normal.shape[0], 4, 4), device=q.device, dtype=q.dtype)
        RM = LM.clone()
        LM[self.face], RM[self.face] = lm, rm
        r0 = r * dt[:, None]
        r, dq = r0.clone(), torch.zeros_like(r0)
        for _ in range(msweep):
            for closed, cells, faces, ex in self.plan:
                A, B, C = self.rows(closed, cells, faces, ex, LM, RM, dt)
                r[cells] = _tridag64(A, B, C, r[cells], closed)
            dq = dq + r
            dL, dR = self.sides(scheme, v, self.gather(dq, torch.zeros_like(fs)))
            g = (lm @ dL[..., None] + rm @ dR[..., None])[..., 0]
            r = r0 - dq + self.scatter(g, dt)
        norms += [r[:, 0].norm() / self.nc, r[:, 0].abs().max()]
        return q + dq, [float(x) for x in norms]

    def rows(self, closed, cells, faces, ex, LM, RM, dt):
        k, n = cells.shape
        A = torch.zeros((k, n, 4, 4), device=dt.device, dtype=dt.dtype)
        B, C = A.clone(), A.clone()
        if closed:   # face i lies between cells i-1 (right) and i (left)
            l, r = LM[faces], RM[faces]
            B += l
            A += r
            B -= r.roll(-1, 1)
            C -= l.roll(-1, 1)
        else:
            l, r = LM[faces[:, :-1]], RM[faces[:, :-1]]
            B += l
            A[:, 1:] += r[:, 1:]
            B[:, :-1] -= r[:, 1:]
            C[:, :-1] -= l[:, 1:]
            B[:, -1] += LM[faces[:, -1]]
            for row, f in ((0, faces[:, 0]), (n - 1, faces[:, -1])):   # a wall mirrors the velocity
                w = (self.right[f] == -2)
                u = self.unit[f]
                M = RM[f].clone()
                mn = M[:, :, 1] * u[:, None, 0] + M[:, :, 2] * u[:, None, 1]
                M[:, :, 1] -= 2 * mn * u[:, None, 0]
                M[:, :, 2] -= 2 * mn * u[:, None, 1]
                B[:, row] += torch.where(w[:, None, None], M, torch.zeros_like(M))
        if len(ex):
            B.index_put_((ex[:, 0], ex[:, 1]), -RM[ex[:, 2]], accumulate=True)
        s = dt[cells][..., None, None]
        return A * s, B * s + torch.eye(4, device=dt.device, dtype=dt.dtype), C * s


_steps = {}


def _march64(case, m, mach, alpha, q):
    if m not in _steps:
        _steps[m] = _Step64(_mesh(*m)[1])
    a = math.radians(alpha)
    u, v = mach * math.cos(a), mach * math.sin(a)
    fs = torch.tensor([1.0, u, v, 1 / GAMMA / (GAMMA - 1) + 0.5 * (u * u + v * v)], device=DEV, dtype=torch.float64)
    q, hist = torch.from_numpy(q).to(DEV), []
    for _ in range(case.get("steps", 1)):
        q, h = _steps[m].step(case["scheme"], _cfl(case), q, fs)
        hist.append(h)
    return q.cpu().numpy(), np.array(hist)


# --- the network and Adam
def _net64(case, seed):
    params, feat, targ = _net_inputs(case, seed)
    p = torch.from_numpy(params).to(DEV).double()
    shapes, w, o = ((256, 5), (256,), (256, 256), (256,), (256, 256), (256,), (4, 256), (4,)), [], 0
    for s in shapes:
        w.append(p[o:o + math.prod(s)].reshape(s).clone().requires_grad_())
        o += math.prod(s)

    def net(x):
        for k in range(0, 6, 2):
            x = torch.nn.functional.gelu(x @ w[k].T + w[k + 1])
        return x @ w[6].T + w[7]
    if case["kind"] == "forward":
        with torch.no_grad():
            return net(feat.double())
    opt, losses = torch.optim.Adam(w, lr=2e-3), []
    mask = (1 << 64) - 1

    def mix(x):   # splitmix64's finaliser, as the framework draws its minibatches
        x = (x + np.uint64(0x9E3779B97F4A7C15))
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return x ^ (x >> np.uint64(31))
    for k in range(case["steps"]):
        i = np.arange(case["batch"], dtype=np.uint64) + np.uint64(k * 0x100000001 & mask)
        rows = torch.from_numpy((mix(np.uint64(seed + 1) ^ mix(i)) % np.uint64(case["n"])).astype(np.int64)).to(DEV)
        loss = ((net(feat[rows].double()) - targ[rows].double()) ** 2).mean()
        opt.zero_grad()
        loss.backward()
        opt.step()
        losses.append(float(loss.detach()))
    return [np.array(losses), torch.cat([t.detach().reshape(-1) for t in w])]
