"""The work that performance is measured on: what a program that uses this library has it do.

Users call the energy/gradient evaluation from their own optimizer (`Solver.objective`, or
`mcg_objective_noalloc` where nothing may be allocated), let the library minimize an increment
(`Solver.minimize`), and evaluate or run many lattices at once (`BatchSolver`), in the FP64 and
in the mixed form.  Sizes are this repository's own workloads (workloads.py, the fixtures and
bench.py) and ragged ones between them; inputs are seeded.

A case holds plain values:
  kind    eval | noalloc | minimize | batch_eval | batch_run
  lattice specimen (the reference's own builder) | cubic | bcc (cubic + body diagonals)
  nx, ny, nz   cells (for a batch: the range of cells per side is lo .. hi, `count` lattices)
  mixed   False: FP64, True: FP32 bulk arithmetic
  trials  the evaluation also returns the beams' trial plastic states
  squeeze evaluation state: affine compression, as a share of the height (0.6: dense contact)
  reuse   True: the default contact skin (a solver's evaluations), False: skin 0, every
          evaluation builds its candidate list (a single evaluation of a new state)
  strain, iterations   minimize: platen travel / height and the iteration cap
  strain, steps        batch_run: compression in `steps` increments after the settling one
"""
import ctypes as C
import math

import numpy as np
import torch

import falling_dice_gb300 as fd
from falling_dice_gb300 import abi, workloads

LARGEST_BEAMS = 3.0e6
COARSE = 0.1  # gradient rms (N) that ends an increment of a sweep's first, coarse pass


def listed():
    e = dict(kind="eval", lattice="bcc", mixed=False, trials=False, squeeze=0.0, reuse=True)
    return [
        # the reference's validation specimen: the smallest call, where launches and latency count
        dict(e, name="specimen_eval", lattice="specimen", nx=2, ny=4, nz=2),
        # a caller with a fixed device-memory budget, on a small ragged lattice
        dict(e, name="small_noalloc_mixed", kind="noalloc", nx=5, ny=4, nz=6, mixed=True, squeeze=0.05),
        # the final evaluation of an increment: the beams' trial states come back with it
        dict(e, name="cubic6_trials", lattice="cubic", nx=6, ny=6, nz=6, trials=True, squeeze=0.1),
        # one evaluation of an outer optimizer's, mid-size and ragged, compressed
        dict(e, name="ragged_eval", nx=19, ny=15, nz=11, squeeze=0.2),
        # densely compressed 32x32x16 specimen: ~42,000 self-contacts, list reused as in a line search
        dict(e, name="dense32_mixed", nx=32, ny=32, nz=16, mixed=True, squeeze=0.6),
        dict(e, name="dense32_fp64", nx=32, ny=32, nz=16, squeeze=0.6, reuse=False),
        # an increment of the 6x6x6 specimen, and of the 32x32x16 specimen in the mixed form, as far
        # as the iterates do not depend on the order of rounding (they are chaotic beyond ~15)
        dict(kind="minimize", name="cubic6_minimize", lattice="cubic", nx=6, ny=6, nz=6, mixed=False, strain=0.002,
             iterations=12),
        dict(kind="minimize", name="bcc32_minimize_mixed", lattice="bcc", nx=32, ny=32, nz=16, mixed=True,
             strain=0.0015, iterations=12),
        # a design sweep: uneven lattices evaluated together, and a short, coarsely converged load run
        dict(kind="batch_eval", name="sweep_eval", lo=4, hi=16, count=48, mixed=False, squeeze=0.1),
        dict(kind="batch_run", name="sweep_run", lo=3, hi=12, count=16, mixed=False, strain=0.006, steps=2),
        # the throughput specimen at a new state, mixed; and the largest call, FP64
        dict(e, name="bcc64_mixed", nx=64, ny=64, nz=32, mixed=True, reuse=False),
        dict(e, name="large_fp64", nx=80, ny=81, nz=41, reuse=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo - 0.49), math.log(hi + 0.49)))))


def draw(rng):
    kind = rng.choice(["eval", "eval", "eval", "noalloc", "minimize", "batch_eval", "batch_run"])
    mixed = rng.random() < 0.5
    if kind == "batch_eval":
        lo = rng.randint(3, 8)
        return dict(kind=kind, lo=lo, hi=lo + rng.randint(1, 8), count=_log(rng, 2, 64), mixed=mixed,
                    squeeze=rng.uniform(0.0, 0.3))
    if kind == "batch_run":
        return dict(kind=kind, lo=3, hi=rng.randint(4, 12), count=_log(rng, 2, 16), mixed=mixed,
                    strain=rng.uniform(0.003, 0.006), steps=rng.randint(1, 2))
    if kind == "minimize":
        lattice = rng.choice(["cubic", "bcc"])
        top = 24 if lattice == "bcc" else 32
        return dict(kind=kind, lattice=lattice, nx=_log(rng, 3, top), ny=_log(rng, 3, top), nz=_log(rng, 3, top),
                    mixed=mixed, strain=rng.uniform(0.001, 0.003), iterations=rng.randint(5, 9))
    case = dict(kind=kind, lattice=rng.choice(["cubic", "bcc"]), mixed=mixed,
                trials=kind == "eval" and rng.random() < 0.25, reuse=rng.random() < 0.5,
                squeeze=rng.choice([0.0, rng.uniform(0.0, 0.3), rng.uniform(0.3, 0.6)]))
    if kind == "noalloc":
        case.update(squeeze=min(case["squeeze"], 0.1), nx=_log(rng, 2, 7), ny=_log(rng, 2, 7), nz=_log(rng, 2, 7))
        return case
    while True:  # cells log-uniform in number, the three sides up to a factor of two apart
        side = math.exp(rng.uniform(math.log(2.5), math.log(80.0)))
        n = [max(2, int(round(side * 2 ** rng.uniform(-0.5, 0.5)))) for _ in range(3)]
        if 11.5 * n[0] * n[1] * n[2] <= LARGEST_BEAMS * (0.2 if case["squeeze"] > 0.3 else 1.0):
            return dict(case, nx=n[0], ny=n[1], nz=n[2])


# ---- inputs ------------------------------------------------------------------------------
def _rng_seed(case, seed):
    return (seed * 1000003 + 12345) & 0x7FFFFFFF


def _setup(case, seed):
    """(cfg, [lattice], [yield]) of a case."""
    s = _rng_seed(case, seed)
    if case["kind"].startswith("batch"):
        r = np.random.default_rng(s)
        cfg, _ = workloads.bcc((4, 4, 4), max_strain=case.get("strain", 0.3), load_steps=case.get("steps", 1),
                               unload_steps=0, contact_stiffness=workloads.CONTACT_STIFF)
        cfg.precision = abi.MCG_MIXED if case["mixed"] else abi.MCG_FP64
        if case["kind"] == "batch_run":
            cfg.gradient_rms_tolerance, cfg.gradient_max_tolerance = COARSE, 100 * COARSE
            cfg.reaction_relative_tolerance = -1.0
        lats, yields = [], []
        for k in range(case["count"]):
            n = case["lo"] + k * (case["hi"] - case["lo"] + 1) // case["count"]  # sizes spread evenly
            _, spec = workloads.bcc((n, n, n), 0.3e-3, min(0.3e-3 + float(r.uniform(0, 0.1e-3)) * n, 0.7e-3), 0.02,
                                    abi.MCG_RADIUS_GRADED_Y)
            spec.seed = s + 7919 * (k + 1)
            lats.append(fd.generate_lattice(spec, cfg))
            yields.append(float(r.uniform(30e6, 70e6)))
        return cfg, lats, yields
    cells = (case["nx"], case["ny"], case["nz"])
    if case["lattice"] == "specimen":
        cfg = abi.default_config()
        cfg.cells_x, cfg.cells_y, cfg.cells_z = cells
        cfg.seed = s
        spec = abi.LatticeSpec()
        spec.kind = abi.MCG_LATTICE_REFERENCE_BCC
    else:
        cfg, spec = workloads.bcc(cells, contact_stiffness=workloads.CONTACT_STIFF,
                                  max_iterations=case.get("iterations", 800))
        if case["lattice"] == "cubic":
            spec.kind = abi.MCG_LATTICE_CUBIC
        spec.seed = s
    cfg.precision = abi.MCG_MIXED if case["mixed"] else abi.MCG_FP64
    lat = fd.generate_lattice(spec, cfg)
    return cfg, [lat], [cfg.material.yield_]


def _states(case, seed, cfg, lats):
    """Concatenated z and plastic states and the platen heights of an evaluation case."""
    z, pl, tops = [], [], []
    for k, lat in enumerate(lats):
        a, b = fd.random_state(lat, 0.05, 0.1, 0.02, _rng_seed(case, seed) + 31 * k + 7)
        if case["squeeze"] > 0:
            y = lat.x0[1::3]
            a[1::6] -= case["squeeze"] * (y - y.min()) / cfg.translation_scale
            a[lat.locked.astype(bool)] = 0
            tops.append(lat.geometry.top0 - case["squeeze"] * lat.geometry.height + 1e-3)
        else:
            tops.append(lat.geometry.top0 + 0.01)
        z.append(a)
        pl.append(b)
    return np.concatenate(z), np.concatenate(pl), tops


def prepare(case, seed):
    cfg, lats, yields = _setup(case, seed)
    st = {"case": case, "cfg": cfg, "lats": lats}
    if case["kind"].startswith("batch"):
        st["sol"] = fd.BatchSolver(cfg, lats, yields=yields)
    else:
        st["sol"] = fd.Solver(cfg, lats[0])
    if case["kind"] in ("eval", "noalloc", "batch_eval"):
        z, pl, tops = _states(case, seed, cfg, lats)
        st["sol"].set_state(plastic=pl)
        st.update(z=z, tops=np.array(tops), top=tops[0])
        if case["kind"] == "eval" and not case["reuse"]:
            st["sol"].set_contact_skin(0.0)
    elif case["kind"] == "minimize":
        g = lats[0].geometry
        st.update(z=np.zeros(6 * lats[0].n_nodes), top=g.top0 - case["strain"] * g.height)
    else:
        st["rest"] = [np.concatenate([getattr(lat, f) for lat in lats]) for f in ("x0", "r0")]
        st["rest"].append(np.zeros(7 * sum(lat.n_beams for lat in lats)))
    return st


FRAME = ("displacement", "reaction_force", "loading_work", "elastic_energy", "plastic_dissipation", "contact_energy",
         "max_penetration", "mean_plastic_strain", "permanent_set")


def _columns(diags):
    return {k: np.array([d[k] for d in diags]) for k in diags[0]}


def run(state):
    case, sol = state["case"], state["sol"]
    kind = case["kind"]
    if kind == "eval":
        return sol.objective(state["z"], state["top"], case["trials"])
    if kind == "noalloc":
        e, grad, diag = C.c_double(), np.empty(6 * sol.n_nodes), abi.Diag()
        dp = C.POINTER(C.c_double)
        rc = sol.lib.mcg_objective_noalloc(sol.h, state["z"].ctypes.data_as(dp), state["top"], C.byref(e),
                                           grad.ctypes.data_as(dp), C.byref(diag))
        if rc:
            raise fd.MCGError(rc, sol.lib.mcg_last_error(sol.h).decode())
        return {"energy": e.value, "grad": grad, "diag": diag.as_dict()}
    if kind == "minimize":
        z, st, energy, diag = sol.minimize(state["top"], state["z"])
        # the mixed form's iterates carry single precision
        t = np.float32 if case["mixed"] else np.float64
        return {"z": z.astype(t), "energy": t(energy), "diag": {k: t(v) for k, v in diag.items() if k != "contacts"},
                "converged": st["converged"]}
    if kind == "batch_eval":
        out = sol.objective(state["z"], state["tops"])
        return dict(out, diag=_columns(out["diag"]))
    sol.set_state(*state["rest"])  # a run starts from the rest state
    status, runs = sol.run()
    t = np.float32 if case["mixed"] else np.float64
    base_x, base_r, plastic = (v.astype(t) for v in sol.get_state())
    frames = np.concatenate([np.array([[f[k] for k in FRAME] for f in fr], t) for fr in runs])
    return {"status": status, "frames": frames, "base_x": base_x, "base_r": base_r, "plastic": plastic}


# ---- what a pass cannot do without ---------------------------------------------------------
def _counts(case):
    if case["kind"].startswith("batch"):
        sides = [case["lo"] + k * (case["hi"] - case["lo"] + 1) // case["count"] for k in range(case["count"])]
        boxes = [(n, n, n) for n in sides]
    else:
        boxes = [(case["nx"], case["ny"], case["nz"])]
    nodes = beams = 0
    for a, b, c in boxes:
        grid = (a + 1) * (b + 1) * (c + 1)
        edges = a * (b + 1) * (c + 1) + (a + 1) * b * (c + 1) + (a + 1) * (b + 1) * c
        kind = case.get("lattice", "bcc")
        if kind == "specimen":  # elements_per_strut elements per strut, interior nodes
            struts = 8 * a * b * c + 2 * (a * (c + 1) + (a + 1) * c)
            nodes += grid + a * b * c + 2 * struts
            beams += 3 * struts
        else:
            nodes += grid + (a * b * c if kind == "bcc" else 0)
            beams += edges + (8 * a * b * c if kind == "bcc" else 0)
    return nodes, beams


def work(case):
    """Bytes: end indices and 15 reals per beam (and its 14 trial values and 3 flags where asked
    for); z, base state, mass, gradient and locks per node.  Operations: about 260 per beam and
    90 per node; self-contact and the solver's vectors are not counted beyond one pass of the
    history per iteration."""
    nodes, beams = _counts(case)
    rb = 4 if case["mixed"] else 8
    nbytes = beams * (8 + 15 * rb) + nodes * (20 * rb + 6)
    flops = 260 * beams + 90 * nodes
    if case.get("trials"):
        nbytes += beams * (14 * rb + 3)
    rounds = 1
    if case["kind"] == "minimize":
        rounds = case["iterations"]
    if case["kind"] == "batch_run":
        rounds = 12 * (case["steps"] + 1)
    if rounds > 1:
        nbytes += nodes * 48 * 20
        flops += nodes * 6 * 4 * 2 * 10
    return {"bytes": nbytes * rounds, "flops": flops * rounds}


# ---- the same results in 64 bits, in plain torch --------------------------------------------
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _qmul(a, b):
    aw, ax, ay, az = a.unbind(1)
    bw, bx, by, bz = b.unbind(1)
    return torch.stack([aw * bw - ax * bx - ay * by - az * bz, aw * bx + ax * bw + ay * bz - az * by,
                        aw * by - ax * bz + ay * bw + az * bx, aw * bz + ax * by - ay * bx + az * bw], 1)


def _dot(a, b):
    return (a * b).sum(1, keepdim=True)


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=1)


def _rot(q, v):
    t = 2 * _cross(q[:, 1:], v)
    return v + q[:, :1] * t + _cross(q[:, 1:], t)


def _conj(q):
    return q * torch.tensor([1.0, -1, -1, -1], dtype=q.dtype, device=q.device)


def _return(total, p, a, k, y, h):
    """Radial return with linear hardening; total and p are scalars or vectors per beam."""
    trial = k * (total - p)
    n = trial.norm(dim=1, keepdim=True)
    f = n - (y + h * a)
    yes = (f > 0) & (n > 1e-20)
    dg = torch.where(yes, f / (k + h), torch.zeros_like(f))
    p = p + trial / n.clamp_min(1e-300) * dg
    a = a + dg
    e = total - p
    return k * e, p, a, dg, 0.5 * k * _dot(e, e), 0.5 * h * a * a, yes


def _closest(p1, q1, p2, q2):
    """Closest points of two segments (either may be a point)."""
    d1, d2, r = q1 - p1, q2 - p2, p1 - p2
    a, e, f, c, b = _dot(d1, d1), _dot(d2, d2), _dot(d2, r), _dot(d1, r), _dot(d1, d2)
    pa, pe = a <= 1e-20, e <= 1e-20
    den = a * e - b * b
    one = torch.ones_like(a)
    sa, se = torch.where(pa, one, a), torch.where(pe, one, e)
    s = torch.where(den.abs() > 1e-20, ((b * f - c * e) / torch.where(den == 0, one, den)).clamp(0, 1), 0 * a)
    t = (b * s + f) / se
    s = torch.where(t < 0, (-c / sa).clamp(0, 1), torch.where(t > 1, ((b - c) / sa).clamp(0, 1), s))
    t = t.clamp(0, 1)
    s = torch.where(pe, (-c / sa).clamp(0, 1), s)
    t = torch.where(pe, 0 * t, t)
    t = torch.where(pa & ~pe, (f / se).clamp(0, 1), t)
    s = torch.where(pa, 0 * s, s)
    return s, t, p1 + d1 * s, p2 + d2 * t


def _pairs(lo, hi, cell):
    """Index pairs (i < j) of the boxes that overlap, found in a uniform grid."""
    org = lo.min(0).values - cell
    c0, c1 = ((lo - org) / cell).floor().long(), ((hi - org) / cell).floor().long()
    dim = c1.max(0).values + 1
    span = c1 - c0 + 1
    cnt = span.prod(1)
    shape = torch.repeat_interleave(torch.arange(len(cnt), device=lo.device), cnt)
    at = torch.arange(len(shape), device=lo.device) - torch.repeat_interleave(cnt.cumsum(0) - cnt, cnt)
    sp = span[shape]
    c = c0[shape] + torch.stack([at % sp[:, 0], at // sp[:, 0] % sp[:, 1], at // (sp[:, 0] * sp[:, 1])], 1)
    key, order = ((c[:, 2] * dim[1] + c[:, 1]) * dim[0] + c[:, 0]).sort()
    shape, c = shape[order], c[order]
    found = []
    for off in range(1, len(key)):
        same = key[off:] == key[:-off]
        if not bool(same.any()):
            break
        w = same.nonzero().squeeze(1)
        i, j = shape[w], shape[w + off]
        first = (torch.maximum(c0[i], c0[j]) == c[w]).all(1)  # each pair in its first common cell only
        ok = first & (lo[i] <= hi[j]).all(1) & (lo[j] <= hi[i]).all(1)
        found.append(torch.stack([torch.minimum(i, j)[ok], torch.maximum(i, j)[ok]], 1))
    return torch.cat(found) if found else torch.zeros((0, 2), dtype=torch.long, device=lo.device)


def _objective64(cfg, lat, sy, plastic, z, top, trials):
    dev = _dev()

    def T(v, *shape):
        return torch.as_tensor(np.ascontiguousarray(v), device=dev).double().reshape(shape or (-1, 1))
    N, m = lat.n_nodes, cfg.material
    E, G = m.young, m.young / (2 * (1 + m.nu))
    locked = torch.as_tensor(lat.locked, device=dev).bool().reshape(N, 6)
    zz = T(z, N, 6).masked_fill(locked, 0.0)
    x = T(lat.x0, N, 3) + cfg.translation_scale * zz[:, :3]
    r = zz[:, 3:]
    ang = r.norm(dim=1, keepdim=True)
    q = torch.cat([torch.cos(ang / 2), 0.5 * torch.sinc(ang / (2 * math.pi)) * r], 1)
    R = _qmul(q, T(lat.r0, N, 4))
    R = R / R.norm(dim=1, keepdim=True)
    a = torch.as_tensor(lat.beam_a, device=dev).long()
    b = torch.as_tensor(lat.beam_b, device=dev).long()
    L0, rad, area, I, J = (T(getattr(lat, f)) for f in ("L0", "radius", "area", "I", "J"))
    pl = T(plastic, lat.n_beams, 7)
    kb, kt = E * I / L0, G * J / L0
    my, ty = sy * I / rad, sy / math.sqrt(3.0) * J / rad
    cs = 0.5 * cfg.shear_correction * G * area * L0
    d = x[b] - x[a]
    L = d.norm(dim=1, keepdim=True)
    t = d / L
    eps = (L - L0) / L0
    fa, pa, aa, dga, ea, ha, ya = _return(eps, pl[:, 0:1], pl[:, 1:2], torch.full_like(eps, E), sy, m.hardening)
    uax, dax = area * L0 * (ea + ha), area * L0 * sy * dga
    e0 = T(lat.e0, lat.n_beams, 3)
    Ra, Rb = R[a], R[b]
    da, db = _rot(Ra, e0), _rot(Rb, e0)
    us = 0.5 * cs * (_dot(da - t, da - t) + _dot(db - t, db - t))
    gt = (2 * t - da - db) * cs
    F = t * (area * fa) + (gt - t * _dot(gt, t)) / L
    Ga, Gb = -cs * _cross(da, t), -cs * _cross(db, t)
    Q = _qmul(_conj(Ra), Rb)
    Q = Q / Q.norm(dim=1, keepdim=True)
    Q = torch.where(Q[:, :1] < 0, -Q, Q)
    sn = Q[:, 1:].norm(dim=1, keepdim=True)
    phi = Q[:, 1:] * torch.where(sn < 1e-12, torch.full_like(sn, 2.0), 2 * torch.atan2(sn, Q[:, :1]) / sn.clamp_min(1e-300))
    axis = _rot(_conj(Ra), t)
    axis = axis / axis.norm(dim=1, keepdim=True)
    rotp = pl[:, 2:5]
    tw, ptw = _dot(phi, axis), _dot(rotp, axis)
    fb, pb, ab, dgb, eb, hb, yb = _return(phi - axis * tw, rotp - axis * ptw, pl[:, 5:6], kb, my, m.bend_hardening * kb)
    ft, pt, at, dgt, et, ht, yt = _return(tw, ptw, pl[:, 6:7], kt, ty, m.torsion_hardening * kt)
    mom = fb + axis * ft
    ur, dr = eb + hb + et + ht, my * dgb + ty * dgt
    ph2 = _dot(phi, phi)
    ph = ph2.sqrt()
    big = ph > 0.05
    phs = torch.where(big, ph, torch.ones_like(ph))
    A = torch.where(big, 1 / phs ** 2 - (1 + torch.cos(phs)) / (2 * phs * torch.sin(phs)),
                    1 / 12 + ph2 * (1 / 720 + ph2 * (1 / 30240 + ph2 * (1 / 1209600 + ph2 / 47900160))))
    c1 = _cross(phi, mom)
    world = _rot(Ra, mom + 0.5 * c1 + A * _cross(phi, c1))
    g = torch.zeros(N, 6, dtype=torch.float64, device=dev)
    g.index_add_(0, a, torch.cat([-F, Ga - world], 1))
    g.index_add_(0, b, torch.cat([F, Gb + world], 1))
    elastic, diss = uax + us + ur, dax + dr
    energy = elastic.sum() + diss.sum()
    mg = T(lat.mass) * cfg.gravity
    energy += (mg * x[:, 1:2]).sum()
    g[:, 1:2] += mg
    mean = x.mean(0)
    energy += 0.5 * cfg.centering_stiffness * (mean[0] ** 2 + mean[2] ** 2)
    g[:, 0] += cfg.centering_stiffness * mean[0] / N
    g[:, 2] += cfg.centering_stiffness * mean[2] / N
    # self-contact: joint spheres, then beam capsules
    kc, jr = cfg.contact_stiffness, cfg.joint_scale * cfg.max_radius
    ids = torch.arange(N, device=dev)
    n0, n1 = torch.cat([ids, a]), torch.cat([ids, b])
    rs = torch.cat([torch.full((N, 1), jr, dtype=torch.float64, device=dev), rad])
    pad = rs + cfg.contact_margin
    lo, hi = torch.minimum(x[n0], x[n1]) - pad, torch.maximum(x[n0], x[n1]) + pad
    p = _pairs(lo, hi, max(2.8 * jr, 0.72 * cfg.cell_size))
    i, j = p[:, 0], p[:, 1]
    conn = torch.as_tensor(lat.connected.astype(np.int64), device=dev).sort().values
    local = torch.zeros(len(i), dtype=torch.bool, device=dev)
    for u in (n0[i], n1[i]):
        for v in (n0[j], n1[j]):
            local |= u == v
            if len(conn):
                k = (torch.minimum(u, v) << 32) | torch.maximum(u, v)
                local |= conn[torch.searchsorted(conn, k).clamp_max(len(conn) - 1)] == k
    i, j = i[~local], j[~local]
    s, u, pa_, pb_ = _closest(x[n0[i]], x[n1[i]], x[n0[j]], x[n1[j]])
    delta = pb_ - pa_
    dist = delta.norm(dim=1, keepdim=True)
    pen = rs[i] + rs[j] + cfg.contact_margin - dist
    hit = (pen > 0).squeeze(1)
    i, j, s, u, pen = i[hit], j[hit], s[hit], u[hit], pen[hit]
    f = delta[hit] / dist[hit] * (kc * pen)
    cap_i, cap_j = (i >= N).unsqueeze(1), (j >= N).unsqueeze(1)
    s, u = torch.where(cap_i, s, 0 * s), torch.where(cap_j, u, 0 * u)
    gx = torch.zeros(N, 3, dtype=torch.float64, device=dev)
    gx.index_add_(0, n0[i], f * (1 - s))
    gx.index_add_(0, n1[i], f * s)
    gx.index_add_(0, n0[j], -f * (1 - u))
    gx.index_add_(0, n1[j], -f * u)
    contact = (0.5 * kc * pen * pen).sum()
    n_contacts = len(i)
    pb0, pt0 = (jr - x[:, 1]).clamp_min(0), (x[:, 1] + jr - top).clamp_min(0)
    gx[:, 1] += kc * (pt0 - pb0)
    contact = contact + (0.5 * kc * (pb0 ** 2 + pt0 ** 2)).sum()
    n_contacts += int((pb0 > 0).sum() + (pt0 > 0).sum())
    g[:, :3] = (g[:, :3] + gx) * cfg.translation_scale
    g = g.masked_fill(locked, 0.0)
    energy = energy + contact
    pens = [float(v.max()) for v in (pen, pb0, pt0) if len(v)]
    out = {"energy": float(energy), "grad": g.reshape(-1).cpu().numpy(),
           "diag": {"elastic": float(elastic.sum()), "plastic": float(diss.sum()), "contact": float(contact),
                    "reaction": float((kc * pt0).sum()), "max_pen": max(pens + [0.0]), "contacts": n_contacts}}
    if trials:
        nrot = pb + axis * pt
        out["trial_next"] = torch.cat([pa, aa, nrot, ab, at], 1).reshape(-1).cpu().numpy()
        out["trial_aux"] = torch.cat([eps, fa, mom, elastic, diss], 1).reshape(-1).cpu().numpy()
        out["trial_flags"] = torch.cat([ya, yb, yt], 1).reshape(-1).to(torch.uint8).cpu().numpy()
    return out


def exact(case, seed):
    if case["kind"] not in ("eval", "noalloc", "batch_eval"):
        return None  # iterates of a minimization have no closed value
    cfg, lats, yields = _setup(case, seed)
    z, pl, tops = _states(case, seed, cfg, lats)
    outs, n, b = [], 0, 0
    for lat, sy, top in zip(lats, yields, tops):
        outs.append(_objective64(cfg, lat, sy, pl[7 * b:7 * (b + lat.n_beams)], z[6 * n:6 * (n + lat.n_nodes)], top,
                                 case.get("trials", False)))
        n += lat.n_nodes
        b += lat.n_beams
    if case["kind"] == "batch_eval":
        return {"energy": np.array([o["energy"] for o in outs]), "grad": np.concatenate([o["grad"] for o in outs]),
                "diag": _columns([o["diag"] for o in outs])}
    return outs[0]
