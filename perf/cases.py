"""The work that users of this framework have it do, as measurable cases.

Five kinds, each through the package's public classes:

  job          one configuration of the FLOW application: its links arrive in
               host memory, are uploaded and flowed with a measurement every
               `every` steps; `save` also downloads the flowed links (a
               checkpoint)
  flow         a segment of a longer flow of a field that is on the device
               already (a program that flows until t^2 E reaches a target, or
               that resumes): `steps` more steps, rows back
  ensemble     the same for many configurations at once
  observables  plaquette, clover energy and charge of one field
  generate     a Metropolis chain from a cold start, links and acceptance back

Every kind returns all that its entry point returns (rows of step, t, plaq,
topc, energy, t^2 E; links).  The mixed forms' rows are returned in single
precision, which is what their links and site arithmetic carry.

exact() is the same computation in complex128 torch, written from the
definitions: staple force, Luscher's third-order Runge-Kutta, e^{iQ} by its
power series, the three neighbouring loops of a clover moved to its site.
"""
import math

import numpy as np
import torch

from latticeyangmills_b200 import Ensemble, GluonField

# Fields above this many sites are drawn on the device by init_links: their
# host copies would be several GB and nobody's 64-bit reference is quick there.
HOST_SITES = 1 << 21
# exact() flows at most this many site-steps (about 10 s of torch).
EXACT_SITE_STEPS = 22_000_000
REAL_BYTES = {"fp64": 8, "fp32_18": 4, "fp32_12": 4}
LINK_REALS = {"fp64": 18, "fp32_18": 18, "fp32_12": 12}


def listed():
    return [
        # The smallest job: an 8^4 thermalised-size lattice, every step
        # measured, as the FLOW application does by default: launches count.
        {"name": "job_8_fp64", "kind": "job", "precision": "fp64", "lattice": "8x8x8x8", "a": 0.35, "eps": 0.01,
         "steps": 100, "every": 1, "reunit": 0, "save": True},
        # The same size in the mixed form, as a scan over many small fields has it.
        {"name": "flow_8_fp32_12", "kind": "flow", "precision": "fp32_12", "lattice": "8x8x8x8", "a": 0.35,
         "eps": 0.01, "steps": 50, "every": 10, "reunit": 10},
        # An ordinary job: 16^3 x 32, eps 0.01 to t = 2, measured every 10 steps.
        {"name": "job_16x32_fp64", "kind": "job", "precision": "fp64", "lattice": "16x16x16x32", "a": 0.35,
         "eps": 0.01, "steps": 160, "every": 10, "reunit": 0, "save": False},
        # Odd extents, a volume that no warp or tile size divides, every step measured.
        {"name": "flow_ragged_fp64", "kind": "flow", "precision": "fp64", "lattice": "15x13x17x21", "a": 0.3,
         "eps": 0.02, "steps": 40, "every": 1, "reunit": 0},
        # The headline size in FP64, the application's default of a row per step.
        {"name": "flow_32_fp64", "kind": "flow", "precision": "fp64", "lattice": "32x32x32x32", "a": 0.35,
         "eps": 0.01, "steps": 10, "every": 1, "reunit": 0},
        # The headline size in the two mixed forms: the long-flow schedule
        # (reunitarised every 10 steps, few rows) and a row per step.
        {"name": "flow_32_fp32_12", "kind": "flow", "precision": "fp32_12", "lattice": "32x32x32x32", "a": 0.35,
         "eps": 0.01, "steps": 20, "every": 10, "reunit": 10},
        {"name": "flow_32_fp32_18", "kind": "flow", "precision": "fp32_18", "lattice": "32x32x32x32", "a": 0.35,
         "eps": 0.01, "steps": 10, "every": 1, "reunit": 10},
        # The largest configuration, 5 % of its links Haar-random, measured every 5 steps.
        {"name": "flow_64_fp32_12", "kind": "flow", "precision": "fp32_12", "lattice": "64x64x64x64", "a": 0.35,
         "haar": 0.05, "eps": 0.02, "steps": 10, "every": 5, "reunit": 10},
        # 64 configurations of four sizes together, in the mixed form.
        {"name": "ensemble_64_fp32_12", "kind": "ensemble", "precision": "fp32_12",
         "lattices": "16*8x8x8x8 16*12x12x12x12 16*16x16x16x16 16*16x16x16x32", "a": 0.35, "eps": 0.01, "steps": 10,
         "every": 10, "reunit": 10},
        # A few small FP64 configurations of uneven sizes together, measured often.
        {"name": "ensemble_12_fp64", "kind": "ensemble", "precision": "fp64",
         "lattices": "6*8x8x8x8 4*6x10x12x14 2*12x12x12x24", "a": 0.35, "eps": 0.01, "steps": 20, "every": 2,
         "reunit": 0},
        # One measurement of a stored field.
        {"name": "observables_24x48_fp64", "kind": "observables", "precision": "fp64", "lattice": "24x24x24x48",
         "a": 0.35},
        # Generating a configuration: 20 sweeps of 30 hits per link at beta = 6.
        {"name": "generate_16_fp64", "kind": "generate", "precision": "fp64", "lattice": "16x16x16x16", "beta": 6.0,
         "su3eps": 0.24, "sweeps": 20, "hits": 30},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _lattice(rng, lo, hi, even=False):
    """Extents of a lattice of about lo..hi sites (spread over the logarithm), no direction over 4 x another."""
    while True:
        side = _log_uniform(rng, lo, hi) ** 0.25
        n = [max(4, round(side * rng.uniform(0.7, 1.4))) for _ in range(4)]
        if even:
            n = [v + v % 2 for v in n]
        if n[0] * n[1] * n[2] * n[3] <= hi:
            return n


def draw(rng):
    kind = rng.choice(["flow", "flow", "flow", "job", "job", "ensemble", "observables", "generate"])
    precision = rng.choice(["fp64", "fp64", "fp32_12", "fp32_18"])
    a = round(rng.uniform(0.25, 0.45), 3)
    text = "x".join
    if kind == "generate":  # the checkerboard needs even extents
        return {"kind": kind, "precision": "fp64", "lattice": text(map(str, _lattice(rng, 256, 65536, True))),
                "beta": round(rng.uniform(5.5, 6.5), 2), "su3eps": 0.24, "sweeps": rng.randint(2, 20),
                "hits": rng.randint(5, 30)}
    if kind == "observables":
        return {"kind": kind, "precision": precision, "lattice": text(map(str, _lattice(rng, 4096, 1 << 20))), "a": a}
    eps = rng.choice([0.005, 0.01, 0.02])
    reunit = 0 if precision == "fp64" else 10
    if kind == "ensemble":
        runs = ["%d*%s" % (rng.randint(1, 8), text(map(str, _lattice(rng, 256, 65536)))) for _ in range(rng.randint(2, 5))]
        return {"kind": kind, "precision": precision, "lattices": " ".join(runs), "a": a, "eps": eps,
                "steps": rng.randint(5, 20), "every": rng.choice([1, 2, 5, 10]), "reunit": reunit}
    n = _lattice(rng, 256, 1 << 20)
    v = n[0] * n[1] * n[2] * n[3]
    case = {"kind": kind, "precision": precision, "lattice": text(map(str, n)), "a": a, "eps": eps,
            "steps": min(100, max(5, EXACT_SITE_STEPS // (2 * v))), "every": rng.choice([1, 1, 5, 10]), "reunit": reunit}
    if kind == "job":
        case["save"] = rng.random() < 0.5
    return case


def _extents(text):
    return tuple(int(v) for v in text.split("x"))


def _lattices(case):
    """Every configuration's extents, in order."""
    if "lattice" in case:
        return [_extents(case["lattice"])]
    out = []
    for run in case["lattices"].split():
        count, n = run.split("*")
        out += [_extents(n)] * int(count)
    return out


def _sites(n):
    return n[0] * n[1] * n[2] * n[3]


# ---- links U = e^{i a H}, H traceless Hermitian with unit-variance normal reals ----

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _mul(a, b):
    """Products of 3x3 matrices held as [3, 3, ...]."""
    return a[:, 0:1] * b[0:1] + a[:, 1:2] * b[1:2] + a[:, 2:3] * b[2:3]


def _dag(a):
    return a.transpose(0, 1).conj()


def _one(like):
    return torch.eye(3, dtype=like.dtype, device=like.device).reshape((3, 3) + (1,) * (like.dim() - 2))


def _exp_i(q, terms, halvings=0):
    """e^{iq} by its power series after `halvings` halvings of q."""
    x = q * (1j / 2 ** halvings)
    one = _one(x)
    e = one + x / terms
    for k in range(terms - 1, 0, -1):
        e = one + _mul(x, e) / k
    for _ in range(halvings):
        e = _mul(e, e)
    return e


def _draw_links(n, a, seed, conf):
    """U_mu as [4][3, 3, t, z, y, x] of configuration `conf`."""
    gen = torch.Generator(device=_device()).manual_seed(seed * 1000 + conf)
    shape = (n[3], n[2], n[1], n[0])
    links = []
    for _ in range(4):
        g = torch.randn((9,) + shape, generator=gen, device=_device(), dtype=torch.float64)
        tr = (g[0] + g[1] + g[2]) / 3
        h = torch.zeros((3, 3) + shape, device=_device(), dtype=torch.complex128)
        for i in range(3):
            h[i, i] = g[i] - tr
        for k, (i, j) in enumerate(((0, 1), (0, 2), (1, 2))):
            h[i, j] = torch.complex(g[3 + 2 * k], g[4 + 2 * k])
            h[j, i] = h[i, j].conj()
        links.append(_exp_i(a * h, 12, 4))
    return links


def _to_host(links):
    """The .bin layout: (t, z, y, x, mu, 18) doubles in host memory."""
    u = torch.stack([torch.view_as_real(m.permute(2, 3, 4, 5, 0, 1).contiguous()).flatten(-3) for m in links], 4)
    return u.cpu().numpy()


# ---- the cases ----

def prepare(case, seed):
    sizes, kind = _lattices(case), case["kind"]
    state = {"case": case, "seed": seed}
    if kind == "ensemble":
        state["ens"] = Ensemble(sizes, case["precision"])
        for c, n in enumerate(sizes):
            state["ens"].upload(c, _to_host(_draw_links(n, case["a"], seed, c)))
        return state
    state["field"] = GluonField(sizes[0], case["precision"])
    if kind == "generate":
        return state
    if _sites(sizes[0]) > HOST_SITES:
        state["field"].init_links("expiah", case["a"], seed, 0, case.get("haar", 0.0))
        return state
    links = _to_host(_draw_links(sizes[0], case["a"], seed, 0))
    if kind == "job":
        state["links"] = links
    else:
        state["field"].upload(links)
    return state


def _rows(case, rows):
    return rows if case["precision"] == "fp64" else np.asarray(rows, dtype=np.float32)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ensemble":
        return {"rows": _rows(case, state["ens"].flow(case["eps"], case["steps"], case["every"], case["reunit"]))}
    field = state["field"]
    if kind == "observables":
        return {"rows": _rows(case, np.array(field.observables().as_tuple()))}
    if kind == "generate":
        acceptance = field.generate_metropolis(case["beta"], case["su3eps"], case["sweeps"], case["hits"],
                                               state["seed"], "cold")
        return {"acceptance": acceptance, "links": field.download()}
    if kind == "job":
        field.upload(state["links"])
    out = {"rows": _rows(case, field.flow(case["eps"], case["steps"], case["every"], case["reunit"]))}
    if case.get("save"):
        out["links"] = _rows(case, field.download())
    return out


def _measurements(case):
    """Rows of a flow, and link-updates per link of it."""
    if case["kind"] == "observables":
        return 1, 0
    every, steps = case["every"], case["steps"]
    return 1 + sum(1 for s in range(1, steps + 1) if s % every == 0 or s == steps), steps


def work(case):
    """A link-update (one link, one Runge-Kutta step) reads and writes the link in each of three stages and
    the 8-real generator twice each way; a measurement reads every link.  The least arithmetic known for
    them: per link and stage 1.5 plaquette generators (about 260 multiply-adds each), three transports of
    one (110), the exponential and the update (240); per site of a measurement 6 planes of a plaquette
    and three transports.  A proposal of a Metropolis update is three sparse SU(2) products on two rows, a
    trace and four Philox calls (about 400 operations)."""
    real, link = REAL_BYTES[case["precision"]], LINK_REALS[case["precision"]]
    sites = sum(_sites(n) for n in _lattices(case))
    if case["kind"] == "generate":
        hits = 4.0 * sites * case["sweeps"] * case["hits"]
        return {"bytes": 4.0 * sites * case["sweeps"] * 2 * link * real + 4.0 * sites * 144,
                "flops": 400.0 * hits + 4.0 * sites * case["sweeps"] * 2 * 1000}
    rows, steps = _measurements(case)
    size = 4.0 * sites * (steps * (6 * link + 4 * 8) + rows * link) * real
    if case["kind"] == "job":
        size += 4.0 * sites * 144 * (2 if case.get("save") else 1)
    per_link = 3 * (1.5 * 260 + 3 * 110 + 240)
    return {"bytes": size, "flops": 2.0 * sites * (4 * steps * per_link + rows * 6 * (260 + 3 * 110 + 30))}


# ---- exact() ----

def _shift(m, mu, sign):
    """m(x + sign mu) of a field [3, 3, ..., t, z, y, x]."""
    return torch.roll(m, -sign, dims=m.dim() - 1 - mu)


def _force(u, mu):
    omega = torch.zeros_like(u[mu])
    for nu in range(4):
        if nu == mu:
            continue
        u_nu_pm = _shift(u[nu], mu, 1)
        omega += _mul(_mul(u_nu_pm, _dag(_shift(u[mu], nu, 1))), _dag(u[nu]))
        omega += _shift(_mul(_mul(_dag(u_nu_pm), _dag(u[mu])), u[nu]), nu, -1)
    x = _mul(u[mu], omega)
    z = 0.5j * (x - _dag(x))
    return z - _one(z) * (z[0, 0] + z[1, 1] + z[2, 2]) / 3


def _step(u, eps):
    z = [torch.zeros_like(m) for m in u]
    for c_new, c_old, e in ((1.0, 0.0, eps / 4), (8 / 9, -17 / 36, eps), (3 / 4, -1.0, eps)):
        z = [c_new * _force(u, mu) + c_old * z[mu] for mu in range(4)]
        u = [_mul(_exp_i(e * z[mu], 14), u[mu]) for mu in range(4)]
    return u


def _trace_sum(a, b):
    """Re tr(a b) summed over the lattice, per configuration."""
    return (a * b.transpose(0, 1)).real.sum(dim=(0, 1, 3, 4, 5, 6))


def _observe(u):
    """plaq, topc, energy per configuration of u, [4][3, 3, conf, t, z, y, x]."""
    sites = u[0][0, 0, 0].numel()
    plaq, energy, g = 0.0, 0.0, {}
    for mu in range(4):
        for nu in range(mu + 1, 4):
            p = _mul(_mul(u[mu], _shift(u[nu], mu, 1)), _dag(_mul(u[nu], _shift(u[mu], nu, 1))))
            plaq = plaq + (p[0, 0] + p[1, 1] + p[2, 2]).real.sum(dim=(1, 2, 3, 4))
            back_nu = _mul(_mul(_dag(u[nu]), p), u[nu])  # the loop of x - nu, moved to x
            c = p + _shift(back_nu, nu, -1)
            c = c + _shift(_mul(_mul(_dag(u[mu]), c), u[mu]), mu, -1)
            c = c - _dag(c)
            g[mu, nu] = c - _one(c) * (c[0, 0] + c[1, 1] + c[2, 2]) / 3
            energy = energy + _trace_sum(g[mu, nu], g[mu, nu])
    topc = _trace_sum(g[0, 1], g[2, 3]) - _trace_sum(g[0, 2], g[1, 3]) + _trace_sum(g[0, 3], g[1, 2])
    return plaq / (18 * sites), -topc / (256 * math.pi ** 2), energy


def _row(step, t, u):
    plaq, topc, energy = (v.cpu().numpy() for v in _observe(u))
    sites = u[0][0, 0, 0].numel()
    return np.stack([np.full_like(plaq, step), np.full_like(plaq, t), plaq, topc, energy,
                     -t * t * energy / (64 * sites)], 1)


def exact(case, seed):
    sizes = _lattices(case)
    # A Metropolis chain is its own definition: accepting or not is what its random stream decides.
    if case["kind"] == "generate":
        return None
    rows, steps = _measurements(case)
    sites = sum(_sites(n) for n in sizes)
    if max(_sites(n) for n in sizes) > HOST_SITES or sites * (steps + 1) > 2 * EXACT_SITE_STEPS:
        return None
    out, saved, first = [], None, 0
    while first < len(sizes):  # configurations of equal extents together
        last = first
        while last < len(sizes) and sizes[last] == sizes[first]:
            last += 1
        fields = [_draw_links(sizes[c], case["a"], seed, c) for c in range(first, last)]
        u = [torch.stack([f[mu] for f in fields], 2) for mu in range(4)]
        t, got = 0.0, [_row(0, 0.0, u)]
        for s in range(1, steps + 1):
            u = _step(u, case["eps"])
            t += case["eps"]
            if s % case["every"] == 0 or s == steps:
                got.append(_row(s, t, u))
        out.append(np.stack(got, 0))  # rows, configurations, 6
        if case.get("save"):
            saved = _to_host([m[:, :, 0] for m in u])
        first = last
    got = np.concatenate(out, 1)
    if case["kind"] == "ensemble":
        return {"rows": got}
    if case["kind"] == "observables":
        return {"rows": got[0, 0]}
    return {"rows": got[:, 0], "links": saved} if case.get("save") else {"rows": got[:, 0]}
