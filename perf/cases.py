"""What a program does with this library, as timed cases.

Every case goes through the package's public binding (nbx.py over the C ABI).
The kinds of call:

  io        Simulation::step on a caller's own body array: one nbx_step_io,
            which uploads, steps once and writes the bodies back.  What the
            drop-in `Simulation` class does on every step.
  steps     A stretch of a run between two output frames: a snapshot goes
            up, `steps` resident steps run, the frame comes back in id order
            (`<n> <steps> <output_every>` on the command line).
  points    accelerations at arbitrary points from a built tree
            (QuadTree::acceleration): field maps, tracer particles.

`scenario` is one of the library's generators (disc, discs = two discs on a
glancing course, square = bodies at rest in a square, many contacts), and
`form` the force law: plain (Barnes-Hut), exact (the same with the
reference's rounding, for runs compared bit for bit), quadrupole and learned
(the corrected forms), naive (all pairs, Plummer law).  `count` > 1 is an
ensemble of independent discs in one handle.
"""
import math
import os
import sys

import numpy as np
import torch

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                   "n-body-simulation_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)
import nbx  # noqa: E402

FORMS = {"plain": {}, "exact": {"exact_math": 1}, "quadrupole": {"use_mlp": 2},
         "learned": {"use_mlp": 1}, "naive": {"force_law": 1}}


def case(name, kind, scenario, n, steps=1, theta=0.5, form="plain", band=0.5, epsilon=1.0,
         collisions=1, count=1, points=0):
    c = {"kind": kind, "scenario": scenario, "n": n, "steps": steps, "theta": theta,
         "form": form, "band": band, "epsilon": epsilon, "collisions": collisions,
         "count": count, "points": points}
    return {"name": name, **c} if name else c


def listed():
    return [
        # a small interactive simulation: the drop-in class, defaults (theta 1)
        case("io_disc_1000", "io", "disc", 1000, theta=1.0),
        # the command line's default size and settings, a frame every 10 steps
        case("disc_10k", "steps", "disc", 10000, steps=10, theta=1.0),
        # an ordinary run at the accuracy the configurations ask for, odd size
        case("disc_99991", "steps", "disc", 99991, steps=10),
        # the headline system through the drop-in call, host bodies every step
        case("io_discs_1m", "io", "discs", 1 << 20),
        # the headline system, resident, a frame every 10 steps
        case("discs_1m", "steps", "discs", 1 << 20, steps=10),
        # contact-heavy collapse at the largest configured size
        case("square_4m", "steps", "square", 1 << 22, steps=3, epsilon=6.144),
        # a parameter sweep: independent discs of uneven size in one handle
        case("ensemble_64", "steps", "disc", 2000, steps=5, count=64),
        # a run to be compared bit for bit with the reference
        case("exact_30011", "steps", "disc", 30011, steps=5, form="exact"),
        # the corrected forms: higher theta at the plain form's accuracy
        case("quadrupole_262147", "steps", "discs", 262147, steps=3, theta=0.65,
             form="quadrupole", band=0.4),
        case("learned_100k", "steps", "disc", 100000, steps=2, theta=0.7, form="learned"),
        # the all-pairs simulation
        case("naive_65537", "steps", "disc", 65537, form="naive", collisions=0),
        # a field map over a built tree
        case("points_200003", "points", "discs", 500000, points=200003),
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["io", "steps", "steps", "steps", "ensemble", "corrected", "naive",
                       "points"])
    scenario = rng.choice(["disc", "discs", "square"])
    theta = rng.choice([0.5, 0.5, 0.7, 1.0])
    if what == "io":
        return case(None, "io", scenario, log_int(rng, 1000, 1200000), theta=theta)
    if what == "steps":
        n = log_int(rng, 1000, 1500000)
        steps = rng.randint(1, max(1, min(10, 6000000 // n)))
        form = rng.choice(["plain", "plain", "plain", "exact"])
        return case(None, "steps", scenario, n, steps=steps, theta=theta, form=form,
                    collisions=rng.choice([1, 1, 1, 0]))
    if what == "ensemble":
        return case(None, "steps", "disc", log_int(rng, 500, 8000), steps=rng.randint(1, 5),
                    theta=theta, count=log_int(rng, 2, 100))
    if what == "corrected":
        form = rng.choice(["quadrupole", "learned"])
        n = log_int(rng, 2000, 400000 if form == "quadrupole" else 150000)
        return case(None, "steps", scenario, n, steps=rng.randint(1, 3),
                    theta=rng.choice([0.6, 0.65, 0.7]), form=form,
                    band=rng.choice([0.4, 0.5]))
    if what == "naive":
        return case(None, "steps", scenario, log_int(rng, 1000, 80000), form="naive",
                    collisions=rng.choice([0, 1]))
    return case(None, "points", scenario, log_int(rng, 5000, 800000), theta=theta,
                points=log_int(rng, 100, 300000))


def sizes(c):
    """Body count of each instance; an ensemble's run over a factor of 12."""
    if c["count"] == 1:
        return [c["n"]]
    return [int(c["n"] * 12.0 ** (i / (c["count"] - 1))) for i in range(c["count"])]


def bodies(c, seed):
    if c["scenario"] == "discs":
        return nbx.two_discs(c["n"], seed, 0.2)
    if c["scenario"] == "square":
        return nbx.cold_square(c["n"], seed)
    return np.concatenate([nbx.uniform_disc(n, seed + i) for i, n in enumerate(sizes(c))])


def field_points(c, seed, b):
    """Points over the bodies' box, a little beyond its edges."""
    rng = np.random.RandomState(seed % (1 << 31))
    u = rng.random_sample((2, c["points"]))
    lo = np.array([b["px"].min(), b["py"].min()], np.float64)
    hi = np.array([b["px"].max(), b["py"].max()], np.float64)
    p = lo[:, None] + (1.1 * u - 0.05) * (hi - lo)[:, None]
    return p.astype(np.float32)


def pinned(n):
    return torch.empty((n, 9), dtype=torch.float32, pin_memory=True)


def prepare(c, seed):
    """The handle, the bodies in pinned memory and room for the result."""
    b = bodies(c, seed)
    n = len(b)
    h = nbx.Handle(sizes(c), theta=c["theta"], epsilon=c["epsilon"], mlp_band=c["band"],
                   collisions=c["collisions"], **FORMS[c["form"]])
    if c["form"] == "learned":
        h.mlp_set_params(np.fromfile(os.path.join(PKG, "weights", "farfield_mlp.f32"),
                                     np.float32))
    s = {"case": c, "handle": h, "n": n}
    if c["kind"] == "points":
        s["points"] = field_points(c, seed, b)
        h.upload(b)
        h.phase("build")
        h.sync()
        return s
    s["in"], s["out"] = pinned(n), pinned(n)
    s["in"].numpy().view(np.uint8)[:] = b.view(np.uint8).reshape(n, 36)
    return s


def records(out):
    """The parts of the 36-byte body records, as views."""
    return {"pos": out[:, 0:2], "vel": out[:, 2:4], "acc": out[:, 4:6],
            "mass_radius": out[:, 6:8], "id": out.view(torch.int32)[:, 8]}


def run(s):
    c, h, n = s["case"], s["handle"], s["n"]
    if c["kind"] == "points":
        ax, ay = h.accel_at(s["points"][0], s["points"][1])
        return {"ax": ax, "ay": ay}
    if c["kind"] == "io":
        h.step_io_ptr(s["in"].data_ptr(), s["out"].data_ptr(), n)
    else:
        h.upload_ptr(s["in"].data_ptr(), n)
        h.step(c["steps"])
        h.download_ptr(s["out"].data_ptr(), n, id_order=True)
    return records(s["out"])


def interactions(c, n):
    """Terms of one target's sum: measured on the two-disc system at theta
    0.5 (334 at 2^20 bodies), with the tree code's log n / theta^2 growth."""
    if c["form"] == "naive":
        return n
    return min(n, 5.2 / c["theta"] ** 2 * max(1.0, math.log2(n / 16)))


def work(c):
    """Bytes: the input and the output once; flops: 20 for each term of the
    force sums (the usual count for one gravitational interaction)."""
    total = sum(sizes(c))
    if c["kind"] == "points":
        return {"bytes": 32.0 * total + 16.0 * c["points"],
                "flops": 20.0 * c["points"] * interactions(c, c["n"])}
    terms = sum(n * interactions(c, n) for n in sizes(c))
    return {"bytes": 72.0 * total, "flops": 20.0 * c["steps"] * terms}


# ------------------------------------------------------------- in 64 bits

def law_sums(tx, ty, x, y, m, eps, naive):
    """Direct sums of the force law at targets (tx, ty) over all bodies."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = [torch.as_tensor(np.asarray(v, np.float64), device=dev) for v in (tx, ty, x, y, m)]
    tx, ty, x, y, m = t
    ax, ay = torch.empty_like(tx), torch.empty_like(ty)
    rows = max(1, (1 << 25) // max(1, len(x)))
    for i in range(0, len(tx), rows):
        dx = x[None, :] - tx[i:i + rows, None]
        dy = y[None, :] - ty[i:i + rows, None]
        d2 = dx * dx + dy * dy
        q = d2 + eps * eps
        f = m / (q * q.sqrt()) if naive else m / (d2.sqrt() * q)
        f = torch.where(d2 > 0, f, torch.zeros_like(f))
        ax[i:i + rows] = (dx * f).sum(1)
        ay[i:i + rows] = (dy * f).sum(1)
    return ax.cpu().numpy(), ay.cpu().numpy()


def contact_pairs(p, r):
    """(later, earlier) of every overlapping box pair in resolution order."""
    n = len(r)
    lox, hix, loy, hiy = p[0] - r, p[0] + r, p[1] - r, p[1] + r
    order = np.lexsort((np.arange(n), lox))
    last = np.searchsorted(lox[order], hix[order], side="right")
    pairs = []
    for a in range(n):  # order[a] is the earlier box
        i = order[a]
        j = order[a + 1:last[a]]
        if len(j):
            j = j[(loy[j] <= hiy[i]) & (loy[i] <= hiy[j])]
            pairs += [(b, i) for b in j]
    rank = np.empty(n, np.int64)
    rank[order] = np.arange(n)
    return sorted(pairs, key=lambda q: (rank[q[0]], rank[q[1]]))


def resolve(p, v, m, r, i, j):
    """One contact between bodies i and j (positions and velocities in place)."""
    d = p[:, j] - p[:, i]
    reach = r[i] + r[j]
    dd = d @ d
    if dd > reach * reach:
        return
    w = v[:, j] - v[:, i]
    w1, w2 = m[j] / (m[i] + m[j]), m[i] / (m[i] + m[j])
    dv, vv = d @ w, w @ w
    apart = dd > 0
    if (dv >= 0 and apart) or vv < 1e-12:
        if dv >= 0 and apart:
            t = d * (reach / math.sqrt(dd) - 1.0)
        else:
            t = (d / math.sqrt(dd) if apart else np.array([1.0, 0.0])) * reach
        p[:, i] -= w1 * t
        p[:, j] += w2 * t
        return
    t = (dv + math.sqrt(max(0.0, dv * dv - vv * (dd - reach * reach)))) / vv
    p[:, i] -= v[:, i] * t
    p[:, j] -= v[:, j] * t
    d = p[:, j] - p[:, i]
    k = d * (1.5 * (d @ w) / (d @ d))
    v[:, i] += k * w1
    v[:, j] -= k * w2
    p[:, i] += v[:, i] * t
    p[:, j] += v[:, j] * t


def exact(c, seed):
    """Each step's motion, contacts and forces in 64 bits, the forces as
    direct sums.  None for the io form (its order of bodies is that of their
    rounded positions), for ensembles, and where it would take long."""
    terms = (c["points"] or c["n"] * c["steps"]) * c["n"]
    if c["kind"] == "io" or c["count"] > 1 or terms > 1.2e11 or c["n"] * c["steps"] > 1100000:
        return None
    b = bodies(c, seed)
    if c["kind"] == "points":
        q = field_points(c, seed, b)
        ax, ay = law_sums(q[0], q[1], b["px"], b["py"], b["mass"], c["epsilon"], False)
        return {"ax": ax, "ay": ay}
    b = b[np.argsort(b["id"])]
    p = np.stack([b["px"], b["py"]]).astype(np.float64)
    v = np.stack([b["vx"], b["vy"]]).astype(np.float64)
    a = np.stack([b["ax"], b["ay"]]).astype(np.float64)
    m, r = b["mass"].astype(np.float64), b["radius"].astype(np.float64)
    dt = float(np.float32(0.05))
    for _ in range(c["steps"]):
        v += a * dt
        p += v * dt
        if c["collisions"]:
            for later, earlier in contact_pairs(p, r):
                resolve(p, v, m, r, later, earlier)
        a = np.stack(law_sums(p[0], p[1], p[0], p[1], m, c["epsilon"], c["form"] == "naive"))
    return {"pos": p.T.copy(), "vel": v.T.copy(), "acc": a.T.copy(),
            "mass_radius": np.stack([m, r], 1), "id": np.arange(len(b), dtype=np.int64)}
