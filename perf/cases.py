"""Performance cases of the HEOM propagator, through its public Python binding of the C ABI.

Every case is one call pattern of a user's program: population dynamics of a single hierarchy
(`Heom.propagate`), the reference's own stepping loop over `solve` and `weighted_add`, save and
restart of a whole hierarchy state, a pump-probe field, ensembles of realisations or of uneven
systems, and adjoint gradients.  Systems are the ones of the benchmark: site energies
U[12100, 12700] cm^-1, couplings N(0, 50 cm^-1), one Drude-Lorentz bath per site (lambda about
35 cm^-1, 1/nu about 50 fs), 300 K.  `exact` restates the method in torch (complex128).
"""
import math
import os
import sys

import numpy as np
import torch
import torch.utils.checkpoint

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dm-heom_b200"))
import heom_b200 as hb  # noqa: E402

HBAR, KB = 1.05457148e-34, 1.380650239684840458953781387048e-23
INVCM = 1.986456217327470903861498336971e-23  # J per cm^-1
FS = 1e-15


def ados(sites, matsubaras, depth):
    return math.comb(sites * matsubaras + depth, depth)


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------

def listed():
    return [
        # the smallest ordinary call: an FMO-like complex at depth 4, populations every 10 fs;
        # launches and latency are all it costs
        {"name": "fmo_depth4", "kind": "propagate", "sites": 7, "matsubaras": 1, "depth": 4, "steps": 100,
         "every": 10, "dt_fs": 1.0, "scheme": "product"},
        # an ordinary production run: 8 sites with one Matsubara term per site, state within L2
        {"name": "n8_m2_depth6", "kind": "propagate", "sites": 8, "matsubaras": 2, "depth": 6, "steps": 20,
         "every": 10, "dt_fs": 0.5, "scheme": "product"},
        # the largest: the benchmark hierarchy, 735,471 ADOs, a state far larger than L2
        {"name": "n8_m2_depth8", "kind": "propagate", "sites": 8, "matsubaras": 2, "depth": 8, "steps": 10,
         "every": 5, "dt_fs": 0.5, "scheme": "product"},
        # a complex of more than eight sites with a Matsubara term (the uneven batch's large members)
        {"name": "n12_m2_depth5", "kind": "propagate", "sites": 12, "matsubaras": 2, "depth": 5, "steps": 10,
         "every": 5, "dt_fs": 1.0, "scheme": "product"},
        # odd site count above eight, no Matsubara term, the Horner order of the RK4 step
        {"name": "n11_m1_depth6_horner", "kind": "propagate", "sites": 11, "matsubaras": 1, "depth": 6,
         "steps": 20, "every": 10, "dt_fs": 1.0, "scheme": "horner"},
        # the drop-in use of the derivative: a program with an RK4 stepper of its own calls solve and
        # weighted_add on hierarchy buffers, as the reference's solver does, and reads the state back
        {"name": "stepper_n7_m2_depth5", "kind": "stepper", "sites": 7, "matsubaras": 2, "depth": 5, "steps": 4,
         "dt_fs": 0.5},
        # restart from a saved state and save again: upload, a few steps, download of every ADO
        {"name": "restart_n6_m2_depth5", "kind": "restart", "sites": 6, "matsubaras": 2, "depth": 5, "steps": 5,
         "dt_fs": 1.0},
        # pump-probe field: a complex, time-dependent Hamiltonian
        {"name": "field_n7_depth7", "kind": "field", "sites": 7, "matsubaras": 1, "depth": 7, "steps": 30,
         "every": 10, "dt_fs": 1.0},
        # static disorder: 256 realisations of the 7-site system at depth 6
        {"name": "disorder_256", "kind": "ensemble", "count": 256, "sites_lo": 7, "sites_hi": 7, "depth_lo": 6,
         "depth_hi": 6, "matsubaras_hi": 1, "steps": 20, "every": 10, "dt_fs": 1.0},
        # systems of uneven size and depth admitted together
        {"name": "uneven_12", "kind": "ensemble", "count": 12, "sites_lo": 4, "sites_hi": 12, "depth_lo": 3,
         "depth_hi": 5, "matsubaras_hi": 2, "steps": 10, "every": 5, "dt_fs": 1.0},
        # gradients of a time-integrated population with respect to H, lambda, gamma and rho0
        {"name": "adjoint_n7_depth8", "kind": "adjoint", "count": 1, "sites": 7, "matsubaras": 1, "depth": 8,
         "steps": 60, "dt_fs": 1.0},
        # the same for a batch of realisations above eight sites
        {"name": "adjoint_batch_n9_depth4", "kind": "adjoint", "count": 4, "sites": 9, "matsubaras": 1,
         "depth": 4, "steps": 40, "dt_fs": 1.0},
    ]


def _size(rng, lo, hi, sites_lo=2, sites_hi=16):
    """(sites, matsubaras, depth) of a hierarchy whose ADO count is near a log-uniform target."""
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    n = rng.randint(sites_lo, sites_hi)
    m = rng.choice([1, 1, 2, 2, 3])
    if n * m > 32:
        m = 1
    d = 1
    while ados(n, m, d + 1) <= want and d < 20:
        d += 1
    return n, m, d


def draw(rng):
    kind = rng.choice(["propagate"] * 5 + ["stepper", "restart", "field", "ensemble", "ensemble", "adjoint"])
    dt = rng.choice([0.5, 1.0]) if kind != "ensemble" else 0.5
    if kind == "propagate":
        n, m, d = _size(rng, 20, 250000)
        if ados(n, m, d) * n * n > 1.6e7:
            d -= 1
        every = rng.choice([1, 2, 5])
        return {"kind": kind, "sites": n, "matsubaras": m, "depth": max(1, d), "steps": every * rng.randint(2, 4),
                "every": every, "dt_fs": 0.5, "scheme": rng.choice(["product", "product", "horner", "reference"])}
    if kind == "stepper":
        n, m, d = _size(rng, 50, 20000)
        return {"kind": kind, "sites": n, "matsubaras": m, "depth": d, "steps": rng.randint(2, 5), "dt_fs": 0.5}
    if kind == "restart":
        n, m, d = _size(rng, 50, 20000)
        return {"kind": kind, "sites": n, "matsubaras": m, "depth": d, "steps": rng.randint(2, 9), "dt_fs": 0.5}
    if kind == "field":
        n, m, d = _size(rng, 50, 20000)
        every = rng.randint(2, 5)
        return {"kind": kind, "sites": n, "matsubaras": m, "depth": d, "steps": every * 3, "every": every,
                "dt_fs": 0.5}
    if kind == "ensemble":
        if rng.random() < 0.5:
            n, d = rng.randint(3, 8), rng.randint(2, 5)
            return {"kind": kind, "count": rng.randint(9, 300), "sites_lo": n, "sites_hi": n, "depth_lo": d,
                    "depth_hi": d, "matsubaras_hi": 1, "steps": 10, "every": 5, "dt_fs": dt}
        lo = rng.randint(2, 8)
        return {"kind": kind, "count": rng.randint(3, 14), "sites_lo": lo, "sites_hi": lo + rng.randint(1, 5),
                "depth_lo": 2, "depth_hi": 4, "matsubaras_hi": 2, "steps": 10, "every": 5, "dt_fs": dt}
    n, m, d = _size(rng, 50, 6000, 3, 11)
    return {"kind": "adjoint", "count": rng.choice([1, 1, 2, 3]), "sites": n, "matsubaras": min(m, 2),
            "depth": min(d, 8), "steps": rng.randint(9, 50), "dt_fs": dt}


# --------------------------------------------------------------------------
# inputs, from the seed alone
# --------------------------------------------------------------------------

def _hamiltonian(rng, n):
    h = np.zeros((n, n))
    iu = np.triu_indices(n, 1)
    h[iu] = rng.normal(0.0, 50.0, size=len(iu[0]))
    h = h + h.T
    h[np.diag_indices(n)] = rng.uniform(12100.0, 12700.0, size=n)
    return h


def _systems(case, seed):
    """Systems of a case as dicts in the config's units (cm^-1, fs, K)."""
    rng = np.random.default_rng(seed)
    out = []
    if case["kind"] == "ensemble":
        for _ in range(case["count"]):
            n = int(rng.integers(case["sites_lo"], case["sites_hi"] + 1))
            out.append((n, int(rng.integers(1, case["matsubaras_hi"] + 1)),
                        int(rng.integers(case["depth_lo"], case["depth_hi"] + 1))))
        if case["sites_lo"] != case["sites_hi"]:  # the work is the case's own, whatever the seed
            shape = np.random.default_rng(case["count"] * 1009 + case["sites_lo"])
            out = [(int(shape.integers(case["sites_lo"], case["sites_hi"] + 1)),
                    int(shape.integers(1, case["matsubaras_hi"] + 1)),
                    int(shape.integers(case["depth_lo"], case["depth_hi"] + 1))) for _ in out]
    else:
        out = [(case["sites"], case["matsubaras"], case["depth"])] * case.get("count", 1)
    base, systems = {}, []
    shared = len(out) > 1  # instances of an ensemble share their baths
    for n, m, d in out:
        if n not in base:
            base[n] = _hamiltonian(rng, n)
        h = base[n].copy()
        if len(out) > 1:
            h[np.diag_indices(n)] += rng.normal(0.0, 100.0, size=n)  # static disorder
        uniform = shared or case["kind"] == "adjoint"
        lam = np.full(n, 35.0) if uniform else rng.uniform(30.0, 40.0, size=n)
        inv = np.full(n, 50.0) if uniform else rng.uniform(45.0, 55.0, size=n)
        systems.append({"n": n, "m": m, "d": d, "h": h, "lam": lam, "inv": inv})
    return systems


def _library_system(s):
    return hb.System(s["h"], s["lam"], s["inv"], np.zeros(s["n"]), s["m"], 300.0, s["d"])


def _top(n, seed):
    """Initial density matrix: a pure state, mostly on the first site."""
    rng = np.random.default_rng(seed + 77)
    v = rng.normal(0.0, 0.1, size=n) + 1j * rng.normal(0.0, 0.1, size=n)
    v[0] += 1.0
    v /= np.linalg.norm(v)
    return np.outer(v, v.conj())


def _flat(a):
    return np.ascontiguousarray(a, dtype=np.complex128).view(np.float64).reshape(-1)


def _saved_state(case, seed):
    """A hierarchy state in mid-run: every ADO filled, magnitudes falling with the order of the ADO."""
    n, nodes = case["sites"], ados(case["sites"], case["matsubaras"], case["depth"])
    rng = np.random.default_rng(seed + 5)
    y = rng.normal(size=(nodes, n * n * 2))
    w = case["sites"] * case["matsubaras"]
    layer = np.repeat(np.arange(case["depth"] + 1), [math.comb(w + k - 1, k) for k in range(case["depth"] + 1)])
    y *= (0.1 * 0.7 ** layer)[:, None]
    y[0] += _flat(_top(n, seed))
    return y.reshape(-1)


def _field(case, seed):
    n = case["sites"]
    rng = np.random.default_rng(seed + 9)
    dm = (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))) * 40.0 * INVCM
    pulses = [(1.0, 15 * FS, 8 * FS, 2.0e14, 0.3), (0.6, 30 * FS, 5 * FS, 1.5e14, -1.1)]
    return dm.conj().T, dm, pulses


def _observable(n):
    o = np.zeros((n, n), np.complex128)
    o[min(2, n - 1), min(2, n - 1)] = 1.0
    return o


def prepare(case, seed):
    systems = _systems(case, seed)
    kind = case["kind"]
    st = {"case": case, "dt": case["dt_fs"] * FS}
    if kind == "ensemble":
        st["ens"] = hb.Ensemble([hb.build_tables(_library_system(s)) for s in systems])
        st["ens"].clear()
        for k, s in enumerate(systems):
            st["ens"].set_top(k, _flat(_top(s["n"], seed)))
        st["ens"].autotune()
        return st
    if kind == "adjoint":
        libs = [_library_system(s) for s in systems]
        st["adj"] = hb.Adjoint(libs if case["count"] > 1 else libs[0])
        st["rho0"], st["obs"] = _top(case["sites"], seed), _observable(case["sites"])
        st["w"] = hb.trapezoid_weights(case["steps"], case["dt_fs"])
        return st
    h = st["heom"] = hb.from_system(_library_system(systems[0]), scheme=case.get("scheme", "product"))
    if kind == "restart":
        st["y0"] = _saved_state(case, seed)
        return st
    if kind == "stepper":
        st["y"], st["tmp"] = h.buffer(), h.buffer()
        st["k"] = [h.buffer() for _ in range(4)]
        st["y0"] = _saved_state(case, seed)
        return st
    h.set_top(_flat(_top(case["sites"], seed)))
    if kind == "field":
        dp, dm, pulses = _field(case, seed)
        h.set_field(dp, dm, pulses[0], pulses[1])
    return st


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------

def run(st):
    case, dt = st["case"], st["dt"]
    kind = case["kind"]
    if kind == "propagate":
        return st["heom"].propagate(dt, case["steps"], case["every"])
    if kind == "field":
        st["heom"].set_time(0.0)
        return st["heom"].propagate(dt, case["steps"], case["every"])
    if kind == "ensemble":
        return np.concatenate([t.reshape(-1) for t in st["ens"].propagate(dt, case["steps"], case["every"])])
    if kind == "adjoint":
        return st["adj"].gradient(st["rho0"], st["obs"], st["w"], dt, case["steps"])
    h = st["heom"]
    if kind == "restart":
        h.set_state(st["y0"])
        h.rk4_steps(dt, case["steps"])
        return h.get_state()
    y, tmp, k = st["y"], st["tmp"], st["k"]
    y.write(st["y0"])
    for _ in range(case["steps"]):  # the classical RK4 of the reference's stepper
        h.solve(y, k[0])
        h.weighted_add(dt, tmp, y, [0.5], k[:1])
        h.solve(tmp, k[1])
        h.weighted_add(dt, tmp, y, [0.0, 0.5], k[:2])
        h.solve(tmp, k[2])
        h.weighted_add(dt, tmp, y, [0.0, 0.0, 1.0], k[:3])
        h.solve(tmp, k[3])
        h.weighted_add(dt, y, y, [1 / 6, 1 / 3, 1 / 3, 1 / 6], k)
    return y.read()


def work(case):
    """Each of a step's four derivative evaluations reads its input and writes its output once; the
    adjoint evaluates the forward operator once and the transposed one once per step, and reads both
    states once more for the gradients.  Operations: the commutator with a real symmetric H and the
    neighbour terms."""
    total_b = total_f = 0.0
    for s in _systems(case, 0):
        n, m, d = s["n"], s["m"], s["d"]
        nodes = ados(n, m, d)
        edges = n * m * ados(n, m, d - 1) if d > 0 else 0
        evals = 4 * case["steps"] * (2 if case["kind"] == "adjoint" else 1)
        per = 8.0 * n ** 3 * (2 if case["kind"] == "field" else 1) + 16.0 * n * n
        total_b += evals * nodes * 32.0 * n * n
        total_f += evals * (nodes * per + edges * 12.0 * 2 * n)
        if case["kind"] in ("restart", "stepper"):
            total_b += nodes * 32.0 * n * n
        if case["kind"] == "adjoint":
            total_b += 4 * case["steps"] * nodes * 32.0 * n * n
            total_f += 4 * case["steps"] * nodes * 16.0 * n ** 3
    return {"bytes": total_b, "flops": total_f}


def tolerance(case):
    """Everything is held and summed in doubles: the present code differs from `exact` (another order of
    the operations, another form of the RK4 polynomial) by up to 7e-15 over these cases; a drawn case
    takes fewer steps but more sites, hence the wider margin."""
    return {"rel": 1e-13, "max": 2e-12}


# --------------------------------------------------------------------------
# the method in plain torch, complex128
# --------------------------------------------------------------------------

def _pade(order):
    """Poles xi (largest first) and residues eta of the [n-1/n] Pade approximant of coth(x/2)/2 - 1/x."""
    bern = {2: (1, 6), 4: (-1, 30), 6: (1, 42), 8: (-1, 30), 10: (5, 66), 12: (-691, 2730)}
    c = [np.longdouble(bern[2 * k + 2][0]) / bern[2 * k + 2][1] / math.factorial(2 * k + 2) for k in range(2 * order)]
    a = np.array([[float(c[order + r - k]) for k in range(1, order + 1)] for r in range(order)])
    b = np.array([-float(c[order + r]) for r in range(order)])
    q = np.linalg.solve(a, b).astype(np.longdouble)
    for _ in range(3):  # refine in extended precision
        res = np.array([-c[order + r] - sum(c[order + r - k] * q[k - 1] for k in range(1, order + 1))
                        for r in range(order)], dtype=np.longdouble)
        q = q + np.linalg.solve(a, res.astype(np.float64)).astype(np.longdouble)
    qc = np.concatenate([[np.longdouble(1)], q])
    pc = [sum(qc[k] * c[m - k] for k in range(m + 1)) for m in range(order)]
    out = []
    for y in np.roots(qc[::-1].astype(np.float64)).real.astype(np.longdouble):
        for _ in range(3):
            f = sum(qc[k] * y ** k for k in range(order + 1))
            y = y - f / sum(k * qc[k] * y ** (k - 1) for k in range(1, order + 1))
        dq = sum(k * qc[k] * y ** (k - 1) for k in range(1, order + 1))
        out.append((float(np.sqrt(-y)), float(sum(pc[m] * y ** m for m in range(order)) / dq / 2)))
    return sorted(out, reverse=True)


def _tuples(width, depth):
    """Every tuple of `width` counts with sum <= depth, in the reference's order: by sum, then by the
    counts sorted downwards, then by the tuple itself."""
    rows = np.zeros((1, 0), np.int16)
    left = np.full(1, depth)
    for _ in range(width):
        reps = left + 1
        start = np.repeat(np.cumsum(reps) - reps, reps)
        t = np.arange(reps.sum()) - start
        rows = np.concatenate([np.repeat(rows, reps, axis=0), t[:, None].astype(np.int16)], axis=1)
        left = np.repeat(left, reps) - t
    down = -np.sort(-rows, axis=1)
    keys = [rows[:, m] for m in range(width - 1, -1, -1)] + [down[:, m] for m in range(width - 1, -1, -1)]
    return rows[np.lexsort(keys + [rows.sum(axis=1)])]


def _neighbours(tup, depth):
    """(plus, minus) indices per mode, -1 where there is none."""
    width = tup.shape[1]
    c = np.array([[math.comb(a, b) if a >= 0 else 0 for b in range(width + 2)] for a in range(width + depth + 2)])

    def rank(t):
        r, used = np.zeros(len(t), np.int64), np.zeros(len(t), np.int64)
        for m in range(width):
            k, v = width - 1 - m, t[:, m].astype(np.int64)
            # sum over x < v of C(k + depth - used - x, k)
            r += c[k + depth - used + 1, k + 1] - c[k + depth - used - v + 1, k + 1]
            used += v
        return r

    place = np.empty(len(tup), np.int64)
    place[rank(tup)] = np.arange(len(tup))
    plus, minus = np.full(tup.shape, -1, np.int64), np.full(tup.shape, -1, np.int64)
    total = tup.sum(axis=1)
    for m in range(width):
        step = np.zeros(width, np.int16)
        step[m] = 1
        ok = total < depth
        plus[ok, m] = place[rank(tup[ok] + step)]
        ok = tup[:, m] > 0
        minus[ok, m] = place[rank(tup[ok] - step)]
    return plus, minus


class _Model:
    """The hierarchy of one system; K Hamiltonians share it (leading axis of every state)."""

    def __init__(self, s, dev, lam=None, gam=None):
        self.n, self.m, self.d, self.dev = s["n"], s["m"], s["d"], dev
        tup = _tuples(s["n"] * s["m"], s["d"])
        plus, minus = _neighbours(tup, s["d"])
        self.nodes = len(tup)
        self.tup = torch.from_numpy(tup.astype(np.float64)).to(dev)
        self.edges = []  # per mode: (ADO with a neighbour above, that neighbour)
        for e in range(tup.shape[1]):
            u = np.nonzero(plus[:, e] >= 0)[0]
            self.edges.append((torch.from_numpy(u).to(dev), torch.from_numpy(plus[u, e]).to(dev)))
            v = np.nonzero(minus[:, e] >= 0)[0]
            assert np.array_equal(np.sort(plus[u, e]), v)
        t = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
        self.lam = (t(s["lam"]) if lam is None else lam.expand(s["n"])) * INVCM
        self.nu = (1.0 / t(s["inv"]) if gam is None else gam.expand(s["n"])) / FS
        self.baths()

    def baths(self):
        beta, n, m = 1.0 / (KB * 300.0), self.n, self.m
        pade = _pade(m)
        nu, lam = self.nu, self.lam
        one = torch.ones_like(nu)
        # the real parts of cbk are scaled by hbar / beta: the exponent of every mode and its coefficient
        total = sum(2 * eta * nu * nu / (xi * xi / (beta * HBAR) ** 2 - nu * nu) for xi, eta in pade)
        self.cbk, rates = [2 * lam / (beta * HBAR) * (1 - total)], [nu]
        for xi, eta in pade[1:]:
            self.cbk.append(4 * lam * nu / (beta * HBAR) ** 2 * eta * xi / (xi * xi / (beta * HBAR) ** 2 - nu * nu))
            rates.append(one * (xi / (beta * HBAR)))
        self.circ = nu * lam / HBAR
        same = 2 * lam / (beta * HBAR * HBAR * nu) - sum(c / (HBAR * r) for c, r in zip(self.cbk, rates))
        tup = self.tup.reshape(self.nodes, n, m)
        self.decay = -sum((tup[:, :, k] * rates[k]).sum(dim=1) for k in range(m))
        off = 1.0 - torch.eye(n, dtype=torch.float64, device=self.dev)
        self.pair = -(same[:, None] + same[None, :]) * off

    def derivative(self, w, h):
        """w: [K, nodes, n, n]; h: [K, n, n] in J."""
        hh = (h / HBAR)[:, None]
        out = 1j * (w @ hh - hh @ w) + (self.decay[:, None, None] + self.pair) * w
        for e, (lo, up) in enumerate(self.edges):
            b, m = divmod(e, self.m)
            c = self.cbk[m][b]
            size = torch.abs(c)
            cp = torch.sqrt((self.tup[lo, e] + 1) * size / HBAR)[None, :, None]
            cm = torch.sqrt((self.tup[lo, e] + 1) * HBAR / size)[None, :, None]
            q = self.circ[b] if m == 0 else torch.zeros_like(c)
            above, below = w[:, up], w[:, lo]
            row = torch.zeros_like(w[:, :, b, :])
            col = torch.zeros_like(row)
            row = row.index_add(1, lo, 1j * cp * above[:, :, b, :]).index_add(
                1, up, cm * (1j * c / HBAR + q) * below[:, :, b, :])
            col = col.index_add(1, lo, -1j * cp * above[:, :, :, b]).index_add(
                1, up, cm * (-1j * c / HBAR + q) * below[:, :, :, b])
            pick = torch.zeros(self.n, dtype=torch.complex128, device=self.dev)
            pick[b] = 1.0
            out = out + row[:, :, None, :] * pick[:, None] + col[:, :, :, None] * pick
        return out

    def step(self, y, dt, hs):
        k1 = self.derivative(y, hs(0.0))
        k2 = self.derivative(y + dt / 2 * k1, hs(0.5))
        k3 = self.derivative(y + dt / 2 * k2, hs(0.5))
        k4 = self.derivative(y + dt * k3, hs(1.0))
        return y + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)


def _start(model, tops):
    y = torch.zeros((len(tops), model.nodes, model.n, model.n), dtype=torch.complex128, device=model.dev)
    y[:, 0] = torch.as_tensor(np.stack(tops), device=model.dev)
    return y


def _floats(t):
    return _flat(t.detach().cpu().numpy())


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    systems = _systems(case, seed)
    cost = sum(ados(s["n"], s["m"], s["d"]) * s["n"] ** 2 * s["n"] * s["m"] for s in systems) * case["steps"]
    if cost > (6e9 if dev == "cuda" else 1e8):
        return None  # would take longer than some seconds
    dt, kind = case["dt_fs"] * FS, case["kind"]
    joule = lambda s: torch.as_tensor(s["h"] * INVCM + 0j, device=dev)  # noqa: E731
    if kind == "ensemble":
        groups, out = {}, [None] * len(systems)
        for k, s in enumerate(systems):
            groups.setdefault((s["n"], s["m"], s["d"]), []).append(k)
        for key, members in groups.items():
            model = _Model(systems[members[0]], dev)
            h = torch.stack([joule(systems[k]) for k in members])
            y = _start(model, [_top(key[0], seed)] * len(members))
            rows = [y[:, 0].clone()]
            for i in range(case["steps"]):
                y = model.step(y, dt, lambda c: h)
                if (i + 1) % case["every"] == 0:
                    rows.append(y[:, 0].clone())
            for q, k in enumerate(members):
                out[k] = _floats(torch.stack([r[q] for r in rows]))
        return np.concatenate(out)
    if kind == "adjoint":
        return _exact_adjoint(case, seed, systems, dev, dt, joule)
    s = systems[0]
    model, n = _Model(s, dev), s["n"]
    h = joule(s)[None]
    if kind in ("restart", "stepper"):
        y = torch.as_tensor(_saved_state(case, seed).view(np.complex128).reshape(1, -1, n, n), device=dev)
        for _ in range(case["steps"]):
            y = model.step(y, dt, lambda c: h)
        return _floats(y)
    y = _start(model, [_top(n, seed)])
    hs, rows = (lambda c: h), [y[0, 0].clone()]
    for i in range(case["steps"]):
        if kind == "field":
            dp, dm, pulses = _field(case, seed)

            def hs(c, t0=i * dt):
                t = t0 + c * dt
                e = sum(a * np.exp(-(t - tc) ** 2 / (2 * w * w)) * np.exp(1j * (ph + om * t))
                        for a, tc, w, om, ph in pulses)
                return h - torch.as_tensor(e * dm + np.conj(e) * dp, device=dev)
        y = model.step(y, dt, hs)
        if (i + 1) % case["every"] == 0:
            rows.append(y[0, 0].clone())
    return _floats(torch.stack(rows)).reshape(len(rows), -1)


def _exact_adjoint(case, seed, systems, dev, dt, joule):
    n, steps = case["sites"], case["steps"]
    obs = torch.as_tensor(_observable(n), device=dev)
    w = np.full(steps + 1, case["dt_fs"])
    w[0] = w[-1] = 0.5 * case["dt_fs"]
    res = {"loss": [], "h": [], "lambda": [], "gamma": [], "rho0": []}
    for s in systems:
        lam = torch.tensor([35.0], dtype=torch.float64, device=dev, requires_grad=True)
        gam = torch.tensor([1.0 / 50.0], dtype=torch.float64, device=dev, requires_grad=True)
        h = torch.as_tensor(s["h"] + 0j, device=dev).requires_grad_(True)
        rho = torch.as_tensor(_top(n, seed), device=dev).requires_grad_(True)
        model = _Model(s, dev, lam, gam)
        pad = torch.zeros((model.nodes - 1, n, n), dtype=torch.complex128, device=dev)
        y = torch.cat([rho[None], pad])[None]
        value = w[0] * (obs.conj() * y[0, 0]).sum().real
        hj = h[None] * INVCM
        for i in range(steps):
            y = torch.utils.checkpoint.checkpoint(lambda v: model.step(v, dt, lambda c: hj), y, use_reentrant=False)
            value = value + w[i + 1] * (obs.conj() * y[0, 0]).sum().real
        value.backward()
        for key, v in (("loss", value), ("h", h.grad), ("lambda", lam.grad[0]), ("gamma", gam.grad[0]),
                       ("rho0", rho.grad)):
            res[key].append(v.detach().cpu().numpy())
    if case["count"] == 1:
        return {k: (v[0] if k in ("h", "rho0") else float(v[0])) for k, v in res.items()}
    return {k: np.stack(v) for k, v in res.items()}
