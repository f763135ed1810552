"""The workloads this library is timed on, through its public entry points.

    listed()            the fixed cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program holds before the call: inputs, matrices, plans
    run(state)          one pass, and its outputs
    work(case)          bytes and operations one pass cannot do without
    exact(case, seed)   the same outputs in 64 bits, from plain torch

Outputs come in the type of the arithmetic behind them: single precision where
the recursion runs in complex64 ("mixed"), double precision otherwise.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

import tight_binding_gb300 as tb
from tight_binding_gb300 import capi
from tight_binding_gb300.serving import model_bounds, model_cell

# one orientation of every nearest-neighbour bond: (from atom, to atom, cell vector)
BONDS = {
    "square": [(0, 0, (1, 0)), (0, 0, (0, 1))],
    "honeycomb": [(0, 1, (0, 0)), (0, 1, (-1, 0)), (0, 1, (0, -1))],
    "kagome": [(0, 1, (0, 0)), (0, 1, (-1, 0)), (0, 2, (0, 0)), (0, 2, (0, -1)), (1, 2, (0, 0)), (1, 2, (1, -1))],
    "lieb": [(0, 1, (0, 0)), (0, 1, (-1, 0)), (0, 2, (0, 0)), (0, 2, (0, -1))],
    "fcc": [(0, 0, v) for v in ((1, 0, 0), (0, 1, 0), (0, 0, 1), (1, -1, 0), (1, 0, -1), (0, 1, -1))],
}
ATOMS = {"square": 1, "honeycomb": 2, "kagome": 3, "lieb": 3, "fcc": 1}
ELEM = {"mixed": 8, "dd": 16, "fp64": 16}          # bytes of a complex vector element
EDGE = 1e-8                                        # margin density_of_states_seq and the Kubo drivers add to the bounds


def listed():
    return [
        # the drop-in call of the reference's GreenFunctionImag on a small lattice: host arrays in and out, latency
        {"name": "braket_square64", "op": "braket", "lattice": "square", "nx": 64, "ny": 64, "R": 8, "M": 256,
         "precision": "fp64"},
        # one whole density of states as the reference's example programs ask for it: build, rescale, moments, spectrum
        {"name": "dos_honeycomb_odd", "op": "dos", "lattice": "honeycomb", "nx": 301, "ny": 253, "R": 4, "M": 512,
         "energies": 1000},
        # the headline workload (graphene-like sheet with on-site disorder), moments of a resident plan
        {"name": "moments_honeycomb1024", "op": "moments", "lattice": "honeycomb", "nx": 1024, "ny": 1024, "R": 32,
         "M": 256, "precision": "mixed", "doubling": True, "vacancies": 0.0, "flux": 0},
        # the same sheet with missing atoms and open edges: every row has its own neighbours; R no power of two
        {"name": "moments_vacancies", "op": "moments", "lattice": "honeycomb", "nx": 701, "ny": 600, "R": 20, "M": 300,
         "precision": "mixed", "doubling": True, "vacancies": 0.03, "flux": 0},
        # a magnetic field: complex hoppings that differ per column, FP64-class accuracy, bras other than kets
        {"name": "moments_flux_dd", "op": "moments", "lattice": "square", "nx": 500, "ny": 333, "R": 6, "M": 256,
         "precision": "dd", "doubling": False, "vacancies": 0.0, "flux": 50},
        # sigma_xy of a strip in a field: the moment matrix of conductivity_Kubo_Bastin on the tensor cores
        {"name": "kubo_bastin_256", "op": "kubo", "form": "bastin", "lattice": "square", "nx": 256, "ny": 256, "nz": 0,
         "R": 16, "M": 512, "tensor": True, "flux": 64, "disorder": 0.0},
        # sigma_xx of a disordered 3D crystal, the largest solve
        {"name": "kubo_greenwood_fcc128", "op": "kubo", "form": "greenwood", "lattice": "fcc", "nx": 128, "ny": 128,
         "nz": 128, "R": 8, "M": 1024, "tensor": True, "flux": 0, "disorder": 2.0},
        # the drivers' default GEMM on a sheet of odd size
        {"name": "kubo_honeycomb_default", "op": "kubo", "form": "greenwood", "lattice": "honeycomb", "nx": 91, "ny": 77,
         "nz": 0, "R": 3, "M": 200, "tensor": False, "flux": 0, "disorder": 1.0},
        # conductivities from a finished moment matrix: Bastin's zeta and its integral, the Greenwood spectrum
        {"name": "spectra_512", "op": "spectra", "M": 512, "energies": 1024},
        # a wave packet followed in time, host vectors in and out
        {"name": "evolve_honeycomb", "op": "evolve", "lattice": "honeycomb", "nx": 400, "ny": 303, "R": 4, "time": 40.0},
        # the spectral range of a new Hamiltonian: GreenFunction(N, HE) without bounds
        {"name": "bounds_honeycomb", "op": "bounds", "lattice": "honeycomb", "nx": 801, "ny": 640},
        # a server working through requests of uneven size, and the density of states of each
        {"name": "serve_20", "op": "serve", "requests": 20, "mix": 3, "side": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["braket", "dos", "moments", "moments", "kubo", "kubo", "spectra", "evolve", "bounds", "serve"])
    kind = rng.choice(["square", "honeycomb", "kagome", "lieb"])
    if op == "braket":
        return {"op": op, "lattice": kind, "nx": _log(rng, 8, 160), "ny": _log(rng, 8, 160), "R": rng.randint(1, 12),
                "M": _log(rng, 32, 512), "precision": rng.choice(["fp64", "fp64", "mixed", "dd"])}
    if op == "dos":
        return {"op": op, "lattice": kind, "nx": _log(rng, 24, 420), "ny": _log(rng, 24, 420), "R": rng.randint(1, 6),
                "M": _log(rng, 64, 768), "energies": _log(rng, 100, 4096)}
    if op == "moments":
        flux = rng.choice([0, 0, 20, 64])
        return {"op": op, "lattice": "square" if flux else kind, "nx": _log(rng, 40, 700), "ny": _log(rng, 40, 700),
                "R": _log(rng, 1, 40), "M": _log(rng, 64, 400), "precision": rng.choice(["mixed", "mixed", "dd", "fp64"]),
                "doubling": rng.random() < 0.7, "vacancies": rng.choice([0.0, 0.0, 0.01, 0.1]), "flux": flux}
    if op == "kubo":
        form = rng.choice(["bastin", "greenwood"])
        fcc = rng.random() < 0.4
        side = _log(rng, 12, 64) if fcc else _log(rng, 24, 300)
        flux = 0 if fcc else rng.choice([0, 32])
        return {"op": op, "form": form, "lattice": "fcc" if fcc else "square" if flux else kind, "nx": side,
                "ny": side + rng.randint(0, 9), "nz": side + rng.randint(0, 5) if fcc else 0, "R": rng.randint(1, 9),
                "M": _log(rng, 32, 600), "tensor": rng.random() < 0.7, "flux": flux, "disorder": rng.choice([0.0, 1.0])}
    if op == "spectra":
        return {"op": op, "M": _log(rng, 32, 1024), "energies": _log(rng, 64, 2048)}
    if op == "evolve":
        return {"op": op, "lattice": kind, "nx": _log(rng, 16, 500), "ny": _log(rng, 16, 500), "R": rng.randint(1, 9),
                "time": round(math.exp(rng.uniform(0.0, math.log(80.0))), 2)}
    if op == "bounds":
        return {"op": op, "lattice": kind, "nx": _log(rng, 32, 900), "ny": _log(rng, 32, 900)}
    return {"op": op, "requests": rng.randint(2, 20), "mix": rng.randint(4, 10 ** 6), "side": _log(rng, 64, 512)}


# ------------------------------------------------------------------ lattices
def _span(c):
    return (c["nx"], c["ny"], c["nz"]) if c["lattice"] == "fcc" else (c["nx"], c["ny"])


def _sites(c):
    return math.prod(_span(c)) * ATOMS[c["lattice"]]


def _gen(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(int(seed))


def _disorder(n, W, seed):
    """On-site energies, uniform in [-W/2, W/2]."""
    return (np.random.default_rng([int(seed), 1]).random(n) - 0.5) * W


def _removed(n, share, seed):
    return (np.random.default_rng([int(seed), 2]).random(n) < share).astype(np.uint8)


def _phases(n, R, seed):
    """R random-phase vectors as an R x n tensor (the columns of an n x R column-major block)."""
    u = torch.rand((R, n), generator=_gen(seed), dtype=torch.float64, device="cuda")
    return torch.polar(torch.full_like(u, 1 / math.sqrt(n)), 2 * math.pi * u)


def _host(block):
    """The block as an n x R column-major host array."""
    return block.cpu().numpy().T


def _lattice(c, W, seed):
    X = tb.PartialLattice(model_cell(c["lattice"]), _span(c))
    if W:
        X.set_scalar_values(_disorder(_sites(c), W, seed))
    if c.get("flux"):
        G = np.zeros((3, 3))
        G[1, 0] = 2 * math.pi / c["flux"]           # Landau gauge: 1 / flux quanta per plaquette
        X.set_gauge_linear(G)
    if c.get("vacancies"):
        X.remove_sites(_removed(_sites(c), c["vacancies"], seed))
    return X


def _periodic(c):
    """Periodic axes: the axis along which the Landau gauge repeats, or all."""
    return [0, 1] if c.get("flux") else [1] * len(_span(c))


def _hamiltonian(c, X):
    scalar = complex if c.get("flux") else float
    if c.get("vacancies"):
        return X.get_Hamiltonian_sparse(scalar)
    return X.get_Hamiltonian_periodic_extend_bare_sparse(_periodic(c), scalar)


DISORDER = 0.5                                     # of the cases that do not say otherwise


def _out(precision, a):
    if precision != "mixed":
        return a
    if isinstance(a, torch.Tensor):
        return a.float()
    return a.astype(np.complex64 if np.iscomplexobj(a) else np.float32)


# ------------------------------------------------------------------ requests of a server
def _requests(c):
    rng = random.Random(c["mix"])
    out = []
    for _ in range(c["requests"]):
        kind = rng.choice(["square", "honeycomb", "kagome", "lieb", "fcc"])
        side = rng.randint(16, max(17, c["side"] // 8)) if kind == "fcc" else rng.randint(32, c["side"])
        out.append({"lattice": kind, "nx": side, "ny": side, "nz": side if kind == "fcc" else 0,
                    "M": rng.choice([256, 512, 1024]), "R": rng.choice([4, 8, 16, 32, 64]), "W": 2 * rng.random(),
                    "precision": "dd" if rng.random() < 0.1 else "mixed"})
    return out


@functools.lru_cache(maxsize=1)
def _server():
    return tb.DosServer()                          # a service has one, for its whole life


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    c, op = case, case["op"]
    s = {"case": c, "seed": int(seed)}
    if op == "spectra":
        s["mu"], s["eps"] = _moment_matrix(c, seed)
        return s
    if op == "serve":
        s["server"], s["jobs"] = _server(), []
        for i, q in enumerate(_requests(c)):
            X = tb.PartialLattice(model_cell(q["lattice"]), _span(q))
            X.set_scalar_values(_disorder(_sites(q), q["W"], seed + i))
            s["jobs"].append((X, q, seed + i, model_bounds(q["lattice"], q["W"])))
        s["e"] = np.cos((np.arange(512) + 0.5) * math.pi / 512)
        return s
    W = c.get("disorder", DISORDER)
    X = _lattice(c, W, seed)
    if op == "dos":
        s["X"], s["bounds"], s["e"] = X, model_bounds(c["lattice"], W), np.linspace(-0.99, 0.99, c["energies"])
        return s
    H = _hamiltonian(c, X)
    if op == "bounds":
        s["H"] = H
        return s
    lo, hi = model_bounds(c["lattice"], W)
    G = tb.GreenFunction(c.get("M", 2), H, lo, hi)
    n = _sites(c)
    if op == "kubo":
        X_a = X.op_position(0)
        s["Ht"], s["va"] = G.scaled_HE, tb.commutator(G.scaled_HE, X_a)
        s["vb"] = tb.commutator(G.scaled_HE, X.op_position(1)) if c["form"] == "bastin" else None
        return s
    kets = _phases(n, c["R"], seed)
    if op == "evolve":
        s["G"], s["kets"] = G, _host(kets)
    elif op == "braket":
        s["M"] = (n, *G.scaled_HE.to_csc())
        s["kets"], s["bras"] = _host(kets), _host(_phases(n, c["R"], seed + 7))
    else:
        s["solver"] = tb.KpmSolver(G.scaled_HE, c["R"], c["precision"], c["doubling"], capi.FLAG_DEVICE_PTRS)
        s["kets"] = kets
        s["bras"] = kets if c["doubling"] else _phases(n, c["R"], seed + 7)
        s["mu"] = torch.empty(c["M"], dtype=torch.float64, device="cuda")
    return s


def _moment_matrix(c, seed):
    """mu_nm of a Kubo solve as the spectra meet it: strongest near the diagonal, kernel-damped, noisy."""
    M, rng = c["M"], np.random.default_rng([int(seed), 3])
    d = np.subtract.outer(np.arange(M), np.arange(M))
    noise = rng.standard_normal((M, M)) + 1j * rng.standard_normal((M, M))
    g = np.sinh(6 * (1 - np.arange(M) / M)) / math.sinh(6)
    mu = np.outer(g, g) * ((0.3 + 0.2j) * np.exp(-np.abs(d) / 8) * np.cos(0.3 * d) + 0.01 * noise)
    return mu, np.cos((np.arange(c["energies"]) + 0.5) * math.pi / c["energies"])


# ------------------------------------------------------------------ run
def run(s):
    c, op = s["case"], s["case"]["op"]
    if op == "braket":
        return _out(c["precision"], tb.Cheb_first_kind_seq_braket(s["M"], c["M"], s["bras"], s["kets"], c["precision"]))
    if op == "dos":
        return tb.density_of_states_seq(s["X"], c["M"], s["e"], *s["bounds"], R=c["R"], seed=s["seed"])
    if op == "moments":
        s["solver"].run_device(c["M"], s["bras"].data_ptr(), s["kets"].data_ptr(), s["mu"].data_ptr())
        return _out(c["precision"], s["mu"])
    if op == "kubo":
        ops = (None, None, s["va"], s["vb"]) if c["form"] == "bastin" else (s["va"], s["va"], None, None)
        return _out("mixed", tb.kubo_mu(s["Ht"], *ops, M=c["M"], R=c["R"], seed=s["seed"], kernel=tb.Lorentz(6.0),
                                        tensor=c["tensor"]))
    if op == "spectra":
        zeta = tb.bastin_zeta(s["mu"], s["eps"], 100.0)
        return [zeta, *tb.bastin_integrate(s["eps"], zeta), tb.greenwood_sigma(s["mu"], s["eps"], 4.0)]
    if op == "evolve":
        return tb.time_evolve(s["G"], c["time"], s["kets"])
    if op == "bounds":
        return list(tb.GreenFunction(256, s["H"]).spectral_range())
    srv = s["server"]
    tickets = [srv.submit(X, q["M"], q["R"], k, *b, precision=q["precision"]) for X, q, k, b in s["jobs"]]
    out = []
    for (X, q, k, b), t in zip(s["jobs"], tickets):
        mu, _ = srv.result(t)
        out += [_out(q["precision"], mu), _out(q["precision"], tb.dos_from_moments(mu, tb.Jackson(), q["R"], s["e"]))]
    return out


# ------------------------------------------------------------------ work
def work(case):
    """Recursions: each step reads v_n and v_{n-1} and writes v_{n+1} once, for all vectors."""
    c, op = case, case["op"]
    if op == "spectra":                             # each entry of mu enters a sum along its two (anti)diagonals
        return {"bytes": 16.0 * c["M"] ** 2 + 24.0 * c["energies"], "flops": 8.0 * c["M"] ** 2 + 24.0 * c["M"] * c["energies"]}
    if op == "serve":
        parts = [_recursion(q, q["M"] / 2, q["R"], q["precision"]) for q in _requests(c)]
        return {k: sum(p[k] for p in parts) for k in parts[0]}
    if op == "bounds":
        return _recursion(c, 200, 1, "fp64")
    if op == "evolve":
        w = _recursion(c, 1.1 * model_bounds(c["lattice"], DISORDER)[1] * c["time"] + 20, c["R"], "dd")
        return {"bytes": w["bytes"] + 32.0 * _sites(c) * c["R"], "flops": w["flops"]}
    if op == "kubo":
        w = _recursion(c, 2 * c["M"], c["R"], "mixed")
        K = float(_sites(c)) * c["R"]
        return {"bytes": w["bytes"] + 32.0 * c["M"] * K, "flops": w["flops"] + 8.0 * c["M"] ** 2 * K}
    steps = c["M"] / 2 if c.get("doubling") else c["M"]
    w = _recursion(c, steps, c["R"], c.get("precision", "fp64"))
    bras = 0.0 if c.get("doubling") or op == "dos" else 16.0 * _sites(c) * c["R"]
    return {"bytes": w["bytes"] + 16.0 * _sites(c) * c["R"] + bras, "flops": w["flops"]}


def _recursion(c, steps, R, precision):
    z = 2 * len(BONDS[c["lattice"]]) / ATOMS[c["lattice"]]
    n = float(_sites(c)) * R * steps
    return {"bytes": 3 * ELEM[precision] * n, "flops": (4 * z + 8) * (2 if c.get("flux") else 1) * n}


# ------------------------------------------------------------------ exact
class _Exact:
    """H~ = (H - b)/a of a case as neighbour tables: (H~ x)_i = d_i x_i + sum_k v_k,i x_(j_k,i)."""

    def __init__(self, c, W, seed, lo, hi):
        span, na, n = _span(c), ATOMS[c["lattice"]], _sites(c)
        cell = np.stack(np.meshgrid(*map(np.arange, span), indexing="ij"), -1).reshape(-1, len(span))
        per = _periodic(c) if not c.get("vacancies") else [0] * len(span)
        flat = lambda v, a: np.ravel_multi_index(tuple(v.T), span) * na + a
        a, b = (hi - lo) / 2, (hi + lo) / 2
        cols, vals = [], []
        for f, t, vec in BONDS[c["lattice"]]:
            to = cell + np.array(vec)
            ok = np.ones(len(cell), bool)
            for x in range(len(span)):
                if not per[x]:
                    ok &= (to[:, x] >= 0) & (to[:, x] < span[x])
            i, j = flat(cell[ok], f), flat(np.mod(to[ok], span), t)
            h = np.exp(1j * (2 * math.pi / c["flux"]) * cell[ok, 0] * vec[1]) if c.get("flux") else np.ones(len(i))
            for p, q, g in ((i, j, h), (j, i, np.conj(h))):
                col, val = np.arange(n), np.zeros(n, h.dtype)
                col[p], val[p] = q, g / a
                cols.append(col)
                vals.append(val)
        diag = (_disorder(n, W, seed) if W else np.zeros(n)) / a - b / a
        if c.get("vacancies"):                      # kept sites first, the rest of the matrix empty
            keep = _removed(n, c["vacancies"], seed) == 0
            k = int(keep.sum())
            pos = np.where(keep, np.cumsum(keep) - 1, -1)
            for q, (col, val) in enumerate(zip(cols, vals)):
                new = pos[col[keep]]
                v = np.where(new < 0, 0, val[keep])
                cols[q] = np.concatenate([np.where(new < 0, 0, new), np.zeros(n - k, int)])
                vals[q] = np.concatenate([v, np.zeros(n - k, v.dtype)])
            diag = np.concatenate([diag[keep], np.full(n - k, -b / a)])
        dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
        self.cell, self.na, self.n = cell, na, n
        self.cols, self.vals, self.diag = [dev(x) for x in cols], [dev(x) for x in vals], dev(diag)

    def velocity(self, x):
        """X H~ - H~ X for the site positions x."""
        v = object.__new__(_Exact)
        x = torch.from_numpy(x).cuda()
        v.cols, v.diag = self.cols, torch.zeros_like(self.diag)
        v.vals = [h * (x - x[j]) for j, h in zip(self.cols, self.vals)]
        return v

    def __call__(self, x):
        y = self.diag * x
        for j, h in zip(self.cols, self.vals):
            y += h * x[..., j]
        return y

    def chebyshev(self, v, n):
        """T_0 v, ..., T_{n-1} v."""
        t0, t1 = v, None
        for _ in range(n):
            yield t0
            t1, t0 = t0, self(t0) if t1 is None else 2 * self(t0) - t1


def _mix64(x):
    m = lambda v, k: (v >> k) & ((1 << (64 - k)) - 1)
    i64 = lambda v: v - (1 << 64) if v >= 1 << 63 else v
    x = x + i64(0x9E3779B97F4A7C15)
    x = (x ^ m(x, 30)) * i64(0xBF58476D1CE4E5B9)
    x = (x ^ m(x, 27)) * i64(0x94D049BB133111EB)
    return x ^ m(x, 31)


def _library_phases(n, R, seed):
    """The seeded random-phase vectors of the library: SplitMix64 of (seed, vector, site)."""
    i64 = lambda v: (v & (1 << 64) - 1) - (1 << 64) if v & 1 << 63 else v & (1 << 64) - 1
    site = torch.arange(n, dtype=torch.int64, device="cuda")
    r = torch.arange(R, dtype=torch.int64, device="cuda")
    key = _mix64(int(seed) ^ _mix64(r + i64(0x632BE59BD9B4E019)))
    h = _mix64(key[:, None] + site[None, :] * i64(0xD1B54A32D192ED03))
    u = ((h >> 11) & ((1 << 53) - 1)).double() * 2.0 ** -53
    return torch.polar(torch.full_like(u, 1 / math.sqrt(n)), 2 * math.pi * u)


def _dot(a, b):
    return float((a.real * b.real + a.imag * b.imag).sum())


def _moments(H, bras, kets, M):
    return np.array([_dot(bras, t) for t in H.chebyshev(kets, M)])


def _spectrum(mu, g, R, e):
    th = torch.from_numpy(np.arccos(e)).cuda()
    w = torch.from_numpy(mu * g).cuda()
    w[1:] *= 2
    k = torch.arange(len(mu), dtype=torch.float64, device="cuda")
    rho = torch.stack([torch.cos(k * t) @ w for t in th]) / torch.sin(th)
    return rho.cpu().numpy() / (R * math.pi)


def _lorentz(M, lam):
    return np.sinh(lam * (1 - np.arange(M) / M)) / math.sinh(lam)


def _jackson(M):
    n, q = np.arange(M), math.pi / (M + 1)
    return ((M + 1 - n) * np.cos(n * q) + np.sin(n * q) / math.tan(q)) / (M + 1)


def _positions(c, H):
    """Cartesian x and y of every site."""
    s3 = math.sqrt(3.0)
    cell = {"square": ([(1, 0), (0, 1)], [(0, 0)]),
            "honeycomb": ([(1.5, -s3 / 2), (1.5, s3 / 2)], [(0, 0), (1, 0)]),
            "kagome": ([(1, 0), (0.5, s3 / 2)], [(0, 0), (0.5, 0), (0.25, s3 / 4)]),
            "lieb": ([(1, 0), (0, 1)], [(0, 0), (0.5, 0), (0, 0.5)]),
            "fcc": ([(0.5, 0.5), (0.5, 0), (0, 0.5)], [(0, 0)])}[c["lattice"]]
    r = (H.cell @ np.array(cell[0], float))[:, None, :] + np.array(cell[1], float)[None]
    return r.reshape(-1, 2).T.copy()


def exact(case, seed):
    c, op = case, case["op"]
    if op == "bounds":                              # Ritz values of the seeded start vector, not of the matrix alone
        return None
    w = work(case)
    if w["bytes"] > 1.5e12 or w["flops"] > 8e12 or (op == "kubo" and 32.0 * c["M"] * _sites(c) * c["R"] > 6e10):
        return None
    if op == "spectra":
        mu, eps = _moment_matrix(c, seed)
        return [_zeta(mu, eps, 100.0), None, None, None, _greenwood(mu, eps, 4.0)]
    if op == "serve":
        out = []
        for i, q in enumerate(_requests(c)):
            kets = _library_phases(_sites(q), q["R"], seed + i)
            H = _Exact(q, q["W"], seed + i, *model_bounds(q["lattice"], q["W"]))
            mu = _doubled(H, kets, q["M"])
            out += [mu, _spectrum(mu, _jackson(q["M"]), q["R"], np.cos((np.arange(512) + 0.5) * math.pi / 512))]
        return out
    W = c.get("disorder", DISORDER)
    lo, hi = model_bounds(c["lattice"], W)
    n, R = _sites(c), c["R"]
    if op == "dos":
        H = _Exact(c, W, seed, lo - EDGE, hi + EDGE)
        kets = _library_phases(n, R, seed)
        return _spectrum(_moments(H, kets, kets, c["M"]), _lorentz(c["M"], 4.0), R, np.linspace(-0.99, 0.99, c["energies"]))
    H = _Exact(c, W, seed, lo, hi)
    if op == "kubo":
        x, y = _positions(c, H)
        kets = _library_phases(n, R, seed)
        va = H.velocity(x)
        if c["form"] == "bastin":
            L, Rt = H.chebyshev(kets, c["M"]), (va(t) for t in H.chebyshev(H.velocity(y)(kets), c["M"]))
        else:
            L, Rt = (va(t) for t in H.chebyshev(va(kets), c["M"])), H.chebyshev(kets, c["M"])
        g = torch.from_numpy(_lorentz(c["M"], 6.0)).cuda()
        L, Rt = (torch.stack([t.reshape(-1) for t in b]) for b in (L, Rt))
        return (torch.outer(g, g) * (L.conj() @ Rt.T)).cpu().numpy()
    kets = _phases(n, R, seed)
    if op == "evolve":
        return _evolved(H, (hi - lo) / 2, (hi + lo) / 2, c["time"], kets)
    if c.get("doubling"):
        return _doubled(H, kets, c["M"])
    return _moments(H, _phases(n, R, seed + 7), kets, c["M"])


def _doubled(H, kets, M):
    """mu_2n = 2 <v_n|v_n> - mu_0, mu_2n-1 = 2 <v_n|v_n-1> - mu_1: half the products."""
    mu, last = np.zeros(M), None
    for n, t in enumerate(H.chebyshev(kets, M // 2 + 1)):
        if n == 0:
            mu[0], mu[1] = _dot(t, t), _dot(t, H(t))
        else:
            if n > 1:
                mu[2 * n - 1] = 2 * _dot(t, last) - mu[1]
            if 2 * n < M:
                mu[2 * n] = 2 * _dot(t, t) - mu[0]
        last = t
    return mu


def _evolved(H, a, b, t, kets):
    """exp(-i H t) by the Chebyshev series; J_k(a t) from the integral over a period (exact to rounding)."""
    z, K = a * t, int(a * t) + 60 + int(10 * (a * t) ** (1 / 3))
    q = (np.arange(4 * K) + 0.5) * math.pi / (2 * K)
    J = (np.cos(np.outer(np.arange(K), q) - z * np.sin(q))).mean(1)
    y = torch.zeros_like(kets)
    for k, v in enumerate(H.chebyshev(kets, K)):
        y += complex((1 if k == 0 else 2) * J[k] * (-1j) ** (k % 4)) * v
    return (y * complex(np.exp(-1j * b * t))).cpu().numpy().T


def _zeta(mu, eps, volume):
    M, th = len(mu), np.arccos(eps)
    n, a = np.arange(M)[:, None], np.where(np.arange(M) == 0, 1.0, 2.0)[:, None]
    s, e = np.sqrt(1 - eps ** 2), eps
    T = a * np.cos(n * th)
    P = a * (e - 1j * n * s) * np.exp(1j * n * th)
    z = (T * (mu @ P)).sum(0) + (a * (e + 1j * n * s) * np.exp(-1j * n * th) * (mu @ T)).sum(0)
    return z / (1 - e ** 2) ** 2 / volume


def _greenwood(mu, eps, R):
    T = np.where(np.arange(len(mu)) == 0, 1.0, 2.0)[:, None] * np.cos(np.arange(len(mu))[:, None] * np.arccos(eps))
    return -(T * (mu.real @ T)).sum(0) / (1 - eps ** 2) / R
