"""Timed cases of the propagator: what programs have it do, through its public Python entry points.

Every propagation case is one call of a run in progress: the context (tables, state) exists, the call advances the
hierarchy by ``steps`` integrator steps and hands back what the caller reads: the trace of rho_0 and <H> of every
step or of <H> alone (``step_trace``), or the final rho_0 (``step`` + ``rho0``), together with the state the caller
can read on the device (``state_device_ptr``).  Two cases cover the closure network and the closure in use.

Families (the ``kind`` of a case):

* ``heom``    one hierarchy: a transverse-field spin glass with sigma_z baths on its spins (``coupling="spin"``), one
              collective diagonal bath (``"collective"``) or one collective bath with spin flips (``"flip"``, the
              reference's compiled model), in double or mixed precision, packed or full slabs
* ``dense``   the same with every entry of H non-zero, on the matrix path
* ``sparse``  random sparse Hermitian H and coupling operators (operators handed over as CSR)
* ``batch``   a disorder average over many small instances of uneven size
* ``closure`` a truncated hierarchy whose missing tier is supplied by the closure network
* ``mlp``     loss and gradients, or the forward pass, of that network on host arrays
"""
from __future__ import annotations

import math

import numpy as np
import torch

from helix_b200 import capi
from helix_b200 import systems as S

DT = {"heom": 0.005, "dense": 0.005, "sparse": 0.01, "batch": 0.01, "closure": 0.01}


def _heom(n, depth, K, baths, coupling="spin", precision="double", full=False, trace="all", steps=10):
    return {"kind": "heom", "n": n, "depth": depth, "K": K, "baths": baths, "coupling": coupling,
            "precision": precision, "full": full, "trace": trace, "steps": steps}


def listed():
    return [
        # the smallest call a program makes: one step of two spins (15 ADOs), with its observables
        dict(_heom(2, 2, 1, 2, steps=1), name="tiny_d4"),
        # four spins with Pade K = 2, depth 3 (455 ADOs): an interactive run, every step recorded
        dict(_heom(4, 3, 2, 4, steps=20), name="spin_d16"),
        # five spins, depth 3 (816 ADOs): the ordinary small production run
        dict(_heom(5, 3, 2, 5, steps=10), name="spin_d32"),
        # six spins, depth 4 (7315 ADOs): the flagship run, final density only
        dict(_heom(6, 4, 2, 6, trace="final", steps=4), name="spin_d64"),
        # eight spins, depth 3 (969 ADOs): larger than the caches, double precision
        dict(_heom(8, 3, 1, 8, trace="final", steps=2), name="spin_d256"),
        # the same hierarchy kept in complex64 with rho_0 in double precision
        dict(_heom(8, 3, 1, 8, precision="mixed", steps=4), name="spin_d256_mixed"),
        # the reference's compiled model: ten spins, one collective bath with spin flips (10 ADOs), energy recorded
        dict(_heom(10, 2, 2, 1, coupling="flip", trace="energy", steps=2), name="flip_d1024"),
        # a dense Hamiltonian (every entry non-zero) at d = 256, 969 ADOs, on the matrix path
        {"kind": "dense", "n": 8, "depth": 3, "K": 1, "baths": 8, "steps": 2, "name": "dense_d256"},
        # general sparse operators for H and for six couplings (91 ADOs)
        {"kind": "sparse", "n": 6, "depth": 2, "K": 1, "baths": 6, "per_row": 3, "steps": 4, "name": "sparse_d64"},
        # a disorder average over 128 realisations of three to five spins
        {"kind": "batch", "count": 128, "n_max": 5, "depth_max": 4, "K": 2, "steps": 5, "name": "batch_128"},
        # depth 2 plus the closure at d = 32, every step recorded
        {"kind": "closure", "n": 5, "depth": 2, "K": 2, "hidden": 512, "steps": 20, "name": "closure_d32"},
        # one optimisation step's gradients of the closure network: 4096 samples, width 512
        {"kind": "mlp", "rows": 4096, "inp": 21, "hidden": 512, "out": 2, "backward": True, "name": "mlp_grad"},
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))


# elements of the whole hierarchy (ADOs x d^2, times the couplings where each has its own operator products)
_MOST = {"heom": 60e6, "flip": 11e6, "dense": 60e6, "sparse": 2.4e6, "closure": 4e6}


def draw(rng):
    while True:
        kind = rng.choice(["spin", "spin", "spin", "band", "mixed", "flip", "dense", "sparse", "batch", "closure",
                           "mlp"])
        steps = rng.randint(1, 12)
        if kind == "spin":
            n = rng.randint(1, 6)
            coupling = rng.choice(["spin", "spin", "collective"])
            baths = rng.randint(1, n) if coupling == "spin" else 1
            c = _heom(n, rng.randint(1, 4 if coupling == "spin" else 9), rng.randint(0, 3), baths, coupling,
                      full=n >= 5 and rng.random() < 0.25, trace=rng.choice(["all", "all", "energy", "final"]), steps=steps)
        elif kind in ("band", "mixed"):
            n = rng.choice([7, 7, 8, 9])
            c = _heom(n, rng.randint(2, 3), rng.randint(0, 2), rng.randint(1, n),
                      precision="mixed" if kind == "mixed" else "double", full=rng.random() < 0.25,
                      trace=rng.choice(["all", "all", "energy", "final"]), steps=min(steps, 4))
        elif kind == "flip":
            c = _heom(rng.randint(2, 10), rng.randint(1, 5), rng.randint(0, 3), 1, "flip", trace=rng.choice(["all", "all", "energy", "final"]),
                      steps=min(steps, 4))
        elif kind == "dense":
            n = rng.choice([7, 8, 9])
            c = {"kind": "dense", "n": n, "depth": rng.randint(2, 3), "K": rng.randint(0, 1),
                 "baths": rng.randint(1, n), "steps": min(steps, 3)}
        elif kind == "sparse":
            n = rng.randint(2, 7)
            c = {"kind": "sparse", "n": n, "depth": rng.randint(1, 3), "K": rng.randint(0, 2),
                 "baths": rng.randint(1, n), "per_row": rng.randint(1, 6), "steps": min(steps, 4)}
        elif kind == "batch":
            return {"kind": "batch", "count": _log_int(rng, 3, 128), "n_max": rng.randint(3, 5),
                    "depth_max": rng.randint(2, 4), "K": rng.randint(1, 2), "steps": rng.randint(1, 5)}
        elif kind == "closure":
            c = {"kind": "closure", "n": rng.randint(2, 6), "depth": rng.randint(1, 2), "K": rng.randint(0, 2),
                 "hidden": rng.choice([64, 96, 256, 512]), "steps": steps}
        else:
            return {"kind": "mlp", "rows": _log_int(rng, 16, 4096), "inp": rng.randint(5, 60),
                    "hidden": rng.choice([32, 64, 96, 200, 256, 512]), "out": rng.choice([2, 2, 2, 7, 64]),
                    "backward": rng.random() < 0.7}
        size = S.hierarchy_size(_modes(c), c["depth"] + 1) * 4 ** c["n"] * (c["baths"] if kind == "sparse" else 1)
        if size <= _MOST.get(kind, _MOST["heom"]):
            return c


def _modes(c):
    return (c["baths"] if "baths" in c else c["n"]) * (c["K"] + 1)


# ---------------------------------------------------------------------------------------------------------------
# models, from the seed alone


def _signs(n):
    r = np.arange(1 << n)
    return np.stack([np.where((r >> i) & 1, 1.0, -1.0) for i in range(n)])


def _glass(rng, n, K, baths, h=1.0, lam=0.1, temperature=1.0):
    """Diagonal and flips of H (J_ij ~ N(0, 1), transverse field h) and one sigma_z bath on each of the first spins."""
    s = _signs(n)
    e = np.zeros(1 << n)
    for i in range(n):
        for j in range(i + 1, n):
            e += rng.standard_normal() * s[i] * s[j]
    bath = dict(beta=1.0 / temperature, gamma=1.0, zeta=2.0 * lam, K=K)
    return {"e": e, "f": np.full(n, float(h)), "h": None, "baths": [dict(bath, v=s[i]) for i in range(baths)]}


def _hermitian(rng, d, per_row, scale):
    """Random sparse Hermitian matrix with a full real diagonal and about 2 per_row other entries in a row."""
    m = np.zeros((d, d), np.complex128)
    for r in range(d):
        for c in rng.integers(0, d, per_row):
            m[r, c] += scale * complex(rng.uniform(-1, 1), rng.uniform(-1, 1))
    return 0.5 * (m + m.conj().T) + np.diag(rng.uniform(-scale, scale, d))


def _model(c, seed):
    rng = np.random.default_rng([seed, 77])
    kind, n = c["kind"], c["n"]
    d = 1 << n
    if kind == "sparse":
        return {"e": np.zeros(d), "f": np.zeros(n), "h": _hermitian(rng, d, c["per_row"], 1.0),
                "baths": [dict(beta=1.0, gamma=1.0, zeta=0.2, K=c["K"], v=_hermitian(rng, d, 2, 0.5))
                          for _ in range(c["baths"])]}
    m = _glass(rng, n, c["K"], c.get("baths", n))
    if kind == "dense":
        g = rng.uniform(-1, 1, (d, d)) + 1j * rng.uniform(-1, 1, (d, d))
        m["h"] = _dense(m, d) + 0.25 * (g + g.conj().T) / math.sqrt(d)
    elif c.get("coupling") == "collective":
        m["baths"] = [dict(m["baths"][0], zeta=0.05, v=_signs(n).T @ rng.uniform(0.4, 0.6, n))]
    elif c.get("coupling") == "flip":
        # the reference's compiled model: diagonal H, V = sum of projections + flips of the spins
        m["f"] = np.zeros(n)
        m["baths"] = [dict(m["baths"][0], zeta=0.01, v=0.5 * _signs(n).sum(0), w=rng.uniform(0.8, 1.2, n))]
        m["e"] = 0.3 * m["e"]
    return m


def _dense(m, d):
    """H as a matrix: the given one, or the diagonal and the flips."""
    return m["h"] if m["h"] is not None else _flips(m["e"], m["f"], d)


def _flips(diag, f, d):
    h = np.diag(diag).astype(np.complex128)
    r = np.arange(d)
    for i, x in enumerate(f):
        h[r, r ^ (1 << i)] += x
    return h


def _csr(m):
    r, c = np.nonzero(m)
    ptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=m.shape[0]))])
    return ptr.astype(np.int32), c.astype(np.int32), m[r, c]


def _problem(m, n, depth, dt):
    baths = []
    for b in m["baths"]:
        args = {k: b[k] for k in ("beta", "gamma", "zeta", "K")}
        if b["v"].ndim == 2:
            baths.append(S.BathSpec(**args, v_csr=_csr(b["v"])))
        else:
            baths.append(S.BathSpec(**args, v_diag=b["v"], v_flip=b.get("w")))
    return S.Problem(dim=1 << n, h_diag=m["e"], h_flip=m["f"], baths=baths, max_depth=depth + 1, dt=dt,
                     h_csr_explicit=None if m["h"] is None else _csr(m["h"]))


def _instances(c, seed):
    """(model, spins, depth) of every realisation of a disorder average; the case alone gives their sizes."""
    out = []
    shape = np.random.default_rng([c["count"], c["n_max"], c["depth_max"]])
    for i in range(c["count"]):
        rng = np.random.default_rng([seed, i])
        n, depth = int(shape.integers(3, c["n_max"] + 1)), int(shape.integers(2, c["depth_max"] + 1))
        out.append((_glass(rng, n, c["K"], n, rng.uniform(0.5, 1.5), rng.uniform(0.05, 0.2), rng.uniform(0.5, 2.0)),
                    n, depth))
    return out


def _mlp_arrays(c, seed):
    rng = np.random.default_rng([seed, 5])
    sizes = [c["inp"], c["hidden"], c["hidden"], c["out"]]
    params = np.concatenate([a.ravel() for i in range(3) for a in (
        rng.uniform(-1, 1, (sizes[i + 1], sizes[i])) * math.sqrt(6.0 / sizes[i]), 0.1 * rng.uniform(-1, 1, sizes[i + 1]))])
    x, t = rng.uniform(-1, 1, (c["rows"], c["inp"])), rng.uniform(-1, 1, (c["rows"], c["out"]))
    return params.astype(np.float32), x.astype(np.float32), t.astype(np.float32)


# ---------------------------------------------------------------------------------------------------------------
# the calls


class _View:
    """A context's device buffer of complex doubles as torch reads it; the tensor keeps the context alive."""

    def __init__(self, ctx, shape):
        self.owner = ctx
        self.__cuda_array_interface__ = {"data": (ctx.state_device_ptr(), False), "shape": shape, "typestr": "<c16",
                                         "version": 3}


def _state_view(ctx):
    """The context's state on the device: [ADOs, elements of a slab], rho_0 alone in mixed precision."""
    d = ctx.dim
    packed = d * (d + 1) // 2 if ctx.hermitian_packed else d * d
    rows = 1 if ctx.mixed else ctx.size
    return torch.as_tensor(_View(ctx, (rows, packed)), device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        params, x, t = _mlp_arrays(case, seed)
        net = capi.MLP(case["inp"], case["hidden"], case["out"])
        net.set_params(params)
        return {"case": case, "net": net, "x": x, "t": t}
    if kind == "batch":
        problems = [_problem(m, n, depth, DT[kind]) for m, n, depth in _instances(case, seed)]
        return {"case": case, "batch": capi.Batch(problems)}
    p = _problem(_model(case, seed), case["n"], case["depth"], DT[kind])
    mixed = kind == "dense" or case.get("precision") == "mixed"
    ctx = capi.Context(p, precision="mixed" if mixed else "double", full_state=case.get("full", False),
                       dense_h=kind == "dense")
    ctx.mixed = mixed
    state = {"case": case, "ctx": ctx}
    if kind == "closure":
        rng = np.random.default_rng([seed, 9])
        closure = capi.Closure(p, case["depth"] + 3, hidden=case["hidden"], capacity=1, seed=seed)
        w = closure.mlp.params()
        closure.mlp.set_params((w * rng.uniform(0.5, 1.0, w.size)).astype(np.float32))
        closure.set_scales(1.0, 0.05)
        closure.attach(ctx)
        state["closure"] = closure
    state["view"] = _state_view(ctx)
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "mlp":
        if case["backward"]:
            return state["net"].gradients(state["x"], state["t"])
        return state["net"].forward(state["x"])
    if case["kind"] == "batch":
        batch = state["batch"]
        sz = batch.step(case["steps"])
        return {"sz": sz, "rho": np.concatenate([batch.rho0(i).ravel() for i in range(batch.count)])}
    ctx = state["ctx"]
    trace = case.get("trace", "all")
    if trace != "final":
        rho, energy = ctx.step_trace(case["steps"], rho0=trace == "all")
        return {"rho": rho, "energy": energy, "state": state["view"]}
    ctx.step(case["steps"])
    return {"rho": ctx.rho0(), "state": state["view"]}


def work(case):
    """Bytes: every step reads the hierarchy and writes it (the Hermitian half of each ADO, as wide as the path
    stores it); flops: four evaluations of the right-hand side a step."""
    kind = case["kind"]
    if kind == "mlp":
        h, passes = case["hidden"], 3 if case["backward"] else 1
        weights = case["inp"] * h + h * h + h * case["out"]
        return {"bytes": 4.0 * (case["rows"] * (case["inp"] + case["out"]) + 2 * weights),
                "flops": 2.0 * passes * case["rows"] * weights}
    if kind == "batch":
        total = [0.0, 0.0]
        for n in range(3, case["n_max"] + 1):  # the mean over the shapes it draws from
            for depth in range(2, case["depth_max"] + 1):
                share = case["count"] / ((case["n_max"] - 2) * (case["depth_max"] - 1))
                for i, v in enumerate(_step_work(n, S.hierarchy_size(n * (case["K"] + 1), depth + 1),
                                                 n * (case["K"] + 1), 16)):
                    total[i] += share * v
        return {"bytes": case["steps"] * total[0], "flops": case["steps"] * total[1]}
    wide = 8 if kind == "dense" or case.get("precision") == "mixed" else 16
    size = S.hierarchy_size(_modes(case), case["depth"] + 1)
    b, f = _step_work(case["n"], size, _modes(case), wide)
    if kind == "dense":
        f += 4.0 * 8.0 * size * 8 ** case["n"]
    if kind == "sparse" or case.get("coupling") == "flip":
        b, f = 2 * b, 3 * f
    return {"bytes": case["steps"] * b, "flops": case["steps"] * f}


def _step_work(n, size, modes, wide):
    d = 1 << n
    half = size * d * (d + 1) // 2
    return 2.0 * wide * half, 4.0 * half * (12 + 8 * n + 4 * modes)


# ---------------------------------------------------------------------------------------------------------------
# the same results in 64 bits, by torch matrix products over the whole hierarchy


def _pade(K):
    """Poles and residues of the [K-1/K] Pade form of the Bose function."""
    def eig(size, shift):
        b = 2.0 * (np.arange(size) + shift) + 1.0
        off = 1.0 / np.sqrt(b[:-1] * b[1:])
        return np.sort(np.linalg.eigvalsh(np.diag(off, 1) + np.diag(off, -1)))[::-1]

    if K == 0:
        return np.zeros(0), np.zeros(0)
    poles = 2.0 / eig(2 * K, 1)[:K]
    xi, zeta = poles ** 2, 4.0 / eig(2 * K - 1, 2)[:K - 1] ** 2
    res = np.full(K, 0.5 * K * (2 * K + 3))
    for i in range(K):
        for j in range(K - 1):
            res[i] *= zeta[j] - xi[i]
        for j in range(K):
            if j != i:
                res[i] /= xi[j] - xi[i]
    return poles, res


def _bath(b):
    """Rates of the modes, their down weights, and the double-commutator, counter and anti-commutator factors."""
    beta, gamma, zeta = b["beta"], b["gamma"], b["zeta"]
    poles, res = _pade(b["K"])
    nu, x = poles / beta, 0.5 * beta * gamma
    pade = 2.0 * res * gamma ** 2 / (nu ** 2 - gamma ** 2)
    down = np.concatenate([[x / math.tan(x) * zeta / beta], zeta / beta * pade])
    return {"nu": np.concatenate([[gamma], nu]), "down": down, "xi": (1.0 - x / math.tan(x) - pade.sum()) * zeta / beta,
            "kappa": zeta * x / beta, "anti": x * zeta / beta}


def _rows(modes, most):
    """Index vectors with sum <= most, the first mode most significant."""
    if modes == 1:
        return [[k] for k in range(most + 1)]
    return [[k] + r for k in range(most + 1) for r in _rows(modes - 1, most - k)]


class _Exact:
    def __init__(self, m, n, depth, dev):
        self.d, self.dev = 1 << n, dev
        bath = [_bath(b) for b in m["baths"]]
        mode = [(j, k) for j, b in enumerate(bath) for k in range(len(b["nu"]))]
        rows = np.array(_rows(len(mode), depth), np.int64)
        at = {r.tobytes(): i for i, r in enumerate(rows)}
        self.size = len(rows)
        step = np.eye(len(mode), dtype=np.int64)
        edge = lambda x: [at.get(r.tobytes(), self.size) for r in rows + x]  # noqa: E731
        t = lambda x: torch.as_tensor(np.asarray(x), device=dev)  # noqa: E731
        nu = np.array([bath[j]["nu"][k] for j, k in mode])
        self.g = t(rows @ nu)[:, None, None]
        self.h = t(_dense(m, self.d))
        self.baths = []
        for j, b in enumerate(bath):
            v = m["baths"][j]["v"]
            if m["baths"][j].get("w") is not None:
                v = _flips(v, m["baths"][j]["w"], self.d)
            modes = [i for i, (jj, _) in enumerate(mode) if jj == j]
            ups = [t(edge(step[i])) for i in modes]
            downs = [(t(edge(-step[i])), t(rows[:, i] * nu[i] * b["down"][mode[i][1]])[:, None, None]) for i in modes]
            anti = t(rows[:, modes[0]] * nu[modes[0]] * b["anti"])[:, None, None]
            self.baths.append((t(v), b["xi"], b["kappa"], ups, downs, anti))

    def sides(self, v, x):
        return (v[:, None] * x, x * v) if v.ndim == 1 else (v @ x, x @ v)

    def rhs(self, x):
        zero = torch.zeros_like(x[:1])
        a = torch.cat([x, zero])
        out = -1j * (self.h @ x - x @ self.h) - self.g * x
        for v, xi, kappa, ups, downs, anti in self.baths:
            left, right = self.sides(v, x)
            s = -1j * xi * (left - right)  # -i [V, s] below makes it -xi [V, [V, x]]
            cl, cr = self.sides(v, left - right)
            out -= 1j * kappa * (cl + cr)
            for up in ups:
                s += a[up]
            for down, w in downs:
                s += w * a[down]
            left, right = self.sides(v, s)
            out -= 1j * (left - right)
            left, right = self.sides(v, a[downs[0][0]])
            out -= anti * (left + right)
        return out

    def steps(self, steps, dt):
        x = torch.zeros(self.size, self.d, self.d, dtype=torch.complex128, device=self.dev)
        x[0, -1, -1] = 1.0
        rho, energy = [], []
        for _ in range(steps):
            cur = x
            x = x.clone()
            for j in range(1, 5):
                cur = self.rhs(cur) * (dt / j)
                x += cur
            rho.append(x[0].clone())
            energy.append(torch.einsum("ij,ji->", self.h, x[0]).real)
        return torch.stack(rho), torch.stack(energy), x


def _packed(x):
    """The upper triangles in the order of the packed device slabs."""
    d = x.shape[-1]
    i = np.arange(d // 2 * (d + 1))
    s, t = i // (d + 1), i % (d + 1)
    first = t < d - s
    r, c = np.where(first, s, d - 1 - s), np.where(first, s + t, t - 1)
    return x.reshape(len(x), -1)[:, torch.as_tensor(r * d + c, device=x.device)]


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "closure":
        return None  # the closure's coefficients are what its 16-bit network says
    if kind == "mlp":
        params, x, t = (torch.as_tensor(a, device=dev).double() for a in _mlp_arrays(case, seed))
        params.requires_grad_(True)
        sizes, y, o = [case["inp"], case["hidden"], case["hidden"], case["out"]], x, 0
        for i in range(3):
            a, b = sizes[i], sizes[i + 1]
            y = y @ params[o:o + a * b].reshape(b, a).T + params[o + a * b:o + a * b + b]
            y = torch.nn.functional.gelu(y) if i < 2 else y
            o += a * b + b
        if not case["backward"]:
            return y.detach().cpu().numpy()
        loss = ((y - t) ** 2).mean()
        loss.backward()
        return float(loss), params.grad.cpu().numpy()
    if kind == "batch":
        sz, rho = np.zeros(case["steps"]), []
        for m, n, depth in _instances(case, seed):
            r, _, _ = _Exact(m, n, depth, dev).steps(case["steps"], DT[kind])
            r = r.cpu().numpy()
            sz += np.einsum("tii,i->t", r, _signs(n)[0]).real
            rho.append(r[-1].ravel())
        return {"sz": sz, "rho": np.concatenate(rho)}
    rho, energy, x = _Exact(_model(case, seed), case["n"], case["depth"], dev).steps(case["steps"], DT[kind])
    mixed = kind == "dense" or case.get("precision") == "mixed"
    # packed slabs: d >= 32, couplings diagonal, not asked to keep full slabs
    packed = case["n"] >= 5 and kind == "heom" and case["coupling"] != "flip" and not case["full"]
    x = x[:1] if mixed else x
    state = _packed(x) if packed else x.reshape(len(x), -1)
    trace = case.get("trace", "all")
    if trace != "final":
        return {"rho": rho.cpu().numpy() if trace == "all" else None, "energy": energy.cpu().numpy(), "state": state}
    return {"rho": rho[-1].cpu().numpy(), "state": state}
