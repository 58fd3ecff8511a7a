"""Performance cases of the field evaluation.

What programs that use this library call, over the sizes they call it with:
the direct sum of small and middling systems, the FP64 FMM with the defaults
of the reference's interface, the FP64 FMM at accuracy settings, the
mixed-precision and learned FMM of large systems, packed batches of
independent systems, a plan evaluated for many multipole sets at fixed
coordinates, and periodic boxes.

A case is a dict:
  kind       "direct", "fmm", "batched", "plan" or "periodic"
  system     "water" (molecules of three sites), "uniform" (random points in
             triplets), "blobs" (Gaussian clusters) or "single" (random points,
             no partners)
  n          particles (batched: of the largest system)
  m, f, p    multipole, field and expansion order
  damp       "", "AMOEBA", "THOLE" or "ERF"
  host       whether the call is made on host arrays
  precision, coef, selector, theta, ncrit   as the library's options

The outputs are the potential column and the field columns.  FP64 calls
return them in FP64.  Mixed-precision fields carry about seven digits, so the
programs that ask for them keep them in 32 bits: those cases return float32.
"""
import math

import numpy as np
import torch

import fmm_gb300
from fmm_gb300 import Options, Plan

_DEFAULT = dict(system="water", m=2, f=1, p=5, damp="", theta=0.5, ncrit=64, host=False, precision="fp64",
                coef="ref", selector="fixed", nsys=0)


def _case(**kw):
    return dict(_DEFAULT, **kw)


def listed():
    return [
        # the field at the sites of one solvated molecule, from a Fortran or
        # Python host program: latency, launches and copies
        _case(name="direct_300_host", kind="direct", n=300, damp="THOLE", host=True),
        # direct sum of 4096 random points with quadrupoles, on the device
        _case(name="direct_4k", kind="direct", system="uniform", n=4096),
        # fields and field gradients of a droplet, the check that every other
        # path is compared with
        _case(name="direct_20k_gradient", kind="direct", n=20001, f=2, damp="AMOEBA"),
        # the reference's own call with its own settings: 4096 points,
        # theta 0.5, ncrit 64, order 5, host arrays
        _case(name="fmm_4k_host", kind="fmm", system="uniform", n=4096, host=True),
        # 66,666 water molecules, Thole damping, order 6, field gradients, FP64
        _case(name="fmm_thole_200k", kind="fmm", n=199998, f=2, p=6, damp="THOLE"),
        # plain FP64 FMM at settings that reach 1e-6: damping-aware lists,
        # exact coefficients, odd particle number
        _case(name="fmm_exact_60k", kind="fmm", n=60003, p=10, damp="AMOEBA", theta=0.3, coef="exact"),
        # mixed precision, fixed rule, 100,000 molecules
        _case(name="mixed_300k", kind="fmm", n=300000, p=8, damp="AMOEBA", precision="mixed", coef="exact"),
        # mixed precision with the learned orders: one million sites of water
        _case(name="learned_1m", kind="fmm", n=999999, p=12, theta=0.3, damp="AMOEBA", precision="mixed",
              coef="exact", selector="learned"),
        # the same on clustered particles (deep, uneven tree)
        _case(name="learned_blobs_250k", kind="fmm", system="blobs", n=250000, p=12, theta=0.3, damp="AMOEBA",
              precision="mixed", coef="exact", selector="learned"),
        # 48 independent systems of 1,000 to 20,000 points in one call, host
        # arrays, erf-damped dipoles
        _case(name="batched_48_erf", kind="batched", system="single", n=20000, nsys=48, m=1, p=6, damp="ERF",
              precision="mixed", coef="exact", host=True),
        # one iteration of an induced-dipole solver: a plan kept for fixed
        # coordinates, new dipoles each pass
        _case(name="plan_dipoles_30k", kind="plan", n=30000, m=1, p=6, damp="AMOEBA", precision="mixed",
              coef="exact"),
        # a periodic box of 1,000 water molecules, host arrays
        _case(name="periodic_3k_host", kind="periodic", n=3000, damp="THOLE", host=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["direct", "fp64", "fp64", "exact", "mixed", "mixed", "learned", "batched", "plan", "periodic"])
    damp = rng.choice(["", "AMOEBA", "THOLE", "ERF"])
    if what == "direct":
        m, f = rng.randint(0, 3), rng.randint(0, 3)
        return _case(kind="direct", system=rng.choice(["water", "uniform"]), m=m, f=f, damp=damp,
                     n=_log(rng, 100, 16000 if m + f < 5 else 5000), host=rng.random() < 0.5)
    if what == "fp64":
        return _case(kind="fmm", system=rng.choice(["water", "uniform"]), n=_log(rng, 3000, 120000),
                     m=rng.randint(0, 2), f=rng.randint(0, 2), p=rng.randint(3, 6), damp=damp,
                     ncrit=rng.choice([32, 64, 100]), host=rng.random() < 0.5)
    if what == "exact":
        return _case(kind="fmm", n=_log(rng, 3000, 60000), f=rng.randint(1, 2), p=rng.randint(6, 10),
                     damp=rng.choice(["", "AMOEBA", "ERF"]), theta=rng.choice([0.3, 0.4, 0.5]), coef="exact",
                     host=rng.random() < 0.5)
    if what == "mixed":
        return _case(kind="fmm", system=rng.choice(["water", "uniform", "blobs"]), n=_log(rng, 10000, 500000),
                     m=rng.randint(1, 2), f=rng.randint(1, 2), p=rng.randint(6, 10),
                     damp=rng.choice(["", "AMOEBA"]), theta=rng.choice([0.4, 0.5]), precision="mixed",
                     coef="exact", host=rng.random() < 0.3)
    if what == "learned":
        return _case(kind="fmm", n=_log(rng, 60000, 800000), p=rng.randint(10, 12), theta=0.3, damp="AMOEBA",
                     precision="mixed", coef="exact", selector="learned", host=rng.random() < 0.3)
    if what == "batched":
        return _case(kind="batched", system="single", n=_log(rng, 3000, 30000), nsys=rng.randint(5, 64),
                     m=rng.randint(0, 1), p=rng.randint(5, 7), damp=rng.choice(["", "ERF"]), precision="mixed",
                     coef="exact", host=True)
    if what == "plan":
        return _case(kind="plan", n=_log(rng, 4000, 150000), m=rng.randint(1, 2), p=rng.randint(5, 8),
                     damp=rng.choice(["AMOEBA", "THOLE"]), precision=rng.choice(["mixed", "mixed", "fp64"]),
                     coef="exact")
    return _case(kind="periodic", n=_log(rng, 500, 6000), p=rng.randint(3, 5), damp=rng.choice(["", "THOLE"]),
                 f=rng.randint(1, 2), host=True)


def _nt(k):
    return (k + 1) * (k + 2) * (k + 3) // 6


# ------------------------------------------------------------------ inputs

def _multipoles(g, n, m, group):
    M = torch.empty(_nt(m), n, dtype=torch.float64, device="cuda")
    for k, sig in enumerate((0.5, 0.1, 0.05, 0.02)[:m + 1]):
        lo, hi = (0 if k == 0 else _nt(k - 1)), _nt(k)
        M[lo:hi] = sig * torch.randn(hi - lo, n, dtype=torch.float64, device="cuda", generator=g)
    q = M[0]
    whole = n // group * group
    v = q[:whole].view(-1, group)
    q[:whole] = (v - v.mean(dim=1, keepdim=True)).reshape(-1)
    return M


def _points(g, system, n):
    u = lambda *s: torch.rand(*s, dtype=torch.float64, device="cuda", generator=g)  # noqa: E731
    if system == "water":
        # one molecule per 59 bohr^3, oxygens at random, random orientations
        k = -(-n // 3)
        box = (59.05 * k) ** (1.0 / 3.0)
        O = u(k, 3) * box
        q = torch.randn(k, 4, dtype=torch.float64, device="cuda", generator=g)
        w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
        half = math.radians(104.5) / 2.0
        a, c = 1.8 * math.sin(half), 1.8 * math.cos(half)
        ex = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y + z * w), 2 * (x * z - y * w)], dim=1)
        ez = torch.stack([2 * (x * z + y * w), 2 * (y * z - x * w), 1 - 2 * (x * x + y * y)], dim=1)
        X = torch.stack([O, O + a * ex + c * ez, O - a * ex + c * ez], dim=1).reshape(-1, 3)[:n]
    elif system == "blobs":
        # 64 Gaussian clusters with Dirichlet weights at a mean density of
        # 2 million particles per (600 bohr)^3
        s = (n / 2e6) ** (1.0 / 3.0)
        cen, sig = u(64, 3) * 600.0 * s, (5.0 + 25.0 * u(64)) * s
        wt = -torch.log(u(64))
        b = torch.multinomial(wt / wt.sum(), n, replacement=True, generator=g)
        X = cen[b] + sig[b, None] * torch.randn(n, 3, dtype=torch.float64, device="cuda", generator=g)
        box = 600.0 * s
    else:
        box = (n / (0.1 if system == "single" else 0.064)) ** (1.0 / 3.0)
        X = u(n, 3) * box
    return X.t().contiguous(), box


def _system(g, case, n):
    X, box = _points(g, case["system"], n)
    group = 1 if case["system"] == "single" else 3
    i = torch.arange(n, device="cuda")
    E = torch.stack([i // group * group + k + 1 for k in range(group)])
    E[E > n] = 0
    u = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    d = 0.3 + 0.5 * u if case["damp"] == "ERF" else math.sqrt(0.39) / (1.0 + 9.0 * u) ** (1.0 / 6.0)
    M = _multipoles(g, n, case["m"], n if group == 1 else 3)
    return dict(X=X, M=M, E=E.to(torch.int32).contiguous(), d=d, box=box)


def _sizes(case):
    if case["kind"] != "batched":
        return [case["n"]]
    # log-spaced from 1000 to n, large and small ones mixed
    k = case["nsys"]
    sizes = [int(1000 * (case["n"] / 1000.0) ** (i / (k - 1.0))) for i in range(k)]
    sizes[1::2] = sizes[1::2][::-1]
    return sizes


def _inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + 17)
    if case["kind"] != "batched":
        return _system(g, case, case["n"])
    return [_system(g, case, n) for n in _sizes(case)]


def _options(case):
    kw = dict(precision=case["precision"], selector=case["selector"])
    if case["coef"] == "exact":
        damping = case["damp"] if case["kind"] == "fmm" and case["damp"] in ("AMOEBA", "ERF") else ""
        return Options.exact(mac_mode="damping" if damping and case["theta"] < 0.5 else "ref", **kw)
    return Options(**kw)


def _host(s):
    # (N, k) arrays in Fortran order, as the reference's interface takes them
    return {k: (np.asfortranarray(v.cpu().numpy().T) if torch.is_tensor(v) else v) for k, v in s.items()}


def prepare(case, seed):
    s = _inputs(case, seed)
    opt = _options(case)
    state = dict(case=case, opt=opt)
    if case["kind"] == "batched":
        state["systems"] = [dict(coordinates=h["X"], multipoles=h["M"], exclusions=h["E"], damping_factors=h["d"])
                            for h in map(_host, s)]
        return state
    if case["kind"] == "plan":
        h = _host(s)
        state["plan"] = Plan(h["X"], _nt(case["m"]), h["E"], case["theta"], case["ncrit"], case["p"], case["f"],
                             case["damp"], h["d"], options=opt)
        state["M"] = s["M"]
        state["F"] = torch.zeros(_nt(case["f"]), case["n"], dtype=torch.float64, device="cuda")
        return state
    if case["host"]:
        state.update(_host(s))
        if case["kind"] == "periodic":
            state["cell"] = np.asfortranarray(np.eye(3) * s["box"])
        return state
    # (N, k) views of column-major device buffers
    state.update({k: (v.t() if v.dim() > 1 else v) for k, v in s.items() if torch.is_tensor(v)})
    state["F"] = torch.zeros(_nt(case["f"]), case["n"], dtype=torch.float64, device="cuda").t()
    return state


def _columns(F):
    # (N, k) field: the potential, and the field (and its gradients) if asked for
    return {"potential": F[:, :1], "field": F[:, 1:]} if F.shape[1] > 1 else {"potential": F}


def run(state):
    case, opt = state["case"], state["opt"]
    kind, f, damp = case["kind"], case["f"], case["damp"]
    rule = (case["theta"], case["ncrit"], case["p"], f)
    if kind == "batched":
        out = fmm_gb300.field_fmm_batched(state["systems"], *rule, damp, options=opt)
        return _columns(np.concatenate(out).astype(np.float32))
    if kind == "plan":
        F = state["plan"].execute_device(state["M"], state["F"]).t()
        return _columns(F.float() if case["precision"] == "mixed" else F)
    d = state["d"] if damp else None
    if case["host"]:
        args = (0, state["X"], state["M"], state["E"])
        if kind == "direct":
            F = fmm_gb300.field_direct(*args, f, damp, d, options=opt)
        elif kind == "periodic":
            F = fmm_gb300.field_fmm(*args, *rule, damp, d, True, state["cell"], options=opt)
        else:
            F = fmm_gb300.field_fmm(*args, *rule, damp, d, options=opt)
        return _columns(F.astype(np.float32) if case["precision"] == "mixed" else F)
    args = (state["X"], state["M"], state["E"])
    if kind == "direct":
        fmm_gb300.field_direct_device(*args, f, state["F"], damp, d, options=opt)
    else:
        fmm_gb300.field_fmm_device(*args, *rule, state["F"], damp, d, options=opt)
    return _columns(state["F"].float() if case["precision"] == "mixed" else state["F"])


def _pair_flops(m, f):
    return 2 * _nt(m) * _nt(f) + 2 * math.comb(m + f + 4, 4) + 12


def work(case):
    """Bytes: inputs read once, the field written once.  Flops: the particle
    pairs of the direct sum, or (estimated for an even density) of the near
    field that the acceptance rule leaves, cells closer than sqrt(6) h / theta,
    and (p + 1)^4 multiply-adds for each far pair."""
    m, f, p = case["m"], case["f"], case["p"]
    n = sum(_sizes(case))
    width = 1 if case["system"] == "single" else 3
    size = n * (8 * (3 + _nt(m) + _nt(f) + (1 if case["damp"] else 0)) + 4 * width)
    if case["kind"] == "direct":
        return {"bytes": size, "flops": n * n * _pair_flops(m, f)}
    flops = 0.0
    for k in _sizes(case):
        side = 2.0 ** math.ceil(math.log(max(1.0, k / (0.8 * case["ncrit"])), 8))  # leaves along the box
        leaf, reach = k / side ** 3, math.sqrt(1.5) / case["theta"]  # particles, near cells' distance in cells

        def inside(r):  # share of a ball of r cells that lies in the box, on average
            return 1.0 if case["kind"] == "periodic" else max(0.125, (1.0 - 0.375 * r / side)) ** 3

        near_cells = 4.0 / 3.0 * math.pi * reach ** 3
        near = min(k * 1.0, near_cells * inside(reach) * leaf)
        far = 8.0 / 7.0 * side ** 3 * min(7.0 * near_cells * inside(2.0 * reach), side ** 3)
        flops += k * near * _pair_flops(m, f) + 2.0 * far * (p + 1) ** 4
    return {"bytes": size, "flops": flops}


# ------------------------------------------------------------------ exact values

def _poly(c, v):
    acc = torch.full_like(v, c[-1])
    for a in reversed(c[:-1]):
        acc = acc * v + a
    return acc


def _numerators(damp, a, r, N):
    """n_j = g_j r^(2j+1), g_j = (r^-1 d/dr)^j phi: the closed form
    A_j K(v) + exp(..) q_j(v), and the power series of small v."""
    if damp == "":
        out, c = [], 1.0
        for j in range(N + 1):
            out.append(torch.full_like(r, c))
            c *= -(2 * j + 1)
        return out
    q_shift = lambda q: [0.0] + list(q)  # noqa: E731
    add = lambda p, q: [(p[i] if i < len(p) else 0.0) + (q[i] if i < len(q) else 0.0)  # noqa: E731
                        for i in range(max(len(p), len(q)))]
    dif = lambda q: [i * q[i] for i in range(1, len(q))] or [0.0]  # noqa: E731
    mul = lambda s, q: [s * x for x in q]  # noqa: E731
    K = 70
    ser, closed = [], []
    if damp == "THOLE":
        v, cut = a * r, 3.0
        e, base = torch.exp(-v), 1.0
        A, q, j0 = 1.0, [-1.0, -0.5], 0
        s = [0.0] + [-((-1.0) ** k / math.factorial(k) + 0.5 * (-1.0) ** (k - 1) / math.factorial(k - 1))
                     for k in range(1, K)]
        step = lambda A, q, j: add(mul(-(2 * j + 1), q), q_shift(add(dif(q), mul(-1.0, q))))  # noqa: E731
        power = lambda k, j: k - 1 - 2 * j  # noqa: E731
    elif damp == "AMOEBA":
        v, cut = (a * r) ** 3, 2.0
        e, base = torch.exp(-v), 1.0
        A, q, j0 = -1.0, [1.0], 1
        s = [0.0] + [(-1.0) ** k / math.factorial(k) for k in range(1, K)]
        step = lambda A, q, j: add(mul(-(2 * j + 1), q), mul(3.0, q_shift(add(dif(q), mul(-1.0, q)))))  # noqa: E731
        power = lambda k, j: 3 * k - 3 - 2 * (j - 1)  # noqa: E731
    else:
        v, cut = torch.sqrt(a) * r, 1.5
        e, base = torch.exp(-v * v), torch.erf(v)
        A, q, j0 = 1.0, [0.0], 0
        tp = 2.0 / math.sqrt(math.pi)
        s = [0.0] * (2 * K)
        for k in range(K):
            s[2 * k + 1] = tp * (-1.0) ** k / (math.factorial(k) * (2 * k + 1))
        step = lambda A, q, j: add(mul(-(2 * j + 1), q),  # noqa: E731
                                   q_shift(add([A * tp], add(dif(q), mul(-2.0, q_shift(q))))))
        power = lambda k, j: k - 1 - 2 * j  # noqa: E731
    small = v < cut
    vs = torch.where(small, v, torch.zeros_like(v))
    out = [torch.zeros_like(r)] if j0 else []
    for j in range(j0, N + 1):
        out.append(torch.where(small, _poly(s, vs), A * base + e * _poly(q, v)))
        s = [c * power(k, j) for k, c in enumerate(s)]
        q, A = step(A, q, j), -(2 * j + 1) * A
    return out


def _components(k):
    return [(x, y, o - x - y) for o in range(k + 1) for x in range(o, -1, -1) for y in range(o - x, -1, -1)]


def _direct64(case, s):
    """The field summed over all pairs but the excluded ones, FP64."""
    m, f, n = case["m"], case["f"], s["X"].shape[1]
    N = m + f
    X, E, damp = s["X"], s["E"].long(), case["damp"]
    src, dst = _components(m), _components(f)
    Mc = [s["M"][i] * ((-1.0) ** (sum(c) + 1) / math.prod(math.factorial(k) for k in c)) for i, c in enumerate(src)]
    F = torch.zeros(len(dst), n, dtype=torch.float64, device="cuda")
    rows = max(1, (1 << 22) // n)
    for i0 in range(0, n, rows):
        i1 = min(n, i0 + rows)
        R = [X[k, i0:i1, None] - X[k, None, :] for k in range(3)]
        skip = torch.zeros(i1 - i0, n, dtype=torch.bool, device="cuda")
        at = torch.arange(i1 - i0, device="cuda")
        skip[at, at + i0] = True
        for row in E:
            e = row[i0:i1]
            skip[at[e > 0], e[e > 0] - 1] = True
        R[0] = torch.where(skip, torch.ones_like(R[0]), R[0])
        r2 = R[0] * R[0] + R[1] * R[1] + R[2] * R[2]
        ir = r2.rsqrt()
        a = s["d"][i0:i1, None] * s["d"][None, :] if damp else None
        g, w = [], torch.where(skip, torch.zeros_like(ir), ir)
        for nj in _numerators(damp, a, r2 * ir, N):
            g.append(nj * w)
            w = w * ir * ir
        T = {(0, 0, 0): g[N]}
        for j in range(N - 1, -1, -1):
            new = {(0, 0, 0): g[j]}
            for c in _components(N - j)[1:]:
                ax = 0 if c[0] else (1 if c[1] else 2)
                down = lambda k: tuple(c[b] - (k if b == ax else 0) for b in range(3))  # noqa: E731
                new[c] = R[ax] * T[down(1)]
                if c[ax] > 1:
                    new[c] += (c[ax] - 1) * T[down(2)]
            T = new
        for k, t in enumerate(dst):
            acc = torch.zeros(i1 - i0, dtype=torch.float64, device="cuda")
            for i, c in enumerate(src):
                acc += T[tuple(x + y for x, y in zip(c, t))] @ Mc[i]
            F[k, i0:i1] = acc
    return F


def exact(case, seed):
    """The direct sum, where it is what the case computes: not for periodic
    boxes, for the reference's 32-bit coefficients above order 5 (they wrap),
    for Thole damping in the FMM (its range exceeds the near field's), nor
    where it takes too long.  AMOEBA damping has no potential of its own: the
    FMM's is the far cells' only."""
    fmm = case["kind"] != "direct"
    if case["kind"] == "periodic" or (fmm and case["damp"] == "THOLE"):
        return None
    if fmm and case["coef"] == "ref" and case["p"] > 5:
        return None
    pairs = sum(n * n for n in _sizes(case))
    if pairs > 4e9 or pairs * _pair_flops(case["m"], case["f"]) > 8e11:
        return None
    s = _inputs(case, seed)
    F = torch.cat([_direct64(case, x) for x in (s if isinstance(s, list) else [s])], dim=1).t()
    out = _columns(F.cpu().numpy() if case["host"] else F)
    if fmm and case["damp"] == "AMOEBA":
        out["potential"] = None
    return out
