"""The measured work of this framework: hafnians and loop hafnians through its public entry points.

A case is a dict of plain values; ``kind`` selects the entry point:

* ``plain``  ``hafnian(A)`` of one n x n matrix, real or complex, in the stated precision
* ``graph``  ``hafnian(A)`` of a 0/1 adjacency matrix: the number of perfect matchings, which
  integer input gets exactly by default
* ``loop``   ``hafnian(A, loop=True)``: even and odd n
* ``gbs``    ``hafnian_repeated(A, rpt, mu, loop=True)``: a photon pattern of a Gaussian state
* ``modes``  ``loop_hafnian_batch(A, D, fixed, cutoff)``: one step of a chain-rule sampler, every
  photon number of the last mode at once
* ``plan``   a device-resident plan over many matrices of uneven size, executed and read
* ``serve``  a ``ProbabilityServer`` answering a burst of Fock-probability requests

Sizes and value distributions are those of ``thewalrus_gb300/workloads.py``, ``bench.py`` and the
tests: the 24 x 24 and 40 x 40 hafnians, the 20-mode state with 40 photons, uneven batches, the
12-mode sampler, 64-mode serving states.
"""
import math

import numpy as np
import torch

import thewalrus_gb300 as tw
from thewalrus_gb300 import _native as nat
from thewalrus_gb300 import workloads as wl
from thewalrus_gb300.serving import GaussianState, ProbabilityServer


def listed():
    return [
        # the smallest useful call, one matrix at a time in a user's loop: latency and launches
        {"name": "plain_c8", "kind": "plain", "n": 8, "matrix": "complex", "precision": "default"},
        # an everyday size, the 24 x 24 complex workload
        {"name": "plain_c24", "kind": "plain", "n": 24, "matrix": "complex", "precision": "default"},
        # the headline: one 40 x 40 complex hafnian
        {"name": "plain_c40", "kind": "plain", "n": 40, "matrix": "complex", "precision": "default"},
        # the largest: a real matrix, a size up from the headline
        {"name": "plain_r44", "kind": "plain", "n": 44, "matrix": "signed", "precision": "default"},
        # perfect matchings of a random graph, exact by default
        {"name": "graph_32", "kind": "graph", "n": 32},
        # loop hafnian of an odd number of vertices
        {"name": "loop_c27", "kind": "loop", "n": 27, "matrix": "complex"},
        # Fock amplitude of a 20-mode Gaussian state: 40 photons, up to 3 in a mode
        {"name": "gbs_20x40", "kind": "gbs", "modes": 20, "photons": 40, "max_rep": 3},
        # one mode's conditional distribution in a chain-rule sampler
        {"name": "modes_12c6", "kind": "modes", "modes": 12, "cutoff": 6, "max_fixed": 2},
        # many matrices of uneven size in one plan, half real and half complex
        {"name": "plan_96x32", "kind": "plan", "count": 96, "n_min": 8, "n_max": 32},
        # a burst of probability requests on a resident 64-mode state
        {"name": "serve_64x28", "kind": "serve", "requests": 64, "modes": 64, "photons": 28, "max_rep": 2},
        # double-double terms, for sums that cancel
        {"name": "plain_c28_dd", "kind": "plain", "n": 28, "matrix": "complex", "precision": "dd"},
        # double-float terms
        {"name": "plain_c34_df", "kind": "plain", "n": 34, "matrix": "complex", "precision": "df"},
    ]


def draw(rng):
    kind = rng.choice(["plain", "plain", "plain", "graph", "loop", "gbs", "modes", "plan", "serve"])
    if kind == "plain":
        matrix = rng.choice(["complex", "complex", "signed", "nonneg"])
        precision = rng.choice(["default", "default", "default", "dd", "df"])
        top = {"default": 40 if matrix == "complex" else 44, "df": 40, "dd": 34}[precision]
        return {"kind": kind, "n": 2 * rng.randint(3, top // 2), "matrix": matrix, "precision": precision}
    if kind == "graph":
        return {"kind": kind, "n": 2 * rng.randint(3, 19)}
    if kind == "loop":
        return {"kind": kind, "n": rng.randint(5, 37), "matrix": rng.choice(["complex", "complex", "signed"])}
    if kind == "gbs":
        modes = rng.randint(4, 20)
        return {"kind": kind, "modes": modes, "photons": 2 * rng.randint(3, min(20, 2 * modes)),
                "max_rep": rng.randint(2, 4)}
    if kind == "modes":
        return {"kind": kind, "modes": rng.randint(4, 14), "cutoff": rng.randint(2, 8),
                "max_fixed": rng.randint(1, 3)}
    if kind == "plan":
        return {"kind": kind, "count": round(math.exp(rng.uniform(math.log(8), math.log(256)))),
                "n_min": 8, "n_max": 2 * rng.randint(6, 16)}
    return {"kind": kind, "requests": round(math.exp(rng.uniform(math.log(8), math.log(128)))),
            "modes": rng.choice([24, 48, 64]), "photons": 2 * rng.randint(5, 14), "max_rep": rng.randint(1, 2)}


# ---------------------------------------------------------------------------------- inputs


def _matrix(matrix, n, seed):
    if matrix == "complex":
        return wl.complex_symmetric(n, seed)
    return wl.real_signed(n, seed) if matrix == "signed" else wl.real_nonneg(n, seed)


def _state_matrix(modes, rng):
    U = wl.haar_unitary(modes, rng)
    return U @ np.diag(np.tanh(rng.uniform(0.3, 0.8, size=modes))) @ U.T


def _inputs(case, seed):
    """The arguments of a case's call (numpy arrays), from the seed alone."""
    rng = np.random.default_rng([seed, 77])
    kind = case["kind"]
    if kind in ("plain", "loop"):
        return (_matrix(case["matrix"], case["n"], seed),)
    if kind == "graph":
        return (wl.adjacency01(case["n"], seed=seed, p=0.5),)
    if kind == "gbs":
        m = case["modes"]
        B = _state_matrix(m, rng)
        Z = np.zeros_like(B)
        A = np.block([[B, Z], [Z, B.conj()]])
        gamma = _displacements(2 * m, rng)
        np.fill_diagonal(A, gamma)
        return A, gamma, _patterns(case)[0]
    if kind == "modes":
        return (_state_matrix(case["modes"], rng), _displacements(case["modes"], rng), _patterns(case)[0],
                case["cutoff"])
    if kind == "plan":
        return ([_matrix("nonneg" if i % 2 else "complex", n, int(rng.integers(1 << 31)))
                 for i, n in enumerate(_sizes(case))],)
    return _state_matrix(case["modes"], rng), _displacements(case["modes"], rng), _patterns(case)


def _displacements(count, rng):
    return (rng.normal(size=count) + 1j * rng.normal(size=count)) * np.sqrt(0.1 / 2)


# The sizes of a plan's matrices and the photon patterns belong to the case, so that every seed of
# it is the same amount of work on other values.


def _sizes(case):
    lo, hi = case["n_min"] // 2, case["n_max"] // 2
    return [2 * (lo + (7 * i) % (hi - lo + 1)) for i in range(case["count"])]


def _patterns(case):
    rng = np.random.default_rng([case["modes"], case.get("photons", 0), case.get("max_rep", 0)])
    if case["kind"] == "gbs":  # the photon pattern on both halves
        nvec = wl.photon_pattern(case["modes"], case["photons"] // 2, case["max_rep"], rng)
        return [np.concatenate([nvec, nvec])]
    if case["kind"] == "modes":
        return [rng.integers(0, case["max_fixed"] + 1, size=case["modes"] - 1)]
    half = case["photons"] // 2 - 1  # even photon numbers 4 .. photons, each as often as the others
    return [wl.photon_pattern(case["modes"], 4 + 2 * ((5 * i) % half), case["max_rep"], rng)
            for i in range(case["requests"])]


def prepare(case, seed):
    args = _inputs(case, seed)
    kind = case["kind"]
    state = {"kind": kind, "args": args}
    if kind == "plain" and case["precision"] != "default":
        state["precision"] = case["precision"]
    if kind == "plan":
        state["plan"] = nat.Plan([tw.prepare_hafnian(M) for M in args[0]])
    if kind == "serve":
        B, alpha, patterns = args
        gs = GaussianState(B, alpha)
        state["server"] = ProbabilityServer([gs])
        state["requests"] = [(0.0, 0, p) for p in patterns]
    return state


def run(state):
    kind, args = state["kind"], state["args"]
    if kind in ("plain", "graph"):
        return tw.hafnian(args[0], precision=state.get("precision"))
    if kind == "loop":
        return tw.hafnian(args[0], loop=True)
    if kind == "gbs":
        A, gamma, rpt = args
        return tw.hafnian_repeated(A, rpt, mu=gamma, loop=True)
    if kind == "modes":
        A, D, fixed, cutoff = args
        return tw.loop_hafnian_batch(A, D, fixed, cutoff)
    if kind == "plan":
        state["plan"].execute()
        return state["plan"].read()
    served = state["server"].serve(state["requests"])
    return np.array([r["amplitude"] for r in served])


# ---------------------------------------------------------------------------------- work


def _pairs(counts):
    """Edges (i, j, multiplicity) over the vertices with their counts, the largest two first, and
    the vertex left over when the total is odd (else None)."""
    left = {i: int(c) for i, c in enumerate(counts) if c}
    edges, odd = [], None
    while left:
        order = sorted(left, key=lambda i: (-left[i], -i))
        i = order[0]
        if len(order) == 1 or left[i] > 2 * left[order[1]]:
            if left[i] == 1:
                odd = i
                break
            edges.append((i, i, left[i] // 2))
            left[i] %= 2
        else:
            j = order[1]
            m = left[j]
            edges.append((i, j, m))
            left[i] -= m
            left[j] = 0
        left = {k: c for k, c in left.items() if c}
    return edges, odd


def _tree_macs(reps, loop, extra):
    """Multiply-adds of the sieve sum over edges of these multiplicities, evaluated as a tree: one
    edge eliminated per level (a symmetric rank-2 update of the remaining vertices' power series
    per order of the edge), the updates shared by the edge's signs, the last two simple edges in
    closed form.  ``extra`` counts unpaired vertices."""
    reps = sorted((int(r) for r in reps if r > 0), reverse=True)
    nodes, macs, deg = 0.5, 0.0, 0
    for q, r in enumerate(reps):
        v = 2 * (len(reps) - q - 1) + extra
        if v <= 2 + extra and r == 1 and len(reps) > 1:
            break
        deg += r
        entries = v * (v - 1) / 2 + (v if loop else 0) + 1
        macs += max(nodes, 1.0) * r * 2 * entries * deg * (deg + 1) / 2
        nodes *= r + 1
    return macs + max(nodes, 1.0) * (10 if loop else 3) * (deg + 1) * (deg + 2) / 2


def work(case):
    kind = case["kind"]
    if kind == "plain":
        n = case["n"]
        per = 8 if case["matrix"] == "complex" else 2
        b = n * n * (16 if case["matrix"] == "complex" else 8) + 16
        return {"bytes": b, "flops": per * _tree_macs([1] * (n // 2), False, 0)}
    if kind == "graph":
        n = case["n"]
        return {"bytes": 8 * n * n + 16, "flops": 2 * _tree_macs([1] * (n // 2), False, 0)}
    if kind == "loop":
        n = case["n"]
        c = case["matrix"] == "complex"
        return {"bytes": n * n * (16 if c else 8) + 16,
                "flops": (8 if c else 2) * _tree_macs([1] * (n // 2), True, n % 2)}
    if kind == "plan":
        b = f = 0.0
        for i, n in enumerate(_sizes(case)):
            b += n * n * (8 if i % 2 else 16) + 16
            f += (2 if i % 2 else 8) * _tree_macs([1] * (n // 2), False, 0)
        return {"bytes": b, "flops": f}
    m, f = case["modes"], 0.0
    patterns = _patterns(case)
    for p in patterns:
        edges, odd = _pairs(p)
        f += 8 * _tree_macs([e[2] for e in edges], True, int(odd is not None) + int(kind == "modes"))
    if kind == "gbs":
        return {"bytes": 16 * (4 * m * m + 2 * m) + 16 * m + 16, "flops": f}
    if kind == "modes":
        return {"bytes": 16 * (m * m + m + case["cutoff"] + 1) + 8 * m, "flops": f}
    return {"bytes": 16 * (m * m + m) + len(patterns) * (8 * m + 16), "flops": f}


# ---------------------------------------------------------------------------------- reference


def _power_trace_sieve(A, v, counts, last=None, cutoff=0, limit=1.2e13):
    """Loop hafnian (plain hafnian: v None) of A with index i repeated counts[i] times, by the
    finite-difference sieve with matrix-power traces in 64 bits:

        2^-K sum over delta of prod_e (-1)^k binom(r_e, k) [eta^K] g(eta),   delta_e = r_e - 2 k,
        g = exp(sum_j (tr((A X_d)^j) / 2j + v X_d (A X_d)^(j-1) v / 2) eta^j),

    with g times the loop series of an unpaired vertex; ``last`` adds an index with 0..cutoff
    photons, whose loop and pair series give every count at once.  None when it costs too much."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    edges, odd = _pairs(counts)
    extras = ([] if odd is None else [odd]) + ([] if last is None else [last])
    E, K = len(edges), sum(e[2] for e in edges)
    cplx = np.iscomplexobj(A) or np.iscomplexobj(v)
    dt = torch.complex128 if cplx else torch.float64
    m = 2 * E
    terms = 1
    for q, e in enumerate(edges):
        terms *= (e[2] + 2) // 2 if q == 0 else e[2] + 1
    half = (K + 1) // 2
    if terms * max(half - 1, 1) * m ** 3 * (8.0 if cplx else 2.0) > limit:
        return None
    At = torch.as_tensor(np.ascontiguousarray(A), dtype=dt, device=dev)
    ends = [e[0] for e in edges] + [e[1] for e in edges]
    idx = torch.as_tensor(ends, dtype=torch.long, device=dev)
    ex = torch.as_tensor(extras, dtype=torch.long, device=dev)
    Am = At[idx][:, idx]
    vt = torch.zeros(A.shape[0], dtype=dt, device=dev) if v is None else torch.as_tensor(
        np.ascontiguousarray(v), dtype=dt, device=dev)
    # columns carried through the powers: the loop weights and the rows of the extra vertices
    cols = torch.cat([vt[idx][:, None], At[idx][:, ex]], dim=1) if m else None
    ncol = 1 + len(extras)
    nout = 1 if last is None else cutoff + 1
    totals = torch.zeros(nout, dtype=dt, device=dev)
    step = 4096 if dev == "cuda" else 256
    for t0 in range(0, terms, step):
        t = torch.arange(t0, min(terms, t0 + step), device=dev)
        B = len(t)
        weight = torch.ones(B, dtype=torch.float64, device=dev)
        delta = torch.zeros(B, E, dtype=torch.float64, device=dev)
        for q, (_, _, r) in enumerate(edges):
            radix = (r + 2) // 2 if q == 0 else r + 1
            k = t % radix
            t = torch.div(t, radix, rounding_mode="floor")
            d = r - 2 * k
            binom = torch.as_tensor([math.comb(r, x) * (-1.0) ** x for x in range(radix)], device=dev)
            weight = weight * binom[k]
            if q == 0:  # delta -> -delta leaves a term's share of the sum unchanged
                weight = weight * torch.where(d > 0, 2.0, 1.0)
            delta[:, q] = d
        g = torch.zeros(B, K + 1, dtype=dt, device=dev)  # log of the series, then the series
        pair = torch.zeros(B, ncol, ncol, K + 1, dtype=dt, device=dev)
        if m:
            d2 = torch.cat([delta, delta], dim=1).to(dt)
            M = torch.cat([Am[:, E:], Am[:, :E]], dim=1)[None] * d2[:, None, :]  # A X_d
            left = torch.cat([cols[E:], cols[:E]], dim=0)[None] * d2[:, :, None]  # X_d cols
            y = cols[None].expand(B, m, ncol)
            powers = [M]
            for _ in range(half - 1):
                powers.append(powers[-1] @ M)
            for j in range(1, K + 1):
                a = min(j, half)
                if j <= half:
                    tr = torch.diagonal(powers[j - 1], dim1=1, dim2=2).sum(-1)
                else:
                    tr = (powers[a - 1] * powers[j - a - 1].transpose(1, 2)).sum((1, 2))
                pair[..., j] = left.transpose(1, 2) @ y
                g[:, j] = tr / (2 * j) + pair[:, 0, 0, j] / 2
                if j < K:
                    y = M @ y
            del powers
        q = g * torch.arange(K + 1, device=dev)
        e = torch.zeros_like(g)
        e[:, 0] = 1
        for j in range(1, K + 1):
            e[:, j] = (q[:, 1:j + 1] * e[:, :j].flip(1)).sum(1) / j

        def times(x, y):
            out = torch.zeros_like(x)
            for s in range(K + 1):
                out[:, s:] += x[:, s:s + 1] * y[:, :K + 1 - s]
            return out

        def loop_of(p):  # series of extra vertex p ending in a loop
            s = pair[:, 1 + p, 0, :].clone()
            s[:, 0] = vt[extras[p]]
            return s

        if last is None:
            series = e if odd is None else times(e, loop_of(0))
            totals[0] += (series[:, K] * weight).sum()
        else:
            b = len(extras) - 1
            lv = loop_of(b)
            lc = pair[:, 1 + b, 1 + b, :].clone()
            lc[:, 0] = At[last, last]
            h = [e, times(e, lv)]
            for k in range(1, cutoff + 1):
                h.append(times(h[k], lv) + k * times(h[k - 1], lc))
            if odd is not None:
                ov, oc = loop_of(0), pair[:, 1, 1 + b, :].clone()
                oc[:, 0] = At[odd, last]
                h = [times(h[k], ov) + (k * times(h[k - 1], oc) if k else 0) for k in range(cutoff + 1)]
            for k in range(cutoff + 1):
                totals[k] += (h[k][:, K] * weight).sum()
    out = (totals * 0.5 ** K).to(torch.complex128).cpu().numpy()
    return out if last is not None else out[0]


def exact(case, seed):
    kind = case["kind"]
    args = _inputs(case, seed)
    if kind in ("plain", "graph"):
        return _power_trace_sieve(args[0], None, [1] * case["n"])
    if kind == "loop":
        return _power_trace_sieve(args[0], np.diag(args[0]), [1] * case["n"])
    if kind == "gbs":
        return _power_trace_sieve(args[0], args[1], args[2])
    if kind == "modes":
        A, D, fixed, cutoff = args
        return _power_trace_sieve(A, D, list(fixed), last=len(A) - 1, cutoff=cutoff)
    if kind == "plan":
        vals = [_power_trace_sieve(M, None, [1] * len(M)) for M in args[0]]
        return None if any(x is None for x in vals) else np.array(vals)
    B, alpha, patterns = args
    eye = np.identity(len(B))
    gamma = alpha - B @ alpha.conj()
    quad = np.vdot(alpha, alpha).real - alpha.conj() @ B @ alpha.conj()
    vacuum = np.exp(0.25 * np.linalg.slogdet(eye - B @ B.conj())[1]) * np.exp(-0.5 * quad)
    out = []
    for p in patterns:
        x = _power_trace_sieve(B, gamma, p)
        if x is None:
            return None
        out.append(x * vacuum / math.sqrt(math.prod(math.factorial(int(c)) for c in p)))
    return np.array(out)
