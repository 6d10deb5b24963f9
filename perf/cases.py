"""The workloads by which this framework's speed is followed: permanents, all-minors
permanents, gradients, samplers and exact distributions, each called as a program
calls it, from single small calls (where launches and latency count) to the largest
ones of the repository's own benchmark.

Everything is host data: the calculators, strategies and the C ABI take host
matrices and occupations and return host results.  Every pass of a sampler starts
from a seeded numpy generator, so the same state gives the same samples.
"""
import math

import numpy as np
import torch

from theboss_gb300 import _native
from theboss_gb300.adjoint import clements_unitary, log_likelihood, probabilities
from theboss_gb300.permanent_calculators import (ChinHuhPermanentCalculator, ClassicPermanentCalculator,
                                                 GlynnGrayPermanentCalculator, RyserPermanentCalculator)
from theboss_gb300.simulation_strategies import (GeneralizedCliffordsBSimulationStrategy,
                                                 GeneralizedCliffordsBUniformLossesSimulationStrategy,
                                                 LossyNetworksGeneralizedCliffordsSimulationStrategy)
from theboss_gb300.submatrices_calculators import (BSCCCHSubmatricesPermanentCalculator,
                                                   BSCCRyserSubmatricesPermanentCalculator)
from theboss_gb300.utilities import haar_unitary, possible_states_array

CALCULATORS = {"ryser": RyserPermanentCalculator, "chin_huh": ChinHuhPermanentCalculator,
               "glynn": GlynnGrayPermanentCalculator, "classic": ClassicPermanentCalculator}
MINORS = {"ryser": BSCCRyserSubmatricesPermanentCalculator, "chin_huh": BSCCCHSubmatricesPermanentCalculator}


def listed():
    return [
        # one small permanent, as a distribution or a test asks for it: all latency
        {"name": "perm_ryser_n8_one", "kind": "perm", "variant": "ryser", "n": 8, "m": 16, "count": 1},
        # the amplitudes of a few dozen patterns at the size where planning and launches still count
        {"name": "perm_glynn_n16_b64", "kind": "perm", "variant": "glynn", "n": 16, "m": 32, "count": 64},
        # one large permanent
        {"name": "perm_chin_huh_n24_one", "kind": "perm", "variant": "chin_huh", "n": 24, "m": 48, "count": 1},
        # a batch of large permanents: sustained arithmetic
        {"name": "perm_glynn_n28_b64", "kind": "perm", "variant": "glynn", "n": 28, "m": 56, "count": 64},
        # one step of a sampler written around the all-minors calculator: small, then large
        {"name": "minors_ryser_k10_one", "kind": "minors", "variant": "ryser", "n": 10, "m": 24},
        {"name": "minors_chin_huh_k21_one", "kind": "minors", "variant": "chin_huh", "n": 21, "m": 42},
        # a handful of lossless samples, some input modes doubly occupied: latency of the sampler
        {"name": "gccb_n8_m16_s16", "kind": "gccb", "n": 8, "m": 16, "eta": 1.0, "samples": 16, "bunched": 2},
        # the benchmark's batch: uniform losses, 10^4 samples
        {"name": "gccb_n20_m40_s10000", "kind": "gccb", "n": 20, "m": 40, "eta": 0.5, "samples": 10000, "bunched": 0},
        # mode-dependent losses: 30 photons in the 120-mode dilation of 60 lossy modes
        {"name": "network_n30_m60_s4", "kind": "network", "n": 30, "m": 60, "samples": 4},
        # one step of fitting a mesh to observed patterns: log-likelihood and its phase gradients
        {"name": "loglik_n12_m24_b256", "kind": "loglik", "n": 12, "m": 24, "count": 256},
        # probabilities of large patterns and their gradient with respect to the matrix
        {"name": "probs_grad_n24_m48_b64", "kind": "probs_grad", "n": 24, "m": 48, "count": 64},
        # the whole output distribution under uniform losses
        {"name": "dist_n8_m16", "kind": "dist", "n": 8, "m": 16},
    ]


def _spread(rng, lo, hi):
    """An integer of [lo, hi], even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["perm", "perm", "minors", "gccb", "gccb", "network", "loglik", "probs_grad", "dist"])
    if kind == "perm":
        # theboss's Ryser formula loses digits with n (its own float64 values agree to 1e-10 at most above this)
        variant = rng.choice(["ryser", "chin_huh", "glynn", "classic"])
        n = rng.randint(2, 14 if variant == "ryser" else 28)
        most = max(1, min(512, 2 ** (33 - n)))
        return {"kind": kind, "variant": variant, "n": n, "m": n + rng.randint(0, n + 5), "count": _spread(rng, 1, most)}
    if kind == "minors":
        n = rng.randint(2, 23)
        return {"kind": kind, "variant": rng.choice(["ryser", "chin_huh"]), "n": n, "m": n + rng.randint(1, n + 3)}
    if kind == "gccb":
        n = rng.randint(3, 24)
        eta = rng.choice([1.0, 0.9, 0.7, 0.5, 0.3])
        # levels grow as 2^k for a sample that keeps k photons: (1 + eta)^n on average
        most = max(1, min(20000, int(4e8 / (n * (1.0 + eta) ** n))))
        return {"kind": kind, "n": n, "m": n + rng.randint(1, 2 * n), "eta": eta, "samples": _spread(rng, 1, most),
                "bunched": rng.randint(0, min(3, n // 3))}
    if kind == "network":
        n = rng.randint(4, 28)
        return {"kind": kind, "n": n, "m": n + rng.randint(0, n), "samples": _spread(rng, 1, max(1, min(1000, 2 ** (31 - n))))}
    if kind == "loglik":
        n = rng.randint(3, 13)
        return {"kind": kind, "n": n, "m": n + rng.randint(2, n + 2), "count": _spread(rng, 8, 400)}
    if kind == "probs_grad":
        n = rng.randint(6, 24)
        return {"kind": kind, "n": n, "m": n + rng.randint(1, n), "count": _spread(rng, 1, max(1, min(256, 2 ** (29 - n))))}
    n = rng.randint(2, 8)
    return {"kind": kind, "n": n, "m": rng.randint(n, 17 - max(n - 7, 0) if n > 6 else 20 - n)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _outputs(g, n, m, count):
    """Output patterns: n photons over m modes, collisions as they fall."""
    T = np.zeros((count, m), dtype=np.int32)
    for k in range(count):
        np.add.at(T[k], g.integers(0, m, size=n), 1)
    return T


def _first_modes(n, m):
    S = np.zeros(m, dtype=np.int32)
    S[:n] = 1
    return S


def prepare(case, seed):
    g = np.random.default_rng(seed)
    kind, n, m = case["kind"], case["n"], case["m"]
    st = {"kind": kind, "case": case}
    if kind in ("perm", "minors"):
        U = haar_unitary(m, seed)
        S = _first_modes(n, m)
        if kind == "perm":
            T = _outputs(g, n, m, case["count"])
            st["calc"] = CALCULATORS[case["variant"]](U, S, T[0])
            st["outputs"] = T
        else:
            st["calc"] = MINORS[case["variant"]](U, S, _outputs(g, n - 1, m, 1)[0])
        st.update(U=U, S=S)
    elif kind == "gccb":
        U = haar_unitary(m, seed)
        S = _first_modes(n, m)
        for b in range(case["bunched"]):  # photon n - 1 - b joins mode b
            S[b] += 1
            S[n - 1 - b] -= 1
        weights = None
        if case["eta"] < 1.0:
            eta = case["eta"]
            weights = [math.comb(n, l) * eta ** l * (1 - eta) ** (n - l) for l in range(n + 1)]
        st.update(U=U, S=S, weights=weights, seed=int(seed) % (2 ** 32))
        if case["samples"] <= 64:
            calc = RyserPermanentCalculator(U, S, None)
            st["strategy"] = (GeneralizedCliffordsBSimulationStrategy(calc) if weights is None else
                              GeneralizedCliffordsBUniformLossesSimulationStrategy(calc, case["eta"]))
    elif kind == "network":
        t = g.uniform(0.3, 0.9, size=m)  # transmissivity of every mode
        U = haar_unitary(m, seed) * np.sqrt(t)[:, None]
        st.update(S=_first_modes(n, m), seed=int(seed) % (2 ** 32),
                  strategy=LossyNetworksGeneralizedCliffordsSimulationStrategy(RyserPermanentCalculator(U)))
    elif kind == "loglik":
        p = m * (m - 1) // 2
        # splitters around 50:50, so that m layers mix every mode
        theta = torch.from_numpy(math.pi / 4 + g.uniform(-0.4, 0.4, size=p))
        phi = torch.from_numpy(g.uniform(0, 2 * math.pi, size=p))
        st.update(theta=theta, phi=phi, S=np.tile(_first_modes(n, m), (case["count"], 1)),
                  T=_outputs(g, n, m, case["count"]))
    elif kind == "probs_grad":
        st.update(U=torch.from_numpy(haar_unitary(m, seed)), S=np.tile(_first_modes(n, m), (case["count"], 1)),
                  T=_outputs(g, n, m, case["count"]), weight=torch.from_numpy(g.uniform(0.5, 1.5, size=case["count"])))
    else:
        st.update(U=haar_unitary(m, seed), S=_first_modes(n, m), outcomes=possible_states_array(n, m, losses=True))
    return st


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(st):
    kind = st["kind"]
    if kind == "perm":
        if len(st["outputs"]) == 1:
            return st["calc"].compute_permanent()
        return st["calc"].compute_permanents_of_outputs(st["outputs"])
    if kind == "minors":
        return np.array(st["calc"].compute_permanents())
    if kind == "gccb":
        np.random.seed(st["seed"])
        if "strategy" in st:
            return np.array(st["strategy"].simulate(st["S"], st["case"]["samples"]))
        return _native.gccb_sample(st["U"], st["S"], st["weights"], st["case"]["samples"])
    if kind == "network":
        np.random.seed(st["seed"])
        return np.array(st["strategy"].simulate(st["S"], st["case"]["samples"]))
    if kind == "loglik":
        theta = st["theta"].clone().requires_grad_(True)
        phi = st["phi"].clone().requires_grad_(True)
        L = log_likelihood(clements_unitary(theta, phi), st["S"], st["T"])
        L.backward()
        return L.detach(), theta.grad, phi.grad
    if kind == "probs_grad":
        U = st["U"].clone().requires_grad_(True)
        p = probabilities(U, st["S"], st["T"])
        (p * st["weight"]).sum().backward()
        return p.detach(), U.grad
    return _native.lossy_probabilities(st["U"], st["S"], st["outcomes"])


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: the matrix and the occupations in, the results out.  Flops: the formulas' own
    (complex add 2, product 6), over the codes of the halved Glynn sum: 8 n - 4 per code of a
    permanent, 9 k - 12 of an all-minors sweep, three products and two sums per factor and code
    of a gradient."""
    kind, n, m = case["kind"], case["n"], case["m"]
    U = 16.0 * m * m
    if kind == "perm":
        c = case["count"]
        return {"bytes": U + c * (8.0 * m + 16), "flops": c * 2.0 ** (n - 1) * (8 * n - 4)}
    if kind == "minors":
        return {"bytes": U + 8.0 * m + 16.0 * m, "flops": 2.0 ** (n - 1) * max(9 * n - 12, 2)}
    if kind in ("gccb", "network"):
        eta = case.get("eta", 1.0)
        modes = 2 * m if kind == "network" else m
        flops = 0.0
        for l in range(n + 1):
            p = math.comb(n, l) * eta ** l * (1 - eta) ** (n - l)
            flops += p * sum(2.0 ** (k - 1) * max(9 * k - 12, 2) + 8.0 * k * modes for k in range(1, l + 1))
        return {"bytes": 16.0 * modes * modes + case["samples"] * 4.0 * m, "flops": case["samples"] * flops}
    if kind in ("loglik", "probs_grad"):
        c = case["count"]
        return {"bytes": 2 * U + c * 8.0 * m, "flops": c * 2.0 ** (n - 1) * n * (8 + 22)}
    flops, rows = 0.0, 0
    for l in range(1, n + 1):
        outcomes = math.comb(m + l - 1, l)
        rows += outcomes
        flops += outcomes * math.comb(n, l) * 2.0 ** (l - 1) * (8 * l - 4)
    return {"bytes": U + rows * (4.0 * m + 8), "flops": flops}


# ---------------------------------------------------------------------------
# The same in plain 64-bit torch: Glynn's formula over all sign vectors
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _signs(n, dev):
    """Sign vectors with the first sign +1: (2^(n-1), n), and their parities."""
    c = torch.arange(2 ** (n - 1), device=dev)
    bits = (c[:, None] >> torch.arange(n - 1, device=dev)) & 1
    d = torch.cat([torch.ones(len(c), 1, dtype=torch.int64, device=dev), 1 - 2 * bits], 1)
    return d.double(), d.prod(1).double()


def _permanent(M):
    """perm of an n x n complex matrix; the low signs as one axis, the high ones in a loop."""
    n = M.shape[0]
    if n == 0:
        return torch.ones((), dtype=M.dtype, device=M.device)
    low = min(n, 22)
    d, par = _signs(low, M.device)
    lo = d.to(M.dtype) @ M[:, :low].T  # (codes, n)
    lo = lo.T.contiguous()
    total = torch.zeros((), dtype=M.dtype, device=M.device)
    for h in range(2 ** (n - low)):
        s = torch.tensor([1 - 2 * ((h >> b) & 1) for b in range(n - low)], dtype=torch.float64, device=M.device)
        shift = (M[:, low:] @ s.to(M.dtype)) if n > low else torch.zeros(n, dtype=M.dtype, device=M.device)
        p = lo[0] + shift[0]
        for f in range(1, n):
            p = p * (lo[f] + shift[f])
        sign = -1.0 if bin(h).count("1") % 2 else 1.0
        total = total + sign * (p * par).sum()
    return total / 2.0 ** (n - 1)


def _modes(occ):
    return np.repeat(np.arange(len(occ)), occ)


def _permanent_and_gradient(M):
    """perm of an n x n matrix and d perm / d M, from the leave-one-out products."""
    n = M.shape[0]
    low = min(n, 18)
    d, par = _signs(low, M.device)
    lo = (d.to(M.dtype) @ M[:, :low].T).T.contiguous()
    perm = torch.zeros((), dtype=M.dtype, device=M.device)
    grad = torch.zeros_like(M)
    for h in range(2 ** (n - low)):
        s = torch.tensor([1 - 2 * ((h >> b) & 1) for b in range(n - low)], dtype=torch.float64, device=M.device)
        f = lo + (M[:, low:] @ s.to(M.dtype))[:, None] if n > low else lo
        sign = (-1.0 if bin(h).count("1") % 2 else 1.0) * par
        pre, suf = [None] * n, [None] * n
        pre[0] = sign.to(M.dtype)
        for a in range(1, n):
            pre[a] = pre[a - 1] * f[a - 1]
        suf[n - 1] = torch.ones_like(pre[0])
        for a in range(n - 2, -1, -1):
            suf[a] = suf[a + 1] * f[a + 1]
        leave = torch.stack([pre[a] * suf[a] for a in range(n)])
        perm = perm + (leave[n - 1] * f[n - 1]).sum()
        grad[:, :low] += leave @ d.to(M.dtype)
        if n > low:
            grad[:, low:] += leave.sum(1)[:, None] * s.to(M.dtype)[None, :]
    return perm / 2.0 ** (n - 1), grad / 2.0 ** (n - 1)


def exact(case, seed):
    kind, n, m = case["kind"], case["n"], case["m"]
    if kind in ("gccb", "network"):
        return None  # samples: whole numbers
    st = prepare(case, seed)
    dev = _device()
    if dev.type == "cpu" and n > 20:
        return None
    if kind == "perm":
        U = torch.from_numpy(st["U"]).to(dev)
        cols = _modes(st["S"])
        out = [complex(_permanent(U[_modes(T)][:, cols])) for T in st["outputs"]]
        return np.complex128(out[0]) if len(out) == 1 else np.array(out)
    if kind == "minors":
        U = torch.from_numpy(st["U"]).to(dev)
        rows = U[_modes(st["calc"].output_state)]
        out = np.zeros(m, dtype=np.complex128)
        for i in np.nonzero(st["S"])[0]:
            S = st["S"].copy()
            S[i] -= 1
            out[i] = complex(_permanent(rows[:, _modes(S)]))
        return out
    if kind in ("loglik", "probs_grad"):
        if kind == "loglik":
            theta, phi = st["theta"].clone().requires_grad_(True), st["phi"].clone().requires_grad_(True)
            U = _mesh(theta, phi, m)
        else:
            U = st["U"].clone()
        Ud = U.detach().to(dev)
        cols = _modes(st["S"][0])
        grad = torch.zeros(m, m, dtype=torch.complex128, device=dev)
        L, probs = 0.0, []
        for k in range(case["count"]):
            rows = _modes(st["T"][k])
            norm = float(np.prod([math.factorial(int(v)) for v in st["T"][k]]))
            p, g = _permanent_and_gradient(Ud[rows][:, cols])
            probs.append(float((p.abs() ** 2).item()) / norm)
            # d|p|^2 = 2 Re(conj(p) dp): torch's gradient of a real function is 2 p conj(dp/dU)
            w = 1.0 / probs[-1] if kind == "loglik" else float(st["weight"][k])
            L += math.log(probs[-1])
            at = torch.zeros(n, m, dtype=torch.complex128, device=dev)
            at[:, torch.from_numpy(cols).to(dev)] = (2.0 * w / norm) * p * g.conj()
            grad.index_add_(0, torch.from_numpy(rows).to(dev), at)
        grad = grad.cpu()
        if kind == "probs_grad":
            return torch.tensor(probs, dtype=torch.float64), grad
        U.backward(grad)
        return torch.tensor(L, dtype=torch.float64), theta.grad, phi.grad
    return _distribution(st, n, m, dev)


def _mesh(theta, phi, m):
    """The rectangular mesh, one splitter after another within each layer's own order."""
    M = torch.eye(m, dtype=torch.complex128)
    at = 0
    for layer in range(m):
        T = torch.eye(m, dtype=torch.complex128)
        for k in range(layer % 2, m - 1, 2):
            e, c, s = torch.exp(1j * phi[at]), torch.cos(theta[at]), torch.sin(theta[at])
            block = torch.stack([torch.stack([e * c, -s + 0j]), torch.stack([e * s, c + 0j])])
            T = T.index_put((torch.tensor([[k, k], [k + 1, k + 1]]), torch.tensor([[k, k + 1], [k, k + 1]])), block)
            at += 1
        M = T @ M
    return M


def _distribution(st, n, m, dev):
    """p(T) = sum over the l-photon sub-inputs of |perm|^2 / C(n, l) / prod T!, l photons detected."""
    import itertools

    U = torch.from_numpy(st["U"]).to(dev)
    T = st["outcomes"]
    counts = T.sum(1)
    out = np.zeros(len(T))
    out[counts == 0] = 1.0
    fact = np.array([math.factorial(k) for k in range(n + 1)], dtype=np.float64)
    for l in range(1, n + 1):
        which = np.nonzero(counts == l)[0]
        rows = torch.from_numpy(np.stack([_modes(T[k]) for k in which])).to(dev)  # (O, l)
        d, par = _signs(l, dev)
        acc = torch.zeros(len(which), dtype=torch.float64, device=dev)
        for cols in itertools.combinations(range(n), l):
            V = (U[:, list(cols)] @ d.T.to(U.dtype)) / 2.0  # (m, codes): every row's signed sums
            for a in range(0, len(which), 1 << 17):
                r = rows[a:a + (1 << 17)]
                p = V[r[:, 0]]
                for f in range(1, l):
                    p = p * V[r[:, f]]
                acc[a:a + (1 << 17)] += ((p * par).sum(1) * 2.0).abs() ** 2
        norm = torch.from_numpy(fact[T[which]].prod(1)).to(dev)
        out[which] = (acc / norm / math.comb(n, l)).cpu().numpy()
    return out
