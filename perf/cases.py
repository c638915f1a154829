"""The calls that users of this framework make, for timing: each case is one pass through
the public entry points, from the smallest calls (latency) to one rank's share of a
20-qubit sweep.

States are seeded i.i.d. complex Gaussian vectors of unit norm (Haar-like), the inputs of
bench.py and of the tests; drawn cases lean them towards |0...0> by a factor exp(-tilt) per
excited site, as partly polarised states are.  The entry points take host arrays, as the reference's do, so a
pass includes the copies to and from the GPU.  SRE results are returned as one array
[value, lost_norm]: lost_norm is 0 up to rounding for these states.

`exact` restates every quantity in 64 bits with plain torch operations from its
definition: dense +-1 (or cube-root-of-unity) matrix products for the transforms.
"""
import math

import numpy as np
import torch

import hadamag_b200 as hm


# ----------------------------------------------------------------------------------
# the cases

def listed():
    return [
        # smallest call: scanning many small states one by one; latency and launches count
        {"name": "sre_n8", "kind": "sre", "n": 8, "q": 2.0, "precision": "fp64"},
        # the reference's 12-qubit example size, called interactively
        {"name": "sre_n12", "kind": "sre", "n": 12, "q": 2.0, "precision": "fp64"},
        # a Renyi index beyond the specialised q = 2, 3
        {"name": "sre_n13_q4", "kind": "sre", "n": 13, "q": 4.0, "precision": "fp64"},
        # an ordinary exact SRE: an odd qubit count in the middle of the range
        {"name": "sre_n17", "kind": "sre", "n": 17, "q": 2.0, "precision": "fp64"},
        # FP32 butterflies, the precision option, at a size where they are worth choosing
        {"name": "sre_n18_fp32", "kind": "sre", "n": 18, "q": 2.0, "precision": "fp32"},
        # the headline sweep, as one of eight ranks runs it: rank 3's share at n = 20
        {"name": "slice_n20", "kind": "slice", "n": 20, "q": 2.0, "precision": "fp64", "world": 8, "rank": 3},
        # many states of uneven sizes and two indices in one call
        {"name": "batched_n8_15", "kind": "batched", "nstates": 48, "nmin": 8, "nmax": 15, "q3": True,
         "precision": "fp32"},
        # value and gradient (backward): one step of an optimisation over states
        {"name": "grad_n14", "kind": "grad", "n": 14, "q": 2},
        # Metropolis estimate with the reference's default chain counts
        {"name": "mc_n16", "kind": "mc", "n": 16, "q": 2.0, "nbeta": 13, "nsamples": 1000},
        # qutrit Mana of a pure state
        {"name": "mana_L9", "kind": "mana", "L": 9},
        # qutrit Mana of a density matrix: the 729 x 729 one of bench.py
        {"name": "mixed_N6", "kind": "mixed", "N": 6},
        # preparing inputs: a brick-wall circuit and the reduced density matrix of its result
        {"name": "circuit_n18", "kind": "circuit", "n": 18, "site": 2, "depth": 8, "NA": 7},
    ]


def draw(rng):
    case = _draw(rng)
    if case["kind"] != "circuit":
        case["tilt"] = round(rng.uniform(0.0, 0.2), 3)
    return case


def _draw(rng):
    kind = rng.choice(["sre", "sre", "sre", "slice", "batched", "grad", "mc", "mana", "mixed", "circuit"])
    if kind == "sre":
        q = rng.choice([2.0, 2.0, 2.0, 3.0, 4.0, 2.5])
        if q in (2.0, 3.0):
            precision = rng.choice(["fp64", "fp64", "fp32"])
            n = rng.randint(6 if precision == "fp64" else 12, 18)
        else:
            precision, n = "fp64", rng.randint(6, 13)
        return {"kind": kind, "n": n, "q": q, "precision": precision}
    if kind == "slice":
        n = rng.randint(19, 21)
        world = int((4 << 2 * (n - 19)) * 2 ** rng.uniform(0, 4)) + 1
        return {"kind": kind, "n": n, "q": rng.choice([2.0, 3.0]), "precision": rng.choice(["fp64", "fp64", "fp32"]),
                "world": world, "rank": rng.randrange(world)}
    if kind == "batched":
        nmin = rng.randint(6, 11)
        precision = rng.choice(["fp32", "fp64"])
        return {"kind": kind, "nstates": int(2 ** rng.uniform(3, 6.5)), "nmin": max(nmin, 8) if precision == "fp32" else nmin,
                "nmax": rng.randint(12, 15), "q3": rng.random() < 0.5, "precision": precision}
    if kind == "grad":
        return {"kind": kind, "n": rng.randint(8, 17), "q": rng.choice([2, 2, 3])}
    if kind == "mc":
        return {"kind": kind, "n": rng.randint(8, 18), "q": 2.0, "nbeta": 2 * rng.randint(3, 10) + 1,
                "nsamples": rng.randint(200, 1500)}
    if kind == "mana":
        return {"kind": kind, "L": rng.randint(5, 10)}
    if kind == "mixed":
        return {"kind": kind, "N": rng.randint(3, 6)}
    site = rng.choice([2, 2, 3])
    n = rng.randint(10, 20) if site == 2 else rng.randint(6, 12)
    return {"kind": kind, "n": n, "site": site, "depth": rng.randint(2, 12), "NA": rng.randint(2, 7 if site == 2 else 5)}


# ----------------------------------------------------------------------------------
# inputs and the calls

def _state(dim, seed, tilt=0.0, site=2):
    g = np.random.default_rng(seed)
    v = g.normal(size=dim) + 1j * g.normal(size=dim)
    if tilt:
        w = np.ones(1)
        while w.size < dim:
            w = np.kron(np.r_[1.0, np.full(site - 1, math.exp(-tilt))], w)
        v *= w
    return v / np.linalg.norm(v)


def _range(case):
    return hm.shard.gray_slice(case["n"], case["rank"], case["world"])


def _inputs(case, seed):
    kind, tilt = case["kind"], case.get("tilt", 0.0)
    if kind in ("sre", "slice", "grad"):
        return {"psi": _state(1 << case["n"], seed, tilt)}
    if kind == "batched":
        # the qubit counts run evenly over the range in a fixed shuffled order
        ns = [case["nmin"] + i % (case["nmax"] - case["nmin"] + 1) for i in range(case["nstates"])]
        ns = np.random.default_rng(case["nstates"]).permutation(ns)
        return {"psis": [_state(1 << int(n), seed * 1000 + i, tilt) for i, n in enumerate(ns)]}
    if kind == "mc":
        pd, rs = hm.proposal_stream(case["n"], case["nbeta"], case["nsamples"], seed)
        return {"psi": _state(1 << case["n"], seed, tilt), "pd": pd, "rs": rs}
    if kind == "mana":
        return {"psi": _state(3 ** case["L"], seed, tilt, 3)}
    if kind == "mixed":
        # a pure state of four more qutrits, traced over those
        m = _state(3 ** (case["N"] + 4), seed, tilt, 3).reshape(3 ** case["N"], 81)
        return {"rho": m @ m.conj().T}
    rng = np.random.default_rng(seed)
    pairs = hm.brick_wall_pairs(case["n"], case["depth"])
    return {"gates": [hm.haar_random_unitary(case["site"], 2, rng) for _ in pairs], "pairs": pairs}


def prepare(case, seed):
    s = dict(case, **_inputs(case, seed))
    kind = case["kind"]
    if kind in ("sre", "grad"):
        s["psi"] = hm.StateVec(s["psi"])
    elif kind == "batched":
        s["psis"] = [hm.StateVec(p) for p in s["psis"]]
    elif kind == "mana":
        s["psi"] = hm.StateVec(s["psi"], q=3)
    elif kind == "mixed":
        s["rho"] = hm.DensityMatrix(s["rho"], q=3)
    elif kind == "slice":
        s["k"] = _range(case)
    s["ctx"] = hm.B200().context()
    return s


def run(s):
    kind = s["kind"]
    if kind == "sre":
        return np.array(hm.SRE(s["psi"], s["q"], precision=s["precision"]))
    if kind == "slice":
        p2, m = s["ctx"].sre_range(s["psi"], s["k"][0], s["k"][1], (s["q"],), hm.PRECISIONS[s["precision"]])
        return {"p2": p2, "m": m}
    if kind == "batched":
        v, lost = hm.SRE_batched(s["psis"], qs=(2, 3) if s["q3"] else (2,), precision=s["precision"])
        return np.concatenate([v, lost[:, None]], axis=1)
    if kind == "grad":
        v, g = hm.SRE_grad(s["psi"], s["q"])
        return {"value": v, "grad": g}
    if kind == "mc":
        m2, M2, M2ADD, P2, mask = s["ctx"].mc_sre(s["psi"], s["q"], s["nbeta"], s["nsamples"], s["pd"], s["rs"])
        return {"m2": m2, "M2": M2, "M2ADD": M2ADD, "P2": P2, "mask": mask.view(np.int64)}
    if kind in ("mana", "mixed"):
        return hm.Mana(s["psi"] if kind == "mana" else s["rho"])
    v = np.zeros(s["site"] ** s["n"], dtype=np.complex128)
    v[0] = 1.0
    sv = hm.apply_brick_wall(hm.StateVec(v, q=s["site"], copy=False), s["depth"], s["gates"])
    return {"psi": sv.data, "rho": hm.reduced_density_matrix(sv, s["NA"]).data}


def _sre_ops(n, q=2.0):
    """One X-string: n 2^n butterfly adds, 2 2^n for the products, 4 2^n for the moments."""
    return (n + 6 + (0 if q == 2.0 else 2)) * float(1 << n)


def work(case):
    kind = case["kind"]
    if kind == "sre":
        n = case["n"]
        return {"bytes": 16.0 * (1 << n) + 16, "flops": _sre_ops(n, case["q"]) * (1 << n)}
    if kind == "slice":
        kb, ke = _range(case)
        return {"bytes": 16.0 * (1 << case["n"]) + 32, "flops": _sre_ops(case["n"], case["q"]) * (ke - kb)}
    if kind == "batched":
        ns = [case["nmin"] + i % (case["nmax"] - case["nmin"] + 1) for i in range(case["nstates"])]
        q = 3.0 if case["q3"] else 2.0
        return {"bytes": sum(16.0 * (1 << n) + 24 for n in ns), "flops": sum(_sre_ops(n, q) * (1 << n) for n in ns)}
    if kind == "grad":
        n = case["n"]  # forward, pointwise powers, backward, two products with psi
        return {"bytes": 32.0 * (1 << n) + 8, "flops": (2 * n + 12) * 4.0 ** n}
    if kind == "mc":
        steps = case["nbeta"] * case["nsamples"]
        return {"bytes": 16.0 * (1 << case["n"]) + 16.0 * steps, "flops": _sre_ops(case["n"]) * steps}
    if kind == "mana":
        L = case["L"]  # 12 operations per 3-point transform, 6 per product, 5 per modulus
        return {"bytes": 16.0 * 3 ** L, "flops": 9.0 ** L * (4 * L + 11)}
    if kind == "mixed":
        N = case["N"]  # 9-term complex sums per output and leg
        return {"bytes": 16.0 * 9 ** N, "flops": 9.0 ** N * (72 * N + 5)}
    q, n = case["site"], case["n"]
    dim, dimA = float(q ** n), float(q ** case["NA"])
    ngates = len(hm.brick_wall_pairs(n, case["depth"]))
    return {"bytes": 16.0 * (2 * dim + dimA * dimA), "flops": 8.0 * dim * (q * q * ngates + dimA)}


# ----------------------------------------------------------------------------------
# the same quantities in 64 bits, from their definitions

_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _along(M, v, size):
    """M applied to every digit group: v (batch, size^...) as matrix products with M."""
    b, dim = v.shape
    step = M.shape[0]
    left = dim
    while left > 1:
        while step > left:  # a smaller remaining group: the leading factor of M
            step //= size
        m = M[:step, :step]
        v = (v.reshape(-1, step) @ m.T).reshape(b, -1, step).transpose(1, 2).reshape(b, dim)
        left //= step
    return v


def _hadamard(bits):
    H = torch.ones(1, 1, dtype=torch.float64, device=_DEV)
    for _ in range(bits):
        H = torch.cat([torch.cat([H, H], 1), torch.cat([H, -H], 1)])
    return H


def _chunks(xs, dim, elems=1 << 27):
    step = max(1, elems // dim)
    for i in range(0, len(xs), step):
        yield xs[i:i + step]


def _transforms(psi, xs):
    """(x, F_x) chunks: F_x = WHT(Re f + Im f), f(r) = conj psi(r) psi(r ^ x)."""
    dim = psi.numel()
    H = _hadamard(5)
    r = torch.arange(dim, device=_DEV)
    for c in _chunks(xs, dim):
        b = psi[r[None, :] ^ c[:, None]]
        g = psi.real * b.real + psi.imag * b.imag
        g += psi.real * b.imag
        g -= psi.imag * b.real
        del b
        yield c, _along(H, g, 2)


def _moments(psi, xs, qs):
    s = [0.0] * (1 + len(qs))
    for _, F in _transforms(psi, xs):
        y = F * F
        s[0] += float(y.sum())
        for i, q in enumerate(qs):
            s[1 + i] += float((y * y if q == 2 else y ** q).sum())
    return s


def _codes(k0, k1):
    k = torch.arange(k0, k1, device=_DEV)
    return k ^ (k >> 1)


def _sre(psi, qs):
    psi = torch.from_numpy(psi).to(_DEV)
    dim = psi.numel()
    s = _moments(psi, _codes(0, dim), qs)
    return [-math.log2(m / dim) for m in s[1:]] + [abs(1.0 - s[0] / dim)]


def _grad(psi, q):
    psi = torch.from_numpy(psi).to(_DEV)
    dim = psi.numel()
    H, r = _hadamard(5), torch.arange(dim, device=_DEV)
    m, grad = 0.0, torch.zeros_like(psi)
    for c, F in _transforms(psi, _codes(0, dim)):
        p = (F * F) ** (q - 1) * F
        m += float((p * F).sum())
        G = _along(H, 2 * q * p, 2)  # dm / dg
        u = r[None, :] ^ c[:, None]
        grad += (1 - 1j) * (G * psi[u]).sum(0)
        grad += (1 + 1j) * (torch.gather(G, 1, u) * psi[u]).sum(0)
    return {"value": -math.log2(m / dim), "grad": (-grad / (m * math.log(2.0))).cpu().numpy()}


def _mc(case, s):
    psi = torch.from_numpy(s["psi"]).to(_DEV)
    dim, nb = psi.numel(), case["nbeta"]
    p2_0, m0 = _moments(psi, _codes(0, 1), (case["q"],))
    H, r = _hadamard(5), torch.arange(dim, device=_DEV)
    beta = torch.arange(nb, device=_DEV, dtype=torch.float64) / (nb - 1)
    pd = torch.from_numpy(s["pd"].astype(np.int64)).to(_DEV)
    rs = torch.from_numpy(s["rs"]).to(_DEV)
    cur = torch.zeros(nb, dtype=torch.int64, device=_DEV)
    prob = torch.full((nb,), 1e-120, dtype=torch.float64, device=_DEV)
    M, P = torch.zeros_like(prob), torch.full_like(prob, p2_0 / dim)
    sM, sP = torch.zeros_like(prob), torch.zeros_like(prob)
    for t in range(case["nsamples"]):
        prop = cur ^ pd[:, t]
        b = psi[r[None, :] ^ prop[:, None]]
        y = _along(H, psi.real * (b.real + b.imag) + psi.imag * (b.imag - b.real), 2) ** 2
        m = (y * y if case["q"] == 2 else y ** case["q"]).sum(1)
        pb = m ** beta
        yes = (rs[:, t] < pb / prob) & (prop != 0)
        cur = torch.where(yes, prop, cur)
        prob = torch.where(yes, pb, prob)
        M = torch.where(yes, -torch.log2(m), M)
        P = torch.where(yes, y.sum(1) / dim, P)
        sM += M
        sP += P
    M2 = (sM / case["nsamples"]).cpu().numpy()
    h = 1.0 / (nb - 1)
    I = h / 3 * (M2[0] + M2[-1] + 4 * M2[1:-1:2].sum() + 2 * M2[2:-1:2].sum())
    return {"m2": -math.log2(2.0 ** -I + m0 / dim), "M2": M2, "M2ADD": np.full(nb, m0 / dim),
            "P2": (sP / case["nsamples"]).cpu().numpy(), "mask": None}


def _mana(psi, L):
    dim = 3 ** L
    psi = torch.from_numpy(psi).to(_DEV)
    w = torch.tensor([[1, 1, 1], [1, -0.5 + 0.75 ** 0.5 * 1j, -0.5 - 0.75 ** 0.5 * 1j],
                      [1, -0.5 - 0.75 ** 0.5 * 1j, -0.5 + 0.75 ** 0.5 * 1j]], dtype=torch.complex128, device=_DEV)
    W = torch.kron(torch.kron(w, w), w)
    pw = 3 ** torch.arange(L, device=_DEV)
    dig = (torch.arange(dim, device=_DEV)[:, None] // pw) % 3
    total = 0.0
    for c in _chunks(torch.arange(dim, device=_DEV), dim, 1 << 25):
        u = torch.zeros(len(c), dim, dtype=torch.int64, device=_DEV)
        v = torch.zeros_like(u)
        for d in range(L):
            xd = dig[c, d][:, None]
            u += (dig[:, d][None, :] + xd) % 3 * pw[d]
            v += (3 - dig[:, d][None, :] + xd) % 3 * pw[d]
        total += float(_along(W, psi[u].conj() * psi[v] / dim, 3).abs().sum())
    return math.log2(total) / math.log2(3.0)


def _mixed(rho, N):
    w = np.exp(2j * np.pi / 3)
    X, Z = np.roll(np.eye(3), 1, axis=0), np.diag([1, w, w * w])
    T = {(a, b): w ** (-2 * a * b % 3) * np.linalg.matrix_power(Z, a) @ np.linalg.matrix_power(X, b)
         for a in range(3) for b in range(3)}
    A0 = sum(T.values()) / 3
    # tr(A_u rho) as a row acting on (i, j) of one qutrit
    M = torch.from_numpy(np.array([(T[u] @ A0 @ T[u].conj().T).T.reshape(9) for u in T])).to(_DEV)
    v = torch.from_numpy(rho).to(_DEV).reshape((3,) * (2 * N))
    v = v.permute([k for i in range(N) for k in (i, N + i)]).reshape(-1)
    for _ in range(N):
        v = (M @ v.reshape(9, -1)).T.reshape(-1)
    return math.log2(float(v.abs().sum()) / 3 ** N)


def _circuit(case, s):
    q, n = case["site"], case["n"]
    v = torch.zeros(q ** n, dtype=torch.complex128, device=_DEV)
    v[0] = 1.0
    for g, (a, _) in zip(s["gates"], s["pairs"]):
        # sites a, a + 1 (1-based, site 1 least significant); the gate index is d_a q + d_(a+1)
        G = torch.from_numpy(g).to(_DEV).reshape(q, q, q, q)
        v = torch.einsum("abcd,xdcy->xbay", G, v.reshape(-1, q, q, q ** (a - 1))).reshape(-1)
    m = v.reshape(q ** case["NA"], -1)
    return {"psi": v.cpu().numpy(), "rho": (m @ m.conj().T).cpu().numpy()}


def exact(case, seed):
    s, kind = _inputs(case, seed), case["kind"]
    if kind == "sre":
        return np.array(_sre(s["psi"], (case["q"],)))
    if kind == "slice":
        kb, ke = _range(case)
        p2, m = _moments(torch.from_numpy(s["psi"]).to(_DEV), _codes(kb, ke), (case["q"],))
        return {"p2": np.array([p2, 0.0]), "m": np.array([[m, 0.0]])}
    if kind == "batched":
        return np.array([_sre(p, (2, 3) if case["q3"] else (2,)) for p in s["psis"]])
    if kind == "grad":
        return _grad(s["psi"], case["q"])
    if kind == "mc":
        return _mc(case, s)
    if kind == "mana":
        return _mana(s["psi"], case["L"])
    if kind == "mixed":
        return _mixed(s["rho"], case["N"])
    return _circuit(case, s)
