"""The work that users of this framework have it do, as measurable cases.

Every case goes through a public entry point of `photonic_engines_b200.clifford`, as a user's program calls
it: the drop-in `fock_sample` (lossless, lossy and partially distinguishable photons, from one shot to many
thousands), `sample_chains` with its marginals, the cofactor step `laplace_cofactors_rows`, the many-circuit
`BatchedSampler` and `emitter_sample`.  Samples come from seeded generators, so one seed is one result.

    listed()           the named cases             prepare(case, seed)   inputs and handles on the GPU
    draw(rng)          one more case               run(state)            one pass; all outputs
    work(case)         bytes and operations        tolerance(case)       how far two correct results may differ
    exact(case, seed)  the floating outputs in plain 64-bit torch
"""
from __future__ import annotations

import math

import torch

from photonic_engines_b200.clifford import (BatchedSampler, emitter_sample, fock_sample, laplace_cofactors_rows,
                                            sample_chains)
from photonic_engines_b200.states import caterpillar, spin_gate

C128 = torch.complex128
BATCH_MODES = (16, 24, 32, 48, 64)


# ------------------------------------------------------------------------------------------------ the cases
def _fock(name, n, m, shots, loss=1.0, indist=1.0, precision="f64"):
    return {"name": name, "kind": "fock", "n": n, "m": m, "shots": shots, "loss": loss, "indist": indist,
            "precision": precision}


def listed() -> list[dict]:
    return [
        # a few small permanent cofactors, as a caller that checks or steps a chain itself asks for them: latency
        {"name": "cofactors_k7_s32", "kind": "cofactors", "K": 7, "m": 49, "S": 32, "precision": "f64"},
        # the cofactor step at 20 columns over a batch of chains
        {"name": "cofactors_k20_s512", "kind": "cofactors", "K": 20, "m": 400, "S": 512, "precision": "f64"},
        # chains with their marginals, given orders and uniforms: validation and resampling programs
        {"name": "marginals_n14_m196", "kind": "marginals", "n": 14, "m": 196, "S": 500, "precision": "f64"},
        # one shot per call: interactive use, feed-forward between shots
        _fock("single_n20_m400", 20, 400, 1),
        # many shots of a small circuit
        _fock("small_n6_m12_10k", 6, 12, 10000),
        # the benchmark's workload: 20 photons in 400 modes
        _fock("fock_n20_m400_2k", 20, 400, 2000),
        # the same through the FP32 block form
        _fock("mixed_n20_m400_2k", 20, 400, 2000, precision="mixed"),
        # a lossy experiment: 30 photons sent, 15 detected on average
        _fock("lossy_n30_m900_100k", 30, 900, 100000, loss=0.5),
        # long chains of a few shots, partially distinguishable photons
        _fock("xmodel_n28_m784_200", 28, 784, 200, indist=0.95),
        # a dense circuit (m = 2n): repeated output modes at every step
        _fock("dense_n24_m48_512", 24, 48, 512),
        # a sweep over many small lossy circuits in one call, in the sampler's default form
        {"name": "batch_256x1000", "kind": "batch", "circuits": 256, "n_max": 12, "shots": 1000},
        # photons from one quantum emitter: the linear cluster state, emitter traced out
        {"name": "emitter_n12_512", "kind": "emitter", "n": 12, "shots": 512},
    ]


def _log_int(rng, lo, hi) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


MOST_FLOPS = 4.0e12                      # a drawn case stays below the largest listed one
MOST_COFACTORS = 512 * 20 * 2.0 ** 18


def draw(rng) -> dict:
    kind = rng.choice(["fock"] * 6 + ["cofactors"] * 3 + ["marginals", "batch", "emitter"])
    if kind == "cofactors":
        K = rng.randint(2, 22)
        S = min(_log_int(rng, 1, 2048), max(1, int(MOST_COFACTORS / (K * 2.0 ** max(0, K - 2)))))
        return {"kind": kind, "K": K, "m": rng.randint(max(3, K), 20 * K), "S": S,
                "precision": rng.choice(["f64", "f64", "f64", "mixed"])}
    if kind == "marginals":
        n = rng.randint(3, 16)
        return {"kind": kind, "n": n, "m": rng.randint(2 * n, 20 * n), "S": _log_int(rng, 4, 1000),
                "precision": rng.choice(["f64", "f64", "mixed"])}
    if kind == "batch":
        return {"kind": kind, "circuits": _log_int(rng, 2, 256), "n_max": rng.randint(5, 12),
                "shots": _log_int(rng, 50, 1000)}
    if kind == "emitter":
        return {"kind": kind, "n": rng.randint(4, 12), "shots": _log_int(rng, 16, 512)}
    n = rng.randint(2, 30)
    m = _log_int(rng, max(n + 1, 4), 1000)
    # lossless, lossy (plain or FP32 form) or partially distinguishable (host-planned: fewer shots)
    form = rng.choice(["lossless", "lossless", "mixed", "lossy", "lossy", "indist"])
    case = {"kind": kind, "n": n, "m": m, "shots": _log_int(rng, 1, 400 if form == "indist" else 100000),
            "loss": rng.choice([0.5, 0.7, 0.9]) if form == "lossy" else 1.0,
            "indist": rng.choice([0.9, 0.95, 0.98]) if form == "indist" else 1.0,
            "precision": "mixed" if form == "mixed" else "f64"}
    while case["n"] > 2 and _fock_flops(dict(case, shots=1)) > MOST_FLOPS / 8:
        case["n"] -= 1
    case["shots"] = max(1, min(case["shots"], int(MOST_FLOPS / _fock_flops(dict(case, shots=1)))))
    return case


# ------------------------------------------------------------------------------------------------ inputs
def _haar(m: int, count: int, gen) -> torch.Tensor:
    """count Haar-random unitaries [count, m, m] on the GPU."""
    z = torch.randn(count, m, m, 2, generator=gen, dtype=torch.float64, device="cuda")
    q, r = torch.linalg.qr(torch.view_as_complex(z))
    d = torch.diagonal(r, dim1=-2, dim2=-1)
    return q * (d / d.abs()).unsqueeze(-2)


def _uniform(gen, *shape):
    return torch.rand(*shape, generator=gen, dtype=torch.float64, device="cuda")


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    st = {"case": case, "seed": seed}
    if kind == "cofactors":
        # per stream K input columns of one circuit and K - 1 chosen output modes
        K, m, S = case["K"], case["m"], case["S"]
        U = _haar(m, 1, gen)[0]
        cols = torch.argsort(_uniform(gen, S, m), dim=1)[:, :K]
        st["A"] = U[:, cols].permute(1, 0, 2).contiguous()
        st["rows"] = torch.randint(0, m, (S, K - 1), generator=gen, device="cuda")
    elif kind == "marginals":
        n, m, S = case["n"], case["m"], case["S"]
        st["U"] = _haar(m, 1, gen)[0]
        st["sigma"] = torch.argsort(_uniform(gen, S, n), dim=1)
        st["uniforms"] = _uniform(gen, S, n)
    elif kind == "fock":
        st["U"] = _haar(case["m"], 1, gen)[0]
        st["generator"] = torch.Generator(device="cuda")
    elif kind == "batch":
        G = case["circuits"]
        ms = [BATCH_MODES[i] for i in torch.randint(0, len(BATCH_MODES), (G,), generator=gen, device="cuda").tolist()]
        fn, fe = torch.rand(2, G, generator=gen, device="cuda").tolist()
        ns = [4 + int(f * (min(case["n_max"], m // 4) - 3)) for f, m in zip(fn, ms)]
        etas = [0.6 + 0.4 * f for f in fe]
        by_m = {m: iter(_haar(m, ms.count(m), gen)) for m in sorted(set(ms))}
        circuits = [(next(by_m[m]), list(range(n))) for m, n in zip(ms, ns)]
        st["sampler"] = BatchedSampler(circuits, shots=case["shots"], loss=etas, seed=seed)
    else:
        n = case["n"]
        st["state"] = caterpillar(n, [spin_gate(math.pi / 2, 0.0)] * n)
        st["U"] = _haar(2 * n, 1, gen)[0]
        st["generator"] = torch.Generator()
    return st


def run(st: dict):
    case = st["case"]
    kind = case["kind"]
    if kind == "cofactors":
        return laplace_cofactors_rows(st["A"], st["rows"], precision=case["precision"])
    if kind == "marginals":
        return sample_chains(st["U"], list(range(case["n"])), st["sigma"], uniforms=st["uniforms"], want_marg=True,
                             precision=case["precision"])
    if kind == "fock":
        st["generator"].manual_seed(st["seed"])
        return fock_sample(st["U"], list(range(case["n"])), case["shots"], generator=st["generator"],
                           loss=case["loss"] if case["loss"] < 1.0 else None,
                           indist=case["indist"] if case["indist"] < 1.0 else None, precision=case["precision"])
    if kind == "batch":
        st["sampler"].gen.manual_seed(st["seed"])
        return st["sampler"].sample()
    st["generator"].manual_seed(st["seed"])
    return emitter_sample(st["state"], st["U"], case["shots"], generator=st["generator"])


# ------------------------------------------------------------------------------------------------ work
def _bose_terms(k1: int, m: int) -> float:
    """Expected terms of the collapsed sum over k1 output modes drawn by bosons in a Haar circuit (every
    occupation equally likely): E[prod (mult + 1)], halved."""
    if k1 < 2:
        return 1.0
    lg = math.lgamma
    return max(1.0, 0.5 * math.exp(lg(2 * m + k1) - lg(2 * m) - lg(m + k1) + lg(m)))


def _iid_terms(k1: int, m: int) -> float:
    """The same for independent uniform output modes."""
    if k1 < 2:
        return 1.0
    t = s = 1.0
    for i in range(1, min(k1, m) + 1):
        t *= (m - i + 1) * (k1 - i + 1) / (i * m)
        s += t
    return max(1.0, 0.5 * s)


def _term_flops(K: int) -> float:
    """One term of a sum with K columns: K column updates (4 operations each) and 3 (K - 2) complex products
    (6 each) for the all-but-one products, K complex additions (2 each)."""
    return 6.0 * K + 18.0 * max(0, K - 2)


def _chain_flops(n: int, m: int) -> float:
    return sum(_bose_terms(k - 1, m) * _term_flops(k) + (8.0 * k + 2.0) * m for k in range(1, n + 1))


def _binomial(n: int, p: float):
    return [(k, math.comb(n, k) * p ** k * (1.0 - p) ** (n - k)) for k in range(n + 1)]


def _fock_flops(case: dict) -> float:
    n, m, p = case["n"], case["m"], case["loss"] * case["indist"]
    per = sum(w * _chain_flops(k, m) for k, w in _binomial(n, p) if w > 1e-12)
    return case["shots"] * per


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "cofactors":
        K, m, S = case["K"], case["m"], case["S"]
        return {"bytes": 16.0 * S * K * (K - 1) + 8.0 * S * (K - 1) + 16.0 * S * K,
                "flops": S * _iid_terms(K - 1, m) * _term_flops(K)}
    if kind == "marginals":
        n, m, S = case["n"], case["m"], case["S"]
        return {"bytes": 16.0 * n * m + 16.0 * S * n + 8.0 * S * (n + m + n * m), "flops": S * _chain_flops(n, m)}
    if kind == "fock":
        return {"bytes": 16.0 * case["n"] * case["m"] + 8.0 * case["shots"] * case["m"], "flops": _fock_flops(case)}
    if kind == "batch":
        # means over the modes, photon numbers (4 to n_max, at most m / 4) and transmissions of prepare()
        G, S = case["circuits"], case["shots"]
        flops = nbytes = 0.0
        for m in BATCH_MODES:
            ns = range(4, min(case["n_max"], m // 4) + 1)
            for n in ns:
                w = 1.0 / (len(BATCH_MODES) * len(ns))
                flops += w * sum(p * _chain_flops(k, m) for k, p in _binomial(n, 0.8))
                nbytes += w * 16.0 * n * m
        return {"bytes": G * nbytes + 8.0 * G * S * max(BATCH_MODES), "flops": G * S * flops}
    # one pure term per step at least: 2^(k - 2) sign vectors, per column and label the 2 x 2 products of the
    # forward and backward chains and the trace (128 operations)
    n, S = case["n"], case["shots"]
    return {"bytes": 16.0 * 4 * n * n + 8.0 * S * 2 * n,
            "flops": S * sum(2.0 ** max(0, k - 2) * k * 256.0 for k in range(1, n + 1))}


# ------------------------------------------------------------------------------------------------ correctness
def _mixed_error(k: int) -> float:
    """FP32 blocks of 2^(k - 2) cancelling terms: about 5e-8 at few columns, growing 1.35 times per column."""
    return min(0.02, 2.0e-7 * 1.35 ** k)


def tolerance(case: dict):
    kind = case["kind"]
    if kind in ("cofactors", "marginals"):
        k = case["K"] if kind == "cofactors" else case["n"]
        if case["precision"] == "mixed":
            return {"rel": _mixed_error(k), "max": min(0.9, 40 * _mixed_error(k)), "differ": 1e-3}
        return {"rel": 1e-11, "max": 1e-9, "differ": 1e-3}
    # whole numbers: a draw within rounding of a step of its cumulative weights may fall on either side of it,
    # which changes the rest of that one shot.  Two shots of a pass may.
    if kind == "batch":
        shots, m, n = case["circuits"] * case["shots"], max(BATCH_MODES), case["n_max"]
    else:
        shots, n = case["shots"], case["n"]
        m = case.get("m", 2 * n)
    return {"differ": min(0.01, 4.0 * n / (shots * m))}


def _cofactors64(B: torch.Tensor) -> torch.Tensor:
    """P [S, K], P[s, c] = permanent of B[s] [K - 1, K] without column c: Glynn's sum over all sign vectors
    (the first sign +), every term formed from scratch."""
    S, k1, K = B.shape
    if k1 == 0:
        return torch.ones(S, 1, dtype=C128, device=B.device)
    total = 1 << (k1 - 1)
    step = max(1, min(total, (1 << 24) // (S * K)))
    P = torch.zeros(S, K, dtype=C128, device=B.device)
    bits = torch.arange(k1 - 1, device=B.device)
    for t0 in range(0, total, step):
        t = torch.arange(t0, min(total, t0 + step), device=B.device)
        d = 1.0 - 2.0 * ((t[:, None] >> bits) & 1).to(torch.float64)
        d = torch.cat([torch.ones(t.shape[0], 1, dtype=torch.float64, device=B.device), d], dim=1)
        s = torch.matmul(d.to(C128), B)                                  # [S, T, K] column sums
        w = d.prod(dim=1).to(C128)
        one = torch.ones_like(s[..., :1])
        left = torch.cat([one, torch.cumprod(s[..., :-1], dim=-1)], dim=-1)
        right = torch.cat([torch.cumprod(s.flip(-1)[..., :-1], dim=-1).flip(-1), one], dim=-1)
        P += (left * right * w[None, :, None]).sum(dim=1)
    return P * 2.0 ** (1 - k1)


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "cofactors":
        st = prepare(case, seed)
        A, rows = st["A"], st["rows"]
        return _cofactors64(torch.gather(A, 1, rows[:, :, None].expand(-1, -1, A.shape[2])))
    if kind == "marginals":
        st = prepare(case, seed)
        n, m, S = case["n"], case["m"], case["S"]
        cols = st["U"][:, :n].t()[st["sigma"]]                            # [S, n, m] columns in chain order
        rows = torch.zeros(S, n, dtype=torch.int64, device="cuda")
        marg = torch.zeros(S, n, m, dtype=torch.float64, device="cuda")
        for k in range(1, n + 1):
            At = cols[:, :k]                                              # [S, k, m]
            B = torch.gather(At, 2, rows[:, None, :k - 1].expand(-1, k, -1)).transpose(1, 2)
            amp = torch.einsum("skm,sk->sm", At, _cofactors64(B))
            w = amp.real ** 2 + amp.imag ** 2
            cw = torch.cumsum(w, dim=1)
            tot = cw[:, -1:]
            marg[:, k - 1] = w / tot
            rows[:, k - 1] = (cw < st["uniforms"][:, k - 1:k] * tot).sum(dim=1).clamp(max=m - 1)
        return {"rows": None, "occ": None, "marg": marg}
    return None                                                           # samples: whole numbers only
