"""Measured workloads of the superblock engine: the calls of one finite-sweep
step as a user's program makes them, from the smallest sector to the largest.

A case is a dict of plain values.  ``prepare`` builds what the program has in
hand (operator blocks, handle, vectors), ``run`` is one pass through the
public entry points, ``exact`` the same result from plain torch in 64 bits.

The sectors have the shapes of the package's generators
(``dmrgpp_b200/superblock.py``): the five Kronecker terms of a spin-1/2 link
over Gaussian Sz histograms ("spin"), and the six or ten terms of a Hubbard
chain or two-leg ladder over (N_up, N_down) histograms ("hubbard", legs 1 or
2).  Entries are N(0, 1); left and right blocks may differ in size.
"""
import math

import numpy as np
import torch

from dmrgpp_b200 import plugin, truncation, wft
from dmrgpp_b200.superblock import KronProblem, gaussian_sector_sizes

DEV = "cuda"


def listed():
    return [
        # a Heisenberg chain at m = 128 (the suite's smallest whole DMRG run):
        # one matvec inside a device solver, where latency is everything
        {"name": "matvec_spin256", "kind": "matvec", "model": "spin", "left": 256, "right": 256, "groups": 13,
         "precision": "fp64", "place": "device"},
        # the synthetic microbench sector through the plugin call of the host
        # program: host vectors in and out
        {"name": "matvec_spin1024_host", "kind": "matvec", "model": "spin", "left": 1024, "right": 1024, "groups": 21,
         "precision": "fp64", "place": "host"},
        # the complex instantiation of the plugin, blocks of unequal odd sizes
        {"name": "matvec_complex701", "kind": "matvec", "model": "spin", "left": 701, "right": 555, "groups": 17,
         "precision": "complex", "place": "device"},
        # a Hubbard chain at m = 1000, tensor-core arithmetic: many patches of
        # ragged sizes below one tile
        {"name": "matvec_chain4000_tf32x3", "kind": "matvec", "model": "hubbard", "legs": 1, "sigma": 2.5,
         "left": 4000, "right": 4000, "precision": "tf32x3", "place": "device"},
        # the two-leg ladder at m = 4000 in both precisions: the largest sector
        {"name": "matvec_ladder16000_fp64", "kind": "matvec", "model": "hubbard", "legs": 2, "sigma": 2.5,
         "left": 16000, "right": 16000, "precision": "fp64", "place": "device"},
        {"name": "matvec_ladder16000_tf32x3", "kind": "matvec", "model": "hubbard", "legs": 2, "sigma": 2.5,
         "left": 16000, "right": 16000, "precision": "tf32x3", "place": "device"},
        # a serving-style batch of independent sectors in one launch
        {"name": "matvec_batch64_fp64", "kind": "batch", "count": 64, "mix": 1, "precision": "fp64"},
        # FP64 Lanczos with full reorthogonalisation (the reference's solver),
        # bounded by its step limit as in the early steps of a sweep
        {"name": "lanczos_chain2500", "kind": "lanczos", "model": "hubbard", "legs": 1, "sigma": 2.5,
         "left": 2500, "right": 2300, "steps": 60},
        # a whole sector solve: TF32x3 Lanczos and FP64 refinement
        {"name": "solve_ladder6000", "kind": "solve", "model": "hubbard", "legs": 2, "sigma": 2.5,
         "left": 6000, "right": 6000},
        # whole mixed-precision solves of a batch, all sectors in lockstep
        {"name": "solve_batch24", "kind": "batch_solve", "count": 24, "mix": 2},
        # the wave-function transformation before a solve ...
        {"name": "wft_ladder16000", "kind": "wft", "sigma": 2.5, "left": 16000, "right": 16000, "left_out": 16000,
         "right_out": 16000},
        # ... and the density-matrix truncation after it, 16000 states to 4000
        {"name": "truncate_ladder16000", "kind": "truncate", "sigma": 2.5, "left": 16000, "right": 16000, "keep": 4000},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "matvec", "batch", "lanczos", "solve", "batch_solve", "wft", "truncate"])
    if kind == "matvec":
        precision = rng.choice(["fp64", "fp64", "tf32x3", "tf32x3", "complex"])
        if precision == "complex" or rng.random() < 0.4:
            left = _spread(rng, 60, 1500)
            return {"kind": kind, "model": "spin", "left": left, "right": max(40, int(left * rng.uniform(0.6, 1.4))),
                    "groups": rng.choice([5, 9, 13, 17, 21]), "precision": precision,
                    "place": rng.choice(["device", "device", "host"])}
        left = _spread(rng, 400, 14000)
        return {"kind": kind, "model": "hubbard", "legs": rng.choice([1, 2]), "sigma": round(rng.uniform(1.2, 3.0), 2),
                "left": left, "right": min(16000, int(left * rng.uniform(0.7, 1.3))), "precision": precision,
                "place": "device"}
    if kind == "batch":
        return {"kind": kind, "count": _spread(rng, 3, 64), "mix": rng.randrange(1 << 16),
                "precision": rng.choice(["fp64", "tf32x3"])}
    if kind == "lanczos":
        left = _spread(rng, 900, 6000)
        return {"kind": kind, "model": "hubbard", "legs": rng.choice([1, 2]), "sigma": round(rng.uniform(1.8, 2.8), 2),
                "left": left, "right": int(left * rng.uniform(0.8, 1.2)), "steps": rng.randrange(30, 61)}
    if kind == "solve":
        left = _spread(rng, 900, 6000)
        return {"kind": kind, "model": "hubbard", "legs": rng.choice([1, 2]), "sigma": round(rng.uniform(1.8, 2.8), 2),
                "left": left, "right": min(6000, int(left * rng.uniform(0.8, 1.2)))}
    if kind == "batch_solve":
        return {"kind": kind, "count": _spread(rng, 3, 24), "mix": rng.randrange(1 << 16)}
    left, right = _spread(rng, 700, 14000), _spread(rng, 700, 14000)
    if kind == "wft":
        return {"kind": kind, "sigma": round(rng.uniform(1.5, 3.0), 2), "left": left, "right": right,
                "left_out": max(200, int(left * rng.choice([1.0, 0.5, 0.25]))),
                "right_out": max(200, int(right * rng.choice([1.0, 0.5, 0.25])))}
    # more environment states than are kept, or the last kept ones were arbitrary
    return {"kind": kind, "sigma": round(rng.uniform(1.5, 3.0), 2), "left": left,
            "right": int(left * rng.uniform(0.5, 1.2)), "keep": max(64, left // 4)}


# ---- sector shapes -------------------------------------------------------

def _spin_shape(left, right, groups):
    """Sizes and terms of an Sz-conserving sector of a spin-1/2 link.  Terms:
    (output patch, input patch, term, kind of A, kind of B) with kinds "sym",
    "eye" or the number of a random matrix, transposed if negative."""
    l = np.maximum(1, gaussian_sector_sizes(left, groups, groups / 5.0))
    r = np.maximum(1, gaussian_sector_sizes(right, groups, groups / 5.0))
    terms, n = [], 0
    for p in range(groups):
        terms += [(p, p, 0, "sym", "eye"), (p, p, 1, "eye", "sym"), (p, p, 2, "sym", "sym")]
    for p in range(groups - 1):
        n += 1
        terms += [(p + 1, p, 3, n, n), (p, p + 1, 4, -n, -n)]
    return l, r, 5, terms


def _hubbard_groups(states, sigma, centre=(0, 0)):
    """(N_up, N_down) histogram: sizes by quantum numbers."""
    reach = int(math.ceil(4 * sigma))
    qs = [(a, b) for a in range(-reach, reach + 1) for b in range(-reach, reach + 1)]
    w = np.array([math.exp(-((a - centre[0]) ** 2 + (b - centre[1]) ** 2) / (2 * sigma * sigma)) for a, b in qs])
    n = np.floor(states * w / w.sum()).astype(np.int64)
    n[int(np.argmax(w))] += states - int(n.sum())
    return {q: int(k) for q, k in zip(qs, n) if k > 0}


def _hubbard_shape(left, right, sigma, legs):
    gl, gr = _hubbard_groups(left, sigma), _hubbard_groups(right, sigma)
    qs = [q for q in gl if (-q[0], -q[1]) in gr]
    index = {q: p for p, q in enumerate(qs)}
    l = np.array([gl[q] for q in qs], dtype=np.int64)
    r = np.array([gr[(-q[0], -q[1])] for q in qs], dtype=np.int64)
    terms, n = [], 0
    for p in range(len(qs)):
        terms += [(p, p, 0, "sym", "eye"), (p, p, 1, "eye", "sym")]
    k = 2
    for step in ((1, 0), (0, 1)):
        for _ in range(legs):
            for p, (a, b) in enumerate(qs):
                q = index.get((a + step[0], b + step[1]))
                if q is not None:
                    n += 1
                    terms += [(q, p, k, n, n), (p, q, k + 1, -n, -n)]
            k += 2
    return l, r, k, terms


def _shape(case):
    if case["model"] == "spin":
        return _spin_shape(case["left"], case["right"], case["groups"])
    return _hubbard_shape(case["left"], case["right"], case["sigma"], case["legs"])


def _batch_shapes(case):
    """Heisenberg and Hubbard sectors, half each, of chains of 16 to 48 sites
    and m in {64, 128, 256, 512}, as in the package's serving batch."""
    g = np.random.default_rng(case["mix"])
    shapes = []
    for _ in range(case["count"]):
        sites, m = int(g.integers(16, 49)), int(g.choice([64, 128, 256, 512]))
        if g.random() < 0.5:
            shapes.append(_spin_shape(2 * m, 2 * m, 2 * int(round(math.sqrt(sites / 2))) + 1))
        else:
            shapes.append(_hubbard_shape(4 * m, 4 * m, 1.0 + sites / 32.0, 1))
    return shapes


def _batch_problems(case, seed):
    return [_problem(s, seed + 1000 * q) for q, s in enumerate(_batch_shapes(case))]


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float64)


def _blocks(shape, g, imaginary=False):
    """The sector's blocks on the GPU, each stored transposed (row-major of the
    transpose = column-major of the block): {(i, j, k): (A^T, B^T)}.  The
    imaginary part of a complex sector is antisymmetric where the real part is
    symmetric, so that H stays Hermitian."""
    l, r, _, terms = shape
    pairs, out, eye = {}, {}, {}

    def one(kind, n_out, n_in, side):
        if kind == "eye":
            if n_out not in eye:
                eye[n_out] = torch.eye(n_out, dtype=torch.float64, device=DEV)
            return torch.zeros_like(eye[n_out]) if imaginary else eye[n_out]
        if kind == "sym":
            a = _randn(g, n_out, n_in)
            return 0.5 * (a - a.T) if imaginary else 0.5 * (a + a.T)
        if kind > 0:
            pairs[kind, side] = _randn(g, n_in, n_out)
            return pairs[kind, side]
        t = pairs[-kind, side].T.contiguous()
        return -t if imaginary else t
    for i, j, k, ka, kb in terms:
        out[i, j, k] = (one(ka, int(l[i]), int(l[j]), 0), one(kb, int(r[i]), int(r[j]), 1))
    return out


def _problem(shape, seed, complex_blocks=False):
    """KronProblem in host memory, as the plugin's caller holds it."""
    g = _generator(seed)
    blocks = _blocks(shape, g)
    if complex_blocks:
        imag = _blocks(shape, g, imaginary=True)
        blocks = {t: tuple(torch.complex(a, b) for a, b in zip(blocks[t], imag[t])) for t in blocks}
    keys = list(blocks)
    flat = torch.cat([m.reshape(-1) for t in keys for m in blocks[t]]).cpu().numpy()
    A, B, at = {}, {}, 0
    for t in keys:
        for table, m in zip((A, B), blocks[t]):
            table[t] = flat[at:at + m.numel()].reshape((m.shape[1], m.shape[0]), order="F")
            at += m.numel()
    return KronProblem(shape[0], shape[1], shape[2], A, B)


def _dim(shape):
    return int(np.sum(shape[0] * shape[1]))


def _work_matvec(shape, per_value=8):
    """Flops and bytes one H*x cannot do without.  A term with an identity
    factor is one product; the others are two, in the cheaper order."""
    l, r, _, terms = shape
    flops = byts = 0
    for i, j, _, ka, kb in terms:
        li, lj, ri, rj = int(l[i]), int(l[j]), int(r[i]), int(r[j])
        if kb == "eye":
            flops += 2 * rj * lj * li
        elif ka == "eye":
            flops += 2 * ri * rj * lj
        else:
            flops += min(2 * ri * lj * (rj + li), 2 * rj * li * (lj + ri))
        byts += per_value * ((0 if ka == "eye" else li * lj) + (0 if kb == "eye" else ri * rj))
    return float(flops), float(byts), _dim(shape)


# ---- the cases -----------------------------------------------------------

_PRECISION = {"fp64": plugin.FP64, "tf32x3": plugin.TF32X3, "complex": plugin.FP64}


def _start(seed, n, dtype=torch.float64):
    g = _generator(seed + 7919)
    return torch.randn(n, generator=g, device=DEV, dtype=dtype)


def _wft_layout(case):
    gl, gr = _hubbard_groups(case["left"], case["sigma"]), _hubbard_groups(case["right"], case["sigma"])
    ol, orr = _hubbard_groups(case["left_out"], case["sigma"]), _hubbard_groups(case["right_out"], case["sigma"])
    qs = [q for q in gl if (-q[0], -q[1]) in gr]
    outs = [q for q in qs if q in ol and (-q[0], -q[1]) in orr]
    at = {q: p for p, q in enumerate(qs)}
    return ([gl[q] for q in qs], [gr[-q[0], -q[1]] for q in qs], [ol[q] for q in outs], [orr[-q[0], -q[1]] for q in outs],
            [at[q] for q in outs])


def _wft_blocks(case, seed):
    l, r, lo, ro, src = _wft_layout(case)
    g = _generator(seed)
    WL = [_randn(g, lo[q], l[p]) / math.sqrt(l[p]) for q, p in enumerate(src)]
    WR = [_randn(g, ro[q], r[p]) / math.sqrt(r[p]) for q, p in enumerate(src)]
    return WL, WR


def _truncation_state(case, seed):
    """Sector vector whose patches have decaying singular values, as the
    Schmidt weights of a ground state."""
    l, r, _, _ = _hubbard_shape(case["left"], case["right"], case["sigma"], 1)
    g, parts = _generator(seed), []
    for lp, rp in zip(l.tolist(), r.tolist()):
        n = min(lp, rp)
        weight = torch.exp(-5.0 * torch.arange(n, device=DEV, dtype=torch.float64) / n)
        parts.append(((_randn(g, lp, n) * weight) @ _randn(g, n, rp)).reshape(-1) / math.sqrt(n))
    psi = torch.cat(parts)
    return l, r, psi / torch.linalg.vector_norm(psi)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "matvec":
        shape, cplx = _shape(case), case["precision"] == "complex"
        bg = plugin.BatchedGemm.from_problem(_problem(shape, seed, cplx), precision=_PRECISION[case["precision"]])
        x = _start(seed, _dim(shape), torch.complex128 if cplx else torch.float64)
        if case["place"] == "host":
            x = x.cpu().numpy()
            return {"do": "apply", "bg": bg, "x": x, "y": np.empty_like(x)}
        return {"do": "apply", "bg": bg, "x": x, "y": torch.empty_like(x)}
    if kind == "batch":
        bg = plugin.BatchedGemm.from_problems(_batch_problems(case, seed), precision=_PRECISION[case["precision"]])
        x = _start(seed, bg.dim)
        return {"do": "apply", "bg": bg, "x": x, "y": torch.empty_like(x)}
    if kind == "batch_solve":
        bg = plugin.BatchedGemm.from_problems(_batch_problems(case, seed), precision=plugin.TF32X3)
        return {"do": kind, "bg": bg, "x": _start(seed, bg.dim)}
    if kind in ("lanczos", "solve"):
        bg = plugin.BatchedGemm.from_problem(_problem(_shape(case), seed),
                                             precision=plugin.FP64 if kind == "lanczos" else plugin.TF32X3)
        return {"do": kind, "bg": bg, "x": _start(seed, bg.dim), "steps": case.get("steps")}
    if kind == "wft":
        l, r, lo, ro, src = _wft_layout(case)
        WL, WR = ([m.cpu().numpy() for m in side] for side in _wft_blocks(case, seed))
        w = wft.WaveFunctionTransform(l, r, lo, ro, src, WL, WR)
        return {"do": kind, "w": w, "x": _start(seed, w.dim_in),
                "y": torch.empty(w.dim_out, dtype=torch.float64, device=DEV)}
    l, r, psi = _truncation_state(case, seed)
    return {"do": kind, "l": l, "r": r, "group": np.arange(len(l)), "psi": psi, "keep": case["keep"]}


def run(state):
    do = state["do"]
    if do == "apply":
        state["bg"].apply_Htarget(state["x"], state["y"])
        return state["y"]
    if do == "lanczos":
        energy, z, _ = state["bg"].lanczos_lowest(state["x"], steps=state["steps"])
        return {"energy": energy, "vector": z}
    if do == "solve":
        energy, z, _ = state["bg"].solve_lowest(state["x"])
        return {"energy": energy, "vector": z}
    if do == "batch_solve":
        energy, z, _ = state["bg"].solve_lowest_group(state["x"])
        return {"energy": energy, "vector": z}
    if do == "wft":
        return state["w"](state["x"], state["y"])
    t = truncation.density_truncate(state["l"], state["r"], state["group"], state["l"], 0, state["psi"], state["keep"])
    # the kept vectors of all groups are views of one packed array
    return {"eigenvalues": np.concatenate(t["eigenvalues"]), "vectors": t["vectors"][0].base, "kept": t["kept"],
            "discarded": t["discarded"]}


def work(case):
    kind = case["kind"]
    if kind == "matvec":
        cplx = case["precision"] == "complex"
        flops, byts, n = _work_matvec(_shape(case), 16 if cplx else 8)
        return {"bytes": byts + 2 * n * (16 if cplx else 8), "flops": flops * (4 if cplx else 1)}
    if kind in ("batch", "batch_solve"):
        each = [_work_matvec(s) for s in _batch_shapes(case)]
        # a whole solve: some 100 matvecs a sector
        times = 100 if kind == "batch_solve" else 1
        return {"bytes": sum(b + 16 * n for _, b, n in each), "flops": times * sum(f for f, _, _ in each)}
    if kind in ("lanczos", "solve"):
        flops, byts, n = _work_matvec(_shape(case))
        steps = case.get("steps", 100)
        # the reorthogonalisation reads the stored vectors twice in each step
        basis = steps * (steps + 1) // 2 if kind == "lanczos" else 0
        return {"bytes": byts + 16 * n * (1 + basis), "flops": steps * flops + 4.0 * n * basis}
    if kind == "wft":
        l, r, lo, ro, src = _wft_layout(case)
        flops = byts = 0
        for q, p in enumerate(src):
            flops += min(2 * ro[q] * l[p] * (r[p] + lo[q]), 2 * r[p] * lo[q] * (l[p] + ro[q]))
            byts += 8 * (lo[q] * l[p] + ro[q] * r[p] + l[p] * r[p] + lo[q] * ro[q])
        return {"bytes": float(byts), "flops": float(flops)}
    l, r, _, _ = _hubbard_shape(case["left"], case["right"], case["sigma"], 1)
    l, r = l.astype(float), r.astype(float)
    share = min(1.0, case["keep"] / l.sum())
    # density matrices (half: symmetric), tridiagonal reduction, kept vectors
    return {"bytes": float(8 * np.sum(l * r + 2 * l * l * share + l)),
            "flops": float(np.sum(l * l * r + 4.0 / 3.0 * l ** 3 + 2 * l ** 3 * share))}


def tolerance(case):
    """About four times what another order of the sums shows; the tensor-core
    sums are kept in 32 bits over up to thousands of terms, and the solves
    stop at a residual of 1e-10 |E|."""
    kind = case["kind"]
    if kind in ("matvec", "batch") and case["precision"] == "tf32x3":
        return {"rel": 1e-4}
    return {"rel": {"matvec": 8e-15, "batch": 8e-15, "wft": 8e-15, "lanczos": 1e-12, "solve": 1e-9, "batch_solve": 1e-9,
                    "truncate": 1e-12}[kind]}


# ---- 64-bit results from plain torch -------------------------------------

def _gpu_blocks(shape, seed, complex_blocks=False):
    g = _generator(seed)
    blocks = _blocks(shape, g)
    if complex_blocks:
        imag = _blocks(shape, g, imaginary=True)
        blocks = {t: tuple(torch.complex(a, b) for a, b in zip(blocks[t], imag[t])) for t in blocks}
    return blocks


def _apply(shape, blocks, x):
    """Y_i = sum B X_j A^T with the patches column-major: as row-major l x r
    matrices, Y_i^T = sum A X_j^T B^T."""
    l, r = shape[0].tolist(), shape[1].tolist()
    at = np.concatenate(([0], np.cumsum(shape[0] * shape[1]))).tolist()
    y = torch.zeros_like(x)
    for (i, j, _), (a_t, b_t) in blocks.items():
        y[at[i]:at[i + 1]].view(l[i], r[i]).addmm_(a_t.T, x[at[j]:at[j + 1]].view(l[j], r[j]) @ b_t)
    return y


def _lanczos(apply, x, steps, tolerance=0.0):
    """Lowest Ritz pair after so many steps, full reorthogonalisation."""
    V = torch.empty(min(steps, x.numel()), x.numel(), dtype=torch.float64, device=DEV)
    alpha, beta, last = [], [], None
    v = x / torch.linalg.vector_norm(x)
    for j in range(V.shape[0]):
        V[j] = v
        w = apply(v)
        alpha.append(float(w @ v))
        w -= alpha[-1] * v
        if j:
            w -= beta[-1] * V[j - 1]
        for _ in range(2):
            w -= V[:j + 1].T @ (V[:j + 1] @ w)
        beta.append(float(torch.linalg.vector_norm(w)))
        v = w / beta[-1]
        if tolerance and j % 10 == 9:
            e = np.linalg.eigvalsh(np.diag(alpha) + np.diag(beta[:-1], 1) + np.diag(beta[:-1], -1))[0]
            if last is not None and abs(e - last) <= tolerance * abs(e):
                break
            last = e
    n = len(alpha)
    e, s = np.linalg.eigh(np.diag(alpha) + np.diag(beta[:n - 1], 1) + np.diag(beta[:n - 1], -1))
    return float(e[0]), torch.from_numpy(s[:, 0]).to(DEV) @ V[:n]


def exact(case, seed):
    kind = case["kind"]
    if kind == "matvec":
        shape, cplx = _shape(case), case["precision"] == "complex"
        y = _apply(shape, _gpu_blocks(shape, seed, cplx), _start(seed, _dim(shape), torch.complex128 if cplx else torch.float64))
        return y.cpu().numpy() if case["place"] == "host" else y
    if kind in ("batch", "batch_solve"):
        shapes = _batch_shapes(case)
        x = _start(seed, sum(_dim(s) for s in shapes)).split([_dim(s) for s in shapes])
        got = []
        for q, shape in enumerate(shapes):
            blocks = _gpu_blocks(shape, seed + 1000 * q)
            if kind == "batch":
                got.append(_apply(shape, blocks, x[q]))
            else:
                got.append(_lanczos(lambda v: _apply(shape, blocks, v), x[q], 300, 1e-15)[0])
        return torch.cat(got) if kind == "batch" else {"energy": np.array(got), "vector": None}
    if kind in ("lanczos", "solve"):
        shape = _shape(case)
        blocks = _gpu_blocks(shape, seed)
        x = _start(seed, _dim(shape))
        steps, tol = (case["steps"], 0.0) if kind == "lanczos" else (400, 1e-15)
        # the sign of a Ritz vector is free
        return {"energy": _lanczos(lambda v: _apply(shape, blocks, v), x, steps, tol)[0], "vector": None}
    if kind == "wft":
        l, r, lo, ro, src = _wft_layout(case)
        WL, WR = _wft_blocks(case, seed)
        n = [a * b for a, b in zip(l, r)]
        x = _start(seed, sum(n)).split(n)
        return torch.cat([(WL[q] @ x[p].view(l[p], r[p]) @ WR[q].T).reshape(-1) for q, p in enumerate(src)])
    l, r, psi = _truncation_state(case, seed)
    sizes = (l * r).tolist()
    eig = [torch.linalg.eigvalsh(m @ m.T) for m in
           (p.view(a, b) for p, a, b in zip(psi.split(sizes), l.tolist(), r.tolist()))]
    eig = torch.cat(eig).cpu().numpy()
    # vectors: free signs
    return {"eigenvalues": eig, "vectors": None, "kept": None, "discarded": float(np.sort(eig)[:-case["keep"]].sum())}
