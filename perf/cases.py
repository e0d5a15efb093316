"""Performance cases: the calls this library is used for, through its Python entry points.

Each case is one unit of a user's work: the twist mesh of one or a few disorder samples (rlm
and hlm, the drivers' loop), the finite-size-scaling graph, or the stage-by-stage form
(assemble, eigensolve, plaquette phases of one pair of theta_1 lines) a program uses that
keeps its own mesh.  Every output is gauge invariant (energies, Chern numbers, plaquette
phases), so it does not depend on the phases of the eigenvectors.

    listed()              the cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   the context, inputs and plan a program holds before the call
    run(state)            one pass
    work(case)            bytes and flops the pass cannot do without
    exact(case, seed)     the same outputs in 64-bit numpy, where that is quick
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "random-landau-model_b200"))
import rlmb  # noqa: E402

# Impurity concentration of every rlm case: the benchmark's, and the drivers' usual one.
IMPURITIES = 16.0


# ------------------------------------------------------------------------------ cases
def _rlm(n_phi, g, samples, mode="fp64", **more):
    return dict(more, kind="rlm", n_phi=n_phi, g=g, samples=samples, mode=mode)


def _hlm(lx, ly, q, band, g, samples, host, mode="fp64", **more):
    return dict(more, kind="hlm", lx=lx, ly=ly, q=q, band=band, g=g, samples=samples, host=host, mode=mode)


def _fss(sizes, g, samples, mode="fp64", **more):
    return dict(more, kind="fss", sizes=sizes, g=g, samples=samples, mode=mode)


def _line(n_phi, g, mode="fp64", **more):
    return dict(more, kind="line", n_phi=n_phi, g=g, mode=mode)


def listed():
    return [
        # the smallest mesh a user runs (a first check, a quick scan over seeds): latency
        _rlm(16, 8, 1, name="rlm16_g8"),
        # plain rlm on a fine mesh: thousands of tiny matrices
        _rlm(16, 64, 2, name="rlm16_g64_s2"),
        # a small odd order on a coarse odd mesh, fewer matrices than it takes to fill the GPU
        _rlm(129, 7, 2, name="rlm129_g7_s2"),
        # many samples of a small lattice, upper band, potentials and results on the host
        _hlm(12, 8, 3, 2, 8, 32, True, name="hlm12x8_b2_g8_s32"),
        # the smallest order of a finite-size-scaling set, all its samples in one call
        _rlm(64, 16, 16, name="rlm64_g16_s16"),
        # the Hofstadter benchmark geometry, a few samples with device-resident data
        _hlm(48, 16, 3, 0, 32, 4, False, name="hlm48x16_g32_s4"),
        # the mid-size rlm benchmark geometry in both precision modes
        _rlm(512, 16, 2, name="rlm512_g16_s2"),
        _rlm(512, 16, 2, "mixed", name="rlm512_g16_s2_mixed"),
        # a finite-size-scaling step: every order of the set in one graph launch
        _fss("64,128,192,256,384,512", 16, 1, name="fss64to512_g16"),
        # one theta_1 line pair solved stage by stage by a program that keeps its own mesh
        _line(300, 8, name="line300_g8"),
        # one sample of a large system, 25 matrices: in double precision, and the largest order
        # in the mixed mode that is meant for it
        _rlm(2500, 4, 1, name="rlm2500_g4"),
        _rlm(3000, 4, 1, "mixed", name="rlm3000_g4_mixed"),
    ]


def draw(rng):
    """A case of the listed ones' ranges: orders 16 .. 2500 spread over their logarithm, as
    much work as a typical call of that order up to that of the largest listed case."""
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["rlm", "rlm", "rlm", "hlm", "hlm", "line", "fss"])
    mode = rng.choice(["fp64", "fp64", "mixed"])
    if kind == "rlm":
        n = log(16, 2500)
        g = 4 if n > 1000 else rng.randint(4, 64 if n <= 64 else 20 if n <= 300 else 8)
        # samples: up to about 16, bounded by the largest listed case's work and by memory
        most = min(16.0, 0.4 * 25 * 3000.0 ** 3 / ((g + 1) ** 2 * n ** 3.0), 2.5e5 / (g + 1) ** 2)
        return _rlm(n, g, log(1, max(1.0, most)), mode)
    if kind == "hlm":
        lx, ly, q = rng.choice([(6, 6, 3), (9, 6, 3), (12, 8, 3), (24, 8, 3), (20, 10, 5), (24, 16, 3),
                                (36, 12, 3), (48, 16, 3)])
        n = lx * ly // q
        g = rng.randint(4, 32)
        most = min(64.0, 1.5e11 / ((g + 1) * g * n ** 3.0), 2.5e5 / ((g + 1) * g))
        return _hlm(lx, ly, q, rng.randrange(q), g, log(1, max(1.0, most)), rng.random() < 0.5, mode)
    if kind == "line":
        return _line(log(16, 1200), rng.randint(4, 12), mode)
    first = rng.randint(24, 96)
    return _fss("%d,%d,%d" % (first, 2 * first + rng.randint(0, 9), 4 * first), rng.randint(6, 16), 1, mode)


# -------------------------------------------------------------------------------- run
def _context(mode):
    ctx = rlmb.Context(0)
    ctx.precision = ctx.MIXED if mode == "mixed" else ctx.FP64   # two refinement steps, the default
    return ctx


def _line_thetas(g):
    """theta indices of two adjacent theta_1 lines (0 and 1), theta_2 = 0 .. g on each."""
    return [0] * (g + 1) + [1] * (g + 1), list(range(g + 1)) * 2


def prepare(case, seed):
    kind, g = case["kind"], case["g"]
    s = dict(case=case, seed=seed)
    if kind == "rlm":
        s["ctx"] = _context(case["mode"])
    elif kind == "hlm":
        s["ctx"] = _context(case["mode"])
        sites, n = case["lx"] * case["ly"], case["lx"] * case["ly"] // case["q"]
        if case["host"]:
            s["pots"] = rlmb.hlm_potentials(seed, sites, case["samples"])
        else:
            s["pots"] = s["ctx"].hlm_potentials_device(seed, sites, 0, case["samples"])
            s["e"] = torch.empty((case["samples"], n), dtype=torch.float64, device="cuda")
            s["c"] = torch.empty_like(s["e"])
    elif kind == "fss":
        sizes = [int(v) for v in case["sizes"].split(",")]
        s["graph"] = rlmb.FssGraph(0, sizes, 1.0, IMPURITIES, g, seed, case["samples"],
                                   1 if case["mode"] == "mixed" else 0)
    else:
        ctx = s["ctx"] = _context(case["mode"])
        p = rlmb.rlm_params(case["n_phi"], 1.0, IMPURITIES)
        cmn, cmt, cjm = rlmb.rlm_coeff_tables(case["n_phi"], p["off_head"], g, p["L1"], p["L2"])
        x, y, st = rlmb.rlm_disorder(p["impurity_num"], p["L1"], p["L2"], seed, 0)
        s["off"] = p["off_head"]
        s["cmn"], s["cmt"], s["cjm"] = (torch.from_numpy(v).cuda() for v in (cmn, cmt, cjm))
        s["imp"] = [torch.from_numpy(v[None]).cuda() for v in (x, y, st)]
        s["t1"], s["t2"] = (np.array(t, dtype=np.int32) for t in _line_thetas(g))
        # (the context's stream, and every handle, is the one run() uses)
        ctx.sync_stream()
    return s


def run(s):
    case = s["case"]
    kind, g = case["kind"], case["g"]
    if kind == "rlm":
        return s["ctx"].rlm_mesh_solve(case["n_phi"], 1.0, IMPURITIES, g, s["seed"], 0, case["samples"])
    if kind == "hlm":
        geom = (case["lx"], case["ly"], case["q"], case["band"], g)
        if case["host"]:
            return s["ctx"].hlm_mesh_solve(*geom, s["pots"])
        s["ctx"].hlm_mesh_solve_device(*geom, s["pots"], s["e"], s["c"])
        return s["e"], s["c"]
    if kind == "fss":
        s["graph"].launch(0)
        return [s["graph"].results(i) for i in range(len(s["graph"].n_phis))]
    ctx, n = s["ctx"], case["n_phi"]
    v = ctx.rlm_potential(*s["imp"], s["cmn"], s["off"])
    h = ctx.rlm_assemble(v, s["cmt"], s["cjm"], n, s["off"], g, s["t1"], s["t2"])
    w = ctx.heevd(h)
    return w, ctx.fhs_line(h[:g + 1], h[g + 1:])


def _orders(case):
    """[(order, matrices, impurities, dim, samples)] of one pass."""
    g = case["g"]
    if case["kind"] == "hlm":
        return [(case["lx"] * case["ly"] // case["q"], (g + 1) * g * case["samples"], 0, 0, case["samples"])]
    sizes = [int(v) for v in case["sizes"].split(",")] if case["kind"] == "fss" else [case["n_phi"]]
    samples = case.get("samples", 1)
    mats = (2 * (g + 1) if case["kind"] == "line" else (g + 1) ** 2) * samples
    out = []
    for n in sizes:
        nimp = int(IMPURITIES * n)
        out.append((n, mats, nimp, 2 * int(math.sqrt(nimp) / 2 + 1) + 1, samples))
    return out


def work(case):
    """Flops: 16/3 n^3 (zhetrd) + 8 n^3 (zunmtr) per eigensolve and the V_mn sums; bytes: the
    inputs (impurities or potentials) read and the results written once."""
    flops = bytes_ = 0.0
    for n, mats, nimp, dim, samples in _orders(case):
        flops += mats * (40.0 / 3.0) * n ** 3.0 + samples * 8.0 * dim * dim * nimp
        bytes_ += samples * (24.0 * nimp + 16.0 * n)
        if case["kind"] == "hlm":
            bytes_ += samples * 8.0 * case["lx"] * case["ly"]
        if case["kind"] == "line":
            bytes_ += mats * 8.0 * n + 8.0 * n * case["g"]
    return {"bytes": bytes_, "flops": flops}


# ------------------------------------------------------------ the same in 64-bit numpy
# Largest sum of matrices * order^3 that is solved here (about 20 s of host LAPACK).
EXACT_MOST = 3e9


def _draws(seed, n):
    """The first n outputs of the seeded 32-bit Mersenne Twister."""
    return np.random.RandomState(seed).randint(0, 2 ** 32, size=n, dtype=np.uint32)


def _plaquettes(prev, cur):
    """-arg of the four-link product / 2 pi of every plaquette and state: prev, cur are
    [g + 1, N, dim] (row = state)."""
    def link(a, b):
        return np.einsum("tnr,tnr->tn", a.conj(), b)

    prod = link(prev[:-1], cur[:-1]) * link(cur[:-1], cur[1:]) * link(cur[1:], prev[1:]) * link(prev[1:], prev[:-1])
    return -np.angle(prod) / (2.0 * math.pi)


def _rlm_matrices(n, g, seed, samples):
    """Yields, per sample, a function (theta_1, theta_2) -> H (numpy, n x n)."""
    nimp = int(IMPURITIES * n)
    o = int(math.sqrt(nimp) / 2 + 1)
    d = 2 * o + 1
    k = np.arange(d) - o
    # the model's coefficients carry a single-precision Gaussian and 1/n
    arg = (-math.pi * (k[:, None] ** 2 + k[None, :] ** 2) / 2.0 / n).astype(np.float32)
    gauss = np.exp(arg.astype(np.float64)).astype(np.float32).astype(np.float64)
    cmn = np.exp(-1j * math.pi * k[:, None] * k[None, :] / n) * gauss * float(np.float32(1.0) / np.float32(n))
    cjm = np.exp(-2j * math.pi * k[None, :] * (np.arange(n)[:, None] + 1) / n)
    side = math.sqrt(n)
    raw = _draws(seed, 3 * nimp * samples).reshape(samples, 3, nimp)
    for r in raw:
        x, y = r[0] * (side / 2.0 ** 32), r[1] * (side / 2.0 ** 32)
        st = np.where(r[2] % 2 == 0, 1.0, -1.0)
        ex = np.exp(-2j * math.pi * np.outer(k, x)) * st
        v = (ex @ np.exp(-2j * math.pi * np.outer(k, y)).T) * cmn

        def build(t1, t2, v=v):
            gm = v * np.exp(2j * math.pi * t1 * k / g / n)[None, :]
            band = np.zeros((d, n), dtype=np.complex128)
            for q in range(d):
                delta = q - o
                for c in (delta, delta + n):
                    if 0 <= c < n:
                        band[:, c] += gm[:, q]
            rows = (np.exp(-2j * math.pi * t2 * k / g / n)[None, :] * cjm) @ band
            i, j = np.triu_indices(n)
            h = np.zeros((n, n), dtype=np.complex128)
            h[i, j] = rows[i, j - i]
            h[j, i] = h[i, j].conj()
            # the solver's matrix is the conjugate of the row-major buffer
            h = h.conj()
            h[np.arange(n), np.arange(n)] = h.diagonal().real
            return h

        yield build


def _solve(build, points):
    """(eigenvalues [k, n], vectors [k, n, n] with row = state) at the given points."""
    w, x = np.linalg.eigh(np.stack([build(*p) for p in points]))
    return w, np.swapaxes(x, 1, 2)


def _rlm_exact(n, g, seed, samples):
    es, cs = [], []
    for build in _rlm_matrices(n, g, seed, samples):
        e, c, prev = np.zeros(n), np.zeros(n), None
        for t1 in range(g + 1):
            w, x = _solve(build, [(t1, t2) for t2 in range(g + 1)])
            e += w.sum(axis=0)
            if prev is not None:
                c += _plaquettes(prev, x).sum(axis=0)
            prev = x
        es.append(e / (g + 1) ** 2)
        cs.append(c + 1.0 / n)
    return np.stack(es), np.stack(cs)


def _hlm_basis(lx, ly, q, band, g, t1, t2):
    """Clean Bloch states of the band as rows [n, sites]."""
    kx, ky = (v.reshape(-1) for v in np.meshgrid(np.arange(lx // q) + t1 / g, np.arange(ly) + t2 / g, indexing="ij"))
    h = np.zeros((kx.size, q, q), dtype=np.complex128)
    for a in range(q):
        h[:, a, a] += -2.0 * np.cos(ky * 2.0 * math.pi / ly + 2.0 * math.pi * a / q)
        if a + 1 < q:
            h[:, a, a + 1] = h[:, a + 1, a] = -1.0
    # (the corner entries close the ring)
    corner = -np.exp(1j * kx * q * 2.0 * math.pi / lx)
    h[:, 0, q - 1], h[:, q - 1, 0] = corner, corner.conj()
    u = np.linalg.eigh(h)[1][:, :, band]
    m, j = np.arange(lx // q) * q, np.arange(ly)
    phase = kx[:, None, None] * (2.0 * math.pi / lx) * m[None, None, :] + ky[:, None, None] * (2.0 * math.pi / ly) * j[None, :, None]
    w = (np.exp(-1j * phase)[..., None] * u[:, None, None, :]).reshape(kx.size, lx * ly)
    return w / np.linalg.norm(w, axis=1, keepdims=True)


def _hlm_exact(case, seed):
    lx, ly, q, band, g = (case[k] for k in ("lx", "ly", "q", "band", "g"))
    n, sites, samples = lx * ly // q, lx * ly, case["samples"]
    pots = _draws(seed, samples * sites).reshape(samples, sites) * (2.0 / 2.0 ** 32) - 1.0
    e, c, prev = np.zeros((samples, n)), np.zeros((samples, n)), None
    for t1 in range(g + 1):
        base = [_hlm_basis(lx, ly, q, band, g, t1, t2) for t2 in range(g)]
        line = np.empty((samples, g + 1, n, sites), dtype=np.complex128)
        for t2, wc in enumerate(base):
            w, u = np.linalg.eigh((wc.conj()[None] * pots[:, None, :]) @ wc.T)
            line[:, t2] = np.swapaxes(u, 1, 2) @ wc
            e += w * (2.0 if t2 == 0 else 1.0)
        line[:, g] = line[:, 0]   # theta_2 = g is the copy of theta_2 = 0
        if prev is not None:
            for s in range(samples):
                c[s] -= _plaquettes(prev[s], line[s]).sum(axis=0)
        prev = line
    return e / (g + 1) ** 2, c


def exact(case, seed):
    kind, g = case["kind"], case["g"]
    small = [mats * n ** 3.0 <= EXACT_MOST and mats <= 20000 for n, mats, _, _, _ in _orders(case)]
    if kind == "fss":
        sizes = [int(v) for v in case["sizes"].split(",")]
        left, out = EXACT_MOST, []
        for n, ok, (_, mats, _, _, _) in zip(sizes, small, _orders(case)):
            ok = ok and mats * n ** 3.0 <= left
            left -= mats * n ** 3.0 if ok else 0.0
            out.append(_rlm_exact(n, g, seed, case["samples"]) if ok else (None, None))
        return out
    if not all(small):
        return None
    if kind == "rlm":
        return _rlm_exact(case["n_phi"], g, seed, case["samples"])
    if kind == "hlm":
        return _hlm_exact(case, seed)
    build = next(_rlm_matrices(case["n_phi"], g, seed, 1))
    w, x = _solve(build, list(zip(*_line_thetas(g))))
    return w, _plaquettes(x[:g + 1], x[g + 1:]).T
