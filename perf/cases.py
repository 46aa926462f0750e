"""Workloads of the density-matrix library, timed through its public entry points.

Each case is one call (or the few calls) that a program built on this library
makes over and over: density evaluations in both precisions, a relaxation
step, whole self-consistent solves, the stochastic DOS and density of the
reference's runs, SP2 purification, a batch of uneven structures, and the two
directions of the learned starting charges.  The cells are the repository's
own (beta-cristobalite SiO2 with seeded Gaussian displacements; the
reference's alpha-quartz slabs).

The C-ABI takes and returns host arrays, so prepare() holds host arrays and a
context (the handle that a program keeps), and run() is the whole call.  The
ABI returns every result as a double; the results of the FP32 form are given
back here in the type in which they were computed, float32.
"""
import numpy as np
import torch

import largetb_gb300 as T
from largetb_gb300 import learned

BOHR = learned.BOHR_PER_ANG
EDGE = 7.16  # angstrom, the conventional cristobalite cell


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest whole solve: the reference's own 36-atom quartz slab,
        # run in FP64 by the small-structure rule; latency and launches count
        dict(name="scc_quartz_36", kind="scc", lattice="quartz", nx=2, ny=2, nz=1, M=120, start="neutral"),
        # the plain FP64 method on its 192-atom configuration
        dict(name="density64_192", kind="density", lattice="cristobalite", nx=2, ny=2, nz=2, M=200, fp64=True,
             sigma=0.05),
        # the same form on an ordinary, ragged cell (1152 atoms)
        dict(name="density64_1152", kind="density", lattice="cristobalite", nx=4, ny=4, nz=3, M=300, fp64=True,
             sigma=0.05),
        # one step of a relaxation or of molecular dynamics: new positions,
        # H and Gamma built from them, one FP32 density (864 atoms)
        dict(name="relax_864", kind="relax", nx=3, ny=3, nz=4, M=200, sigma=0.05),
        # the headline cell's density evaluation (5184 atoms, order 400)
        dict(name="density32_5184", kind="density", lattice="cristobalite", nx=6, ny=6, nz=6, M=400, fp64=False,
             sigma=0.05),
        # a whole learned-start solve in the FP32 form on a middle cell (1440 atoms)
        dict(name="scc_learned_1440", kind="scc", lattice="cristobalite", nx=5, ny=4, nz=3, M=300, start="learned",
             sigma=0.08),
        # the DOS of the reference's logged 4608-atom run: 500 vectors, 1000 moments
        dict(name="dos_quartz_4608", kind="dos", nx=8, ny=8, nz=8, moments=1000, vectors=500, points=2000),
        # the reference's default density on its long slabs: 20 vectors (27000 atoms)
        dict(name="stochastic_quartz_27000", kind="stochastic", nx=10, ny=10, nz=30, M=200, moments=1000, vectors=20,
             points=2000),
        # SP2 purification of the 1536-atom cell, FP32 blocks, drop 1e-5
        dict(name="sp2_1536", kind="sp2", nx=4, ny=4, nz=4, sigma=0.08),
        # a batch of uneven cells, every side in {2, 3, 4}, solved together
        dict(name="batch_10_uneven", kind="batch", count=10, M=300, pick=7),
        # learned starting charges of the 12288-atom cell: features and prediction
        dict(name="charges_12288", kind="charges", nx=8, ny=8, nz=8, sigma=0.08),
        # forward and backward of the charge network over many samples
        dict(name="mlp_grad_65536", kind="grad", samples=65536),
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread evenly over its logarithm."""
    return int(min(hi, max(lo, round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    """A further case of the listed ranges."""
    kind = rng.choice(["scc", "density64", "density32", "relax", "learned", "dos", "stochastic", "sp2", "batch",
                       "charges", "grad"])
    sig = rng.choice([0.02, 0.05, 0.08, 0.12])
    side = lambda lo, hi: rng.randint(lo, hi)  # noqa: E731
    order = lambda lo, hi: _log(rng, lo, hi)  # noqa: E731
    if kind == "scc":
        return dict(kind="scc", lattice="quartz", nx=side(1, 4), ny=side(1, 4), nz=side(1, 2), M=order(80, 200),
                    start="neutral")
    if kind == "density64":
        return dict(kind="density", lattice=rng.choice(["cristobalite", "cristobalite", "quartz"]), nx=side(1, 4),
                    ny=side(1, 4), nz=side(1, 4), M=order(60, 300), fp64=True, sigma=sig)
    if kind == "density32":
        return dict(kind="density", lattice="cristobalite", nx=side(3, 6), ny=side(3, 6), nz=side(2, 6),
                    M=order(100, 400), fp64=False, sigma=sig)
    if kind == "relax":
        return dict(kind="relax", nx=side(2, 4), ny=side(2, 5), nz=side(2, 4), M=order(100, 300), sigma=sig)
    if kind == "learned":
        return dict(kind="scc", lattice="cristobalite", nx=side(3, 4), ny=side(3, 5), nz=side(2, 4),
                    M=order(150, 300), start="learned", sigma=sig)
    if kind == "dos":
        return dict(kind="dos", nx=side(2, 8), ny=side(2, 8), nz=side(2, 8), moments=order(200, 1000),
                    vectors=order(10, 500), points=2000)
    if kind == "stochastic":
        return dict(kind="stochastic", nx=side(3, 10), ny=side(3, 10), nz=side(4, 30), M=order(100, 200),
                    moments=order(300, 1000), vectors=order(8, 40), points=2000)
    if kind == "sp2":
        return dict(kind="sp2", nx=side(2, 4), ny=side(2, 4), nz=side(2, 4), sigma=rng.choice([0.05, 0.08]))
    if kind == "batch":
        return dict(kind="batch", count=side(2, 10), M=order(100, 300), pick=rng.randint(0, 999))
    if kind == "charges":
        return dict(kind="charges", nx=side(2, 8), ny=side(2, 8), nz=side(2, 8), sigma=sig)
    return dict(kind="grad", samples=_log(rng, 500, 131072))


# ---------------------------------------------------------------------------
# what a program has in hand
# ---------------------------------------------------------------------------
def _plus_u(m):
    """+U on the diagonal of the reference's quartz Gamma (with -U its SCC runs away)."""
    rows = np.repeat(np.arange(m.natoms), np.diff(m.g_rowptr))
    m.g_vals = np.where(rows == m.g_colidx, np.abs(m.g_vals), m.g_vals)
    return m


def _model(case, seed):
    """The case's cell.  The quartz slab is a fixed lattice: its seed goes into
    a small diagonal disorder of H (a few meV, as strain would give)."""
    if case.get("lattice", "cristobalite") == "cristobalite":
        return T.model_cristobalite(case["nx"], case["ny"], case["nz"], sigma_ang=case["sigma"], seed=seed + 1)
    m = _plus_u(T.model_quartz(case["nx"], case["ny"], case["nz"]))
    rows = np.repeat(np.arange(m.n), np.diff(m.rowptr))
    on = np.random.default_rng(seed).normal(0.0, 2e-4, m.n)
    m.vals = m.vals + np.where(rows == m.colidx, on[rows], 0.0)
    return m


def _box(case):
    return learned.cell_box((case["nx"], case["ny"], case["nz"]))


def _batch_cells(case, seed):
    r = np.random.default_rng(case["pick"])
    return [(tuple(int(v) for v in r.integers(2, 5, 3)), float(r.uniform(0.02, 0.12)), 1000 * (seed + 1) + i)
            for i in range(case["count"])]


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "density":
        m = _model(case, seed)
        s["ctx"] = T.Context(M=case["M"], precision=T.PREC_FP64 if case["fp64"] else T.PREC_FP32)
        s["ctx"].set_model(m)
    elif kind == "relax":
        m = _model(case, seed)
        s.update(xyz=m.xyz, species=m.species, box=_box(case))
        s["ctx"] = T.Context(M=case["M"], precision=T.PREC_FP32)
    elif kind == "scc":
        m = _model(case, seed)
        # the learned start is nearer to the fixed point and mixes best with its own step;
        # a short history where the slab has few atoms (as in the tests of these slabs)
        mix = dict(mix_beta=learned.MIX_BETA) if case["start"] == "learned" else dict(mix_history=4)
        s["ctx"] = T.Context(M=case["M"], precision=T.PREC_FP32, **mix)
        s["ctx"].set_model(m)
        if case["start"] == "learned":
            s.update(model=m, box=_box(case), mlp=learned.load())
    elif kind in ("dos", "stochastic"):
        m = _model(dict(case, lattice="quartz"), seed)
        s["seed"] = seed + 17
        s["ctx"] = T.Context(M=case.get("M", 200), kT=0.0)
        s["ctx"].set_model(m)
    elif kind == "sp2":
        m = _model(case, seed)
        s["ctx"] = T.Context(precision=T.PREC_FP32)
        s["ctx"].set_model(m)
    elif kind == "batch":
        ms = [T.model_cristobalite(*d, sigma_ang=sg, seed=sd) for d, sg, sd in _batch_cells(case, seed)]
        s["batch"] = T.Batch(ms, M=case["M"])
    elif kind == "charges":
        m = _model(case, seed)
        s.update(xyz=m.xyz, species=m.species, box=_box(case), mlp=learned.load())
    else:
        s["feat"], s["target"] = _samples(case, seed)
        s["mlp"] = learned.load()
    return s


def _samples(case, seed):
    """Features of distorted cells (non-negative, a few tenths, many near zero)
    and net charges around those of SiO2."""
    r = np.random.default_rng(seed)
    n = case["samples"]
    feat = (r.gamma(0.6, 0.6, (n, T.api.MLP_NFEAT)) * (r.random((n, T.api.MLP_NFEAT)) < 0.8)).astype(np.float32)
    target = np.where(r.random(n) < 1 / 3, -1.1, 0.55) + r.normal(0, 0.1, n)
    return feat, target.astype(np.float32)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _f32(r, *keys):
    return {k: np.asarray(r[k], np.float32) for k in keys}


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "density":
        r = s["ctx"].density()
        keys = ("diagP", "q", "moments", "e_band", "mu")
        return {k: np.asarray(r[k]) for k in keys} if case["fp64"] else _f32(r, *keys)
    if kind == "relax":
        s["ctx"].set_geometry(s["xyz"], s["species"], s["box"])
        return _f32(s["ctx"].density(), "diagP", "q", "moments", "e_band", "mu")
    if kind == "scc":
        q0 = learned.warm_start(s["mlp"], s["model"], s["box"]) if case["start"] == "learned" else None
        return _f32(s["ctx"].scc_solve(q0), "q", "diagP", "e_band", "mu")
    if kind == "dos":
        r = s["ctx"].kpm_dos(n_moments=case["moments"], n_random=case["vectors"], seed=s["seed"],
                             npts=case["points"])
        return {k: r[k] for k in ("moments", "energies", "dos")}
    if kind == "stochastic":
        r = s["ctx"].density_stochastic(n_probes=case["vectors"], seed=s["seed"], dos_moments=case["moments"],
                                        dos_points=case["points"])
        return {k: np.asarray(r[k]) for k in ("diagP", "q", "mu")}
    if kind == "sp2":
        return _f32(s["ctx"].sp2(), "diagP", "q", "e_band")
    if kind == "batch":
        r = s["batch"].scc_solve()
        return dict(q=np.concatenate(r["q"]).astype(np.float32), **_f32(r, "e_band", "mu"))
    if kind == "charges":
        feat = T.mlp_features(s["xyz"], s["species"], s["box"])
        return dict(feat=feat, charge=s["mlp"].predict(feat))
    g, loss = s["mlp"].grad(s["feat"], s["target"])
    return dict(grad=g, loss=loss)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
_SCC_ITERS = 20  # density evaluations of an ordinary solve


def _blocks(case):
    """(atoms, stored 4x4 blocks): Si has four neighbours, O two."""
    per = 24 if case.get("lattice", "cristobalite") == "cristobalite" else 9
    na = per * case["nx"] * case["ny"] * case["nz"]
    return na, 11 * na // 3


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = [dict(kind="scc", start="neutral", nx=d[0], ny=d[1], nz=d[2], M=case["M"])
                 for d, _, _ in _batch_cells(case, 0)]
        ws = [work(c) for c in parts]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    if kind == "grad":
        n, p = case["samples"], T.api.MLP_NPARAM
        return dict(bytes=4.0 * (33 * n + 2 * p), flops=6.0 * n * p)
    if kind == "charges":
        na, _ = _blocks(case)
        return dict(bytes=na * (28.0 + 128 + 4), flops=na * (80.0 * 32 * 20 + 2 * T.api.MLP_NPARAM))
    if kind in ("dos", "stochastic"):
        na, nnzb = _blocks(dict(case, lattice="quartz"))
        n, nv = 4 * na, case["vectors"]
        # moments up to 2k from T_k; the density's T_k x need every order
        steps = case["moments"] / 2 + (case["M"] if kind == "stochastic" else 0)
        return dict(bytes=132.0 * nnzb + 8.0 * (n + 3 * case["points"]), flops=steps * nv * (32.0 * nnzb + 4 * n))
    na, nnzb = _blocks(case)
    n = 4 * na
    if kind == "sp2":
        # each of ~25 steps squares a matrix of ~300 blocks a row, its upper half
        return dict(bytes=132.0 * nnzb + 8.0 * n, flops=25 * 64.0 * na * min(na, 300) * min(na, 150))
    evals = _SCC_ITERS if kind == "scc" else 1
    # moments up to order 2k from T_k on all n unit vectors, and two dot products a column
    flops = evals * (case["M"] / 2) * n * (32.0 * nnzb + 4 * n)
    return dict(bytes=132.0 * nnzb + 8.0 * (2 * n + case["M"]), flops=flops)


# ---------------------------------------------------------------------------
# the same results in 64 bits, in plain torch and numpy
# ---------------------------------------------------------------------------
def _sparse(m, a, b):
    """X = (H - b)/a as a CSR tensor on the GPU, H symmetrised, and H's Gershgorin bounds if a is None."""
    rows = np.repeat(np.arange(m.n), np.diff(m.rowptr))
    i = torch.tensor(np.stack([np.concatenate([rows, m.colidx]), np.concatenate([m.colidx, rows])]), device="cuda")
    v = torch.tensor(np.concatenate([m.vals, m.vals]) / 2, device="cuda")
    h = torch.sparse_coo_tensor(i, v, (m.n, m.n)).coalesce()
    (r, c), v = h.indices(), h.values()
    if a is None:
        dg = torch.zeros(m.n, dtype=torch.float64, device="cuda").index_add_(0, r[r == c], v[r == c])
        rad = torch.zeros_like(dg).index_add_(0, r[r != c], v[r != c].abs())
        lo, hi = float((dg - rad).min()), float((dg + rad).max())
        a, b = (hi - lo) / 2, (hi + lo) / 2
    k = torch.arange(m.n, device="cuda")
    x = torch.sparse_coo_tensor(torch.cat([h.indices(), torch.stack([k, k])], 1),
                                torch.cat([v, torch.full((m.n,), -b, dtype=torch.float64, device="cuda")]) / a,
                                (m.n, m.n)).coalesce()
    return x.to_sparse_csr(), a, b


def _jackson(N):
    k = np.arange(N)
    t = np.pi / (N + 1)
    g = ((N - k + 1) * np.cos(t * k) + np.sin(t * k) / np.tan(t)) / (N + 1)
    g[0] = 1.0
    return g


def _diag_moments(x, M):
    """d[k][i] = T_k(X)_ii for k = 0..M."""
    n = x.shape[0]
    d = torch.empty(M + 1, n, dtype=torch.float64, device="cuda")
    xd = torch.zeros(n, dtype=torch.float64, device="cuda")
    coo = x.to_sparse_coo().coalesce()
    (r, c), v = coo.indices(), coo.values()
    xd.index_add_(0, r[r == c], v[r == c])
    for c0 in range(0, n, 2048):
        cols = torch.arange(c0, min(n, c0 + 2048), device="cuda")
        t0 = torch.zeros(n, len(cols), dtype=torch.float64, device="cuda")
        t0[cols, cols - c0] = 1.0
        t1 = x @ t0
        for k in range((M + 2) // 2):
            if 2 * k <= M:
                d[2 * k, cols] = 2 * (t0 * t0).sum(0) - 1
            if 2 * k + 1 <= M:
                d[2 * k + 1, cols] = 2 * (t0 * t1).sum(0) - xd[cols]
            t0, t1 = t1, 2 * (x @ t1) - t0
    return d.cpu().numpy()


def _coeffs(mu_x, beta, M):
    if beta <= 0:
        th, k = np.arccos(mu_x), np.arange(1, M)
        return np.concatenate([[1 - th / np.pi], -2 * np.sin(k * th) / (k * np.pi)])
    nq = 1 << int(np.ceil(np.log2(max(4 * M, 13 * beta, 256))))
    th = np.pi * (np.arange(nq) + 0.5) / nq
    f = 0.5 * (1 - np.tanh(0.5 * beta * (np.cos(th) - mu_x)))
    c = 2 * (np.cos(np.outer(np.arange(M), th)) @ f) / nq
    c[0] /= 2
    return c


def _density(m, M, kT=0.01, shift=None):
    if shift is not None:
        rows = np.repeat(np.arange(m.n), np.diff(m.rowptr))
        vals, m.vals = m.vals, m.vals + np.where(rows == m.colidx, shift[rows], 0.0)
    x, a, b = _sparse(m, None, None)
    if shift is not None:
        m.vals = vals
    d = _diag_moments(x, M)
    mom, g, ne = d.sum(1), _jackson(M), m.n_electrons
    lo, hi = -1.0, 1.0
    for _ in range(60):
        mid = (lo + hi) / 2
        lo, hi = (mid, hi) if 2 * (_coeffs(mid, a / kT, M) * g) @ mom[:M] < ne else (lo, mid)
    mu = (lo + hi) / 2
    w = _coeffs(mu, a / kT, M) * g
    p = w @ d[:M]
    tx = np.concatenate([[mom[1]], 0.5 * (mom[2:M + 1] + mom[:M - 1])])
    return dict(diagP=p, q=2 * p.reshape(-1, 4).sum(1), moments=mom, e_band=np.float64(2 * w @ (a * tx + b * mom[:M])),
                mu=np.float64(a * mu + b))


def _scc(m, M):
    """The fixed point of the charges by Anderson mixing on densities in 64 bits."""
    gam = np.zeros((m.natoms, m.natoms))
    gam[np.repeat(np.arange(m.natoms), np.diff(m.g_rowptr)), m.g_colidx] = m.g_vals
    q, hist = m.q0.copy(), []
    for _ in range(60):
        r = _density(m, M, shift=np.repeat(gam @ (q - m.q0), 4))
        res = r["q"] - q
        if np.abs(res).max() < 1e-10:
            break
        hist = (hist + [(q, res)])[-5:]
        dq = np.array([q - h[0] for h in hist[:-1]]).reshape(-1, m.natoms)
        dr = np.array([res - h[1] for h in hist[:-1]]).reshape(-1, m.natoms)
        c = np.linalg.lstsq(dr.T, res, rcond=1e-10)[0] if len(dr) else np.zeros(0)
        q = q - c @ dq + 0.2 * (res - c @ dr)
    return {k: r[k] for k in ("q", "diagP", "e_band", "mu")}


def _probes(n, nv, seed):
    """The library's counter-based Gaussian stream (splitmix64, Box-Muller): deviate t n + i is entry i of vector t."""
    def mix(k):
        z = np.uint64(seed) + (k + np.uint64(1)) * np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return (z ^ (z >> np.uint64(31))) >> np.uint64(11)
    with np.errstate(over="ignore"):
        k = np.uint64(2) * np.arange(n * nv, dtype=np.uint64)
        u1 = (mix(k).astype(np.float64) + 1) / 2.0 ** 53
        u2 = mix(k + np.uint64(1)).astype(np.float64) / 2.0 ** 53
    return torch.tensor((np.sqrt(-2 * np.log(u1)) * np.cos(2 * np.pi * u2)).reshape(nv, n).T.copy(), device="cuda")


def _dos(m, nmom, nv, seed, npts):
    x, a, b = _sparse(m, None, None)
    r = _probes(m.n, nv, seed)
    mom, t0, t1 = np.zeros(nmom), r, x @ r
    for k in range((nmom + 1) // 2):  # r.T_2k r = 2 |T_k r|^2 - |r|^2, and the odd orders likewise
        mom[2 * k] = 2 * float((t0 * t0).sum()) - (mom[0] if k else float((r * r).sum()))
        if 2 * k + 1 < nmom:
            mom[2 * k + 1] = 2 * float((t0 * t1).sum()) - (mom[1] if k else float((r * t1).sum()))
        t0, t1 = t1, 2 * (x @ t1) - t0
    th = np.pi * (np.arange(npts) + 0.5) / npts
    wk = _jackson(nmom) * mom
    wk[1:] *= 2
    rho = (np.cos(np.outer(th, np.arange(nmom))) @ wk) / (np.pi * np.sin(th))
    return dict(moments=mom, energies=a * np.cos(th) + b, dos=rho)


def _stochastic(m, case, seed):
    npts, M = case["points"], case["M"]
    s = _dos(m, case["moments"], case["vectors"], seed, npts)
    e, dos = s["energies"], s["dos"]
    xq = np.cos(np.pi * (np.arange(npts) + 0.5) / npts)
    area = ((xq[:-1] - xq[1:]) * (dos[1:] + dos[:-1]) / 2)[::-1]  # from the bottom of the spectrum
    cum = np.cumsum(area)
    mi = npts - 1 - int(np.argmax(cum >= m.n_electrons * area.sum() / (2 * m.n)))
    on = np.nonzero(dos / m.n >= 0.001)[0]
    emin = e[on[-1]] if on.size and on[-1] > 0 else -10.0
    emax = e[on[0]] if on.size else 10.0
    a, b = (emax - emin) / 2, (emax + emin) / 2
    w = _coeffs((e[mi] - b) / a, 0.0, M) * _jackson(M)
    x = _sparse(m, a, b)[0]
    r = _probes(m.n, case["vectors"], seed + 1)
    t0, t1 = r, x @ r
    p = w[0] * (r * t0).sum(1)
    for k in range(1, M):
        p += w[k] * (r * t1).sum(1)
        t0, t1 = t1, 2 * (x @ t1) - t0
    p = (p / (r * r).sum(1)).cpu().numpy()
    return dict(diagP=p, q=2 * p.reshape(-1, 4).sum(1), mu=np.float64(e[mi]))


def _projector(m):
    """Zero-temperature density matrix by purification of the dense matrix, nothing dropped."""
    x, a, b = _sparse(m, None, None)
    h = x.to_dense() * a + b * torch.eye(m.n, dtype=torch.float64, device="cuda")
    p = (0.5 * (torch.eye(m.n, dtype=torch.float64, device="cuda") - x.to_dense()))
    best = np.inf
    for _ in range(60):
        p2 = p @ p
        err = float((p2 - p).square().sum().sqrt())
        if err < 1e-10 or (err < 1e-6 and err >= best):
            break
        best = err
        p = p2 if 2 * float(torch.trace(p)) > m.n_electrons else 2 * p - p2
    dg = torch.diagonal(p).cpu().numpy()
    return dict(diagP=dg, q=2 * dg.reshape(-1, 4).sum(1), e_band=np.float64(2 * float((p * h).sum())))


def _features(m, box):
    x, bx = torch.tensor(m.xyz, device="cuda"), torch.tensor(box, device="cuda")
    si = torch.tensor(m.species == 14, device="cuda")
    mu = 0.8 + 0.28 * torch.arange(16, dtype=torch.float64, device="cuda")
    f = torch.zeros(m.natoms, 32, dtype=torch.float64, device="cuda")
    for a0 in range(0, m.natoms, 1024):
        d = x[None] - x[a0:a0 + 1024, None]
        d -= bx * torch.round(d / bx)
        r = d.square().sum(-1).sqrt() / BOHR
        i, j = torch.nonzero((r < 5.0) & (r > 0), as_tuple=True)
        rij = r[i, j]
        v = torch.exp(-12.5 * (rij[:, None] - mu).square()) * (0.5 * (torch.cos(np.pi * rij / 5) + 1))[:, None]
        for first, sel in ((0, si[j]), (16, ~si[j])):
            f[:, first:first + 16].index_add_(0, i[sel] + a0, v[sel])
    return f


def _network(mlp):
    p, nrm = mlp.get()
    w = torch.tensor(p).bfloat16().double().cuda().requires_grad_()
    nrm = torch.tensor(nrm, dtype=torch.float64, device="cuda")
    parts = torch.split(w, [2048, 64, 4096, 64, 64, 1])

    def f(feat):
        h = torch.nn.functional.silu((feat - nrm[:32]) * nrm[32:] @ parts[0].view(64, 32).T + parts[1])
        h = torch.nn.functional.silu(h @ parts[2].view(64, 64).T + parts[3])
        return h @ parts[4] + parts[5]
    return w, f


def exact(case, seed):
    kind = case["kind"]
    if kind == "density":
        return _density(_model(case, seed), case["M"])
    if kind == "relax":
        return _density(_model(case, seed), case["M"])
    if kind == "scc":
        # dozens of density evaluations: within seconds only for the small slabs
        return _scc(_model(case, seed), case["M"]) if case["start"] == "neutral" else None
    if kind == "dos":
        return _dos(_model(dict(case, lattice="quartz"), seed), case["moments"], case["vectors"], seed + 17,
                    case["points"])
    if kind == "stochastic":
        return _stochastic(_model(dict(case, lattice="quartz"), seed), case, seed + 17)
    if kind == "sp2":
        return _projector(_model(case, seed))
    if kind == "batch":
        return None  # hundreds of density evaluations
    w, f = _network(learned.load())
    if kind == "charges":
        feat = _features(_model(case, seed), _box(case))
        with torch.no_grad():
            return dict(feat=feat, charge=f(feat))
    feat, target = (torch.tensor(v, dtype=torch.float64, device="cuda") for v in _samples(case, seed))
    loss = (f(feat) - target).square().mean()
    loss.backward()
    return dict(grad=w.grad, loss=loss.detach())
