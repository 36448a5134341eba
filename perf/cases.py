"""The work that programs built on this package have it do, as measurable cases.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare``/``run`` do the work through the public entry points and ``exact``
computes the same outputs in plain FP64 torch without the package's kernels.
Geometry is the reference's two-plate patch antenna; a seed moves every
dimension, the band and (for the network) the data by a few percent.

Kinds of case:

* ``call``      one ``patch_sweep_fastquad_cuda`` call from host arrays, the
                drop-in use (geometry upload, set-up, sweep, release);
* ``plan``      ``SweepPlan.run`` on resident geometry, repeated sweeps;
* ``extract``   the same with the analytic-extraction scheme of the design family;
* ``family``    ``sweep_family``: several designs meshed, planned and swept in flight;
* ``assemble``  ``ggassemble_ZV_EFIE_RWG_DIFF_GPU_FAST``: Z and V to the host;
* ``centroid``  ``patch_sweep_cuda``: the one-point assembly's sweep;
* ``train``     the surrogate network: a few epochs and a prediction.
"""
import importlib
import math

import numpy as np
import torch

PKG = "matlab-cuda-efief-vs-cpu_b200"
m = importlib.import_module(PKG)
sur = importlib.import_module(PKG + ".surrogate")

MU0 = 4.0 * math.pi * 1e-7
C0 = 299792458.0
EPS0 = 1.0 / (MU0 * C0 * C0)
# the reference's two option sets (its GPU drivers' and its accurate one)
OPTS = {
    "gpu": dict(quad_order=2, near_sing_eps=1.2, self_subdiv=2, self_alpha=0.20, near_subdiv=1, near_alpha=0.15,
                near_order=2),
    "accurate": dict(quad_order=4, near_sing_eps=2.5, self_subdiv=2, self_alpha=0.20, near_subdiv=2, near_alpha=0.15,
                     near_order=4),
}

# Patch cells (px, py) over ground cells (gx, gy); lengths in mm, band in GHz.
_BENCH = dict(Lp=30.0, Wp=38.0, G=60.0, h=1.6, feed=-7.0, f0=2.0, f1=3.0, er=1.0, tand=0.0, opts="gpu", order="grid",
              spacing="even")
# the reference's own sweep: 20.1 mm patch over a 0.2 m ground, er 2.59, 538 unknowns, its vertex order
_REF = dict(Lp=20.1, Wp=20.1, G=200.0, h=1.59, feed=3.15, f0=1.0, f1=1.4, er=2.59, tand=1e-4, opts="gpu",
            order="reference", spacing="even", px=8, py=6, gx=12, gy=12)
# one design of the benchmark's family (patch pitch 1.5 mm, ground pitch 3 mm)
_DESIGN = dict(W=35.0, L=30.0, h=1.6, feed=-6.0, pitch=1.5, gpitch=3.0)


def listed():
    return [
        # one frequency of the reference's own design in one call: the smallest use, all latency
        dict(_REF, name="call_ref_1", kind="call", nf=1),
        # the reference's published run: its design, 41 points, one call
        dict(_REF, name="call_ref_41", kind="call", nf=41),
        # the benchmark's small configuration on resident geometry
        dict(_BENCH, name="plan_1k_11", kind="plan", px=12, py=10, gx=16, gy=16, nf=11, dev=False),
        # a lossy substrate, the accurate option set and a logarithmic frequency list
        dict(_BENCH, name="call_1k_lossy_21", kind="call", px=12, py=10, gx=16, gy=16, nf=21, er=4.4, tand=0.02,
             f0=1.0, f1=2.0, opts="accurate", spacing="log"),
        # a handful of unsorted points on a mid-size design, prepack made on the GPU: an adaptive sweep's round
        dict(_BENCH, name="plan_4k_8", kind="plan", px=25, py=19, gx=31, gy=30, nf=8, dev=True, spacing="random"),
        # the headline: a dense sweep of a 7k-unknown design on resident geometry
        dict(_BENCH, name="plan_7k_101", kind="plan", px=32, py=24, gx=40, gy=40, nf=101, dev=False),
        # a large design, a few points, one call
        dict(_BENCH, name="call_20k_8", kind="call", px=80, py=64, gx=40, gy=40, nf=8, Lp=32.0, Wp=40.0, G=90.0),
        # a dense sweep of one family design with the analytic extraction (7-point rule)
        dict(_DESIGN, name="extract_2k_41", kind="extract", nf=41),
        # designs of uneven size in flight together, from dimensions to Zin
        dict(name="family_4x41", kind="family", n=4, nf=41, pitch=1.5, gpitch=3.0, workers=3),
        # assembly only, Z and V brought to the host
        dict(_BENCH, name="assemble_3k", kind="assemble", px=21, py=17, gx=27, gy=26, nf=1),
        # the one-point entry point's sweep
        dict(_BENCH, name="centroid_1k_21", kind="centroid", px=12, py=10, gx=16, gy=16, nf=21),
        # training of the surrogate on solver samples, and its prediction of a dense band
        dict(name="train_20k", kind="train", rows=20000, hidden=256, layers=4, batch=1024, epochs=3, query=801),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["call", "call", "plan", "plan", "plan", "extract", "family", "assemble", "centroid", "train"])
    if kind == "train":
        return dict(kind=kind, rows=log(2000, 20000), hidden=rng.choice([64, 128, 256]), layers=rng.randint(2, 4),
                    batch=rng.choice([256, 512, 1024]), epochs=rng.randint(1, 3), query=log(100, 800))
    if kind == "family":
        return dict(kind=kind, n=rng.randint(2, 5), nf=log(8, 41), pitch=rng.choice([1.5, 2.0, 2.5]),
                    gpitch=rng.choice([3.0, 4.0, 5.0]), workers=rng.randint(2, 3))
    if kind == "extract":
        return dict(_DESIGN, kind=kind, nf=log(5, 60), W=rng.uniform(25, 45), L=rng.uniform(20, 40),
                    h=rng.uniform(0.8, 3.2), feed=rng.uniform(-6, 6), pitch=rng.uniform(1.5, 2.5),
                    gpitch=rng.uniform(3.0, 5.0))
    top = {"call": 7000, "plan": 7000, "assemble": 3500, "centroid": 2000}[kind]
    ne = log(500, top)
    # unknowns are about three per cell; a bit over half of the cells lie on the ground
    cells = ne / 3.0
    gx = max(4, int(round(math.sqrt(0.62 * cells) * rng.uniform(0.9, 1.1))))
    gy = max(4, int(round(0.62 * cells / gx)))
    px = max(3, int(round(math.sqrt(0.38 * cells) * rng.uniform(0.95, 1.25))))
    py = max(3, int(round(0.38 * cells / px)))
    nf = 1 if kind == "assemble" else log(1, 101) if ne < 3000 else log(1, 48)
    c = dict(_BENCH, kind=kind, px=px, py=py, gx=gx, gy=gy, nf=nf)
    if kind in ("call", "plan") and rng.random() < 0.3:
        c.update(er=rng.uniform(2.0, 4.5), tand=rng.choice([0.0, 1e-4, 0.02]), f0=1.2, f1=2.0)
    if kind in ("call", "plan") and ne < 1500 and rng.random() < 0.3:
        c.update(opts="accurate")
    if kind != "assemble":
        c.update(spacing=rng.choice(["even", "even", "log", "random"]))
    if kind == "plan":
        c.update(dev=rng.random() < 0.5)
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _dims(c, seed):
    r = np.random.default_rng(seed)
    s = 1.0 + 0.02 * r.uniform(-1, 1, 6)
    d = dict(Lp=c["Lp"] * s[0] * 1e-3, Wp=c["Wp"] * s[1] * 1e-3, Lg=c["G"] * s[2] * 1e-3, Wg=c["G"] * s[3] * 1e-3,
             h=c["h"] * s[4] * 1e-3, feed=(0.0, c["feed"] * s[5] * 1e-3))
    if c["order"] == "reference":
        d["feed"] = (-0.5 * d["Wp"] + 1e-3, c["feed"] * s[5] * 1e-3)
    a, b = c["f0"] * 1e9 * (1 + 0.01 * r.uniform(-1, 1)), c["f1"] * 1e9 * (1 + 0.01 * r.uniform(-1, 1))
    n = c["nf"]
    if c["spacing"] == "log":
        f = np.geomspace(a, b, n) if n > 1 else np.array([a])
    elif c["spacing"] == "random":
        f = r.uniform(a, b, n)
    else:
        f = np.linspace(a, b, n) if n > 1 else np.array([0.5 * (a + b)])
    er = c["er"]
    eps = EPS0 * er * (1 - 1j * c["tand"])   # the medium around the plates
    return d, f, (eps if c["tand"] else eps.real)


def _family(c, seed):
    one = sur.sample_designs(c["n"], seed=seed, pitch=c["pitch"] * 1e-3, ground_pitch=c["gpitch"] * 1e-3)
    return one


def _design(c, seed):
    s = 1.0 + 0.02 * np.random.default_rng(seed).uniform(-1, 1, 4)
    return sur.PatchDesign(c["W"] * s[0] * 1e-3, c["L"] * s[1] * 1e-3, c["h"] * s[2] * 1e-3, c["feed"] * s[3] * 1e-3,
                           c["pitch"] * 1e-3, c["gpitch"] * 1e-3)


def _train_data(c, seed):
    r = np.random.default_rng(seed)
    X = r.uniform(-1, 1, (c["rows"], 5)).astype(np.float32)
    # a resonance curve over the band, as the solver's samples show
    q = X[:, 4] - 0.3 * X[:, 1] + 0.1 * X[:, 2]
    z = (0.3 + 1.5 / (0.15 + 1j * (q - 0.1 * X[:, 3]))).astype(np.complex128)
    return X, sur.zin_to_target(50.0 * z), r.uniform(-1, 1, (c["query"], 5)).astype(np.float32)


def prepare(case, seed):
    c, k = case, case["kind"]
    if k == "train":
        X, T, Q = _train_data(c, seed)
        net = sur.Surrogate(n_hidden=c["hidden"], n_layers=c["layers"], seed=1 + seed % 1000)
        return dict(k=k, c=c, net=net, p0=net.get_params(), X=X, T=T, Q=Q)
    if k == "family":
        return dict(k=k, c=c, designs=_family(c, seed))
    if k == "extract":
        d = _design(c, seed)
        return dict(k=k, plan=sur.design_plan(d, nfreq=c["nf"]), freqs=d.band(c["nf"]))
    d, f, eps = _dims(c, seed)
    V, F, _, _ = m.make_patch_with_ground_mesh(d["Lp"], d["Wp"], d["Lg"], d["Wg"], d["h"], c["px"], c["py"], c["gx"],
                                               c["gy"], vertex_order=c["order"])
    r = m.build_rwg_interior({"V": V, "F": F})
    pe = m.pick_port_edge_by_point_and_layer(r, (*d["feed"], +d["h"] / 2), +1)
    ge = m.pick_port_edge_by_point_and_layer(r, (*d["feed"], -d["h"] / 2), -1)
    mesh = [V, F, r["edge"], r["plusTri"], r["minusTri"], r["plusSign"], r["minusSign"], r["rp"], r["rm"], r["Ap"],
            r["Am"], r["len"]]
    spread = 1.5 * float(np.mean(r["len"]))
    tail = [MU0, eps, pe, ge, 1.0, spread, 50.0]
    if k == "centroid":
        return dict(k=k, args=mesh + [f] + tail)
    if k == "plan":
        dev = c["dev"]
        pre = None if dev else m.efie_precompute_pack({"V": V, "F": F}, OPTS[c["opts"]], gpu=True)
        plan = m.SweepPlan(*mesh, pre, *tail, opts=m.sweep_opts(nfreq_hint=c["nf"]),
                           precompute=OPTS[c["opts"]] if dev else None)
        return dict(k=k, plan=plan, freqs=f)
    pre = m.efie_precompute_pack({"V": V, "F": F}, OPTS[c["opts"]], gpu=True)
    if k == "assemble":
        w = 2.0 * math.pi * f[0]
        return dict(k=k, args=mesh + [pre, w * np.sqrt(complex(MU0) * eps), w, MU0, eps,
                                      np.array([pe, ge, 1.0, spread])])
    return dict(k=k, args=mesh + [pre, f] + tail)


def run(s):
    k = s["k"]
    if k == "call":
        Zin, S11 = m.patch_sweep_fastquad_cuda(*s["args"])
    elif k == "centroid":
        Zin, S11 = m.patch_sweep_cuda(*s["args"])
    elif k == "assemble":
        Z, V = m.ggassemble_ZV_EFIE_RWG_DIFF_GPU_FAST(*s["args"])
        return dict(Z=Z, V=V)
    elif k == "family":
        return dict(Zin=[z for _, z in sur.sweep_family(s["designs"], s["c"]["nf"], workers=s["c"]["workers"])])
    elif k == "train":
        c, net = s["c"], s["net"]
        net.set_params(s["p0"])
        hist = net.train(s["X"], s["T"], epochs=c["epochs"], batch=c["batch"], seed=3)
        return dict(loss=hist, params=net.get_params(), pred=net.forward(s["Q"]))
    else:
        Zin, S11 = s["plan"].run(s["freqs"])
    return dict(Zin=Zin, S11=S11)


# ---------------------------------------------------------------------------
# Work
# ---------------------------------------------------------------------------
def _edges(px, py, gx, gy):
    return sum(3 * a * b - a - b for a, b in ((px, py), (gx, gy))), 2 * (px * py + gx * gy)


def _sweep_work(ne, nt, nf, nq):
    """Geometry in, Zin and S11 out; per frequency a complex point-pair
    evaluation (about 40 operations) for every regular pair of the symmetric
    matrix and one complex factorization of it (4/3 N^3)."""
    return dict(bytes=nt * nq * 32.0 + ne * 150.0 + nf * 40.0,
                flops=nf * (20.0 * nq * nq * nt * nt + 4.0 / 3.0 * float(ne) ** 3))


def work(case):
    c, k = case, case["kind"]
    if k == "train":
        h, l = c["hidden"], c["layers"]
        w = 5 * h + (l - 1) * h * h + 3 * h
        return dict(bytes=32.0 * c["rows"] + 24.0 * w, flops=6.0 * w * c["rows"] * c["epochs"] + 2.0 * w * c["query"])
    if k in ("extract", "family"):
        n = c.get("n", 1)
        W, L = (c["W"], c["L"]) if k == "extract" else (35.0, 30.0)
        G = 1.6 * max(W, L)
        ne, nt = _edges(W / c["pitch"], L / c["pitch"], G / c["gpitch"], G / c["gpitch"])
        w = _sweep_work(ne, nt, c["nf"], 7)
        return {x: n * y for x, y in w.items()}
    ne, nt = _edges(c["px"], c["py"], c["gx"], c["gy"])
    nq = 3 if c["opts"] == "gpu" else 6
    if k == "assemble":
        return dict(bytes=16.0 * ne * ne + nt * nt + 150.0 * ne, flops=20.0 * nq * nq * nt * nt)
    return _sweep_work(ne, nt, c["nf"], 1 if k == "centroid" else nq)


# ---------------------------------------------------------------------------
# The same outputs in FP64 torch, from the dimensions on
# ---------------------------------------------------------------------------
_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _plate(W, L, z, nx, ny, offset, order):
    def lin(a, b, n):
        y = a + (np.arange(n + 1, dtype=np.float64) * (b - a)) / n
        y[0], y[-1] = a, b
        return y

    X, Y = np.meshgrid(lin(-W / 2, W / 2, nx), lin(-L / 2, L / 2, ny))
    o = "F" if order == "reference" else "C"   # the reference numbers vertices y-fastest
    V = np.stack([X.flatten(o), Y.flatten(o), np.full(X.size, z)], axis=1)
    j, i = np.meshgrid(np.arange(ny), np.arange(nx), indexing="ij")
    v1 = (offset + j * (nx + 1) + i).reshape(-1)
    v2, v3, v4 = v1 + 1, v1 + nx + 1, v1 + nx + 2
    return V, np.stack([v1, v2, v4, v1, v4, v3], axis=1).reshape(-1, 3)


def _mesh(d, px, py, gx, gy, order):
    Vp, Fp = _plate(d["Wp"], d["Lp"], +d["h"] / 2, px, py, 0, order)
    Vg, Fg = _plate(d["Wg"], d["Lg"], -d["h"] / 2, gx, gy, len(Vp), order)
    return np.vstack([Vp, Vg]), np.vstack([Fp, Fg])


def _rwg(V, F):
    """Interior edges in (lower, higher vertex) order; sides in triangle order."""
    nt = len(F)
    a, b = F.reshape(-1), F[:, [1, 2, 0]].reshape(-1)
    tri = np.repeat(np.arange(nt), 3)
    lo, hi = np.minimum(a, b), np.maximum(a, b)
    o = np.lexsort((np.arange(a.size), hi, lo))
    same = (lo[o][1:] == lo[o][:-1]) & (hi[o][1:] == hi[o][:-1])
    i = np.nonzero(same)[0]
    r = [o[i], o[i + 1]]
    ea, eb = lo[r[0]], hi[r[0]]
    c, free, t = [], [], []
    ln = np.sqrt(((V[eb] - V[ea]) ** 2).sum(1))
    for s, x in enumerate(r):
        tv = F[tri[x]]
        opp = tv.sum(1) - ea - eb
        A = 0.5 * np.linalg.norm(np.cross(V[tv[:, 1]] - V[tv[:, 0]], V[tv[:, 2]] - V[tv[:, 0]]), axis=1)
        sg = np.where(a[x] == ea, 1.0, -1.0)
        c.append((sg if s == 0 else -sg) * ln / (2.0 * A))
        free.append(V[opp])
        t.append(tri[x])
    return dict(ea=ea, eb=eb, center=0.5 * (V[ea] + V[eb]), len=ln, tri=t, c=c, free=free)


def _norm(v):
    return np.sqrt(v[..., 0] * v[..., 0] + v[..., 1] * v[..., 1] + v[..., 2] * v[..., 2])


def _port(r, p, up):
    c = r["center"]
    zmid = 0.5 * (c[:, 2].max() + c[:, 2].min())
    i = np.nonzero((c[:, 2] > zmid) == up)[0]
    return int(i[np.argmin(_norm(c[i] - np.asarray(p)))])


def _weights(r, e, spread):
    c = r["center"]
    zmid = 0.5 * (c[:, 2].max() + c[:, 2].min())
    w = np.exp(-(_norm(c - c[e]) / spread) ** 2) * ((c[:, 2] > zmid) == (c[e, 2] > zmid))
    return w / w.sum()


def _rule(n):
    """Points (u, v) and weights (sum 1/2) of the 1-, 3-, 6- and Dunavant's 7-point rule."""
    if n == 1:
        return np.array([[1 / 3, 1 / 3]]), np.array([0.5])
    if n == 3:
        return np.array([[1 / 6, 1 / 6], [2 / 3, 1 / 6], [1 / 6, 2 / 3]]), np.ones(3) / 6
    if n == 6:
        a, b, w1, w2 = 0.445948490915965, 0.108103018168070, 0.111690794839005, 0.054975871827661
        q = [[a, a], [a, 1 - 2 * a], [1 - 2 * a, a], [b, b], [b, 1 - 2 * b], [1 - 2 * b, b]]
        return np.array(q), np.array([w1] * 3 + [w2] * 3)
    s = math.sqrt(15.0)
    a, b = (6 - s) / 21, (6 + s) / 21
    q = [[1 / 3, 1 / 3], [a, a], [1 - 2 * a, a], [a, 1 - 2 * a], [b, b], [1 - 2 * b, b], [b, 1 - 2 * b]]
    return np.array(q), 0.5 * np.array([9 / 40] + [(155 - s) / 1200] * 3 + [(155 + s) / 1200] * 3)


def _points(T, rule, depth=0):
    """Rule points [Nt, 4^depth, Q, 3] and weights of the subdivided triangles T [Nt, 3, 3]."""
    S = T[:, None]
    for _ in range(depth):
        A, B, C = S[:, :, 0], S[:, :, 1], S[:, :, 2]
        AB, BC, CA = 0.5 * (A + B), 0.5 * (B + C), 0.5 * (C + A)
        S = np.stack([np.stack(x, 2) for x in ((A, AB, CA), (AB, B, BC), (CA, BC, C), (AB, BC, CA))], 2)
        S = S.reshape(len(T), -1, 3, 3)
    q, w = rule
    e1, e2 = S[:, :, 1] - S[:, :, 0], S[:, :, 2] - S[:, :, 0]
    a2 = np.linalg.norm(np.cross(e1, e2), axis=-1)
    P = S[:, :, None, 0] + q[None, None, :, 0, None] * e1[:, :, None] + q[None, None, :, 1, None] * e2[:, :, None]
    return P, w[None, None, :] * a2[:, :, None], a2


def _t(x):
    return torch.as_tensor(np.ascontiguousarray(x), device=_DEV)


def _sums(p1, w1, p2, w2, off, green):
    """S0, S1, S2, S3 of point pairs (coordinates about each triangle's centroid)."""
    d = (off[:, None] + p1)[:, :, None] - p2[:, None]
    G = green((d * d).sum(-1)) * (w1[:, :, None] * w2[:, None])
    t0, t1 = G.sum(2), G.sum(1)
    c1, c2 = p1.to(G.dtype), p2.to(G.dtype)
    S1 = (t0[..., None] * c1).sum(1)
    S2 = (t1[..., None] * c2).sum(1)
    S3 = ((G[..., None] * c2[:, None]).sum(2) * c1).sum((1, 2))
    return torch.cat([t0.sum(1)[:, None], S1, S2, S3[:, None]], 1)


def _potential(v, r):
    """int 1/R and int (r' - r)/R over the triangles v [P, 3, 3] seen from r [P, Q, 3]
    (Wilton et al. 1984, Graglia 1993)."""
    n = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    n = (n / torch.linalg.norm(n, dim=-1, keepdim=True))[:, None]
    d = ((r - v[:, None, 0]) * n).sum(-1)
    rho = r - d[..., None] * n
    I, J, ad = torch.zeros_like(d), torch.zeros_like(r), d.abs()
    for i in range(3):
        p, q = v[:, None, i], v[:, None, (i + 1) % 3]
        l = (q - p) / torch.linalg.norm(q - p, dim=-1, keepdim=True)
        u = torch.linalg.cross(l, n)
        P0, lp, lm = ((p - rho) * u).sum(-1), ((q - rho) * l).sum(-1), ((p - rho) * l).sum(-1)
        R0 = P0 * P0 + d * d
        Rp, Rm = (R0 + lp * lp).sqrt(), (R0 + lm * lm).sqrt()
        on = R0 < 1e-30 * (lp * lp + lm * lm)
        num = torch.where(lp >= 0, Rp + lp, R0 / (Rp - lp))
        den = torch.where(lm >= 0, Rm + lm, R0 / (Rm - lm))
        f = torch.where(on, torch.zeros_like(d), (num / den).log())
        beta = torch.where(ad > 0, torch.atan(P0 * lp / (R0 + ad * Rp)) - torch.atan(P0 * lm / (R0 + ad * Rm)),
                           torch.zeros_like(d))
        I = I + P0 * f - ad * beta
        J = J + u * (0.5 * (R0 * f + lp * Rp - lm * Rm))[..., None]
    return I, J - (d * I)[..., None] * n


class _Problem:
    """Geometry, pair lists and edges on the device; z(k, omega, mu, eps) assembles Z."""

    def __init__(self, V, F, scheme, opts=None):
        T = V[F]
        r = _rwg(V, F)
        o = T.mean(1)
        nt = len(F)
        self.r, self.nt, self.scheme, self.o = r, nt, scheme, _t(o)
        loc = lambda P: _t((P - o[:, None, None]).reshape(nt, -1, 3))  # noqa: E731
        area2 = np.linalg.norm(np.cross(T[:, 1] - T[:, 0], T[:, 2] - T[:, 0]), axis=1)
        if scheme == "ref":
            nq = {1: 1, 2: 3}
            P, w, _ = _points(T, _rule(nq.get(opts["quad_order"], 6)))
            near = _rule(nq.get(opts["near_order"], 6))
            Pn, wn, _ = _points(T, near, opts["near_subdiv"])
            Ps, ws, a2 = _points(T, near, opts["self_subdiv"])
            self.near, self.self_ = (loc(Pn), _t(wn.reshape(nt, -1))), (loc(Ps), _t(ws.reshape(nt, -1)))
            h = np.sqrt(2.0 * area2 / math.sqrt(3.0))
            D = _norm(o[:, None] - o[None])
            a, b = np.nonzero(D < opts["near_sing_eps"] * 0.5 * (h[:, None] + h[None]))
            self.pairs = _t(np.stack([a, b], 1)[a < b])
            aeq = opts["near_alpha"] * np.sqrt(0.5 * area2 / math.pi)
            self.soft = _t(aeq)
            sub = np.repeat(np.arange(a2.shape[1]), len(near[1]))
            self.same = _t((sub[:, None] == sub[None]).astype(np.float64))
            self.aS2 = _t((opts["self_alpha"] ** 2 * 0.5 * a2 / math.pi)[:, sub])
        elif scheme == "centroid":
            P, w, _ = _points(T, _rule(1))
            self.soft = _t(0.04 * 0.5 * area2 / math.pi)   # selfAlpha 0.20
        else:
            P, w, _ = _points(T, _rule(7))
            self.vtx = _t(T - o[:, None])
            inc = np.zeros((nt, len(V)), np.float32)
            inc[np.arange(nt)[:, None], F] = 1
            inc = _t(inc)
            self.pairs = torch.nonzero(torch.triu(inc @ inc.T > 0))
        self.reg = (loc(P), _t(w.reshape(nt, -1)))
        self.tri = [_t(x.astype(np.int64)) for x in r["tri"]]
        self.c = [_t(x) for x in r["c"]]
        self.d = [_t(f - o[x]) for f, x in zip(r["free"], r["tri"])]

    def _set(self, S, a, b, v):
        S[a, b] = v
        S[b, a] = torch.cat([v[:, :1], v[:, 4:7], v[:, 1:4], v[:, 7:]], 1)

    def z(self, k, omega, mu, eps):
        kc = complex(k)

        def green(R2):
            R = R2.sqrt().clamp_min(1e-15)
            return torch.exp(-1j * kc * R) / (4.0 * math.pi * R)

        def smooth(R2):
            R = R2.sqrt()
            x = torch.where(R > 0, R, torch.ones_like(R))
            em = torch.expm1(kc.imag * x)
            g = torch.complex(em * torch.cos(kc.real * x) - 2 * torch.sin(0.5 * kc.real * x) ** 2,
                              -(1 + em) * torch.sin(kc.real * x)) / (4 * math.pi * x)
            return torch.where(R > 0, g, torch.full_like(g, -1j * kc / (4 * math.pi)))

        nt, (P, w), o = self.nt, self.reg, self.o
        q = P.shape[1]
        S = torch.empty(nt, nt, 8, dtype=torch.complex128, device=_DEV)
        step = max(1, int(3e7 / (nt * q * q)))
        for i in range(0, nt, step):
            n = min(step, nt - i)
            a = torch.arange(i, i + n, device=_DEV).repeat_interleave(nt)
            b = torch.arange(nt, device=_DEV).repeat(n)
            S[i:i + n] = _sums(P[a], w[a], P[b], w[b], o[a] - o[b], green).reshape(n, nt, 8)
        own = torch.arange(nt, device=_DEV)
        if self.scheme == "centroid":
            S[own, own] = _sums(P, w, P, w, 0 * o, lambda R2: green(R2 + self.soft[:, None, None]))
        elif self.scheme == "ref":
            (Pn, wn), (Ps, ws) = self.near, self.self_
            step = max(1, int(3e7 / Pn.shape[1] ** 2))
            for i in range(0, len(self.pairs), step):
                a, b = self.pairs[i:i + step].T
                s2 = torch.minimum(self.soft[a], self.soft[b]) ** 2
                self._set(S, a, b, _sums(Pn[a], wn[a], Pn[b], wn[b], o[a] - o[b],
                                         lambda R2: green(R2 + s2[:, None, None])))
            step = max(1, int(3e7 / Ps.shape[1] ** 2))
            for i in range(0, nt, step):
                x = own[i:i + step]
                s2 = self.aS2[x][:, :, None] * self.same
                S[x, x] = _sums(Ps[x], ws[x], Ps[x], ws[x], 0 * o[x], lambda R2: green(R2 + s2))
        else:
            step = 100000
            for i in range(0, len(self.pairs), step):
                a, b = self.pairs[i:i + step].T
                v = _sums(P[a], w[a], P[b], w[b], o[a] - o[b], smooth)
                r = P[a] + (o[a] - o[b])[:, None]
                I, J = _potential(self.vtx[b], r)
                Sp = J + r * I[..., None]
                wa = w[a] / (4 * math.pi)
                st = torch.cat([(wa * I).sum(1)[:, None], ((wa * I)[..., None] * P[a]).sum(1),
                                (wa[..., None] * Sp).sum(1), (wa * (P[a] * Sp).sum(-1)).sum(1)[:, None]], 1)
                v = v + st
                mean = 0.5 * (v[:, 1:4] + v[:, 4:7])
                eq = (a == b)[:, None]
                v = torch.cat([v[:, :1], torch.where(eq, mean, v[:, 1:4]), torch.where(eq, mean, v[:, 4:7]), v[:, 7:]],
                              1)
                self._set(S, a, b, v)
        al, be = 1j * omega * mu, 1.0 / (1j * omega * complex(eps))
        Z = 0
        for a in range(2):
            da = self.d[a].to(S.dtype)
            for b in range(2):
                db = self.d[b].to(S.dtype)
                M = S[self.tri[a]][:, self.tri[b]]
                v = M[..., 7] - (M[..., 1:4] * db[None]).sum(-1) - (M[..., 4:7] * da[:, None]).sum(-1)
                v = v + (da @ db.T) * M[..., 0]
                Z = Z + (al * v + 4 * be * M[..., 0]) * (self.c[a][:, None] * self.c[b][None])
        return Z


def _solve(p, freqs, eps, feed, h, edge_port=False):
    r = p.r
    pe, ge = _port(r, (*feed, +h / 2), True), _port(r, (*feed, -h / 2), False)
    spread = 1.5 * float(np.mean(r["len"]))
    wP, wG = _weights(r, pe, spread), _weights(r, ge, spread)
    rhs = _t(0.5 * wP - 0.5 * wG).to(torch.complex128)
    port = np.zeros(len(wP))
    if edge_port:
        port[pe] += 1.0
        port[ge] -= 1.0
    else:
        port = (wP - wG) * r["len"]
    port = _t(port).to(torch.complex128)
    out = []
    for f in freqs:
        w = 2.0 * math.pi * f
        Z = p.z(w * np.sqrt(complex(MU0) * eps), w, MU0, eps)
        out.append((port * torch.linalg.solve(Z, rhs)).sum())
        del Z
    Zin = 1.0 / torch.stack(out).cpu().numpy()
    return Zin, (Zin - 50.0) / (Zin + 50.0)


def _exact_design(d, nf):
    px, py, gx, gy = d.cells()
    G = d.ground_factor * max(d.W, d.L)
    V, F = _mesh(dict(Wp=d.W, Lp=d.L, Wg=G, Lg=G, h=d.h), px, py, gx, gy, "grid")
    return _solve(_Problem(V, F, "extract"), d.band(nf), EPS0, (0.0, d.feed), d.h)


def exact(case, seed):
    c, k = case, case["kind"]
    if k == "train":
        return None   # a training run in 16-bit weights has no 64-bit counterpart
    if k == "extract":
        Zin, S11 = _exact_design(_design(c, seed), c["nf"])
        return dict(Zin=Zin, S11=S11)
    if k == "family":
        return dict(Zin=[_exact_design(d, c["nf"])[0] for d in _family(c, seed)])
    ne, nt = _edges(c["px"], c["py"], c["gx"], c["gy"])
    if ne > 4500 or c["nf"] * (float(ne) ** 3 * 2e-12 + nt * nt * (2e-8 if c["opts"] == "gpu" else 2e-7)) > 10:
        return None   # over about 20 seconds
    d, f, eps = _dims(c, seed)
    V, F = _mesh(d, c["px"], c["py"], c["gx"], c["gy"], c["order"])
    p = _Problem(V, F, "centroid" if k == "centroid" else "ref", OPTS[c["opts"]])
    if k == "assemble":
        w = 2.0 * math.pi * f[0]
        Z = p.z(w * np.sqrt(complex(MU0) * eps), w, MU0, eps)
        # the signs of an interior edge's two sides come with the edge: same basis, same matrix
        pe, ge = _port(p.r, (*d["feed"], +d["h"] / 2), True), _port(p.r, (*d["feed"], -d["h"] / 2), False)
        spread = 1.5 * float(np.mean(p.r["len"]))
        V = 0.5 * _weights(p.r, pe, spread) - 0.5 * _weights(p.r, ge, spread)
        return dict(Z=Z.cpu().numpy(), V=V.astype(np.complex128))
    Zin, S11 = _solve(p, f, eps, d["feed"], d["h"], k == "centroid")
    return dict(Zin=Zin, S11=S11)
