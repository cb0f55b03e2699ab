"""The work a user of this framework has it do, as timed cases.

Kinds of case (``case["kind"]``), each one public call or the short sequence of calls a program makes:

``particle``  one particle and its orientations through the classes of ``bl_dda.scatterer``: DiscreteDipoles,
              set_interaction_matrix (the Green's spectrum), solve_matrix_equation, the observables.  What
              run_dda.py does for every condition.
``bicgstab``  ``bl_krylov.bl_bicgstab_jacobi_mvp_fft`` on resident spectrum, occupancy and right-hand sides.
``cocg``      ``bl_krylov.bl_cocg_rq_jacobi_mvp_fft``, likewise, on general excitations: the bilinear forms of the
              circularly polarised plane waves nearly vanish, and the method often breaks down on them.
``batch``     ``bl_krylov.bl_bicgstab_jacobi_mvp_fft_batch`` over small particles of a sweep.
``product``   ``mvp_fft.fft_mvp`` on the whole cuboid, complex128 or complex64.  The complex64 product is what
              the complex64 and mixed solves spend their time on; their solutions are defined to the
              tolerance only, so the arithmetic is measured here.
``green``     ``mvp_fft.fft_init`` and a first product with it: the cost of a new wavelength or lattice.
``infer``     the learned warm start's network on one particle: features and forward pass.
``train``     one training sample of that network: features, forward, loss, every parameter's gradient.

Solves run to the classes' own default stopping rule (tol 1e-2, itermax 25): X after a few iterations of a block
method is a function of its inputs to rounding.  Particles are smooth deformed ellipsoids inscribed in their
lattice, the lattice spacing a sixteenth of the wavelength in the medium, the refractive indices those of a
slightly birefringent, slightly absorbing silicate grain in water.
"""
import math
import os
import random  # noqa: F401  (draw() takes a random.Random)
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "block-dda_py_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

WL_0, M_M = 1.0, 1.33
M_P = (1.45 + 0.01j, 1.48 + 0.01j, 1.42 + 0.01j)
LF = WL_0 / M_M / 16.0
K = 2.0 * math.pi * M_M / WL_0
TOL, ITERMAX = 1e-2, 25
ITERATIONS = 4              # of a solve to TOL, about: for work()
LAYERS, MODES = 4, 12       # the warm start's shipped network
NET = (13, 32, 6, 64)       # its input channels, width, output channels, projection


def listed():
    return [
        # one small particle, ten orientations: the notebook's example, all launch latency
        dict(name="particle_small", kind="particle", nx=17, ny=17, nz=17, L=10),
        # the size-parameter-5 sphere's lattice with block-COCG-rq
        dict(name="cocg_28", kind="cocg", nx=28, ny=28, nz=28, L=8),
        # one incident direction on a middling particle: no block to hide behind
        dict(name="bicgstab_one_column", kind="bicgstab", nx=52, ny=60, nz=71, L=1),
        # a sweep's ordinary particle with its block of orientations, uneven odd lattice
        dict(name="bicgstab_mid", kind="bicgstab", nx=45, ny=55, nz=83, L=32),
        # the benchmark's size-parameter-20 lattice and block, from host arrays to observables
        dict(name="particle_large", kind="particle", nx=93, ny=112, nz=174, L=64),
        # a sweep's small particles advanced together
        dict(name="batch_sweep", kind="batch", nx=20, ny=25, nz=31, L=16, count=8),
        # products: small, ragged, large
        dict(name="product_c64_small", kind="product", nx=24, ny=20, nz=30, L=4, c64=True),
        dict(name="product_c128_ragged", kind="product", nx=61, ny=47, nz=85, L=11, c64=False),
        dict(name="product_c64_large", kind="product", nx=93, ny=112, nz=174, L=64, c64=True),
        # a new wavelength on a lattice of the sweep
        dict(name="green_mid", kind="green", nx=64, ny=75, nz=105, L=2),
        # the warm start's network: one particle's inference, one training sample
        dict(name="infer_mid", kind="infer", nx=45, ny=55, nz=70, L=16),
        dict(name="train_sample", kind="train", nx=30, ny=36, nz=44, L=16),
    ]


def draw(rng):
    def lattice(lo, hi):   # edges spread over the logarithm, a mean edge first, the aspect of the shapes around it
        e = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        return {a: max(lo, min(hi, round(e * math.exp(rng.uniform(-0.35, 0.35))))) for a in ("nx", "ny", "nz")}

    def columns(n, hi=64):   # a particle of few wavelengths has few independent responses: fewer columns
        hi = min(hi, max(1, int(round((n["nx"] * n["ny"] * n["nz"]) ** (1 / 3) * 0.6))))
        return int(round(math.exp(rng.uniform(0.0, math.log(hi)))))

    kind = rng.choice(["particle", "cocg", "bicgstab", "bicgstab", "batch", "product", "product", "green", "infer",
                       "train"])
    if kind == "batch":
        n = lattice(16, 40)
        return dict(kind=kind, **n, L=rng.choice([8, 16] if min(n.values()) > 20 else [8]), count=rng.randint(3, 12))
    if kind == "product":
        return dict(kind=kind, **(n := lattice(12, 120)), L=int(round(math.exp(rng.uniform(0.0, math.log(64))))),
                    c64=rng.random() < 0.5)
    if kind == "green":
        return dict(kind=kind, **lattice(16, 110), L=rng.randint(1, 4))
    if kind == "infer":
        return dict(kind=kind, **lattice(16, 72), L=rng.randint(4, 20))
    if kind == "train":
        return dict(kind=kind, **lattice(14, 40), L=rng.randint(2, 16))
    if kind == "cocg":   # block-COCG-rq converges on small particles and narrow blocks only
        return dict(kind=kind, **(n := lattice(14, 28)), L=columns(n, 8))
    return dict(kind=kind, **(n := lattice(14, 105)), L=columns(n))


# ---- inputs ----------------------------------------------------------------------------------
def _rng(case, seed):
    return np.random.default_rng([int(seed), case["nx"], case["ny"], case["nz"], case["L"]])


def _shape(n):
    """(occupied mask (cells,), cell centres (cells, 3)) of a deformed ellipsoid inscribed in the lattice."""
    rng = np.random.default_rng(list(n))
    axes = [(np.arange(m) - 0.5 * (m - 1)) * LF for m in n]
    half = [0.5 * m * LF for m in n]
    ph, amp = rng.uniform(0, 2 * np.pi, 3), rng.uniform(0.03, 0.1, 3)
    X, Y, Z = np.meshgrid(*axes, indexing="ij")
    x, y, z = X / half[0], Y / half[1], Z / half[2]
    r2 = x * x + y * y + z * z
    lim = 0.97 - sum(a * (1 + np.sin(3 * c + p)) / 2 for a, c, p in zip(amp, (y, z, x), ph))
    return (r2 <= lim * lim).ravel(), np.stack([X.ravel(), Y.ravel(), Z.ravel()], axis=1)


def _euler(L, rng):
    return np.column_stack([rng.uniform(0, 2 * np.pi, L), np.arccos(rng.uniform(-1, 1, L)),
                            rng.uniform(0, 2 * np.pi, L)])


def _rotation(euler):
    def rz(t):
        c, s, o, i = np.cos(t), np.sin(t), np.zeros_like(t), np.ones_like(t)
        return np.stack([c, -s, o, s, c, o, o, o, i], axis=-1).reshape(-1, 3, 3)

    def ry(t):
        c, s, o, i = np.cos(t), np.sin(t), np.zeros_like(t), np.ones_like(t)
        return np.stack([c, o, s, o, i, o, -s, o, c], axis=-1).reshape(-1, 3, 3)
    return rz(-euler[:, 2]) @ ry(-euler[:, 1]) @ rz(-euler[:, 0])


def _physics(pos, euler):
    """diag_A (3N,), eps_r (3,) and B (3N, L) of the particle, complex128 on the GPU."""
    mp = np.array(M_P, dtype=np.complex128)
    er = mp ** 2 / M_M ** 2
    vol = LF ** 3
    a = np.cbrt(3 * vol / (4 * np.pi))
    mt = (8 * np.pi / 3) * ((1 - 1j * K * a) * np.exp(1j * K * a) - 1)
    cm = 3 / (4 * np.pi) * (er - 1) / (er + 2) * vol
    diag = torch.from_numpy(np.tile((1 - mt * cm / vol) / cm, pos.shape[0])).cuda()
    R = _rotation(euler)
    e0 = (R[:, :, 0] + 1j * R[:, :, 1]) / np.sqrt(2)
    p, u, e = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (pos, R[:, :, 2], e0))
    B = torch.exp(1j * K * (p @ u.T))[:, None, :] * e.T[None]
    return diag, er, B.reshape(3 * pos.shape[0], -1)


def _system(n, L, rng):
    is_in, grid = _shape(n)
    address = np.flatnonzero(is_in)
    euler = _euler(L, rng)
    diag, er, B = _physics(grid[address], euler)
    return dict(n=n, is_in=is_in, grid=grid, address=address, euler=euler, diag=diag, er=er, B=B)


def _excite(s, L, rng):
    """General right-hand sides in the place of the plane waves."""
    B = rng.standard_normal((3 * s["address"].size, L, 2))
    return dict(s, B=torch.from_numpy(B).cuda().view(torch.complex128)[..., 0])


def _lattices(case, rng):
    """The lattices of a sweep's particles: the case's and others up to a fifth smaller."""
    out = []
    for i in range(case["count"]):
        f = 1.0 - 0.2 * i / case["count"]
        out.append(tuple(max(8, int(round(case[a] * f))) for a in ("nx", "ny", "nz")))
    return out


def _dense(case, seed, dtype):
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + case["nx"] * case["nz"] + case["L"])
    rows = 3 * case["nx"] * case["ny"] * case["nz"]
    return torch.randn((rows, case["L"]), dtype=dtype, device="cuda", generator=g)


def _net_shapes():
    cin, w, cout, proj = NET
    out = [(cin, w), (w,)]
    for _ in range(LAYERS):
        out += [(MODES ** 3, w, w, 2), (w, w), (w,)]
    return out + [(w, proj), (proj,), (proj, cout), (cout,)]


def _net_params(seed):
    """Every parameter of the network, flat float32: scaled as for training, the biases small."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 17)
    parts = []
    for s in _net_shapes():
        std = 0.05 if len(s) == 1 else 1.0 / (s[1] * math.sqrt(2.0)) if len(s) == 4 else 1.0 / math.sqrt(s[0])
        parts.append(torch.randn(math.prod(s), device="cuda", generator=g) * std)
    return torch.cat(parts)


def _n(case):
    return (case["nx"], case["ny"], case["nz"])


def prepare(case, seed):
    from bdda_b200 import runtime
    from bl_dda import scatterer
    from mvp_fft import mvp_fft
    kind, n, L, rng = case["kind"], _n(case), case["L"], _rng(case, seed)
    scatterer.DiscreteDipoles.verbose = False

    def occupancy(green, s):
        return runtime.Occupancy(green.plan, s["address"])

    if kind == "particle":
        is_in, grid = _shape(n)
        target = scatterer.Target("ellipsoid", np.array(n), LF, grid, is_in, np.array(M_P))
        return dict(case=case, target=target, field=scatterer.IncidentField(WL_0, M_M, _euler(L, rng)))
    if kind in ("bicgstab", "cocg"):
        s = _system(n, L, rng)
        if kind == "cocg":
            s = _excite(s, L, rng)
        green = mvp_fft.fft_init(n, 3, LF, K)
        return dict(case=case, args=(n, 3, occupancy(green, s), green, s["diag"], s["B"], TOL, ITERMAX))
    if kind == "batch":
        problems = []
        for m in _lattices(case, rng):
            s = _system(m, L, rng)
            green = mvp_fft.fft_init(m, 3, LF, K)
            problems.append((m, occupancy(green, s), green, s["diag"], s["B"]))
        return dict(case=case, problems=problems)
    if kind == "product":
        P = _dense(case, seed, torch.complex64 if case["c64"] else torch.complex128)
        green = mvp_fft.fft_init(n, 3, LF, K)
        green.ghat(runtime.PREC["c64" if case["c64"] else "c128"])
        return dict(case=case, green=green, P=P)
    if kind == "green":
        k = K * float(rng.uniform(0.8, 1.25))
        return dict(case=case, k=k, P=_dense(case, seed, torch.complex128))
    from bdda_b200 import warmstart
    s = _system(n, L, rng)
    plan = runtime.Plan(n)
    model = warmstart.WarmStartFNO(layers=LAYERS, modes=MODES)
    model.params.copy_(_net_params(seed))
    state = dict(case=case, model=model, occ=runtime.Occupancy(plan, s["address"]), diag=s["diag"], B=s["B"],
                 er=s["er"])
    if kind == "train":
        state["X"] = _bicgstab(s)[0]
    return state


def run(state):
    from bl_dda import scatterer
    from bl_krylov import bl_krylov
    from mvp_fft import mvp_fft
    case = state["case"]
    kind, n = case["kind"], _n(case)
    if kind == "particle":
        d = scatterer.DiscreteDipoles(state["target"], state["field"])
        d.set_interaction_matrix()
        d.solve_matrix_equation()
        c_abs, c_ext = d.compute_C_abs(), d.compute_C_ext()
        fw_theta, fw_phi = d.compute_PCAS_observable_S_fw()
        return [c_abs, c_ext, fw_theta, fw_phi, d.compute_OCBS_observable_S_bk(), d.iter_fin, d.err_fin]
    if kind == "bicgstab":
        return bl_krylov.bl_bicgstab_jacobi_mvp_fft(*state["args"])
    if kind == "cocg":
        return bl_krylov.bl_cocg_rq_jacobi_mvp_fft(*state["args"])
    if kind == "batch":
        return bl_krylov.bl_bicgstab_jacobi_mvp_fft_batch(state["problems"], TOL, ITERMAX)
    if kind == "product":
        return mvp_fft.fft_mvp(n, 3, state["green"], state["P"], precision="c64" if case["c64"] else None)
    if kind == "green":
        return mvp_fft.fft_mvp(n, 3, mvp_fft.fft_init(n, 3, LF, state["k"]), state["P"])
    model, L = state["model"], case["L"]
    if kind == "infer":
        work, scale = model.features(n, state["occ"], state["diag"], state["B"], state["er"])
        model.forward(work, L, n)
        return [model.buffer(work, L, n, 1, L * math.prod(n) * NET[2]), scale]
    loss = model.loss_and_grad(n, state["occ"], state["diag"], state["B"], state["er"], state["X"])
    return [loss, model.grads]


# ---- what a pass cannot do without ------------------------------------------------------------
def work(case):
    n, L, kind = _n(case), case["L"], case["kind"]
    cells = math.prod(n)
    occ = 0.45 * cells

    def product(c, columns):   # pruned transforms on the doubled grid, and the 3 x 3 multiply
        a, b, d = c
        lines = a * b * 2 * d * math.log2(2 * d) + a * 2 * d * 2 * b * math.log2(2 * b) \
            + 4 * b * d * 2 * a * math.log2(2 * a)
        return columns * (2 * 5 * 3 * lines + 66 * 8 * a * b * d)

    def green(c):
        return 8 * math.prod(c) * (6 * 5 * math.log2(8 * math.prod(c)) + 60)

    def solve(c, o, products=2, blocks=6):
        vec = 3 * o * L
        return dict(bytes=16.0 * (2 * vec + 3 * o) + 8 * 6 * 16.0 * math.prod(c) * ITERATIONS + 4 * math.prod(c),
                    flops=ITERATIONS * (products * product(c, L) + blocks * 8.0 * vec * L))

    if kind in ("bicgstab", "cocg"):
        return solve(n, occ) if kind == "bicgstab" else solve(n, occ, 1, 9)
    if kind == "particle":
        w = solve(n, occ)
        return dict(bytes=24.0 * occ + 96.0 * L + 33.0 * cells + 8 * 6 * 16.0 * cells * ITERATIONS,
                    flops=w["flops"] + green(n))
    if kind == "batch":
        ws = [solve(c, 0.45 * math.prod(c)) for c in _lattices(case, None)]
        return dict(bytes=sum(w["bytes"] for w in ws), flops=sum(w["flops"] for w in ws))
    if kind == "product":
        cb = 8.0 if case["c64"] else 16.0
        return dict(bytes=cb * (2 * 3 * cells * L + 6 * 8 * cells), flops=product(n, L))
    if kind == "green":
        return dict(bytes=16.0 * (2 * 3 * cells * L + 6 * 8 * cells), flops=green(n) + product(n, L))
    cin, w, cout, proj = NET
    rows, params = cells * L, 4.0 * sum(math.prod(s) for s in _net_shapes())
    spectral = 2 * 2 * 2.0 * MODES * w * rows * (1 + 2.0 * MODES / n[2] + 2.0 * MODES ** 2 / (n[1] * n[2]))
    flops = rows * 2.0 * (cin * w + LAYERS * w * w + w * proj + proj * cout) + LAYERS * spectral \
        + LAYERS * 8.0 * L * MODES ** 3 * w * w
    inputs = 16.0 * 3 * occ * L + 4.0 * cells + params
    if kind == "infer":
        return dict(bytes=inputs + 4.0 * cout * rows, flops=flops)
    return dict(bytes=inputs + 16.0 * 3 * occ * L + params, flops=3.0 * flops)


# ---- the same in 64 bits, plain torch ------------------------------------------------------------
def _green_spectrum(n, k=K):
    """The six unique components' spectrum of A'(r) on the doubled grid."""
    m = [2 * v for v in n]
    d = []
    for N, M in zip(n, m):
        i = torch.arange(M, device="cuda")
        d.append((torch.where(i < N, i, i - M).double() * LF, i != N))
    (X, Y, Z) = torch.meshgrid(*[v for v, _ in d], indexing="ij")
    (a, b, c) = torch.meshgrid(*[v for _, v in d], indexing="ij")
    r = torch.sqrt(X * X + Y * Y + Z * Z)
    ok = a & b & c & (r > 0)
    r = torch.where(ok, r, torch.ones_like(r))
    u = (X / r, Y / r, Z / r)
    g = torch.exp(1j * k * r) / r * ok
    f = (1 - 1j * k * r) / r ** 2
    out = []
    for p, q in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)):
        uu, delta = u[p] * u[q], 1.0 if p == q else 0.0
        out.append(torch.fft.fftn(g * (k * k * (uu - delta) + f * (delta - 3 * uu))))
    return out


def _apply(G, n, P):
    """The dense product, columns in turn: (3 cells, L) -> (3 cells, L)."""
    m = tuple(2 * v for v in n)
    out = torch.empty_like(P)
    step = max(1, min(P.shape[1], int(2e8 // (3 * math.prod(m)))))
    for c in range(0, P.shape[1], step):
        f = torch.fft.fftn(P[:, c:c + step].T.reshape(-1, *n, 3).movedim(-1, 0), s=m, dim=(2, 3, 4))
        y = [G[0] * f[0] + G[1] * f[1] + G[2] * f[2], G[1] * f[0] + G[3] * f[1] + G[4] * f[2],
             G[2] * f[0] + G[4] * f[1] + G[5] * f[2]]
        del f
        for a in range(3):
            v = torch.fft.ifftn(y[a], dim=(1, 2, 3))[:, :n[0], :n[1], :n[2]]
            out[a::3, c:c + step] = v.reshape(v.shape[0], -1).T
    return out


def _operator(s):
    """M^-1 A of the particle, and M^-1."""
    G, j = _green_spectrum(s["n"]), 1.0 / s["diag"][:, None]
    rows = (3 * torch.from_numpy(s["address"]).cuda()[:, None] + torch.arange(3, device="cuda")).reshape(-1)

    def product(v):
        full = torch.zeros((3 * math.prod(s["n"]), v.shape[1]), dtype=v.dtype, device=v.device)
        full[rows] = v
        return v + j * _apply(G, s["n"], full)[rows]
    return product, j


def _bicgstab(s):
    A, j = _operator(s)
    R = s["B"] * j
    bnorm = torch.linalg.norm(R)
    X, P, R0, it, err = torch.zeros_like(R), R, R, 0, math.inf
    for it in range(ITERMAX):
        V = A(P)
        RV = R0.conj().T @ V
        alpha = torch.linalg.solve(RV, R0.conj().T @ R)
        T = R - V @ alpha
        Z = A(T)
        zeta = (Z.conj() * T).sum() / (Z.conj() * Z).sum()
        X = X + P @ alpha + zeta * T
        R = T - zeta * Z
        err = float(torch.linalg.norm(R) / bnorm)
        if err < TOL:
            break
        P = R + (P - zeta * V) @ torch.linalg.solve(RV, -(R0.conj().T @ Z))
    return X, it, err


def _cocg(s):
    A, j = _operator(s)
    W = s["B"] * j
    bnorm = torch.linalg.norm(W)
    Q, xi = torch.linalg.qr(W)
    X, S, it, err = torch.zeros_like(W), Q, 0, math.inf
    for it in range(ITERMAX):
        AS = A(S)
        alpha = torch.linalg.solve(S.T @ AS, Q.T @ Q)
        X = X + S @ (alpha @ xi)
        Qn, tau = torch.linalg.qr(Q - AS @ alpha)
        xi = tau @ xi
        err = float(torch.linalg.norm(xi) / bnorm)
        if err < TOL:
            break
        S = Qn + S @ torch.linalg.solve(Q.T @ Q, tau.T @ (Qn.T @ Qn))
        Q = Qn
    return X, it, err


def _observables(s, X):
    L, vol = X.shape[1], LF ** 3
    P = X.reshape(-1, 3, L)
    pos = torch.from_numpy(s["grid"][s["address"]]).cuda()
    R = torch.from_numpy(_rotation(s["euler"])).cuda()
    er = torch.from_numpy(s["er"]).cuda()[None, :, None]
    E = 4 * math.pi * P / ((er - 1) * vol)
    c_abs = 4 * math.pi * K * (P * E.conj()).imag.sum((0, 1))
    c_ext = 4 * math.pi * K * (P * s["B"].reshape(-1, 3, L).conj()).imag.sum((0, 1))

    def far(u, theta, phi):
        e = math.sqrt(2.0) * torch.exp(1j * K * (pos @ u.T))
        t, p = torch.einsum("ncl,lc->nl", P, theta + 0j), torch.einsum("ncl,lc->nl", P, phi + 0j)
        return K * K * (t * e.conj()).sum(0), K * K * (p * (1j * e).conj()).sum(0)
    fw = far(R[:, :, 2], R[:, :, 0], R[:, :, 1])
    bk = far(-R[:, :, 2], -R[:, :, 0], R[:, :, 1])
    return [v.cpu().numpy() for v in (c_abs, c_ext, fw[0], fw[1], (bk[1] - bk[0]) / math.sqrt(2.0))]


def _network(s, L, params):
    """(features (L, cells, cin), scale, J (3N, L), output (L, cells, cout)) in float64; params a flat float64 array."""
    n, cells = s["n"], math.prod(s["n"])
    cin, w, cout, proj = NET
    p, off = [], 0
    for shape in _net_shapes():
        p.append(params[off:off + math.prod(shape)].reshape(shape))
        off += math.prod(shape)
    J = s["B"] / s["diag"][:, None]
    scale = torch.sqrt((J.abs() ** 2).mean(0))
    x = torch.zeros((L, cells, cin), dtype=torch.float64, device="cuda")
    at = torch.from_numpy(s["address"]).cuda()
    chi = torch.from_numpy((s["er"] - 1) / (s["er"] + 2)).cuda()
    x[:, at, 0] = 1.0
    x[:, at, 1:7] = torch.view_as_real(chi).reshape(-1)
    x[:, at, 7:13] = torch.view_as_real((J / scale).reshape(-1, 3, L).permute(2, 0, 1).contiguous()).reshape(L, -1, 6)
    F = []
    for N in n:
        f = torch.cat([torch.arange(MODES // 2), torch.arange(N - MODES // 2, N)]).double()
        F.append(torch.exp(-2j * math.pi * torch.outer(torch.arange(N).double(), f) / N).cuda())
    v = (x @ p[0] + p[1]).reshape(L, *n, w)
    for l in range(LAYERS):
        Rl, Wl, bl = p[2 + 3 * l:5 + 3 * l]
        A = torch.einsum("bxyzc,zk->bxykc", v + 0j, F[2])
        A = torch.einsum("bxjkc,xi->bijkc", torch.einsum("bxykc,yj->bxjkc", A, F[1]), F[0])
        S = torch.einsum("bki,kio->bko", A.reshape(L, -1, w), torch.view_as_complex(Rl)).reshape(A.shape)
        S = torch.einsum("bijkc,xi->bxjkc", S, F[0].conj())
        S = torch.einsum("bxykc,zk->bxyzc", torch.einsum("bxjkc,yj->bxykc", S, F[1].conj()), F[2].conj())
        z = v @ Wl + bl + S.real / cells
        v = torch.nn.functional.gelu(z) if l + 1 < LAYERS else z
    h = torch.nn.functional.gelu(v.reshape(L, cells, w) @ p[-4] + p[-3])
    return scale, J, h @ p[-2] + p[-1]


def exact(case, seed):
    kind, n, L, rng = case["kind"], _n(case), case["L"], _rng(case, seed)
    if kind == "product":
        P = _dense(case, seed, torch.complex64 if case["c64"] else torch.complex128).to(torch.complex128)
        return _apply(_green_spectrum(n), n, P)
    if kind == "green":
        k = K * float(rng.uniform(0.8, 1.25))
        return _apply(_green_spectrum(n, k), n, _dense(case, seed, torch.complex128))
    if kind == "batch":
        return [_bicgstab(_system(m, L, rng)) for m in _lattices(case, rng)]
    s = _system(n, L, rng)
    if kind == "bicgstab":
        return _bicgstab(s)
    if kind == "cocg":
        return _cocg(_excite(s, L, rng))
    if kind == "particle":
        if math.prod(n) * L > 6e7:   # over twenty seconds
            return None
        X, it, err = _bicgstab(s)
        return _observables(s, X) + [it, err]
    params = _net_params(seed).double()
    if kind == "infer":
        with torch.no_grad():
            scale, _, y = _network(s, L, params)
        return [y.reshape(-1), scale]
    params.requires_grad_(True)
    scale, J, y = _network(s, L, params)
    X = _bicgstab(s)[0]
    at = torch.from_numpy(s["address"]).cuda()
    t = torch.view_as_real(((X - J) / scale).reshape(-1, 3, L).permute(2, 0, 1).contiguous()).reshape(L, -1, 6)
    loss = (((y[:, at] - t) ** 2).sum((1, 2)) / (t ** 2).sum((1, 2))).mean()
    loss.backward()
    return [float(loss), params.grad]
