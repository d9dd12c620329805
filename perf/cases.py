"""Performance cases of the solver's main path: advancing curvilinear blocks in time.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same
ranges, ``prepare`` makes the inputs and the resident block, ``run`` is one pass
through the public calls, ``work`` the bytes and operations the pass cannot do
without, and ``exact`` the pass in plain FP64 torch for the schemes restated
below.

A pass is what a host program does between two exchanges with the solver: hand
over a state, run some time steps, take the result back.  Blocks of ordinary
size use the streaming calls with pinned host arrays (as the benchmark's
end-to-end loop), the small block, the block set and the single right-hand side
the blocking calls.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from chimera_comp_les_b200 import Block
from chimera_comp_les_b200 import batch as B
from chimera_comp_les_b200 import workloads as W

GAMMA = 1.4
CUDA = "cuda:0"

# the benchmark's option sets: MUSCL + Rusanov with Smagorinsky (RK2), the
# WENO3 / 4-point central blend (RK3), WENO5-JS + Roe (RK3), the inviscid
# WENO5-JS + Rusanov vortex, and the dynamic model on the blend
SCHEMES = {
    "muscl": dict(les=1, fluxorder=2, s=0.0, ren=1600.0, ma=0.1, pr=0.71),
    "blend": dict(les=1, fluxorder=3, s=0.5, ren=1600.0, ma=0.1, pr=0.71),
    "central": dict(les=1, fluxorder=3, s=1.0, ren=1600.0, ma=0.1, pr=0.71),
    "weno5_roe": dict(les=1, fluxorder=3, weno_order=5, flux="roe", s=0.0, ren=10000.0, ma=0.4, pr=0.71,
                      cs_const=0.17 ** 2),
    "vortex": dict(les=0, inviscid=1, fluxorder=3, weno_order=5, s=0.0, ren=1600.0, ma=0.1, pr=0.71),
    "dynamic": dict(les=2, fluxorder=3, s=1.0, ren=1600.0, ma=0.1, pr=0.71, max_cs=0.1),
    "sphere": dict(les=1, fluxorder=3, weno_order=5, flux="roe", s=0.0, ren=300.0, ma=0.3, pr=0.71, cs_const=0.01),
    "channel": dict(les=1, fluxorder=3, s=1.0, ren=3000.0, ma=0.5, pr=0.71, calc_sigma=1, isothermal=1),
}
# operations per interior node and stage, counted on a C restatement of the
# schemes (additions, multiplications, divisions and square roots)
FLOPS = {"muscl": 2250, "blend": 2996, "central": 2050, "weno5_roe": 4669, "vortex": 2575, "dynamic": 4426,
         "sphere": 4669, "channel": 2996}


def listed():
    """The cases; sizes are unique points per direction (DMDA nodes of the sphere)."""
    return [
        # a coarse block advanced step by step by a host program: launches and latency
        dict(name="tgv_32_fp64", kind="small", scheme="muscl", nx=32, ny=32, nz=32, precision="fp64", steps=20),
        # the benchmark's headline block in both forms
        dict(name="tgv_128_mixed", kind="block", scheme="muscl", nx=128, ny=128, nz=128, precision="mixed", steps=20),
        dict(name="tgv_128_fp64", kind="block", scheme="muscl", nx=128, ny=128, nz=128, precision="fp64", steps=10),
        # the reference's hybrid scheme with both fluxes on every face, a ragged block
        dict(name="blend_97x75x61_fp64", kind="block", scheme="blend", nx=97, ny=75, nz=61, precision="fp64", steps=10),
        # isotropic turbulence with WENO5-JS + Roe: the size sweep's scheme, both forms
        dict(name="turbulence_192_mixed", kind="block", scheme="weno5_roe", nx=192, ny=192, nz=192, precision="mixed",
             steps=10),
        dict(name="turbulence_96_fp64", kind="block", scheme="weno5_roe", nx=96, ny=96, nz=96, precision="fp64",
             steps=5),
        # inviscid vortex advection
        dict(name="vortex_64_fp64", kind="block", scheme="vortex", nx=64, ny=64, nz=64, precision="fp64", steps=10),
        # flow past a sphere: immersed boundary, slip sides, inflow and outflow
        dict(name="sphere_96x96x128_mixed", kind="sphere", scheme="sphere", nx=96, ny=96, nz=128, precision="mixed",
             steps=5),
        # uneven blocks advanced together, halos from a donor permutation
        dict(name="blocks_8_mixed", kind="blocks", scheme="blend", nx=112, ny=88, nz=64, blocks=8, precision="mixed",
             steps=20),
        # dynamic Smagorinsky model on the central scheme
        dict(name="dynamic_96x80x72_fp64", kind="block", scheme="dynamic", nx=96, ny=80, nz=72, precision="fp64",
             steps=5),
        # wall-bounded block with isothermal walls and the shock sensor's hybrid weights
        dict(name="channel_64x65x96_fp64", kind="channel", scheme="channel", nx=64, ny=65, nz=96, precision="fp64",
             steps=5),
        # one right-hand side for a host program's own integrator
        dict(name="rhs_48x40x44_fp64", kind="rhs", scheme="blend", nx=48, ny=40, nz=44, precision="fp64", steps=1),
    ]


def draw(rng):
    """One more case of the listed ranges."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["small", "block", "block", "block", "block", "sphere", "blocks", "channel", "rhs"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "sphere":
        return dict(kind=kind, scheme="sphere", nx=size(72, 104), ny=size(72, 104), nz=size(88, 136), precision=prec,
                    steps=3)
    if kind == "channel":
        return dict(kind=kind, scheme="channel", nx=size(24, 96), ny=size(33, 97), nz=size(24, 128), precision=prec,
                    steps=rng.randint(3, 5))
    if kind == "blocks":
        return dict(kind=kind, scheme=rng.choice(["blend", "muscl"]), nx=size(40, 112), ny=size(36, 88),
                    nz=size(36, 64), blocks=rng.randint(3, 8), precision=prec,
                    steps=rng.randint(4, 6) if prec == "fp64" else rng.randint(8, 16))
    if kind == "rhs":
        return dict(kind=kind, scheme=rng.choice(["blend", "muscl", "central", "weno5_roe"]), nx=size(20, 80),
                    ny=size(20, 80), nz=size(20, 80), precision=prec, steps=1)
    if kind == "small":
        return dict(kind=kind, scheme=rng.choice(["muscl", "central", "vortex"]), nx=size(16, 48), ny=size(16, 48),
                    nz=size(16, 48), precision=prec, steps=rng.randint(10, 20))
    scheme = rng.choice(["muscl", "muscl", "blend", "central", "weno5_roe", "vortex", "dynamic"])
    hi = 144 if prec == "mixed" or scheme in ("muscl", "central") else 112
    return dict(kind=kind, scheme=scheme, nx=size(48, hi), ny=size(48, hi), nz=size(48, hi), precision=prec,
                steps=rng.randint(4, 7))


# ------------------------------------------------------------------ inputs --
def _options(case, dt):
    o = dict(SCHEMES[case["scheme"]])
    s = o.pop("s")
    return dict(inviscid=0, s_x=s, s_y=s, s_z=s, gamma=GAMMA, dt=dt) | o


def _rng(seed):
    return np.random.default_rng([int(seed), 77])


def _axis(m, n, length):
    return (torch.arange(m, dtype=torch.float64, device=CUDA) - 1.0) * (length / n)


def _mesh(n, length):
    """Node coordinates x, y, z (each (nz+2, ny+2, nx+2)) of a periodic box."""
    ax = [_axis(n[d] + 2, n[d], length) for d in range(3)]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    return x, y, z


def _conserved(rho, u, v, w, p):
    return torch.stack([rho, rho * u, rho * v, rho * w, p / (GAMMA - 1) + 0.5 * rho * (u * u + v * v + w * w)], dim=-1)


def _distorted(n, length, amp, rng):
    """Periodic box moved by two seeded sine modes per coordinate."""
    xyz = _mesh(n, length)
    th = [2 * math.pi * c / length for c in xyz]
    out = []
    for c in range(3):
        f = torch.zeros_like(xyz[0])
        for _ in range(2):
            k = rng.integers(0, 3, size=3)
            k[c] = max(int(k[c]), 1)
            f += torch.sin(float(k[0]) * th[0] + float(k[1]) * th[1] + float(k[2]) * th[2] + rng.uniform(0, 2 * math.pi))
        out.append(xyz[c] + 0.5 * amp * f)
    return torch.stack(out, dim=-1)


def _tgv(case, seed):
    """Taylor-Green vortex on the perturbed box, shifted and disturbed by seed."""
    n = (case["nx"], case["ny"], case["nz"])
    r = _rng(seed)
    x, y, z = _mesh(n, 2 * math.pi)
    X = torch.stack([x + 0.05 * torch.sin(y) * torch.sin(z), y + 0.05 * torch.sin(z) * torch.sin(x),
                     z + 0.05 * torch.sin(x) * torch.sin(y)], dim=-1)
    sx, sy, sz = (X[..., a] + r.uniform(0, 2 * math.pi) for a in range(3))
    ma = 0.1
    p = 100.0 + (torch.cos(2 * sx) + torch.cos(2 * sy)) * (torch.cos(2 * sz) + 2.0) / 16.0
    u = torch.sin(sx) * torch.cos(sy) * torch.cos(sz)
    v = -torch.cos(sx) * torch.sin(sy) * torch.cos(sz)
    w = 0.02 * torch.sin(2 * sx + sy) * torch.cos(3 * sz)
    rho = GAMMA * p * ma * ma
    q = _conserved(rho, u / rho, v / rho, w / rho, p)
    steps_dt = (1e-3 if case["scheme"] == "muscl" else 2e-3) * 128.0 / max(n)
    return X, q, steps_dt


def _turbulence(n, seed, mach_t, u_rms=None):
    """Solenoidal random field with a Passot-Pouquet spectrum (k0 = 4)."""
    nx, ny, nz = n
    g = torch.Generator(device=CUDA)
    g.manual_seed(int(seed) % (1 << 62) + 11)
    kx, ky, kz = (torch.fft.fftfreq(m, 1.0 / m, dtype=torch.float64, device=CUDA) for m in (nx, ny, nz))
    KZ, KY, KX = torch.meshgrid(kz, ky, kx, indexing="ij")
    k2 = KX * KX + KY * KY + KZ * KZ
    ok = (k2 > 0) & (2 * KX.abs() < nx) & (2 * KY.abs() < ny) & (2 * KZ.abs() < nz)
    k2s = torch.where(ok, k2, torch.ones_like(k2))
    amp = torch.where(ok, (k2s / 16) * torch.exp(-k2s / 16) / torch.sqrt(k2s), torch.zeros_like(k2))
    uh = [amp * torch.complex(torch.randn(k2.shape, dtype=torch.float64, device=CUDA, generator=g),
                              torch.randn(k2.shape, dtype=torch.float64, device=CUDA, generator=g)) for _ in range(3)]
    div = (KX * uh[0] + KY * uh[1] + KZ * uh[2]) / k2s
    uh = [uh[0] - KX * div, uh[1] - KY * div, uh[2] - KZ * div]
    u = [torch.fft.ifftn(a).real for a in uh]
    tot = math.sqrt(float((u[0] ** 2 + u[1] ** 2 + u[2] ** 2).mean()))
    c = 1.0 if u_rms is None else math.sqrt(3.0) * u_rms / mach_t
    u = [a * (mach_t * c / tot) for a in u]
    idx = [(torch.arange(m + 2, device=CUDA) - 1) % m for m in (nz, ny, nx)]
    u = [a[idx[0]][:, idx[1]][:, :, idx[2]] for a in u]
    one = torch.ones_like(u[0])
    return _conserved(one, u[0], u[1], u[2], one * (c * c / GAMMA))


def _cfl_dt(q, spacing, cfl):
    r = q[..., 0]
    c = torch.sqrt(GAMMA * (GAMMA - 1) * (q[..., 4] - 0.5 * (q[..., 1:4] ** 2).sum(-1) / r) / r)
    lam = sum(float(((q[..., 1 + a] / r).abs() + c).max()) / spacing[a] for a in range(3))
    return math.floor(cfl / lam * 1e7) / 1e7


def _inputs(case, seed):
    """Coordinates and state (device tensors, natural order) and dt of a block."""
    n = (case["nx"], case["ny"], case["nz"])
    s = case["scheme"]
    if case["kind"] == "rhs":
        X = _distorted(n, 2 * math.pi, 0.04, _rng(seed))
        return X, _turbulence(n, seed, 0.3), 2e-3
    if s == "weno5_roe":
        X = torch.stack(_mesh(n, 2 * math.pi), dim=-1)
        q = _turbulence(n, seed, 0.4, u_rms=1.0)
        return X, q, _cfl_dt(q, [2 * math.pi / m for m in n], 0.4)
    if s == "vortex":
        L = 10.0
        X = torch.stack(_mesh(n, L), dim=-1)
        c0 = _rng(seed).uniform(4.0, 6.0, size=2)
        dx, dy = X[..., 0] - c0[0], X[..., 1] - c0[1]
        r2 = dx * dx + dy * dy
        f = 5.0 / (2 * math.pi) * torch.exp(0.5 * (1 - r2))
        t = 1 - (GAMMA - 1) * 25.0 / (8 * GAMMA * math.pi ** 2) * torch.exp(1 - r2)
        rho = t ** (1 / (GAMMA - 1))
        q = _conserved(rho, 1 - f * dy, 1 + f * dx, torch.zeros_like(rho), rho ** GAMMA)
        return X, q, _cfl_dt(q, [L / m for m in n], 0.5)
    return _tgv(case, seed)


def _channel(case, seed):
    """Channel: walls in j (tanh-clustered), periodic i and k (streamwise)."""
    n = (case["nx"], case["ny"], case["nz"])
    r = _rng(seed)
    lx, lz = math.pi, 2 * math.pi
    xs, zs = _axis(n[0] + 2, n[0], lx), _axis(n[2] + 2, n[2], lz)
    s = torch.linspace(-1, 1, n[1], dtype=torch.float64, device=CUDA)
    ys = 1 + torch.tanh(1.8 * s) / math.tanh(1.8)
    z, y, x = torch.meshgrid(zs, ys, xs, indexing="ij")
    ma = SCHEMES["channel"]["ma"]
    p = torch.full_like(x, 1 / (GAMMA * ma * ma))
    env = y * (2 - y)
    w = 1.5 * env
    u, v = torch.zeros_like(x), torch.zeros_like(x)
    for _ in range(4):
        kx, kz = int(r.integers(1, 4)), int(r.integers(1, 4))
        a, b = r.uniform(0, 2 * math.pi, size=2)
        e = 0.05 * env * torch.cos(kx * 2 * math.pi * x / lx + a) * torch.cos(kz * 2 * math.pi * z / lz + b)
        u, v, w = u + e, v + 0.5 * env * e, w + e
        p = p * (1 + 0.2 * e)
    q = _conserved(torch.ones_like(x), u, v, w, p)
    dy = float((ys[1:] - ys[:-1]).min())
    return torch.stack([x, y, z], dim=-1), q, _cfl_dt(q, [lx / n[0], dy, lz / n[2]], 0.3)


def _block_sizes(case):
    """Uneven sizes around (nx, ny, nz) and a donor permutation, the same for every seed."""
    r = np.random.default_rng([case["nx"], case["ny"], case["nz"], case["blocks"]])
    uniq = [tuple(max(16, int(m * r.uniform(0.45, 1.35))) for m in (case["nx"], case["ny"], case["nz"]))
            for _ in range(case["blocks"])]
    perm = np.roll(np.arange(case["blocks"]), 1 + int(r.integers(0, case["blocks"] - 1)))
    return uniq, [int(x) for x in perm]


def _block_set(case, seed):
    uniq, perm = _block_sizes(case)
    coords, qs, dt = [], [], 1.0
    for b, n in enumerate(uniq):
        coords.append(_distorted(n, 2 * math.pi, 0.03, np.random.default_rng([int(seed), 5, b])))
        qs.append(_turbulence(n, int(seed) * 64 + b, 0.3))
        dt = min(dt, _cfl_dt(qs[-1], [2 * math.pi / m / 1.2 for m in n], 0.4))
    return uniq, perm, coords, qs, dt


def _pinned(t):
    out = torch.empty(t.shape, dtype=torch.float64, pin_memory=True)
    out.copy_(t)
    return out.numpy()


def _host(t):
    return t.cpu().numpy()


# -------------------------------------------------------------- the passes --
def prepare(case, seed):
    kind = case["kind"]
    prec, steps = case["precision"], case["steps"]
    if kind == "blocks":
        uniq, perm, coords, qs, dt = _block_set(case, seed)
        dims = [tuple(m + 2 for m in n) for n in uniq]
        bt = B.Batch(dims, precision=prec, **_options(case, dt))
        for k in range(len(dims)):
            bt.FormMetrics(k, _host(coords[k]))
        bt.set_halo_maps(B.halo_maps_donor(dims, perm))
        q = [_pinned(x) for x in qs]
        for k in range(len(dims)):
            bt.SetInitialCondition(k, q[k])
        bt.sync()
        return dict(kind=kind, batch=bt, q=q, steps=steps)
    if kind == "sphere":
        n = (case["nx"], case["ny"], case["nz"])
        sc = W.sphere_case(n=n, h_min=0.03, seed=int(seed) % (1 << 31))
        blk = Block(*n, bctype=sc["bctype"], precision=prec, **_options(case, 1e-3))
        blk.FormMetrics(sc["coords"])
        blk.set_nvert(sc["nvert"])
        blk.set_ibm_surface(0, sc["surface"])
        blk.set_ibm_list(0, sc["info"], sc["coords"])
        q = torch.from_numpy(sc["q"])
    else:
        X, q, dt = _channel(case, seed) if kind == "channel" else _inputs(case, seed)
        mz, my, mx = q.shape[:3]
        more = dict(bctype=(7, 7, 1, 1, 7, 7)) if kind == "channel" else {}
        blk = Block(mx, my, mz, precision=prec, **more, **_options(case, dt))
        blk.FormMetrics(_host(X))
    q = _pinned(q)
    blk.SetInitialCondition(q)
    state = dict(kind=kind, block=blk, q=q, steps=steps)
    if kind not in ("small", "rhs"):
        state["out"] = torch.empty(q.shape, dtype=torch.float64, pin_memory=True).numpy()
    return state


def run(state):
    kind, q, steps = state["kind"], state["q"], state["steps"]
    if kind == "blocks":
        bt = state["batch"]
        for k in range(len(q)):
            bt.SetInitialCondition(k, q[k])
        bt.RungeKutta(steps)
        return [bt.Q(k) for k in range(len(q))]
    blk = state["block"]
    if kind == "small":
        blk.SetInitialCondition(q)
        blk.RungeKutta(steps)
        return blk.Q()
    if kind == "rhs":
        blk.SetInitialCondition(q)
        blk.CalcUCat()
        blk.Compute_eddy_viscosity_LES()
        return blk.formRHS(0)
    blk.upload_async(q)
    blk.RungeKutta(steps, sync=False)
    blk.download_async(state["out"])
    blk.join_transfers()
    return state["out"]


def work(case):
    """Per step and stage: Q, Qold and the result once (120 B), the metric
    vectors and aj (80 B; 44 B as FP32 vectors), nu_t; per pass the state in
    and out."""
    fo = SCHEMES[case["scheme"]]["fluxorder"]
    if case["kind"] == "blocks":
        cells = sum(n[0] * n[1] * n[2] for n in _block_sizes(case)[0])
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "rhs":
        return {"bytes": cells * (40 + 40 + 80 + 8.0), "flops": cells * float(FLOPS[case["scheme"]])}
    node = (208 if case["precision"] == "fp64" else 172) + (8 if case["scheme"] == "sphere" else 0)
    visits = cells * fo * case["steps"]
    return {"bytes": visits * node + cells * 80.0, "flops": visits * float(FLOPS[case["scheme"]])}


# ------------------------------------------------- the pass in plain FP64 ---
# Arrays are padded boxes (..., mz+4, my+4, mx+4) of FP64 torch tensors, node
# (i, j, k) at index + 2; d = 0, 1, 2 is the i, j, k direction.  Written for
# periodic blocks and blocks that take every halo node from a donor.
def _wrap_index(m):
    return (torch.arange(m + 4, device=CUDA) - 2) % m


def _ghosts(own):
    mz, my, mx = own.shape[-3:]
    return own[..., _wrap_index(mz), :, :][..., _wrap_index(my), :][..., _wrap_index(mx)].contiguous()


def _faces(a, d, off, e=None, t=0):
    """Nodes pos + off of the faces pos = 0 .. m-2 along d, interior across,
    shifted by t along e."""
    ix = []
    for ax in range(3):
        m = a.shape[-1 - ax] - 4
        lo, hi = (2 + off, 1 + off + m) if ax == d else (3, m + 1)
        if e == ax:
            lo, hi = lo + t, hi + t
        ix.append(slice(lo, hi))
    return a[..., ix[2], ix[1], ix[0]]


def _inner(a, e=None, t=0):
    ix = []
    for ax in range(3):
        m = a.shape[-1 - ax] - 4
        s = t if e == ax else 0
        ix.append(slice(3 + s, m + 1 + s))
    return a[..., ix[2], ix[1], ix[0]]


def _diff(f, d):
    return f.narrow(-1 - d, 1, f.shape[-1 - d] - 1) - f.narrow(-1 - d, 0, f.shape[-1 - d] - 1)


def _metrics(X):
    """csi, eta, zet (3, 3, ...) and aj by central differences, padded."""
    mz, my, mx = X.shape[:3]
    x = X.permute(3, 0, 1, 2)
    D = torch.zeros((3, 3, mz, my, mx), dtype=torch.float64, device=CUDA)  # [direction][component]
    for d in range(3):
        n = x.shape[-1 - d]
        D[d].narrow(-1 - d, 1, n - 2).copy_(0.5 * (x.narrow(-1 - d, 2, n - 2) - x.narrow(-1 - d, 0, n - 2)))
    c, e, z = D
    cross = lambda a, b: torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])  # noqa: E731
    met = torch.stack([cross(e, z), cross(z, c), cross(c, e)])
    det = (c * cross(e, z)).sum(0)
    aj = torch.where(det != 0, 1.0 / torch.where(det != 0, det, torch.ones_like(det)), torch.zeros_like(det))
    for d in range(3):  # the two other vectors and aj from the inward neighbour
        n = aj.shape[-1 - d]
        for dst, src in ((0, 1), (n - 1, n - 2)):
            for a in [met[q] for q in range(3) if q != d] + [aj]:
                a.select(-1 - d, dst).copy_(a.select(-1 - d, src))
    return _ghosts(met), _ghosts(aj)


def _minmod(a, b):
    return torch.where(a * b < 0, torch.zeros_like(a), torch.sign(a) * torch.minimum(a.abs(), b.abs()))


def _weno3(a, b, c, d0, d1):
    """Value at the face beyond b, from a, b, c = v_{i-1}, v_i, v_{i+1} (the
    solver's right states carry the two weights the other way round)."""
    t0, t1 = (1e-6 + (c - b) ** 2) ** 2, (1e-6 + (a - b) ** 2) ** 2
    a0, a1 = d0 / t0, d1 / t1
    return (a0 * (0.5 * b + 0.5 * c) + a1 * (1.5 * b - 0.5 * a)) / (a0 + a1)


def _weno5(a, b, c, d, e):
    b0 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    b1 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    b2 = 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    a0, a1, a2 = 0.1 / (1e-6 + b0) ** 2, 0.6 / (1e-6 + b1) ** 2, 0.3 / (1e-6 + b2) ** 2
    return (a0 * (2 * a - 7 * b + 11 * c) + a1 * (-b + 5 * c + 2 * d) + a2 * (2 * c + 5 * d - e)) / (6 * (a0 + a1 + a2))


def _upwind(o, V, d, h, shape):
    """Reconstruction of (rho, momenta, energy, p) and the numerical flux; V: nodes -2 .. 3."""
    m = shape[-1 - d] + 1
    pos = torch.arange(m - 1, device=CUDA).view([-1 if ax == 2 - d else 1 for ax in range(3)])
    a, b, c, e = V[1], V[2], V[3], V[4]
    if o["fluxorder"] == 2:
        L, R = b + 0.5 * _minmod(c - b, b - a), c - 0.5 * _minmod(e - c, c - b)
    else:
        L, R = _weno3(a, b, c, 0.6666667, 0.3333333), _weno3(e, c, b, 0.3333333, 0.6666667)
        if o.get("weno_order") == 5:
            in5 = (pos >= 2) & (pos <= m - 4)
            L = torch.where(in5, _weno5(V[0], a, b, c, e), L)
            R = torch.where(in5, _weno5(V[5], e, c, b, a), R)
    if not o["les"]:
        end = (pos == 0) | (pos == m - 2)
        L, R = torch.where(end, b, L), torch.where(end, c, R)
    UL, UR = (h * L[1:4]).sum(0) / L[0], (h * R[1:4]).sum(0) / R[0]
    hh = (h * h).sum(0)
    jump = R[:5] - L[:5]
    if o.get("flux") == "roe":
        area = hh.sqrt()
        nv = h / area
        sl, sr = L[0].sqrt(), R[0].sqrt()
        wl, wr = sl / (sl + sr), sr / (sl + sr)
        vl, vr = L[1:4] / L[0], R[1:4] / R[0]
        vt = wl * vl + wr * vr
        H = wl * (L[4] + L[5]) / L[0] + wr * (R[4] + R[5]) / R[0]
        q2 = (vt * vt).sum(0)
        c2 = (GAMMA - 1) * (H - 0.5 * q2)
        ct = c2.abs().sqrt()
        un = (vt * nv).sum(0)
        dp, dv = R[5] - L[5], vr - vl
        dun, rt = (dv * nv).sum(0), sl * sr
        a1, a2, a3 = (dp - rt * ct * dun) / (2 * c2), jump[0] - dp / c2, (dp + rt * ct * dun) / (2 * c2)
        lam = [(un - ct).abs(), un.abs(), (un + ct).abs()]
        dl = 0.1 * ct
        fix = lambda l: torch.where(l < dl, (l * l + dl * dl) / (2 * dl), l)  # noqa: E731
        s1, s2, s3, ss = fix(lam[0]) * a1, lam[1] * a2, fix(lam[2]) * a3, lam[1] * rt
        D = torch.cat([(s1 + s2 + s3)[None], s1 * (vt - ct * nv) + s2 * vt + s3 * (vt + ct * nv) + ss * (dv - dun * nv),
                       (s1 * (H - un * ct) + s2 * 0.5 * q2 + s3 * (H + un * ct) + ss * ((vt * dv).sum(0) - un * dun))[None]])
        D = area * D
    else:
        sa = [u.abs() + (GAMMA * s[5] / s[0] * hh).abs().sqrt() for u, s in ((UL, L), (UR, R))]
        D = torch.maximum(sa[0], sa[1]) * jump
    F = 0.5 * (L[:5] * UL + R[:5] * UR)
    F[1:4] += 0.5 * (L[5] + R[5]) * h
    F[4] += 0.5 * (L[5] * UL + R[5] * UR)
    return F - 0.5 * D


def _central(V, Ms, d, h):
    """4-point skew-symmetric flux, 2-point average on the faces next to the ends."""
    m = V[2].shape[-1 - d] + 1
    pos = torch.arange(m - 1, device=CUDA).view([-1 if ax == 2 - d else 1 for ax in range(3)])
    Q = V[1:5]
    U = [(Ms[s] * Q[s][1:4]).sum(0) / Q[s][0] for s in range(4)]
    G = [torch.cat([q[:4], (q[4] + q[5])[None]]) for q in Q]
    four = (G[1] + G[2]) * (U[1] + U[2]) / 3 - (G[0] * (U[0] + U[2]) + G[1] * (U[1] + U[3]) + G[2] * (U[2] + U[0]) +
                                               G[3] * (U[1] + U[3])) / 24
    four[1:4] += (-Q[0][5] + 7 * Q[1][5] + 7 * Q[2][5] - Q[3][5]) / 12 * h
    A = 0.5 * (Q[1] + Q[2])
    Uc = (h * A[1:4]).sum(0) / A[0]
    two = torch.cat([(A[0] * Uc)[None], A[1:4] * Uc + A[5] * h, (Uc * (A[4] + A[5]))[None]])
    return torch.where((pos > 0) & (pos < m - 2), four, two)


def _viscous(o, prim, rho, met, aj, d2, nut, d):
    """Viscous and subgrid fluxes (momenta and energy) and the subgrid stress."""
    D = [None] * 3
    for e in range(3):
        if e == d:
            D[e] = _faces(prim, d, 1) - _faces(prim, d, 0)
        else:
            D[e] = 0.25 * (_faces(prim, d, 1, e, 1) + _faces(prim, d, 0, e, 1) - _faces(prim, d, 1, e, -1) -
                           _faces(prim, d, 0, e, -1))
    mh = [0.5 * (_faces(met[e], d, 0) + _faces(met[e], d, 1)) for e in range(3)]
    md = mh[d]
    g = [(mh[e] * md).sum(0) for e in range(3)]
    grad = sum(D[e][:3, None] * mh[e][None] for e in range(3))  # [velocity][x]
    ajc = 0.5 * (_faces(aj, d, 0) + _faces(aj, d, 1))
    nu = 1.0 / o["ren"]
    if o["les"]:
        nu = nu * 0.5 * (_faces(rho, d, 0) + (_faces(rho, d, 1) if d == 0 else _faces(rho, d, 0, 0, 1)))
    div = 2.0 / 3.0 * (grad[0, 0] + grad[1, 1] + grad[2, 2])
    t = sum(g[e] * D[e][:3] for e in range(3)) + (grad * md[:, None]).sum(0) - div * md
    F = t * ajc * nu
    vel = 0.5 * (_faces(prim[:3], d, 0) + _faces(prim[:3], d, 1))
    heat = sum(g[e] * D[e][3] for e in range(3)) * ajc * (GAMMA * nu / o["pr"] / (GAMMA - 1))
    energy = (F * vel).sum(0) + heat
    A = torch.zeros_like(F)
    if o["les"] and o["s"]:
        s = o["s"]
        rc = 0.5 * (_faces(rho, d, 0) + _faces(rho, d, 1))
        nt = 0.5 * s * (_faces(nut, d, 0) + _faces(nut, d, 1))
        S = grad.clone()
        for a in range(3):
            S[a, a] -= div
        ks = -0.5 * (S * S).sum((0, 1)) * _faces(d2, d, 0) * (0.06 * 2.0 / 3.0)
        A = t * ajc * nt * rc + ks * md * rc * s
    return F + A, energy, A


def _rhs(o, P, met, aj, d2, nut):
    """Right-hand side at the interior nodes from the padded state P (5, ...)."""
    rho = P[0]
    safe = torch.where(rho != 0, rho, torch.ones_like(rho))
    vel = P[1:4] / safe
    p = (GAMMA - 1) * (P[4] - 0.5 * (P[1:4] * vel).sum(0))
    W6 = torch.cat([P, p[None]])
    prim = torch.cat([vel, (p / safe)[None]])
    conv = visc = le = 0.0
    for d in range(3):
        V = [_faces(W6, d, s) for s in range(-2, 4)]
        h = 0.5 * (_faces(met[d], d, 0) + _faces(met[d], d, 1))
        s = o["s"] if o["les"] else 0.0
        F = 0.0
        if s != 1.0:
            F = (1 - s) * _upwind(o, V, d, h, V[0].shape)
        if s != 0.0:
            F = F + s * _central(V, [_faces(met[d], d, t) for t in range(-1, 3)], d, h)
        conv = conv + _diff(F, d)
        del V, F
        if not o.get("inviscid"):
            Fm, en, A = _viscous(o, prim, rho, met, aj, d2, nut, d)
            visc = visc + _diff(torch.cat([torch.zeros_like(en)[None], Fm, en[None]]), d)
            if o["les"]:
                le = le + _diff(0.5 * (_faces(rho, d, 0) + _faces(rho, d, 1)) * A, d)
            del Fm, en, A
    r = visc - conv
    if o["les"] and not o.get("inviscid"):
        my = P.shape[-2] - 4
        j = torch.arange(1, my - 1, device=CUDA).view(1, -1, 1)
        r[4] += torch.where((j > 2) & (j < my - 2), (_inner(vel) * le).sum(0), torch.zeros_like(r[4]))
    return r * _inner(aj)


def _eddy(o, P, met, aj, d2):
    """Constant-coefficient Smagorinsky viscosity at the interior nodes."""
    rho = torch.where(P[0] != 0, P[0], torch.ones_like(P[0]))
    vel = P[1:4] / rho
    D = [0.5 * (_inner(vel, e, 1) - _inner(vel, e, -1)) for e in range(3)]
    g = sum(D[e][:, None] * _inner(met[e])[None] for e in range(3)) * _inner(aj)
    tr = 2.0 / 3.0 * (g[0, 0] + g[1, 1] + g[2, 2])
    S = 0.5 * (g + g.transpose(0, 1))
    for a in range(3):
        S[a, a] -= tr
    return o.get("cs_const", 0.03) * _inner(d2) * torch.sqrt(2 * (S * S).sum((0, 1)))


class _Periodic:
    """Halo rule of independent periodic blocks."""

    def start(self, own):
        return [_ghosts(a) for a in own]

    def nut(self, inner):
        return [_ghosts(torch.nn.functional.pad(a, (1,) * 6)) for a in inner]

    def stage(self, inner, P):
        """Boundary nodes keep the stage input two nodes across (k over j over i faces)."""
        out = []
        for a, p in zip(inner, P):
            mz, my, mx = (s + 2 for s in a.shape[-3:])
            own = torch.nn.functional.pad(a, (1,) * 6)
            box = p[:, 2:-2, 2:-2, 2:-2]
            assert box.shape[-3:] == (mz, my, mx)
            own[..., 0], own[..., mx - 1] = p[:, 2:-2, 2:-2, 0], p[:, 2:-2, 2:-2, mx + 3]
            own[..., 0, :], own[..., my - 1, :] = p[:, 2:-2, 0, 2:-2], p[:, 2:-2, my + 3, 2:-2]
            own[..., 0, :, :], own[..., mz - 1, :, :] = p[:, 0, 2:-2, 2:-2], p[:, mz + 3, 2:-2, 2:-2]
            out.append(_ghosts(own))
        return out


class _Donor:
    """Halo rule of blocks whose non-interior nodes come from a donor's interior."""

    def __init__(self, perm):
        self.perm = perm

    def _fill(self, inner):
        out = []
        for b, a in enumerate(inner):
            don = inner[self.perm[b]]
            full, ix = don, []
            for ax in (-3, -2, -1):
                m, md = a.shape[ax] + 2, don.shape[ax] + 2
                x = torch.arange(-2, m + 2, device=CUDA)
                ix.append(torch.where(x < 1, md - 2 + x, torch.where(x > m - 2, x - (m - 2), 1 + (x - 1) % (md - 2))) - 1)
            full = don[..., ix[0], :, :][..., ix[1], :][..., ix[2]].contiguous()
            full[..., 3:-3, 3:-3, 3:-3] = a
            out.append(full)
        return out

    def start(self, own):
        return self._fill([a[..., 1:-1, 1:-1, 1:-1] for a in own])

    def nut(self, inner):
        return self._fill(inner)

    def stage(self, inner, P):
        return self._fill(inner)


def _advance(o, dt, coords, qs, steps, halo, rhs_only=False):
    geo = []
    for X in coords:
        met, aj = _metrics(X)
        d2 = torch.where(aj != 0, torch.where(aj != 0, 1 / aj, torch.ones_like(aj)) ** (1.0 / 3.0), torch.zeros_like(aj)) ** 2
        geo.append((met, aj, d2))
    P = halo.start([q.permute(3, 0, 1, 2).contiguous() for q in qs])
    blocks = range(len(P))
    zero = [torch.zeros_like(g[1]) for g in geo]
    sgs = o["les"] and not o.get("inviscid")
    if rhs_only:
        nut = halo.nut([_eddy(o, P[b], *geo[b]) for b in blocks]) if sgs else zero
        out = torch.zeros_like(qs[0])
        out[1:-1, 1:-1, 1:-1] = _rhs(o, P[0], *geo[0], nut[0]).permute(1, 2, 3, 0)
        return [out]
    ns = o["fluxorder"]
    alfa, beta = ([1.0, 0.25, 2.0 / 3.0], [1.0, 0.75, 1.0 / 3.0]) if ns == 3 else ([1.0, 0.5], [1.0, 0.5])
    seen = None  # the state whose velocity the eddy viscosity reads: the last stage input
    for _ in range(steps):
        nut = zero
        if sgs and seen is not None and o["s"]:
            nut = halo.nut([_eddy(o, seen[b], *geo[b]) for b in blocks])
        old, cur = P, P
        for s in range(ns):
            new = []
            for b in blocks:
                r = _rhs(o, cur[b], *geo[b], nut[b])
                if s == 0:
                    new.append(_inner(old[b]) + alfa[s] * dt * r)
                else:
                    new.append(beta[s] * _inner(old[b]) + alfa[s] * dt * r + alfa[s] * _inner(cur[b]))
                del r
            seen, cur = cur, halo.stage(new, cur)
        P = cur
    return [p[:, 2:-2, 2:-2, 2:-2].permute(1, 2, 3, 0).contiguous() for p in P]


def exact(case, seed):
    """The pass in FP64 torch operations; None for the sphere, the channel and
    the dynamic model, whose rules are not restated here."""
    if case["kind"] in ("sphere", "channel") or case["scheme"] == "dynamic":
        return None
    o = SCHEMES[case["scheme"]]
    if case["kind"] == "blocks":
        _, perm, coords, qs, dt = _block_set(case, seed)
        return _advance(o, dt, coords, qs, case["steps"], _Donor(perm))
    X, q, dt = _inputs(case, seed)
    return _advance(o, dt, [X], [q], case["steps"], _Periodic(), rhs_only=case["kind"] == "rhs")[0]
