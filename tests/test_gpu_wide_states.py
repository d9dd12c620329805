"""States beyond the range in which the kernels' branch-free quotients hold
(cb_div.cuh), where IEEE division still gives a finite result: jumps whose
square overflows (a WENO weight of 0), squared smoothness measures and
densities above 2^1022, subnormal densities.  One right-hand side (the general
kernel) and one step (the no-IBM kernels), with and without a body, against the
restatement.  The bar is the FP64 form's, 1e-12, on the largest value of each
field (squares of these values overflow), near the jump and away from it."""
import numpy as np
import pytest

import oracle as O
from _common import RTOL_L2, gpu_block, oracle_run
from chimera_comp_les_b200 import workloads as W

pytestmark = pytest.mark.gpu

N = (40, 17, 18)  # two tiles in i, three to four in j
SCHEMES = {
    "muscl": dict(les=1, fluxorder=2, s_x=0.0, s_y=0.0, s_z=0.0),
    "muscl_roe": dict(les=0, fluxorder=2, flux=1, inviscid=1),
    "first_blend": dict(les=1, fluxorder=1, s_x=0.5, s_y=0.5, s_z=0.5),
    "weno3_blend": dict(les=1, fluxorder=3, s_x=0.5, s_y=0.5, s_z=0.5),
    "weno3_roe": dict(les=1, fluxorder=3, flux=1, s_x=0.0, s_y=0.0, s_z=0.0),
    "std_weno3": dict(les=0, fluxorder=3),
    "weno5": dict(les=1, fluxorder=3, weno_order=5, s_x=0.0, s_y=0.0, s_z=0.0),
    "weno5_roe": dict(les=0, fluxorder=3, weno_order=5, flux=1, inviscid=1),
    "central": dict(les=1, fluxorder=3),
    "central_two_point": dict(les=1, fluxorder=3, central=1),
}
# steps small enough that the stages' states stay on the restatement's finite side
DT = {"jump": 1e-20, "dense": 1e-150, "dense_even": 1e-150}
CASES = ([(s, f"jump{a}") for s in ("weno3_blend", "weno3_roe", "std_weno3", "weno5", "weno5_roe") for a in (0, 1, 2)]
         + [(s, f"ramp{a}") for s in ("weno3_roe", "weno5") for a in (0, 1)]
         + [(s, "dense") for s in ("muscl", "muscl_roe", "first_blend")]
         + [(s, "dense_even") for s in ("weno3_blend", "weno3_roe", "std_weno3", "central", "central_two_point")]
         + [(s, "subnormal") for s in ("muscl_roe", "std_weno3", "weno5_roe", "central_two_point")])


def _state(shape, kind):
    """The state and the nodes on its far side of a jump (None without one)."""
    q = W.random_smooth_state(shape, seed=9)
    if kind[:-1] in ("jump", "ramp"):
        ax = 2 - int(kind[-1])
        m = shape[ax]
        g = np.ones(m)
        if kind[:-1] == "jump":  # 1 -> 1e80 -> 1: its square's square overflows
            g[m // 3:2 * m // 3] = 1e80
        else:  # 1 -> 1e75 -> 1e77 -> 1: (1e77)^4 = 1e308 lies above 2^1022, (1e75)^4 below
            g[m // 3:2 * m // 3] = 1e77
            g[m // 3] = 1e75
        far = np.broadcast_to((g > 1).reshape([m if a == ax else 1 for a in range(3)]), shape)
        q[far] = (np.array([1.0, 0.3, -0.2, 0.1, 7.0]) * np.broadcast_to(
            g.reshape([m if a == ax else 1 for a in range(3)]), shape)[..., None])[far]
        return q, far
    if kind == "dense":  # densities in 5.6e307 .. 8e307, momentum and sound speed of one size
        q = np.concatenate([8e307 * q[..., :1] / q[..., :1].max(), 1e153 * q[..., 1:4], q[..., 4:]], axis=-1)
    elif kind == "dense_even":
        q = np.concatenate([np.full(shape + (1,), 5e307), 1e70 * q[..., 1:4], q[..., 4:]], axis=-1)
    else:
        q = q * 1e-310
    return q, None


def _worst(got, ref, far):
    parts = [np.ones(ref.shape[:3], bool)]
    if far is not None:  # the far side, the nodes a stencil reaches from it, the rest
        near = far.copy()
        for ax in range(3):
            for s in (-3, -2, -1, 1, 2, 3):
                near |= np.roll(far, s, axis=ax)
        parts = [far, near & ~far, ~near]
    err = 0.0
    for m in parts:
        for f in range(5):
            a, b = got[m][:, f], ref[m][:, f]
            top = np.abs(b).max()
            if top > 0:
                err = max(err, float(np.abs(a / top - b / top).max()))
            else:
                assert not a.any()
    return err


@pytest.mark.parametrize("body", [False, True], ids=["clean", "body"])
@pytest.mark.parametrize("scheme,kind", CASES, ids=["-".join(c) for c in CASES])
def test_fp64_matches_the_restatement(scheme, kind, body):
    coords = W.periodic_grid(N, 2 * np.pi, amp=0.04)
    shape = coords.shape[:3]
    cfg = O.Config(mx=N[0] + 2, my=N[1] + 2, mz=N[2] + 2, ren=500.0, ma=0.3, pr=0.71,
                   dt=DT.get(kind.rstrip("012"), 1e-4), **{"inviscid": 0, **SCHEMES[scheme]})
    q, far = _state(shape, kind)
    nv = np.zeros(shape)
    if body:
        nv[8:10, 7:9, 20:23] = 3.0
    with np.errstate(all="ignore"):
        ref = oracle_run(cfg, coords, q, nv, steps=1)
    assert np.isfinite(ref["rhs"]).all()
    with gpu_block(cfg) as b:
        b.FormMetrics(coords)
        if body:
            b.set_nvert(nv)
        b.SetInitialCondition(q)
        if cfg.les and not cfg.inviscid:
            b.CalcUCat()
            b.Compute_eddy_viscosity_LES()
        rhs = b.formRHS(0)
        assert _worst(rhs, ref["rhs"], far) <= RTOL_L2
        if np.isfinite(ref["q_steps"]).all():  # (not the blend's energy beside a jump of 1e80)
            b.SetInitialCondition(q)
            b.RungeKutta(1)
            assert _worst(b.Q(), ref["q_steps"], far) <= RTOL_L2


# ------------------------------------------- model and sensor kernels -------
def _momentum(shape, rho, u):
    """Density rho (scaled to its maximum) and velocities of size u; energy 1."""
    q = W.random_smooth_state(shape, seed=9)
    r = rho * (q[..., :1] / q[..., :1].max())
    return np.concatenate([r, r * (u * q[..., 1:4]), q[..., 4:]], axis=-1)


@pytest.mark.parametrize("les", [1, 2])
@pytest.mark.parametrize("rho,scale", [(8e307, 1.0), (1e-310, 1.0), (1.0, 8.2e-103)], ids=["dense", "subnormal", "fine_grid"])
def test_eddy_viscosity_beyond_the_quotients_range(les, rho, scale):
    """nu_t and the dynamic coefficient; fine_grid: 1 / aj of aj above 2^1022."""
    coords = scale * W.periodic_grid(N, 2 * np.pi, amp=0.01)
    shape = coords.shape[:3]
    cfg = O.Config(mx=N[0] + 2, my=N[1] + 2, mz=N[2] + 2, ren=500.0, ma=0.3, pr=0.71, inviscid=0, les=les, max_cs=0.1)
    if les == 2 and rho > 1e300:
        pytest.skip("the test filter's sum of densities overflows in the reference too")
    q = _momentum(shape, rho, 0.3)
    with np.errstate(all="ignore"):
        ref = oracle_run(cfg, coords, q, np.zeros(shape))
    if scale != 1.0:
        assert ref["metrics"]["aj"].min() > 2.0 ** 1022
    with gpu_block(cfg) as b:
        b.FormMetrics(coords)
        b.SetInitialCondition(q)
        b.CalcUCat()
        b.Compute_eddy_viscosity_LES()
        nut = b.nu_t()
        cs = b.CS() if les == 2 else None
    assert np.isfinite(ref["nut"]).all() and ref["nut"].max() > 0.0
    assert np.abs(nut - ref["nut"]).max() <= RTOL_L2 * ref["nut"].max()
    if les == 2:
        assert np.abs(cs - ref["cs"]).max() <= RTOL_L2 * ref["cs"].max()


@pytest.mark.parametrize("kind", ["jump", "dense"])
def test_sensor_beyond_the_quotients_range(kind):
    """jump: a pressure jump of 1e160, whose square overflows on one side; dense: the EOS of densities above 2^1022."""
    coords = W.periodic_grid(N, 2 * np.pi, amp=0.04)
    shape = coords.shape[:3]
    cfg = O.Config(mx=N[0] + 2, my=N[1] + 2, mz=N[2] + 2, ma=0.3, pr=0.71, inviscid=1, les=1, fluxorder=2, calc_sigma=1,
                   s_x=1.0, s_y=1.0, s_z=1.0)
    far = None
    if kind == "jump":
        q = W.random_smooth_state(shape, seed=9)
        far = np.zeros(shape, bool)
        far[:, :, shape[2] // 3:2 * shape[2] // 3] = True
        q[far] = [1.0, 0.3, -0.2, 0.1, 1e160]
    else:
        q, far = _state(shape, "dense")
    with np.errstate(all="ignore"):
        ref = oracle_run(cfg, coords, q, np.zeros(shape))["rhs"]
    assert np.isfinite(ref).all()
    with gpu_block(cfg) as b:
        b.FormMetrics(coords)
        b.SetInitialCondition(q)
        assert _worst(b.formRHS(0), ref, far) <= RTOL_L2


# ------------------------------------------------------------- mixed form ---
# (ramp_e in the other schemes and heavy in the blend lie a little outside the form's bar whatever the quotients are)
MIXED_CASES = ([("weno3_roe", "ramp_e")] + [(s, "heavy") for s in ("muscl", "muscl_roe")]
               + [(s, "fine") for s in ("muscl_inviscid", "muscl_roe")])


@pytest.mark.parametrize("scheme", ["weno3_blend", "weno5", "weno5_roe"])
def test_mixed_weno_of_steep_energies_is_finite(scheme):
    """The state ramp_e of the next test in the schemes that the bar leaves out."""
    coords = W.periodic_grid(N, 2 * np.pi, amp=0.04)
    shape = coords.shape[:3]
    cfg = O.Config(mx=N[0] + 2, my=N[1] + 2, mz=N[2] + 2, ren=500.0, ma=0.3, pr=0.71, **{"inviscid": 0, **SCHEMES[scheme]})
    q = W.random_smooth_state(shape, seed=9)
    x = np.arange(shape[2])
    q[..., 4] += 3.6e9 * np.minimum(x, shape[2] - 1 - x)
    with gpu_block(cfg, precision="mixed") as b:
        b.FormMetrics(coords)
        b.SetInitialCondition(q)
        if cfg.les and not cfg.inviscid:
            b.CalcUCat()
            b.Compute_eddy_viscosity_LES()
        assert np.isfinite(b.formRHS(0)).all()


@pytest.mark.parametrize("body", [False, True], ids=["clean", "body"])
@pytest.mark.parametrize("scheme,kind", MIXED_CASES, ids=["-".join(c) for c in MIXED_CASES])
def test_mixed_matches_the_restatement(scheme, kind, body):
    """The mixed form's bar, 1e-5.  ramp_e: an energy that changes by 3.6e9 from node to node, so that every
    (eps + beta)^2 lies in 2^126 .. 2^128, where the flushing reciprocal gives 0; heavy: densities of 1.0e38 .. 1.5e38,
    above 2^126; fine: cells of 1.7e-10, whose squared face areas are subnormal."""
    scale = 1.1e-9 if kind == "fine" else 1.0
    coords = scale * W.periodic_grid(N, 2 * np.pi, amp=0.04)
    shape = coords.shape[:3]
    kw = {"inviscid": 0, **({"les": 0, "fluxorder": 2, "inviscid": 1} if scheme == "muscl_inviscid" else SCHEMES[scheme])}
    cfg = O.Config(mx=N[0] + 2, my=N[1] + 2, mz=N[2] + 2, ren=500.0, ma=0.3, pr=0.71,
                   dt={"ramp_e": 1e-8, "heavy": 1e-3, "fine": 1e-13}[kind], **kw)
    q = W.random_smooth_state(shape, seed=9)
    if kind == "ramp_e":
        x = np.arange(shape[2])
        q[..., 4] += 3.6e9 * np.minimum(x, shape[2] - 1 - x)
    elif kind == "heavy":
        rho, u = 1.5e38 * q[..., 0] / q[..., 0].max(), 0.3 * q[..., 1:4]
        q[..., 0], q[..., 1:4] = rho, rho[..., None] * u
        q[..., 4] = rho * (0.125 + 0.5 * (u * u).sum(axis=-1))
    nv = np.zeros(shape)
    if body:
        nv[8:10, 7:9, 20:23] = 3.0
    ref = oracle_run(cfg, coords, q, nv, steps=1)
    assert np.isfinite(ref["rhs"]).all() and np.isfinite(ref["q_steps"]).all()
    with gpu_block(cfg, precision="mixed") as b:
        b.FormMetrics(coords)
        if body:
            b.set_nvert(nv)
        b.SetInitialCondition(q)
        if cfg.les and not cfg.inviscid:
            b.CalcUCat()
            b.Compute_eddy_viscosity_LES()
        rhs = b.formRHS(0)
        b.SetInitialCondition(q)
        b.RungeKutta(1)
        step = b.Q()
    for got, want in ((rhs, ref["rhs"]), (step, ref["q_steps"])):
        for f in range(5):
            top = np.abs(want[..., f]).max()
            assert O.rel_l2(got[..., f] / top, want[..., f] / top) <= 1e-5


def test_mixed_eddy_viscosity_of_heavy_states():
    coords = W.periodic_grid(N, 2 * np.pi, amp=0.04)
    shape = coords.shape[:3]
    cfg = O.Config(mx=N[0] + 2, my=N[1] + 2, mz=N[2] + 2, ren=500.0, ma=0.3, pr=0.71, inviscid=0, les=1)
    q = _momentum(shape, 1.5e38, 0.3)
    ref = oracle_run(cfg, coords, q, np.zeros(shape))["nut"]
    with gpu_block(cfg, precision="mixed") as b:
        b.FormMetrics(coords)
        b.SetInitialCondition(q)
        b.CalcUCat()
        b.Compute_eddy_viscosity_LES()
        assert O.rel_l2(b.nu_t(), ref) <= 1e-5
