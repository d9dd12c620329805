"""Stage kernel on states of plateaus and jumps: zero slopes, slopes of opposite
sign on a node's two sides and extrema of one node (the branches of minmod, here
also as the mixed form's median), at sizes that end on, one short of and one
beyond a tile in i and j, for each blend weight (upwind flux only, both fluxes,
central flux only).  Against the restatement: FP64 RTOL_L2, mixed 1e-5, the
forms' own bars."""
import numpy as np
import pytest

import oracle as O
from _common import RTOL_L2, gpu_block, oracle_run, per_field_rel_l2
from chimera_comp_les_b200 import workloads as W

pytestmark = pytest.mark.gpu

SCHEMES = {"muscl": dict(fluxorder=2), "weno3": dict(fluxorder=3), "weno5": dict(fluxorder=3, weno_order=5)}
SIZES = [(32, 7, 9), (33, 13, 8), (31, 15, 6)]


def _state(shape):
    z, y, x = np.meshgrid(*(np.arange(m) for m in shape), indexing="ij")
    step = ((x // 3) % 2) + 2 * ((y // 2) % 2) + ((z // 4) % 2) + ((x + y + z) % 7 == 0)
    rho = 1.0 + 0.1 * step
    u, v, w = 0.2 * (step % 2), -0.1 * (step % 3), 0.05 * (z % 2)
    p = 5.0 + 0.3 * ((step * 3) % 4)
    return np.stack([rho, rho * u, rho * v, rho * w, p / 0.4 + 0.5 * rho * (u * u + v * v + w * w)], axis=-1)


@pytest.mark.parametrize("n", SIZES, ids=str)
@pytest.mark.parametrize("sigma", [0.0, 0.5, 1.0])
@pytest.mark.parametrize("scheme", SCHEMES)
def test_plateaus_match_the_restatement(scheme, sigma, n):
    coords = W.periodic_grid(n, 2 * np.pi, amp=0.04)
    shape = coords.shape[:3]
    cfg = O.Config(mx=n[0] + 2, my=n[1] + 2, mz=n[2] + 2, les=1, inviscid=0, ren=500.0, ma=0.3, pr=0.71, dt=1e-4,
                   s_x=sigma, s_y=sigma, s_z=sigma, **SCHEMES[scheme])
    q = _state(shape)
    ref = oracle_run(cfg, coords, q, np.zeros(shape), steps=1)["q_steps"]
    for prec, tol in (("fp64", RTOL_L2), ("mixed", 1e-5)):
        with gpu_block(cfg, precision=prec) as b:
            b.FormMetrics(coords)
            b.SetInitialCondition(q)
            b.RungeKutta(1)
            assert max(per_field_rel_l2(b.Q(), ref)) <= tol
