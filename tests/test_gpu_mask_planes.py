"""Stage kernel with an immersed body: the planes of a tile column that no
nonzero nvert reaches run the no-IBM tile code.  Bodies on tile edges, at the
i = 1 column (which the zeta-face test of every column reads) and at the ends
of k, with one chunk over all planes (split around the body), short chunks and
balanced segments, against the restatement (FP64 1e-12, mixed 1e-5)."""
import numpy as np
import pytest

import oracle as O
from _common import RTOL_L2, gpu_block, oracle_run, per_field_rel_l2
from chimera_comp_les_b200 import workloads as W

pytestmark = pytest.mark.gpu

N = (70, 19, 40)  # 3 x 3 tile columns (3 x 4 with WENO5-JS)
SCHEMES = {
    "muscl": dict(les=1, fluxorder=2, s_x=0.0, s_y=0.0, s_z=0.0),
    "weno5_roe": dict(les=1, fluxorder=3, weno_order=5, flux=1, s_x=0.0, s_y=0.0, s_z=0.0),
    "weno3_blend": dict(les=1, fluxorder=3, s_x=0.3, s_y=0.6, s_z=0.5),
    "central": dict(les=1, fluxorder=3),
    "std_weno3": dict(les=0, fluxorder=3),
}
BODIES = {"tile_edge": (33, 8, 20), "i1": (2, 14, 22), "k_low": (50, 10, 3), "k_high": (64, 5, 38)}


def _mask(shape, centre):
    z, y, x = np.meshgrid(*(np.arange(m) for m in shape), indexing="ij")
    r = np.sqrt((x - centre[0]) ** 2 + (y - centre[1]) ** 2 + (z - centre[2]) ** 2)
    return np.where(r < 1.8, 3.0, np.where(r < 2.9, 1.0, 0.0))


@pytest.mark.parametrize("body", BODIES)
@pytest.mark.parametrize("scheme", SCHEMES)
def test_planes_without_nvert_match_the_restatement(scheme, body):
    coords = W.periodic_grid(N, 2 * np.pi, amp=0.04)
    shape = coords.shape[:3]
    cfg = O.Config(mx=N[0] + 2, my=N[1] + 2, mz=N[2] + 2, inviscid=0, ren=500.0, ma=0.3, pr=0.71, dt=0.002,
                   **SCHEMES[scheme])
    q, nv = W.random_smooth_state(shape, seed=17), _mask(shape, BODIES[body])
    ref = oracle_run(cfg, coords, q, nv, steps=1)
    for prec, tol in (("fp64", RTOL_L2), ("mixed", 1e-5)):
        first = None
        for kchunk in (40, 7, 0):
            with gpu_block(cfg, precision=prec) as b:
                b.FormMetrics(coords)
                b.set_nvert(nv)
                b.SetInitialCondition(q)
                b.autotune([kchunk])
                b.RungeKutta(1)
                got = b.Q()
                if cfg.les:
                    b.SetInitialCondition(q)
                    b.CalcUCat()
                    b.Compute_eddy_viscosity_LES()
                rhs = b.formRHS(0)
            assert max(per_field_rel_l2(got, ref["q_steps"])) <= tol
            if cfg.les:
                assert max(per_field_rel_l2(rhs, ref["rhs"])) <= tol
            if prec == "fp64":
                assert first is None or np.array_equal(got, first)
                first = got
