"""A block with an immersed body runs the planes no nonzero nvert reaches through
the no-IBM tile code; which planes those are depends on the k-chunk (runs shorter
than MASK_MIN_RUN stay with the body's).  In the mixed form the two codes differ
in more than the nvert tests (packed FP32, a metric slot), so the bits of a step
must not depend on the chunk."""
import numpy as np
import pytest

import oracle as O
from _common import gpu_block
from chimera_comp_les_b200 import workloads as W
from test_gpu_mask_planes import BODIES, N, SCHEMES, _mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("body", ["tile_edge", "k_low"])
@pytest.mark.parametrize("scheme", SCHEMES)
def test_mixed_bits_do_not_depend_on_the_chunk(scheme, body):
    coords = W.periodic_grid(N, 2 * np.pi, amp=0.04)
    shape = coords.shape[:3]
    cfg = O.Config(mx=N[0] + 2, my=N[1] + 2, mz=N[2] + 2, inviscid=0, ren=500.0, ma=0.3, pr=0.71, dt=0.002, **SCHEMES[scheme])
    q, nv = W.random_smooth_state(shape, seed=17), _mask(shape, BODIES[body])
    first = None
    for kchunk in (40, 13, 7, 3, 0):  # 3: no clean run is long enough beside the body
        with gpu_block(cfg, precision="mixed") as b:
            b.FormMetrics(coords)
            b.set_nvert(nv)
            b.SetInitialCondition(q)
            b.autotune([kchunk])
            b.RungeKutta(1)
            got = b.Q()
        assert first is None or np.array_equal(got, first), kchunk
        first = got
