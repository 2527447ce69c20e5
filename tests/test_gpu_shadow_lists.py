"""The shadow kernel's leaf lists and sample rounds where they turn (needs a B200).

One warp takes a face's samples 32 at a time against the leaves its rays can enter; a face that can
enter more leaves than the list holds walks the tree ray by ray. The sample counts lie around one
and two rounds, the face counts around a warp's and a block's share, and a large plate over a dense
mesh overflows the list. Bar, as for the other meshes: shadow counts equal to the oracle's (which
tests every triangle with the same FP32 arithmetic) for 99.9 % of the entries, never more than one
sample apart."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_raytrace import _c6, _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nmonte", [1, 31, 32, 33, 65])
@pytest.mark.parametrize("nface", [7, 8, 65, 320])
def test_sample_rounds_and_face_shares(ctx, N, O, nmonte, nface):
    from dsmc_suite_b200 import workloads as W
    spot, facet = W.cratered_mesh(2, craters=6, depth=0.4, width=0.4)
    facet = facet[:nface]
    n = N.mesh_normals(spot, facet)["normal"]
    _compare(ctx.shadow_flux(spot, facet, n, 0.4, 5, nmonte), O.shadow_flux(spot, facet, n, 0.4, 5, nmonte),
             _c6(n, 0.4, 5), nmonte)


def test_plate_over_a_dense_mesh_overflows_the_list(ctx, N, O):
    from dsmc_suite_b200 import workloads as W
    spot, facet = W.cratered_mesh(4, craters=20, depth=0.3, width=0.2)
    k = len(spot)
    plate = np.array([[-3.0, -0.2, -2.5], [3.0, -0.2, -2.5], [0.0, -0.2, 4.0], [0.0, 0.2, 4.0]])
    spot = np.vstack([spot, plate])
    facet = np.vstack([facet, [[k, k + 1, k + 2], [k, k + 1, k + 3]]]).astype(np.int32)
    n = N.mesh_normals(spot, facet)["normal"]
    G = ctx.shadow_flux(spot, facet, n, 0.3, 6, 40)
    O_ = O.shadow_flux(spot, facet, n, 0.3, 6, 40, nthreads=8)
    assert _compare(G, O_, _c6(n, 0.3, 6), 40) > 0
    lit = _c6(n, 0.3, 6)[-2:] > 0
    assert np.any((G[-2:] < _c6(n, 0.3, 6)[-2:]) & lit)   # the plate itself is shadowed by the body
