"""tracer_2d, tracer_2d_1L and tracer_2d_nested (not nested) on the parts of a face that ranks own, against the FP64
oracle: quadrants, blocks 0 to 3 cells from an edge (halo rows cross it, the block does not), bands along one edge,
odd offsets, and blocks of one cell; one substep, and two with the halos as they were."""
import functools

import numpy as np
import pytest

import oracle as O
import oracle.oracle as OO
from fv3atm_gb300 import api
from fv3atm_gb300 import synth as S

from ._helpers import rel_l2, sub_domain

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-12
N, NG = 40, 3
BLOCKS = [(1, 20, 1, 20), (21, 40, 1, 20), (1, 20, 21, 40), (21, 40, 21, 40), (9, 31, 11, 30), (2, 17, 3, 30),
          (3, 17, 2, 30), (4, 20, 4, 39), (5, 38, 4, 38), (1, 40, 1, 3), (1, 3, 1, 40), (38, 40, 1, 40), (1, 40, 38, 40),
          (1, 40, 2, 39), (2, 39, 1, 40), (7, 40, 6, 40), (1, 2, 38, 39), (1, 1, 1, 1), (40, 40, 40, 40), (17, 17, 23, 23),
          (2, 2, 2, 2), (39, 39, 2, 2)]


@pytest.fixture(scope="module")
def prob():
    return S.make_problem(N, 2, 3, seed=5, cmax=0.9)


@pytest.mark.parametrize("q_split", [1, 2])
@pytest.mark.parametrize("hord", [8, 5, 1])
@pytest.mark.parametrize("block", BLOCKS)
def test_part_of_a_face_matches_oracle(cuda, monkeypatch, prob, block, hord, q_split):
    P, (i0, i1, j0, j1) = prob, block
    geom, args = sub_domain(P, 2, *block)
    corners = (int(i0 == 1 and j0 == 1), int(i1 == N and j0 == 1), int(i0 == 1 and j1 == N), int(i1 == N and j1 == N))
    da = float(np.min(P.geoms[2].area[NG:NG + N, NG:NG + N]))
    bounds = (i0, i1, j0, j1, i0 - NG, i1 + NG, j0 - NG, j1 + NG, NG)
    monkeypatch.setattr(OO, "GridRef", functools.partial(OO.GridRef, corners=corners))
    ref = O.tracer_2d_nested(*args, geom, None, hord=hord, q_split=q_split, nested=0, bounds=O.Bounds(*bounds),
                             npx=N + 1, npy=N + 1, da_min=da)
    gs, bd = api.GridStruct(geom, corners=corners, da_min=da), api.Bounds(*bounds)
    inner = np.s_[..., NG:NG + j1 - j0 + 1, NG:NG + i1 - i0 + 1]
    for entry in (api.tracer_2d, api.tracer_2d_1L, api.tracer_2d_nested):
        q, dp, mfx, mfy, cx, cy = (a.copy() for a in args)
        entry(q, dp, mfx, mfy, cx, cy, gs, bd, N + 1, N + 1, P.npz, P.nq, hord, q_split, P.dt)
        assert rel_l2(q[inner], ref[0][inner]) <= FP64_TOL
        assert rel_l2(dp[inner], ref[1][inner]) <= FP64_TOL
