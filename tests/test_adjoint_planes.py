"""The replay and the backward step march up several planes a CTA where the
domain has enough columns of tiles: ragged domains whose columns take 3 and 6
planes, the last column of a tile row short."""
from __future__ import annotations

import pytest

import mumatscale_b200 as M
import test_adjoint_shapes as S

pytestmark = pytest.mark.gpu


def _planes(dims):
    tiles = -(-dims[0] // 32) * -(-dims[1] // 8)
    return max(1, min(6, tiles * dims[2] // (148 * 3)))


@pytest.mark.parametrize("dims,planes", [((65, 63, 61), 3), ((97, 71, 75), 6)])
def test_gradient_of_several_planes(built, cuda_device, tmp_path, dims, planes):
    assert _planes(dims) == planes and dims[2] % planes != 0
    steps, every = 30, 12
    with S._domain(tmp_path, dims, M.PREC_F64, 1.1) as other:
        other.step(steps)
        target = other.download("ce")
    with S._domain(tmp_path, dims, M.PREC_F64) as dom:
        dom.adjoint_record(steps, every)
        assert dom.adjoint_replay_loss(dom.download("ce")) == 0.0  # the unscaled replay is the recorded run
        g = dom.adjoint_gradient(target)
        assert g == dom.adjoint_gradient(target)
        assert abs(g["loss"] - dom.adjoint_replay_loss(target)) <= 1e-13 * g["loss"]
        for n, name in ((0, "Dliq"), (1, "part_coef")):
            up, dn = [1.0] * 3, [1.0] * 3
            up[n] += S.FD_STEP
            dn[n] -= S.FD_STEP
            base = (dom.params.Dliq, dom.params.part_coef)[n]
            fd = (dom.adjoint_replay_loss(target, up) - dom.adjoint_replay_loss(target, dn)) / (2 * S.FD_STEP)
            assert abs(g[name] * base - fd) <= S.FD_TOL * abs(fd), name
    with S._domain(tmp_path, dims, M.PREC_F32) as dom:
        dom.adjoint_record(steps, every)
        assert dom.adjoint_replay_loss(dom.download("ce")) == 0.0
        h = dom.adjoint_gradient(target)
        for name in ("Dliq", "part_coef"):
            assert abs(h[name] - g[name]) <= 2e-2 * abs(g[name]), name  # as in test_adjoint
