"""The replay and the backward step march columns of 32 x 8 cells through a few
planes: domains that end inside a column, a plane run or a checkpoint segment."""
from __future__ import annotations

import numpy as np
import pytest

import mumatscale_b200 as M
from mumatscale_b200 import workloads as W

pytestmark = pytest.mark.gpu

FD_STEP, FD_TOL = 1e-4, 1e-4  # central differences and their agreement, as in test_adjoint


def _domain(tmp_path, dims, prec, scale=1.0):
    deck, _, thr, rot = W.one_grain(64, tip_curv=0)
    f = tmp_path / "a.in"
    f.write_text(deck.replace("NCellsPerSB 64 64 64", "NCellsPerSB %d %d %d" % dims))
    p = M.read_deck(f)
    p.initialTemperature -= 5.0
    p.Dliq *= scale
    p.part_coef *= scale
    d = M.Domain(p, precision=prec)
    W.setup_one_grain(d, np.array([[n // 2 for n in dims]], dtype=np.int32), thr, rot)
    return d


@pytest.mark.parametrize("dims,every", [((33, 9, 7), 1), ((5, 17, 40), 100), ((64, 8, 13), 7), ((31, 33, 1 + 6 * 4), 30)])
def test_gradient_of_odd_domains(built, cuda_device, tmp_path, dims, every):
    steps = 60
    with _domain(tmp_path, dims, M.PREC_F64, 1.1) as other:
        other.step(steps)
        target = other.download("ce")
    with _domain(tmp_path, dims, M.PREC_F64) as dom:
        dom.adjoint_record(steps, every)
        ce = dom.download("ce")
        assert dom.adjoint_replay_loss(ce) == 0.0  # the unscaled replay is the recorded run
        g = dom.adjoint_gradient(target)
        assert g == dom.adjoint_gradient(target)
        assert abs(g["loss"] - dom.adjoint_replay_loss(target)) <= 1e-13 * g["loss"]
        for n, name in ((0, "Dliq"), (1, "part_coef")):
            up, dn = [1.0] * 3, [1.0] * 3
            up[n] += FD_STEP
            dn[n] -= FD_STEP
            base = (dom.params.Dliq, dom.params.part_coef)[n]
            fd = (dom.adjoint_replay_loss(target, up) - dom.adjoint_replay_loss(target, dn)) / (2 * FD_STEP)
            assert abs(g[name] * base - fd) <= FD_TOL * abs(fd), name
    with _domain(tmp_path, dims, M.PREC_F32) as dom:
        dom.adjoint_record(steps, every)
        assert dom.adjoint_replay_loss(dom.download("ce")) == 0.0
        h = dom.adjoint_gradient(target)
        assert abs(h["Dliq"] - g["Dliq"]) <= 2e-2 * abs(g["Dliq"])  # as in test_adjoint
