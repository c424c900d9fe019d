"""Domains of more planes than a launch can have layers of tiles at the default
planes per tile (grid.z is at most 65,535)."""
from __future__ import annotations

import numpy as np
import pytest

import mumatscale_b200 as M
from mumatscale_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _domain(tmp_path, dims, prec):
    deck, _, thr, rot = W.one_grain(64, tip_curv=0)
    f = tmp_path / "tall.in"
    f.write_text(deck.replace("NCellsPerSB 64 64 64", "NCellsPerSB %d %d %d" % dims))
    p = M.read_deck(f)
    p.initialTemperature -= 5.0
    p.site_setup = 1
    d = M.Domain(p, precision=prec)
    W.setup_one_grain(d, np.array([[n // 2 for n in dims]], dtype=np.int32), thr, rot)
    return d


def test_default_tile_of_a_tall_domain(built, cuda_device, tmp_path):
    dims = (3, 3, 65535 * 8 + 100)
    with _domain(tmp_path, dims, M.PREC_F32) as dom:
        assert dom.stencil_tile() == (2, 0)
        dom.step(3)
        gr, ce = dom.download("gr"), dom.download("ce")
        assert dom.num_grains == 2
    with _domain(tmp_path, dims, M.PREC_F32) as dom:
        dom.set_stencil_tile(1, 32)
        dom.step(3)
        assert np.array_equal(gr, dom.download("gr")) and np.array_equal(ce, dom.download("ce"))


def test_adjoint_of_a_tall_domain(built, cuda_device, tmp_path):
    dims = (3, 3, 65535 * 6 + 50)
    with _domain(tmp_path, dims, M.PREC_F64) as dom:
        target = dom.download("ce")
        dom.step(2)
        dom.adjoint_record(4, 2)
        assert dom.adjoint_replay_loss(dom.download("ce")) == 0.0
        g = dom.adjoint_gradient(target)
        assert g["loss"] > 0 and g["Dliq"] != 0
        assert abs(g["loss"] - dom.adjoint_replay_loss(target)) <= 1e-13 * g["loss"]
        up, dn = (dom.adjoint_replay_loss(target, (1 + s, 1.0, 1.0)) for s in (1e-4, -1e-4))
        fd = (up - dn) / 2e-4
        assert abs(g["Dliq"] * dom.params.Dliq - fd) <= 1e-4 * abs(fd)  # as in test_adjoint
