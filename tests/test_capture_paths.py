"""Capture in small domains, eight lanes per list entry, against a batch, where a
thread takes an entry: from lists that leave lanes idle to lists that every warp
goes through several rounds of."""
from __future__ import annotations

import numpy as np
import pytest

import mumatscale_b200 as M
from mumatscale_b200 import workloads as W
import test_active_tiles as T
from digests import mismatches, state_digests

pytestmark = pytest.mark.gpu

ROUND = 148 * 3 * 256 // 8  # entries in flight at once


def _list_length(dom):
    s = dom.download("gr") > 0
    near = np.zeros_like(s)
    for ax in range(3):
        for sh in (1, -1):
            near |= np.roll(s, sh, ax)
    return int((near & ~s)[1:-1, 1:-1, 1:-1].sum())


@pytest.mark.parametrize("prec", [M.PREC_F64, M.PREC_F32])
@pytest.mark.parametrize("dims,sites", [((64, 64, 64), 20000), ((63, 61, 66), 1500)])
def test_capture_at_every_list_length(built, cuda_device, tmp_path, monkeypatch, prec, dims, sites):
    monkeypatch.setattr(T, "DIMS", dims)
    p = T._params(tmp_path, "cooling")
    p.initialTemperature = W.T_LIQ - 3.0
    p.maxTotalGrains = 40000
    p.maxGrainDensity = 4e17  # orientations drawn ahead for every cell
    p.site_setup = 1
    rng = np.random.default_rng(3)
    cells = np.unique(rng.integers(0, dims[0] * dims[1] * dims[2], sites))
    xyz = np.stack([cells % dims[0], cells // dims[0] % dims[1], cells // (dims[0] * dims[1])], 1).astype(np.int32)
    thr = np.maximum(0.05, rng.normal(2.0, 0.5, len(cells))).astype(np.float32)
    rot = np.stack([W.quat_to_rotmat(q).ravel() for q in W.random_quaternions(rng, len(cells))])
    lengths = []
    with M.Domain(p, precision=prec) as dom, M.Batch([p], precision=prec) as b:
        for d in (dom, b.domains[0]):
            d.set_sites(xyz, thr)
            d.set_site_orientations(xyz, rot)
        for n in (1, 2, 47, 60, 40, 150, 400, 300):
            dom.step(n)
            b.step(n)
            assert mismatches(state_digests(b.domains[0]), state_digests(dom)) == [], dom.timestep
            lengths.append(_list_length(dom))
    assert max(lengths) > 3 * ROUND, lengths
    if sites < 2000:
        assert min(lengths) < ROUND, lengths
