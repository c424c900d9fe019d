"""Steps that leave tiles at rest out (the tile map) against steps that visit
every tile: a z-slab split, or the same domain in tiles too few for a map.  Both
must agree bit for bit in every state a tile can rest in or be woken from.  Each
test asserts that the map is on and that tiles were left out, so that it cannot
pass on the kernel without one."""
from __future__ import annotations

import numpy as np
import pytest

import mumatscale_b200 as M
from mumatscale_b200 import workloads as W
import test_active_tiles as T

pytestmark = pytest.mark.gpu

FIELDS = T.FIELDS
DIMS = (150, 100, 80)  # ragged in x and y at both tile widths
MAP_MIN = 148 * 4      # a lone domain's map is on above this many tiles
#: (cells per thread, planes): 1040, 1053 and 780 tiles, ragged in z too, and
#: a tile whose last layer is one plane
TILES = [(1, 5), (2, 3), (2, 4)]


def _tiles(cpt, zc, dims=DIMS):
    return -(-dims[0] // (32 * cpt)) * -(-dims[1] // 8) * -(-dims[2] // zc)


def _params(tmp_path, monkeypatch, kind, dims=DIMS):
    monkeypatch.setattr(T, "DIMS", dims)
    return T._params(tmp_path, kind)


def _setup(doms, kind, dims=DIMS):
    _, _, _, planes, thr = T.KINDS[kind]
    rot = np.stack([W.quat_to_rotmat(q).ravel() for q in W.random_quaternions(np.random.default_rng(1), 6)])
    gr = np.zeros(tuple(n + 2 for n in dims[::-1]), dtype=np.int32)
    gr[1:planes + 1, 1:-1, 1:dims[0] // 2 + 1] = 1
    gr[1:planes + 1, 1:-1, dims[0] // 2 + 1:-1] = 2
    for d in doms:
        d.set_sites(T.SITES, np.array(thr, dtype=np.float32))
        d.set_site_orientations(T.SITES, rot[:4])
        if planes:
            d.set_grains(rot[4:])
            d.upload("gr", gr)
            d.upload("fs", (gr > 0).astype(np.float64))


def _same(a, b, at, fields=FIELDS):
    for f in fields:
        assert np.array_equal(a.download(f), b.download(f)), (at, f)


def _disturb(doms):
    """Somewhere far from every front."""
    ce = doms[-1].download("ce")
    ce[60, 75, 100:104] *= 1.01
    for d in doms:
        d.upload("ce", ce)


def _left_out(counts, kind):
    """Tiles rested, and in the kinds whose temperature or fronts reach resting
    tiles some of those woke."""
    assert max(counts) > 0, counts
    if kind != "cooling":
        assert min(counts) < max(counts), counts


@pytest.mark.parametrize("kind", list(T.KINDS))
@pytest.mark.parametrize("prec", [M.PREC_F64, M.PREC_F32])
@pytest.mark.parametrize("cpt,zc", TILES)
def test_map_equals_visiting_every_tile(built, cuda_device, tmp_path, monkeypatch, kind, prec, cpt, zc):
    p = _params(tmp_path, monkeypatch, kind)
    with M.Domain(p, precision=prec) as dom, M.SlabGroup(p, 2, precision=prec) as every:
        dom.set_stencil_tile(cpt, zc)
        assert dom.test_tile_map()[0] == _tiles(cpt, zc) > MAP_MIN
        assert every.slabs[0].test_tile_map() == (0, 0)
        _setup((dom, every), kind)
        counts = []
        for part, n in enumerate((1, 2, 37, 60, 80, 1, 90)):
            if part == 4:
                before = dom.test_tile_map()[1]
                _disturb((dom, every))
                dom.step(1)
                every.step(1)
                assert dom.test_tile_map()[1] == 0  # an upload wakes every tile
                assert before > 0
            got = dom.step_reduce(n)
            every.step(n)
            counts.append(dom.test_tile_map()[1])
            _same(dom, every, part)
            # sums of at most 1.2 million terms in [0, 1], in different orders
            assert abs(got - every.reduce("fs_fraction")) <= 1e-12
        assert dom.num_grains == every.num_grains
        _left_out(counts, kind)


@pytest.mark.parametrize("kind", list(T.KINDS))
@pytest.mark.parametrize("prec", [M.PREC_F64, M.PREC_F32])
def test_map_in_a_batch(built, cuda_device, tmp_path, monkeypatch, kind, prec):
    """Two domains of different sizes; the smaller, whose fronts
    soon reach all of its tiles, has a map only in a batch."""
    small = T.DIMS
    p, q = _params(tmp_path, monkeypatch, kind), _params(tmp_path, monkeypatch, kind, small)
    with M.Batch([p, q], precision=prec) as b, M.SlabGroup(p, 2, precision=prec) as e0, \
            M.SlabGroup(q, 2, precision=prec) as e1:
        b.set_stencil_tile(2, 3)
        _setup((b.domains[0], e0), kind)
        _setup((b.domains[1], e1), kind, small)
        counts = [[], []]
        for part, n in enumerate((1, 50, 70, 1, 90)):
            if part == 2:
                _disturb((b.domains[0], e0))
            b.step(n)
            for i, (dom, every) in enumerate(zip(b.domains, (e0, e1))):
                every.step(n)
                _same(dom, every, (part, i))
                assert abs(dom.reduce("fs_fraction") - every.reduce("fs_fraction")) <= 1e-12
                counts[i].append(dom.test_tile_map()[1])
        assert [d.test_tile_map()[0] for d in b.domains] == [_tiles(2, 3), _tiles(2, 3, small)]
        _left_out(counts[0], kind)


@pytest.mark.parametrize("prec", [M.PREC_F64, M.PREC_F32])
def test_map_with_curvature_and_between_other_calls(built, cuda_device, tmp_path, monkeypatch, prec):
    """Curvature (which slabs refuse), a record, a checkpoint, a new tile and
    tuning between steps: against the same calls on tiles too large for a map."""
    p = _params(tmp_path, monkeypatch, "cooling")
    p.tip_curv = 1
    p.gibbs_coef = W.GIBBS
    with M.Domain(p, precision=prec) as dom, M.Domain(p, precision=prec) as every:
        dom.set_stencil_tile(1, 5)
        every.set_stencil_tile(2, 64)
        assert every.test_tile_map() == (0, 0)
        _setup((dom, every), "cooling")
        ck = str(tmp_path / "tiles.ckpt")
        for part in range(6):
            for d in (dom, every):
                if part == 1:
                    d.adjoint_record(20, 10)
                if part == 2:
                    d.adjoint_release()
                    d.checkpoint_save(ck)
                if part == 4:
                    d.checkpoint_load(ck)
                d.step(35)
            if part == 3:
                dom.set_stencil_tile(2, 3)
            if part == 4:
                dom.autotune(reps=1)
                dom.set_stencil_tile(1, 4)
            _same(dom, every, part)
            if part != 4 and part != 3:
                assert dom.test_tile_map()[1] > 0, part


@pytest.mark.parametrize("prec", [M.PREC_F64, M.PREC_F32])
def test_map_with_resumed_steps(built, cuda_device, tmp_path, monkeypatch, prec):
    """More grains between two refills than a rank has orientations drawn ahead:
    the step that runs out resumes at activation."""
    p = _params(tmp_path, monkeypatch, "cooling")
    rng = np.random.default_rng(2)
    cells = np.unique(rng.integers(0, 150 * 100 * 79, 900))
    xyz = np.stack([cells % 150, cells // 150 % 100, cells // 15000], 1).astype(np.int32)
    # T = Tliq - 2 falling: a few of them in every step
    per_step = 400 * p.ts_delt
    thr = (2.0 + per_step * rng.uniform(1, 200, len(cells))).astype(np.float32)
    with M.Domain(p, precision=prec) as dom, M.Domain(p, precision=prec) as every:
        dom.set_stencil_tile(1, 5)
        every.set_stencil_tile(2, 64)
        for d in (dom, every):
            d.set_sites(xyz, thr)
        for n in (1, 250, 20):
            dom.step(n)
            every.step(n)
            assert dom.test_tile_map()[0] == _tiles(1, 5)
            _same(dom, every, n)
        assert dom.num_grains == every.num_grains > 600


@pytest.mark.parametrize("prec", [M.PREC_F64, M.PREC_F32])
def test_map_without_sites(built, cuda_device, tmp_path, monkeypatch, prec):
    """A microstructure that only grows and melts."""
    p = _params(tmp_path, monkeypatch, "heating")
    planes = T.KINDS["heating"][3]
    rot = np.stack([W.quat_to_rotmat(q).ravel() for q in W.random_quaternions(np.random.default_rng(1), 1)])
    gr = np.zeros(tuple(n + 2 for n in DIMS[::-1]), dtype=np.int32)
    gr[1:planes + 1, 1:-1, 1:-1] = 1
    with M.Domain(p, precision=prec) as dom, M.SlabGroup(p, 2, precision=prec) as every:
        dom.set_stencil_tile(2, 3)
        for d in (dom, every):
            d.set_grains(rot)
            d.upload("gr", gr)
            d.upload("fs", (gr > 0).astype(np.float64))
        counts = []
        for n in (1, 60, 90, 60):
            dom.step(n)
            every.step(n)
            counts.append(dom.test_tile_map()[1])
            _same(dom, every, n)
        _left_out(counts, "heating")


@pytest.mark.parametrize("kind", ["cooling", "heating", "laser"])
@pytest.mark.parametrize("prec", [M.PREC_F64, M.PREC_F32])
def test_slabs_with_wide_default_tiles(built, cuda_device, tmp_path, monkeypatch, kind, prec):
    """Slabs large enough for two cells per thread by default, against one
    domain with one."""
    dims = (250, 128, 126)
    p = _params(tmp_path, monkeypatch, kind, dims)
    with M.Domain(p, precision=prec) as dom, M.SlabGroup(p, 2, precision=prec) as every:
        dom.set_stencil_tile(1, 16)
        assert every.slabs[0].stencil_tile() == (2, 0)
        _setup((dom, every), kind, dims)
        for n in (1, 2, 67, 70):
            dom.step(n)
            every.step(n)
            _same(dom, every, n)
