"""The step leaves stencil tiles at rest out; a z-slab split visits every tile.
Both must agree bit for bit in every state a tile can rest in or be woken
from: melt no solute has reached, solid below its kept-solid limit, a limit
that the temperature crosses, nucleation and capture in a resting tile, an
upload, faces without mold."""
from __future__ import annotations

import numpy as np
import pytest

import mumatscale_b200 as M
from mumatscale_b200 import workloads as W

pytestmark = pytest.mark.gpu

FIELDS = ("ce", "cl", "fs", "gr", "dc", "temperature")
DIMS = (150, 20, 40)  # ragged in x and y at both tile widths
SITES = np.array([[3, 3, 2], [140, 12, 3], [70, 9, 35], [71, 10, 36]], dtype=np.int32)
LASER = """AnalyticalThermal 1
LaserPower 40
LaserSpeed 0.5
LaserSpotSize 20e-6
LaserAbsorption 0.4
LaserHatchSpacing 8e-6
LaserStartLocation -1e-5 5e-6 34e-6
NoOfLayers 1
NoOfTracks 4
SubInitialTemp 300
ThermalConductivity 100
SpecificHeat 395
Density 7594.94
"""
#: (temperature lines, faces, time step factor, solid planes, undercoolings of the sites)
KINDS = {
    "cooling": (f"InitialTemperature {W.T_LIQ - 2!r}\nGradient 0\nVelocity 0\nCoolingRate 400\n", "1 1 1 1 1 1", 1, 0,
                (0.5, 2.2, 1.0, 2.6)),
    # solid that stays, then passes its limit, then melts
    "heating": (f"InitialTemperature {W.T_SOL - 3!r}\nGradient 0\nVelocity 0\nCoolingRate -80000\n", "1 1 1 1 1 1", 1,
                12, (500.0,) * 4),
    "gradient, open x and y": (f"InitialTemperature {W.T_LIQ - 3!r}\nGradient 6e4\nVelocity 2e-3\nCoolingRate 0\n",
                               "0 0 0 0 1 1", 1, 6, (0.5, 1.5, 0.9, 2.0)),
    "laser": (LASER, "1 1 1 1 1 1", 4, 34, (3.0,) * 4),
}


def _params(tmp_path, kind):
    temp, faces, slower, _, _ = KINDS[kind]
    dx = 1e-6
    f = tmp_path / "tiles.in"
    f.write_text(f"""BaseFileName tiles
NSubblocks 1 1 2
NCellsPerSB {DIMS[0]} {DIMS[1]} {DIMS[2] // 2}
FaceCtrl {faces}
CellSize {dx!r}
FSGrow 0.66
TimeStep {W.FOURIER / slower * dx * dx / W.D_LIQ!r}
RandSeedVal 5
LiquidusTemp {W.T_LIQ!r}
SolidusTemp {W.T_SOL!r}
Cinit {W.C0!r}
m_solute0 0 0 {W.SLOPE!r}
part_coef0 0 0 {W.K_PART!r}
Dsol {W.D_SOL!r}
Dliq {W.D_LIQ!r}
MaxTotGrains 1000
GNOriented 1
{temp}""")
    return M.read_deck(f)


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("prec,cpt,zchunk", [(M.PREC_F64, 1, 5), (M.PREC_F64, 2, 3), (M.PREC_F32, 1, 8),
                                             (M.PREC_F32, 2, 4)])
def test_steps_equal_visiting_every_tile(built, cuda_device, tmp_path, kind, prec, cpt, zchunk):
    p = _params(tmp_path, kind)
    _, _, _, planes, thr = KINDS[kind]
    rot = np.stack([W.quat_to_rotmat(q).ravel() for q in W.random_quaternions(np.random.default_rng(1), 6)])
    shape = tuple(n + 2 for n in DIMS[::-1])
    gr = np.zeros(shape, dtype=np.int32)
    gr[1:planes + 1, 1:-1, 1:76] = 1
    gr[1:planes + 1, 1:-1, 76:-1] = 2
    with M.Domain(p, precision=prec) as dom, M.SlabGroup(p, 2, precision=prec) as every:
        dom.set_stencil_tile(cpt, zchunk)
        for d in (dom, every):
            d.set_sites(SITES, np.array(thr, dtype=np.float32))
            d.set_site_orientations(SITES, rot[:4])
            if planes:
                d.set_grains(rot[4:])
                d.upload("gr", gr)
                d.upload("fs", (gr > 0).astype(np.float64))
        for part, n in enumerate((1, 2, 37, 60, 80, 1, 90)):
            if part == 4:  # a disturbance far from every front
                ce = every.download("ce")
                ce[30, 15, 100:104] *= 1.01
                dom.upload("ce", ce)
                every.upload("ce", ce)
            got = dom.step_reduce(n)
            every.step(n)
            for f in FIELDS:
                assert np.array_equal(dom.download(f), every.download(f)), (part, f)
            # sums of at most 120,000 terms in [0, 1], in different orders
            assert abs(got - every.reduce("fs_fraction")) <= 1e-12
        assert dom.num_grains == every.num_grains
