"""The FP64 temperature contraction (tiles of 64 x cells by 128 rows, the halo
columns apart where they would need another column of tiles) against the
quadrature summed node by node in 64 bits."""
from __future__ import annotations

import numpy as np
import pytest

import mumatscale_b200 as M
from mumatscale_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _quadrature(p, ts):
    """temperature.c:62-123 for a single track, on the halo'd grid."""
    gx, gy, gz = p.grid
    t = ts * p.ts_delt
    alpha, s = p.lthcon / (p.rho * p.lcp), p.lsd / (2.0 * 1.414)
    ldt = 20 * alpha / p.lv / p.lv / 400
    front = p.lab * (0.0 if t < 1e-4 else p.lpow) * alpha / (5.568328 * p.lthcon)
    lx = (np.arange(gx + 2) + 0.5) * p.cellSize - (p.x0 + t * p.lv)
    ly = (np.arange(gy + 2) + 0.5) * p.cellSize - p.y0
    z = (np.arange(gz + 2) + 0.5) * p.cellSize
    total = np.zeros((gz + 2, gy + 2, gx + 2))
    for i in range(400):
        lt = (0.5 + i) * ldt
        a = s * s + 4 * alpha * lt
        flat = ((lx + p.lv * lt) ** 2)[None, None, :] + (ly ** 2)[None, :, None]
        deep = ((z - p.z0) ** 2)[:, None, None] / (4 * alpha * lt)
        total += ldt * np.exp(-flat / a - deep) / (np.sqrt(alpha * lt) * a)
    return np.where((z <= p.z0 + p.cellSize)[:, None, None], p.liniT + front * total, 0.0)


@pytest.mark.parametrize("dims", [(64, 7, 5), (63, 14, 14), (62, 6, 14), (65, 30, 9), (1, 3, 2), (128, 126, 3)])
def test_temperature_of_ragged_domains(built, cuda_device, tmp_path, dims):
    f = tmp_path / "am.in"
    f.write_text(W.am_track(dims, 1e-6))
    p = M.read_deck(f)
    p.x0, p.z0 = -20e-6, (dims[2] - 1) * 1e-6  # the top of the substrate inside the domain
    with M.Domain(p, precision=M.PREC_F64) as dom:
        dom.step(12)
        got, want = dom.download("temperature"), _quadrature(p, 12)
    assert want.max() > 400  # the source is on
    # 400 terms, each with the rounding of its exponentials and products
    assert np.abs(got - want).max() <= 1e-12 * want.max()
