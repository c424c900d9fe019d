"""Batches of many domains: a stencil CTA finds its tile's
domain in rounds of 64 parts, one round to 64 domains, two to 4096."""
from __future__ import annotations

import pytest

import mumatscale_b200 as M
from mumatscale_b200 import workloads as W
from digests import mismatches, state_digests

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 65, 130, 1030])
def test_every_domain_is_found(built, cuda_device, tmp_path, n):
    f = tmp_path / "d.in"
    decks = W.ensemble(n, seed=9, edges=(8, 11, 20))
    ps = []
    for d in decks:
        f.write_text(d)
        ps.append(M.read_deck(f))
    with M.Batch(ps, precision=M.PREC_F32) as b:
        b.set_stencil_tile(1, 3)
        b.step(25)
        for i in {0, 1, 31, 32, 33, 62, 63, 64, 65, n // 2, 1022, 1023, 1024, n - 2, n - 1} & set(range(n)):
            with M.Domain(ps[i], precision=M.PREC_F32) as d:
                d.step(25)
                assert mismatches(state_digests(b.domains[i]), state_digests(d)) == [], i
