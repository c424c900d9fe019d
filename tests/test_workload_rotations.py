"""Rotations of the seeded workloads are the same on every host."""
from __future__ import annotations

import math
from fractions import Fraction

import numpy as np

from mumatscale_b200 import workloads as W


def test_norm_rounds_once_per_component():
    q = W.random_quaternions(np.random.default_rng(4), 3000) * np.array([1.0, 1e-3, 7.0, 1e5])
    for row in q:
        s = 0.0
        for v in row:
            s = float(Fraction(v) ** 2 + Fraction(s))
        assert W._norm(row) == math.sqrt(s)
