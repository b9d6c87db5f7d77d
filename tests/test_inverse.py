"""Division-step inversion and the sums over lane quads: the arithmetic on the host, the kernels on the GPU."""
import os
import random

import numpy as np
import pytest

import oracle_lib as ora
import pyref
from pyref import R, fr_array
from test_host_arith import ROOT, _run

G = np.frombuffer(pyref.g1_bytes((pyref.GX, pyref.GY)), dtype=np.uint8).copy()


def test_division_step_inverse_matches_oracle_on_host():
    _run(os.path.join(ROOT, "tests", "host", "inverse_host_check.cpp"))


@pytest.fixture(scope="module")
def be():
    from project_b200 import Backend

    b = Backend(0)
    yield b
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("count", [1, 2, 1023, 1024, 1025])  # one CTA per point up to 1024 points
def test_same_base_batch_sizes(be, count):
    rng = random.Random(count)
    sparse = [0, 1, 255, 1 << 248, 0xFF << 120, (1 << 255) % R, R - 1]  # single windows, neighbouring ones empty
    scalars = (sparse + pyref.rand_fr(rng, count))[:count] if count > 2 else pyref.rand_fr(rng, count)
    assert np.array_equal(be.g1_mul_same_base(G, fr_array(scalars)), ora.g1_mul_same_base(G, fr_array(scalars)))


@pytest.mark.gpu
def test_same_base_of_order_three(be):
    """(0, 2) has order 3: every sum of the tree meets coinciding, opposite and vanishing operands."""
    x = bytes(48)
    point, opposite = x + (2).to_bytes(48, "little"), x + (pyref.P - 2).to_bytes(48, "little")
    rng = random.Random(3)
    scalars = list(range(12)) + [3 << 248, (1 << 16) + 2, (1 << 200) + 1, R - 1] + pyref.rand_fr(rng, 40)
    got = be.g1_mul_same_base(np.frombuffer(point, dtype=np.uint8).copy(), fr_array(scalars))
    want = [(bytes(96), point, opposite)[s % 3] for s in scalars]
    assert [bytes(p) for p in got] == want


@pytest.mark.gpu
@pytest.mark.parametrize("log2n", [2, 3, 10, 12, 18, 19])  # one CTA, ragged CTAs, one and four quartets per thread
def test_weights_through_the_cta_inversion(be, log2n):
    x = fr_array([0x123456789ABCDEF0123456789 + log2n])[0]
    assert np.array_equal(be.bary_weights(log2n, x).download(), ora.bary_weights(x, 1 << log2n))


def test_host_point_arithmetic():
    _run(os.path.join(ROOT, "tests", "host", "host_g1_check.cpp"))
