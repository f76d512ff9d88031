"""The sweep at the edges of its tiles, against the oracle (GPU): velocity
counts around whole 32- and 16-velocity segments, element counts that leave a
ragged last block, every edge kind and mass matrix, and meshes whose blocks
have so wide a halo that one tile buffer only fits, or no 128-element tile.

Tolerances as in test_gpu_parity.py: FP64 1e-10 (roundoff over a few steps),
FP32 against the FP64 oracle 1e-5."""
import numpy as np
import pytest

from dgbgk import cavity_case, channel_case
from helpers import rel_l2
from test_gpu_parity import TOL64, compare_macros, pair

pytestmark = pytest.mark.gpu


def tol(prec):
    return TOL64 if prec == 64 else 1e-5


@pytest.mark.parametrize("nr,nt", [(3, 5), (2, 8), (4, 8), (3, 11), (7, 9), (8, 8), (5, 13)])
@pytest.mark.parametrize("prec,tile", [(64, 64), (64, 128), (32, 64), (32, 128)])
def test_velocity_and_block_remainders(nr, nt, prec, tile):
    # V = 15, 16, 32, 33, 63, 64, 65; 98 elements (a ragged block of 34 or 98)
    s, o, _ = pair(cavity_case(7, nr, nt, mach=0.3, kn=0.1), prec=prec, tile_elems=tile)
    r, q = s.advance(3), o.advance(3)
    assert rel_l2(s.get_state(), o.get_state()) <= tol(prec)
    assert rel_l2(r["res_linf"], q["res_linf"]) <= (1e-9 if prec == 64 else 1e-4)
    assert rel_l2(r["res_l2"], q["res_l2"]) <= (1e-9 if prec == 64 else 1e-4)


@pytest.mark.parametrize("sides", ["outflow", "freestream", "wall"])
@pytest.mark.parametrize("immat,alpha", [(1, 1.0), (0, 1.0), (1, 0.9), (0, 0.9)])
@pytest.mark.parametrize("prec", [64, 32])
def test_edge_kinds(sides, immat, alpha, prec):
    c = channel_case(-2.0, 4.0, -2.0, 2.0, 21, 15, 12, 12, mach=2.0, kn=0.05, obstacle_side=1.0, sides=sides)
    c.immat, c.alpha = immat, alpha
    s, o, _ = pair(c, prec=prec)
    r, q = s.advance(4), o.advance(4)
    assert rel_l2(s.get_state(), o.get_state()) <= tol(prec)
    # the largest increment includes those of nodes on inflow sides
    assert rel_l2(r["res_linf"], q["res_linf"]) <= (1e-9 if prec == 64 else 1e-4)
    assert rel_l2(r["res_l2"], q["res_l2"]) <= (1e-9 if prec == 64 else 1e-4)


def sheets(case, k):
    """k disconnected copies of the case's mesh at the same place: the element
    order interleaves them, so a block's halo grows with k."""
    m = case.mesh
    E, NP = m.nelem, m.npoin
    m.intma = np.concatenate([m.intma + NP * i for i in range(k)])
    m.coord = np.concatenate([m.coord] * k)
    b = [m.bsido.copy() for _ in range(k)]
    for i in range(k):
        b[i][:, :2] += NP * i
        b[i][:, 2] += E * i
    m.bsido = np.concatenate(b)
    if m.wall_velocity is not None:
        m.wall_velocity = np.concatenate([m.wall_velocity] * k)
    return case


@pytest.mark.parametrize("k", [6, 24, 64])
@pytest.mark.parametrize("prec,tile", [(64, 0), (64, 64), (64, 128), (32, 0), (32, 64), (32, 128)])
def test_wide_halos(k, prec, tile):
    s, o, _ = pair(sheets(cavity_case(6, 4, 9, mach=0.3, kn=0.1), k), prec=prec, tile_elems=tile)
    s.advance(3)
    o.advance(3)
    assert rel_l2(s.get_state(), o.get_state()) <= tol(prec)
    compare_macros(s, o, tol(prec))
    # the halo does grow; past what a 128-element tile can hold, 64 are taken
    assert s.info()["max_halo"] >= min(2 * k, 100)
    assert s.info()["tile_elems"] in (64, 128)


@pytest.mark.parametrize("nt", [8, 9, 10, 13])
def test_default_fp64_tile_follows_the_tile_count(nt):
    # 2048 elements: 16 blocks of 128 at V = 16 * nt, so 128, 144, 160 and 208
    # tiles; a chip with more SMs than tiles takes 64 elements
    import torch

    s, o, _ = pair(cavity_case(32, 16, nt, mach=0.3, kn=0.1))
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    assert s.info()["tile_elems"] == (64 if 16 * nt <= nsm else 128)
    s.advance(2), o.advance(2)
    assert rel_l2(s.get_state(), o.get_state()) <= TOL64


@pytest.mark.parametrize("immat", [1, 0])
@pytest.mark.parametrize("prec,n", [(64, 12), (64, 17), (32, 18)])
def test_specular_chains_of_corner_elements(prec, n, immat):
    # ALPHA < 1: a corner element's velocities wait on one another in chains of
    # several levels, taken level by level
    c = cavity_case(6, n, n, mach=0.4, kn=0.5)
    c.immat, c.alpha = immat, 0.9
    s, o, _ = pair(c, prec=prec)
    r, q = s.advance(4), o.advance(4)
    assert rel_l2(s.get_state(), o.get_state()) <= tol(prec)
    assert rel_l2(r["res_l2"], q["res_l2"]) <= (1e-9 if prec == 64 else 1e-4)
