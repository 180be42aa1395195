"""Every wide form of csrc/rt_list.h, and the layouts next to the entries' reach (GPU).

A pass runs an entry's wide form when its grid has 152 CTAs or more, so each wide form takes
enough lines: x entries by depth, z entries by width.  Windows wider than 4608 or deeper than 3072
points keep the Stockham passes in that direction: x on the entries over z on Stockham plans (fields
and half spectra row by row) and both on Stockham plans.  States and gathers against the FP64 oracle
after two steps from a random state, relative L2 <= 1e-4 as everywhere.
"""
import numpy as np
import pytest

import oracle as O
import qpstd
from cases import rel_l2
from test_gpu_rt_lines import SCALE, TOL, _check, _shot

pytestmark = pytest.mark.gpu
KINDS = [qpstd.APS, qpstd.VAPS]


# the longest line of each x entry, 152 CTAs deep (lines of up to 128 points would need windows
# deeper than any z plan takes)
@pytest.mark.parametrize("nxx,nzz", [(192, 1214), (256, 1213), (384, 607), (512, 606), (640, 609), (768, 611),
                                     (1024, 605), (1152, 606), (1280, 607), (1536, 606), (1680, 605), (2048, 607)])
@pytest.mark.parametrize("kind", KINDS)
def test_wide_x_entries(kind, nxx, nzz):
    _check(kind, nxx, nzz, steps=2)


# each z entry below 512 points or its own length, 152 CTAs wide
@pytest.mark.parametrize("nxx,nzz", [(2419, 180), (2418, 200), (2420, 256), (1211, 320), (1212, 400), (607, 512),
                                     (606, 640), (607, 660), (608, 800), (2421, 79), (2422, 127), (1213, 191),
                                     (605, 255), (606, 383), (609, 511)])
@pytest.mark.parametrize("kind", KINDS)
def test_wide_z_entries(kind, nxx, nzz):
    _check(kind, nxx, nzz, steps=2)


# depths with an entry of their own for the constant-Q step and no quick form (acoustic: padded); a
# last group with one row, with a full pair
@pytest.mark.parametrize("nzz", [392, 420, 432, 448, 450, 480, 500, 540, 560, 576, 588, 600, 630, 648, 672, 700, 720, 768,
                                 784, 810, 840, 864, 882, 896, 900, 960, 980, 1000, 1024, 1050, 1080, 1120, 1296, 1344,
                                 1600, 1680, 1728, 1792, 1800])
@pytest.mark.parametrize("kind,nxx", [(qpstd.APS, 41), (qpstd.VAPS, 41), (qpstd.VAPS, 42)])
def test_exact_depths(kind, nxx, nzz):
    _check(kind, nxx, nzz, steps=2)


# x on an entry and z on a Stockham plan; both on Stockham plans
@pytest.mark.parametrize("nxx,nzz", [(60, 3200), (61, 3201), (70, 3074), (5040, 42), (5040, 60)])
@pytest.mark.parametrize("kind", KINDS)
def test_lines_beyond_the_entries(kind, nxx, nzz):
    _check(kind, nxx, nzz, steps=2)


@pytest.mark.parametrize("nxx,nzz", [(60, 3201), (5040, 42)])
@pytest.mark.parametrize("kind", [qpstd.ARTM, qpstd.QRTM])
def test_images_beyond_the_entries(kind, nxx, nzz):
    d = _shot(kind, nxx, nzz, nt=10, snaps=3)
    obs = O.OracleShot(dict(d, kind=O.VAPS if kind == qpstd.QRTM else O.APS)).model()
    ref_img, ref_ssg, _ = O.OracleShot(d).rtm(obs)
    img, ssg = qpstd.rtm_shot(d, obs)
    assert rel_l2(ssg, ref_ssg) < TOL
    assert rel_l2(img, ref_img) < TOL


@pytest.mark.parametrize("nxx,nzz", [(60, 3201), (5040, 42)])
def test_lowrank_beyond_the_entries(nxx, nzz):
    d = _shot(qpstd.VAPS, nxx, nzz)
    f = qpstd.lowrank_decompose(nxx, nzz, d["dx"], d["dz"], d["dt"], d["vp"], d["tao"], d["gam"], 3, 3)
    rng = np.random.default_rng(nxx)
    st0 = rng.standard_normal((8, nxx, nzz)) * SCALE[:, None, None]
    ref_st, ref_g = O.OracleShot(dict(d, lowrank=f)).steps(st0, 0, 2)
    sh = qpstd.Shot(d)
    sh.set_lowrank(f)
    sh.set_state(st0.astype(np.float32))
    g, st = sh.advance(0, 2), sh.get_state()
    sh.close()
    for k in range(8):
        assert rel_l2(st[k], ref_st[k]) < TOL, (k, rel_l2(st[k], ref_st[k]))
    assert rel_l2(g, ref_g) < TOL
