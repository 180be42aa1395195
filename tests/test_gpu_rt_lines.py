"""Register-to-register line passes at the edges of their lengths (GPU).

Every entry of csrc/rt_list.h serves a range of line lengths; the cases take the ends of the
ranges (the longest line of an entry and the first of the next), the z lengths with a direct
entry, ragged sizes (odd widths and depths: the last tile and the last row pair are partial)
and grids with enough lines for the wide forms.  States and gathers against the FP64 oracle
after a few steps from a random state, relative L2 <= 1e-4 as everywhere.
"""
import numpy as np
import pytest

import oracle as O
import qpstd
import workloads as W
from cases import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-4
SCALE = np.array([1.0, 1e-3, 1e-3, 1e-4, 1e-4, 1e-4, 1e-4, 1e-2])


def _shot(kind, nxx, nzz, nt=8, snaps=0, pml=4):
    nx, nz = nxx - 2 * pml, nzz - 2 * pml
    parent = W.parent_model(nx, nz, nxx + nzz, nlayers=3, nanom=1)
    d = W.window_of_parent(kind, parent, 0, nx, pml, nt, 0.0005, 20.0, snaps)
    assert (d["nxx"], d["nzz"]) == (nxx, nzz)
    return d


def _check(kind, nxx, nzz, steps=3):
    visco = kind in (qpstd.VAPS, qpstd.QRTM)
    d = _shot(kind, nxx, nzz)
    rng = np.random.default_rng(nxx * nzz)
    st0 = rng.standard_normal((8, nxx, nzz)) * SCALE[:, None, None]
    if not visco:
        st0[7] = 0.0
    ref_st, ref_g = O.OracleShot(d).steps(st0, 0, steps)
    sh = qpstd.Shot(d)
    sh.set_state(st0.astype(np.float32))
    g, st = sh.advance(0, steps), sh.get_state()
    sh.close()
    for f in range(8 if visco else 7):
        assert rel_l2(st[f], ref_st[f]) < TOL, (f, rel_l2(st[f], ref_st[f]))
    assert rel_l2(g, ref_g) < TOL


@pytest.mark.parametrize("nxx", [11, 80, 81, 129, 193, 256, 385, 512, 513, 641, 769, 1025, 1152, 1281, 1537, 1681, 2049,
                                 2561, 3073, 3601, 4321, 4608])
@pytest.mark.parametrize("kind", [qpstd.APS, qpstd.VAPS])
def test_x_lengths(kind, nxx):
    _check(kind, nxx, 27 if nxx % 2 else 28)


@pytest.mark.parametrize("nzz", [11, 80, 81, 128, 129, 180, 193, 200, 257, 320, 385, 400, 513, 640, 641, 660, 769, 800,
                                 1025, 1153, 1281, 1537, 2049, 2561])
@pytest.mark.parametrize("kind", [qpstd.APS, qpstd.VAPS])
def test_z_lengths(kind, nzz):
    _check(kind, 43 if nzz % 2 else 42, nzz)


@pytest.mark.parametrize("kind,nxx,nzz", [(qpstd.APS, 2449, 181), (qpstd.VAPS, 2450, 200), (qpstd.VAPS, 1219, 320),
                                          (qpstd.APS, 613, 401), (qpstd.VAPS, 190, 1217), (qpstd.APS, 250, 1219),
                                          (qpstd.VAPS, 380, 611), (qpstd.VAPS, 901, 613), (qpstd.APS, 1300, 770)])
def test_wide_forms(kind, nxx, nzz):
    _check(kind, nxx, nzz, steps=2)


@pytest.mark.parametrize("nxx,nzz", [(129, 81), (190, 1217)])
def test_filter_that_changes_every_step(nxx, nzz):
    """Exact transforms along x (Bluestein on the padded entry), image and illumination."""
    d = dict(_shot(qpstd.QRTM, nxx, nzz, nt=12, snaps=3), etas=1e4, etar=1e4)
    obs = O.OracleShot(dict(d, kind=O.VAPS)).model()
    ref_img, ref_ssg, _ = O.OracleShot(d).rtm(obs)
    img, ssg = qpstd.rtm_shot(d, obs)
    assert rel_l2(ssg, ref_ssg) < TOL
    assert rel_l2(img, ref_img) < TOL


@pytest.mark.parametrize("kind", [qpstd.APS, qpstd.VAPS])
@pytest.mark.parametrize("nzz", [27, 29, 30])
def test_state_after_an_overflow(kind, nzz):
    """A clean state brings a shot back whose fields have overflowed, at depths with padded rows."""
    d = _shot(kind, 41, nzz)
    rng = np.random.default_rng(nzz)
    st0 = (rng.standard_normal((8, 41, nzz)) * SCALE[:, None, None]).astype(np.float32)
    sh, new = qpstd.Shot(d), qpstd.Shot(d)
    sh.set_state(np.full((8, 41, nzz), np.nan, dtype=np.float32))
    sh.advance(0, 2)
    for s in (sh, new):
        s.set_state(st0)
    np.testing.assert_array_equal(sh.advance(0, 3), new.advance(0, 3))
    np.testing.assert_array_equal(sh.get_state(), new.get_state())


@pytest.mark.parametrize("nxx,nzz", [(300, 200), (400, 256), (439, 200), (800, 200), (1000, 400)])
def test_spectral_operator_error(nxx, nzz):
    """The (k^2)^0.505 operator of a step against 64 bits, beside a plain FP32 transform with the exact multipliers:
    tables rounded once leave a step at 1.0 - 1.4 times its error, tables built in FP32 at 1.7 - 1.9 (widths that
    transform directly)."""
    import scipy.fft as sf
    d = _shot(qpstd.VAPS, nxx, nzz)
    rng = np.random.default_rng(nxx)
    kx, kz = np.fft.fftfreq(nxx), np.fft.fftfreq(nzz)
    low = np.exp(-2 * (4.0 * np.pi) ** 2 * (kx[:, None] ** 2 + kz[None, :] ** 2))
    st0 = np.zeros((8, nxx, nzz))
    st0[0] = np.fft.ifft2(np.fft.fft2(rng.standard_normal((nxx, nzz))) * low).real
    sh = qpstd.Shot(d)
    sh.set_state(st0.astype(np.float32))
    sh.advance(0, 1)
    st = sh.get_state().astype(np.float64)
    sh.close()
    k = lambda n, h: np.minimum(np.arange(n), n - np.arange(n)) * (2 * W.REF_PI / (n * h))
    sym = (k(nxx, d["dx"])[:, None] ** 2 + k(nzz, d["dz"])[None, :] ** 2) ** 0.505
    ref = np.fft.ifft2(np.fft.fft2(st[0]) * sym).real
    fp32 = sf.ifft2(sf.fft2(st[0].astype(np.complex64)) * sym.astype(np.float32)).real
    assert rel_l2(st[7], ref) < 1.5 * rel_l2(fp32, ref)


@pytest.mark.parametrize("nxx,nzz", [(300, 300), (337, 240), (512, 512), (800, 180)])
def test_illumination_has_no_bias(nxx, nzz):
    """A homogeneous medium whose coefficients are powers of two (their rounding stays out of it): the illumination is
    proportional to the fourth power of the wave speed's inverse, so derivatives short by 5e-8 would show as 2e-7.
    Left by the mean gain that the multipliers take back: 1e-8 a derivative, 4e-8, and as much for rounding."""
    d = _shot(qpstd.ARTM, nxx, nzz, nt=60, snaps=5, pml=20)
    one = np.ones(nxx * nzz, dtype=np.float32)
    d = dict(d, vp=2048 * one, rho=256 * one, bbx=one / 256, bbz=one / 256, dt=2.0 ** -10)
    obs = np.zeros((d["nt"], len(d["gxg"])))
    _, ref, _ = O.OracleShot(d).rtm(obs)
    _, ssg = qpstd.rtm_shot(d, obs)
    ref, ssg = np.asarray(ref, dtype=np.float64).ravel(), ssg.astype(np.float64).ravel()
    bias = (ssg * ref).sum() / (ref * ref).sum() - 1
    assert abs(bias) < 8e-8, bias
