"""ME-AWENO passes at the edges of their tiles: the default build (two points
a thread) against the FP64 run of the same model.

The x pass has tiles of 58 points x 8 rows, the y and z passes of 26 points x
16 columns, taken in pairs of rows or columns, so sizes run over one tile, one
point more, odd remainders and the smallest model the scheme accepts.  The
bound is the distance the same algorithm in FP32 with every operation rounded
keeps from FP64 (the exact build's), doubled.
"""

import numpy as np
import pytest

import parity_util as pu
from cgfdm import Session, cases


def _run(nx, ny, nz, source, tmp):
    c = cases.halfspace_case(NX=nx, NY=ny, NZ=nz, nPML=5, steps=24, n_stations=3, depth_m=300.0, courant=0.4)
    c.fault = []
    c.gauss_hill = 1
    at = (nx // 2, ny // 2, nz // 2)
    if source == "ricker":
        c.ricker_point = at + (8.0,)
    else:
        c.double_couple = dict(X=at[0], Y=at[1], Z=at[2], strike=40.0, dip=55.0, rake=70.0, Mw=8.0, duration=0.6)
    c.stations = [(at[0], at[1], nz - 1), (at[0] - 3, at[1] + 3, nz // 2), (nx - 1, ny - 1, nz - 1)]
    return cases.write_case(c, str(tmp / "run"), scheme="SCFDM")


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz,source", [(8, 7, 8, "couple"), (26, 26, 26, "ricker"), (27, 25, 27, "couple"),
                                             (58, 16, 13, "couple"), (59, 17, 15, "ricker"), (33, 53, 9, "couple"),
                                             (15, 9, 53, "couple")])
def test_passes_match_fp64(tmp_path, nx, ny, nz, source):
    d = _run(nx, ny, nz, source, tmp_path)
    err = {}
    with Session(d) as s:
        st64, _, W64 = s.run_precise(24, bits=64, wavefield=True)
    assert np.abs(W64[3:-3, 3:-3, 3:-3]).max() > 0
    for flavor in ("fast", "exact"):
        with Session(d, flavor=flavor) as s:
            s.run(24)
            W, st = s.wavefield(), s.stations()
        # momentum and strain have their own scales; halo layers are compared too
        err[flavor] = pu.errors_by_quantity(W, W64, st, st64)
    print(f"{nx}x{ny}x{nz} {source}: " + ", ".join(f"{q} fast {err['fast'][q]:.2e} exact {e:.2e}"
                                                   for q, e in err["exact"].items()))
    for q, e in err["exact"].items():
        assert err["fast"][q] <= 2 * e + 1e-7, q


def _waves(shape, amp, rng):
    z, y, x = np.meshgrid(*[np.arange(n) for n in shape], indexing="ij")
    w = np.zeros(shape + (9,))
    for f in range(9):
        for _ in range(4):
            k = rng.normal(size=3)
            k *= 2 * np.pi / (np.linalg.norm(k) * rng.uniform(8, 20))
            w[..., f] += amp[f] * rng.normal() * np.cos(k[0] * x + k[1] * y + k[2] * z + rng.uniform(0, 6.3))
    return w.astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [1, 2, 3, 8, 16])
def test_passes_scale_with_the_field(tmp_path, shift):
    """The scheme is homogeneous but for the 1e-6 in the smoothness indicators:
    a field 2^shift times as large stays finite and gives 2^shift times the
    result.  Momentum of 5e8 gives indicators of 1e16 to 1e17; three more
    powers of two take them past 9e18, where the reciprocal of an unscaled
    square is subnormal.  Strains of 40 have indicators of 1 at least almost
    everywhere, so the 1e-6 moves a weight by 1e-6 there; the states' spread
    over the sub-stencils is a tenth of the field or less."""
    d = _run(37, 29, 31, "ricker", tmp_path)
    out = []
    with Session(d) as s:
        i = s.info
        w = _waves((i.nzp, i.nyp, i.nxp), [5e8] * 3 + [40.0] * 6, np.random.default_rng(3))
        for n in (0, shift):
            s.set_wavefield(w * np.float32(2.0**n))
            s.run(1)
            out.append(s.wavefield().astype(np.float64) / 2.0**n)
    assert np.isfinite(out[1]).all()
    for part in (slice(0, 3), slice(3, 9)):
        assert pu.rel_l2(out[1][..., part], out[0][..., part]) <= 1e-6
