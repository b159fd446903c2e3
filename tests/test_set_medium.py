"""cgfdm_set_medium against a session created with that medium.

set_medium makes the coordinates again on the device from the height map, by
the grid's own formula (flat, terrain in float, terrain in double; a part's
block of the volume is uploaded), and rescales the fault's moment rates.  The
metric, the matrices behind it and a short run must be those of a fresh session
on the same medium, bit for bit, whatever ran before the call.
"""

import numpy as np
import pytest

import parity_util as pu
from cgfdm import CgfdmError, Session, cases, configs
from cgfdm.domain import Part

STEPS = 11


def _medium(shape, seed):
    """Smooth +-5 % around a half-space, [nzp][nyp][nxp][3] (Vs, Vp, rho)."""
    rng = np.random.default_rng(seed)
    z, y, x = np.meshgrid(*[np.arange(n) for n in shape], indexing="ij")
    m = np.empty(shape + (3,))
    for c, v in enumerate((3464.0, 6000.0, 2670.0)):
        k = rng.uniform(0.1, 0.5, 3)
        m[..., c] = v * (1 + 0.05 * np.sin(k[0] * x + k[1] * y + k[2] * z + rng.uniform(0, 6)))
    return m.astype(np.float32)


def _dirs(tmp_path, grid, source):
    """Two run directories that differ in their medium file only, and the media."""
    if source == "fault":
        c = pu.multi_fault(steps=STEPS, courant=0.4)
    else:
        c = pu.small_halfspace(steps=STEPS, NX=34, NY=30, NZ=26, courant=0.4)
        c.fault = []
        c.ricker_point = (17, 15, 18, 6.0)
    c.extra = dict(c.extra, mediumFile="medium.bin", useMedium=1)
    if grid == "hill":
        c.gauss_hill = 1
    elif grid == "double":
        # the same hill by the formula of the reference's useTerrain path
        c.gauss_hill = 1
        c.extra = dict(c.extra, useTerrain=1, SRTM90=0)
    out = []
    for n in range(2):
        d = tmp_path / f"run{n}"
        d.mkdir()
        if grid == "file":
            configs.gaussian_hills(c.NX, c.NY, c.DH, np.random.default_rng(5), hrange=(20.0, 0.04 * c.NZ * c.DH),
                                   wrange=(800.0, 3000.0)).tofile(str(d / "terrain.bin"))
            c.extra = dict(c.extra, terrainFile="terrain.bin")
        med = _medium((c.NZ + 6, c.NY + 6, c.NX + 6), 20 + n)
        med.tofile(str(d / "medium.bin"))
        out.append((cases.write_case(c, str(d)), med))
    return out


def _state(s):
    return s.cjm(), s.stations(), s.wavefield(), s.pgv()


@pytest.mark.gpu
@pytest.mark.parametrize("flavor", ["fast", "exact"])
@pytest.mark.parametrize("source", ["point", "fault"])
@pytest.mark.parametrize("grid", ["flat", "hill", "file", "double"])
def test_set_medium_is_a_fresh_session(tmp_path, grid, source, flavor):
    (d0, m0), (d1, m1) = _dirs(tmp_path, grid, source)
    with Session(d1, flavor=flavor) as s:
        s.run(STEPS)
        ref = _state(s)
    assert np.abs(ref[2]).max() > 0
    with Session(d0, flavor=flavor) as s:
        s.run(5)
        s.set_medium(m1)
        assert s.info.steps_done == 0
        s.run(STEPS)
        for a, r in zip(_state(s), ref):
            np.testing.assert_array_equal(a, r)
        # and back, from a finished run
        s.set_medium(m0)
        s.run(STEPS)
        back = _state(s)
    with Session(d0, flavor=flavor) as s:
        s.run(STEPS)
        for a, r in zip(back, _state(s)):
            np.testing.assert_array_equal(a, r)


@pytest.mark.gpu
def test_set_medium_on_a_part_and_refusals(tmp_path):
    """A part of the whole grid takes its coordinates from its block of the
    volume; a medium past the CFL limit is refused and changes nothing."""
    (d0, m0), (d1, m1) = _dirs(tmp_path, "file", "fault")
    with Session(d1) as s:
        s.run(STEPS)
        ref = _state(s)
    p = Part(d0, (1, 1, 1), (0, 0, 0))
    try:
        p.run(3)
        p.set_medium(m1)
        p.run(STEPS)
        for a, r in zip(_state(p), ref):
            np.testing.assert_array_equal(a, r)
    finally:
        p.close()
    fast = m1.copy()
    fast[10, 10, 10, 1] *= 5
    with Session(d1) as s:
        s.run(4)
        with pytest.raises(CgfdmError) as e:
            s.set_medium(fast)
        assert e.value.code == 110 and s.info.steps_done == 4
        s.run(STEPS)
        for a, r in zip(_state(s), ref):
            np.testing.assert_array_equal(a, r)
