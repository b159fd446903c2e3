"""The bounded waits of the stage kernel and of the ME-AWENO passes, made to
run out on purpose.

Every wait of the CGFDM stage kernel for a plane copy, and of a pass for its
tile's, is bounded; a wait
that gives up sets a device error word, the CTA waits (bounded) for the
copies it did issue and returns, and the next cgfdm_run reports
CGFDM_E_TIMEOUT.  The reference has no such path: its CHECK macro prints a
CUDA error and carries on (src/macro.h:94-103).

The test hook cgfdm_test_stall makes one work item leave one plane copy
unissued: nothing is in flight for that slot and its barrier phase never
completes, so the wait runs out after a short limit (about 2 ms here).  The
drain then waits for the copies that were issued, including the one for the
same slot's missing plane, which also runs out.  No copy is left landing in
shared memory, and the device stays usable: a fresh session on it then
matches the golden fixture of the reference's CPU build.
"""

import os
import tempfile

import numpy as np
import pytest

import golden_cases
from cgfdm import CgfdmError, Session, cases

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
E_TIMEOUT = 20002
WAIT_CYCLES = 1 << 22


def _fresh_session_matches_golden():
    mk, scheme = golden_cases.CASES["cg_halfspace"]
    gold = np.load(os.path.join(ROOT, "tests", "golden", "cg_halfspace.npz"))
    with tempfile.TemporaryDirectory() as d:
        cases.write_case(mk(), d, scheme=scheme)
        with Session(d, device=0, flavor="exact") as s:
            s.run(s.info.NT)
            st = s.stations()
    assert np.array_equal(st, gold["stations"])


@pytest.mark.gpu
@pytest.mark.parametrize("fill", [2, 7], ids=["first_window", "in_loop"])
def test_stage_wait_gives_up_and_device_recovers(tmp_path, fill):
    # fill 2: a plane of the item's first window (issued before the loop);
    # fill 7: a plane the loop issues, with later copies already in flight
    c = cases.halfspace_case(NX=64, NY=60, NZ=40, nPML=6, steps=16, n_stations=2)
    cases.write_case(c, str(tmp_path))
    with Session(str(tmp_path), device=0) as s:
        s.run(1)
        s.test_stall(item=0, fill=fill, wait_cycles=WAIT_CYCLES)
        with pytest.raises(CgfdmError) as e:
            s.run(9)
        assert e.value.code == E_TIMEOUT
        assert "gave up" in str(e.value)
    _fresh_session_matches_golden()


def _sc_run(tmp_path, name):
    # 86 x 61 x 40: 2 x 8 x 40 tiles in the x pass (more than two a CTA), 6 x 3 x 40
    # in y, 6 x 61 x 2 in z
    c = cases.halfspace_case(NX=86, NY=61, NZ=40, nPML=6, steps=16, n_stations=2, depth_m=500.0, courant=0.4)
    c.fault = []
    c.gauss_hill = 1
    c.ricker_point = (43, 30, 20, 6.0)
    c.stations = [(43, 30, 39), (20, 40, 10)]
    return cases.write_case(c, str(tmp_path / name), scheme="SCFDM")


@pytest.mark.gpu
@pytest.mark.parametrize("tile", [0, 300, 599], ids=["first", "second", "third"])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_pass_wait_gives_up_and_device_recovers(tmp_path, axis, tile):
    """A CTA's first tile (copy issued before the loop) and later ones (issued
    while the tile before is computed): the status, and a fresh session that
    then gives what an undisturbed one gives, bit for bit."""
    d = _sc_run(tmp_path, "run")
    with Session(d, device=0) as s:
        s.run(16)
        ref = (s.stations(), s.wavefield(), s.pgv())
    with Session(d, device=0) as s:
        s.run(1)
        s.test_stall(item=tile, fill=axis, wait_cycles=WAIT_CYCLES)
        with pytest.raises(CgfdmError) as e:
            s.run(9)
        assert e.value.code == E_TIMEOUT
        assert "gave up" in str(e.value) and "word 3" in str(e.value)
    with Session(d, device=0) as s:
        s.run(16)
        for a, r in zip((s.stations(), s.wavefield(), s.pgv()), ref):
            np.testing.assert_array_equal(a, r)


@pytest.mark.gpu
def test_pass_stall_hook_checks_its_arguments(tmp_path):
    d = _sc_run(tmp_path, "run")
    with Session(d, device=0) as s:
        for bad in (dict(item=-1, fill=0), dict(item=640, fill=0), dict(item=720, fill=1), dict(item=732, fill=2),
                    dict(item=0, fill=3), dict(item=0, fill=-1)):
            with pytest.raises(CgfdmError) as e:
                s.test_stall(wait_cycles=WAIT_CYCLES, **bad)
            assert e.value.code == 20003
    with Session(d, device=0, flavor="exact") as s:
        with pytest.raises(CgfdmError) as e:
            s.test_stall(item=0, fill=0, wait_cycles=WAIT_CYCLES)
        assert e.value.code == 180
