"""Grids of vertical columns: the metric terms the kernels leave out are zero,
and leaving them out changes nothing.

Every grid this library builds has x a function of i alone and y of j alone,
so grad xi = (xi_x, 0, 0) and grad eta = (0, eta_y, 0).  The stage kernels
read neither the four zero terms nor the derivatives they multiply; the
reference-form run (cgfdm_run_precise) reads all nine terms and takes all
derivatives, so the two must agree: bit for bit in the exact build with the
run's FP32 form.  Sizes sit at the edges of tiles and of the pencils, with
absorbing layers that overlap at the smallest ones.
"""

import json

import numpy as np
import pytest

import parity_util as pu
from cgfdm import Session, cases, configs

ZERO_TERMS = [1, 2, 3, 5]     # xi_y xi_z et_x et_z of the packed metric


def _case(nx, ny, nz, nPML, grid, steps, tmp, scheme="CGFDM"):
    c = cases.halfspace_case(NX=nx, NY=ny, NZ=nz, nPML=nPML, steps=steps, n_stations=3, depth_m=500.0, courant=0.4)
    c.fault = []
    c.ricker_point = (nx // 2, ny // 2, nz // 2, 6.0)
    c.stations = [(nx // 2, ny // 2, nz - 1), (1, ny - 2, nz // 2), (nx - 1, 0, 1)]
    d = tmp / f"{grid}_{nx}x{ny}x{nz}_{scheme}"
    d.mkdir()
    if grid == "hill":
        c.gauss_hill = 1
    elif grid == "file":
        rng = np.random.default_rng(nx * 1000 + ny)
        configs.gaussian_hills(nx, ny, c.DH, rng, hrange=(20.0, 0.04 * nz * c.DH),
                               wrange=(800.0, 3000.0)).tofile(str(d / "terrain.bin"))
        c.extra["terrainFile"] = "terrain.bin"
    return cases.write_case(c, str(d), scheme=scheme)


def _waves(shape, seed, amp):
    rng = np.random.default_rng(seed)
    w = np.zeros(shape + (9,), np.float32)
    z, y, x = np.meshgrid(*[np.arange(n) for n in shape], indexing="ij")
    for f in range(9):
        for _ in range(3):
            k = rng.normal(size=3)
            k *= 2 * np.pi / (np.linalg.norm(k) * rng.uniform(6, 20))
            w[..., f] += amp[f] * rng.normal() * np.cos(k[0] * x + k[1] * y + k[2] * z + rng.uniform(0, 6.3))
    w[:3] = 0
    w[-3:] = 0
    w[:, :3] = 0
    w[:, -3:] = 0
    w[:, :, :3] = 0
    w[:, :, -3:] = 0
    return w


@pytest.mark.gpu
@pytest.mark.parametrize("scheme", ["CGFDM", "SCFDM"])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("grid", ["flat", "hill", "file"])
def test_left_out_metric_terms_are_zero(tmp_path, grid, precision, scheme):
    d = _case(37, 29, 23, 5, grid, 8, tmp_path, scheme)
    with Session(d, options=f'{{"metricPrecision": "{precision}"}}') as s:
        c = s.cjm()
    assert (c[..., ZERO_TERMS] == 0).all()
    assert (c[3:-3, 3:-3, 3:-3, [0, 4, 8]] != 0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("options", ['{"stageTile": 8}', '{"stageTile": 4}', '{"stagePipeline": "ring"}',
                                     '{"PML": 0}'])
@pytest.mark.parametrize("nx,ny,nz,nPML,grid", [(32, 8, 16, 3, "file"), (33, 9, 17, 4, "hill"), (63, 31, 9, 4, "file"),
                                                (13, 41, 19, 8, "file"), (66, 11, 25, 6, "flat")])
def test_stage_matches_all_terms_run_bit_for_bit(tmp_path, nx, ny, nz, nPML, grid, options):
    d = _case(nx, ny, nz, nPML, grid, 17, tmp_path)
    with Session(d, options=options, flavor="exact") as s:
        st_p, pgv_p, W_p = s.run_precise(17, bits=32, wavefield=True)
        s.run(17)
        assert np.abs(W_p).max() > 0
        np.testing.assert_array_equal(W_p.astype(np.float32), s.wavefield())
        np.testing.assert_array_equal(st_p.astype(np.float32), s.stations())
        np.testing.assert_array_equal(pgv_p.astype(np.float32), s.pgv()[:, :, :2])


@pytest.mark.gpu
@pytest.mark.parametrize("options", ['{}', '{"stagePipeline": "ring"}'])
@pytest.mark.parametrize("nx,ny,nz,nPML,grid", [(33, 9, 17, 4, "hill"), (13, 41, 19, 8, "file"), (66, 11, 25, 6, "flat")])
def test_default_build_stays_as_close_to_fp64(tmp_path, nx, ny, nz, nPML, grid, options):
    """The default build ends a step from its three stage values instead of a
    running sum and factors the sums: no further from the FP64 run than twice
    the exact build, with a source whose cube reaches into the halo (those
    cells are held in all four stage buffers)."""
    d = _case(nx, ny, nz, nPML, grid, 17, tmp_path)
    p = tmp_path / f"{grid}_{nx}x{ny}x{nz}_CGFDM" / "params.json"
    q = json.loads(p.read_text())
    q.update(sourceX=1, sourceY=2)
    p.write_text(json.dumps(q))
    err = {}
    for flavor in ("exact", "fast"):
        with Session(d, options=options, flavor=flavor) as s:
            st64, _, W64 = s.run_precise(17, bits=64, wavefield=True)
            s.run(17)
            W, st = s.wavefield(), s.stations()
        err[flavor] = pu.errors_by_quantity(W, W64, st, st64)
    for q, e in err["exact"].items():
        assert e < 1e-5, q
        assert err["fast"][q] <= 2 * e + 1e-7, q


@pytest.mark.gpu
def test_halo_of_an_initial_wavefield_is_held_in_every_stage(tmp_path):
    """set_wavefield keeps its halo through all stages: the default build
    (four stage buffers) and the exact one (three) agree, 1e-6 over nine steps
    of about ten roundings each."""
    d = _case(33, 21, 17, 4, "hill", 9, tmp_path)
    out = {}
    for flavor in ("exact", "fast"):
        with Session(d, flavor=flavor) as s:
            i = s.info
            rng = np.random.default_rng(4)
            w = _waves((i.nzp, i.nyp, i.nxp), 4, [0.05] * 3 + [5e5] * 6)
            w[:, :3] = w[:, 3:6] + rng.normal(size=w[:, :3].shape) * w.std(axis=(0, 1, 2)) * 0.1
            s.set_wavefield(w.astype(np.float32))
            s.run(9)
            out[flavor] = s.wavefield()
    for part in (slice(0, 3), slice(3, 9)):
        assert pu.rel_l2(out["fast"][..., part], out["exact"][..., part]) <= 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("options", [None, '{"storage": "fp16"}', '{"PML": 0}'])
def test_default_build_needs_no_more_memory(tmp_path, options):
    """The default build's other RK form holds as much on the device as the
    exact build's running sum, absorbing layers included."""
    d = _case(37, 29, 23, 6, "hill", 8, tmp_path)
    held = {}
    for flavor in ("exact", "fast"):
        with Session(d, options=options, flavor=flavor) as s:
            held[flavor] = s.info.device_bytes
    assert held["fast"] == held["exact"] > 0
