"""GPU parity of the TG RK3 substep (libchapsim, sm_100a) against the FP64
CPU oracle and the golden fixtures.  Tolerance: FP64 form within 1e-10
relative (max |a-b| / max |b|) on u, v, w, p after every checked stage."""
import math
import os

import numpy as np
import pytest

from tests.conftest import relerr

pytestmark = pytest.mark.gpu

TOL = 1e-10
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


def _need_gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def pair(nx, ny, nz, lx=4 * math.pi, lz=4 * math.pi / 3, ren=2800.0, dt=1e-3, seed=0, amp=0.1, **kw):
    _need_gpu()
    from chapsim1ww_b200 import TGChannel
    from oracle.pyoracle import OracleTG
    g = TGChannel(nx, ny, nz, lx=lx, lz=lz, ren=ren, dt=dt, **kw)
    o = OracleTG(nx, ny, nz, lx=lx, lz=lz, ren=ren, dt=dt, **kw)
    g.random_fl_fld_tg(seed, amp, project=False)
    o.init_random(seed, amp)
    return g, o


def compare(g, o, names=("u", "v", "w", "p"), tol=TOL, tag=""):
    errs = {n: relerr(g.get_field(n), o.get(n)) for n in names}
    bad = {n: e for n, e in errs.items() if not e <= tol}
    assert not bad, f"{tag}: relative errors above {tol}: {errs}"
    return errs


@pytest.mark.parametrize("dims", [(16, 12, 8), (24, 16, 12), (64, 64, 64), (48, 20, 40), (60, 18, 36)])
def test_substep_parity(dims):
    g, o = pair(*dims)
    compare(g, o, ("u", "v", "w"), tol=1e-14, tag="init")
    g.solverrk3_mom_tg(0)
    o.substep(0)
    compare(g, o, tag="ns0")
    for step in range(2):
        for ns in (1, 2, 3):
            g.solverrk3_mom_tg(ns)
            o.substep(ns)
            compare(g, o, tag=f"step{step} ns{ns}")
    compare(g, o, ("h0u", "h0v", "h0w"), tag="h0")
    assert g.divgck_tg() < 1e-11
    assert abs(g.bulk_velocity_tg() - o.bulk()) < 1e-12


@pytest.mark.parametrize("dims", [(112, 16, 176), (80, 12, 96)])
def test_radix_7_11_lengths(dims):
    # lengths outside FFT99's 2/3/5 support (112 = 7*16, 176 = 11*16)
    g, o = pair(*dims, seed=3)
    g.solverrk3_mom_tg(0)
    o.substep(0)
    for ns in (1, 2, 3):
        g.solverrk3_mom_tg(ns)
        o.substep(ns)
    compare(g, o, tag="radix")


def test_graph_step_matches_eager_bitwise():
    _need_gpu()
    from chapsim1ww_b200 import TGChannel
    a = TGChannel(32, 24, 16)
    b = TGChannel(32, 24, 16)
    for s in (a, b):
        s.random_fl_fld_tg(7, 0.1, project=True)
    a.step(3)
    for _ in range(3):
        for ns in (1, 2, 3):
            b.solverrk3_mom_tg(ns)
    for n in ("u", "v", "w", "p"):
        assert np.array_equal(a.get_field(n), b.get_field(n)), n


def test_async_transfers_match_blocking_copies():
    """Stream-ordered uploads, a step and downloads queued on one context's
    stream give the same bits as blocking copies around the same step, with
    pinned and with pageable host buffers."""
    _need_gpu()
    import torch
    from chapsim1ww_b200 import TGChannel
    a = TGChannel(32, 24, 16)
    b = TGChannel(32, 24, 16)
    a.random_fl_fld_tg(5, 0.1, project=True)
    names = ("u", "v", "w", "p")
    start = {n: a.get_field(n) for n in names}
    for pinned in (True, False):
        host = {}
        for n in names:
            h = (torch.empty(a.shape, dtype=torch.float64, pin_memory=True).numpy() if pinned
                 else np.empty(a.shape))
            h[...] = start[n]
            host[n] = h
            b.set_field_async(n, h)
        b.step(2)
        for n in names:
            b.get_field_async(n, out=host[n])
        b.sync()
        for n in names:
            a.set_field(n, start[n])
        a.step(2)
        for n in names:
            assert np.array_equal(host[n], a.get_field(n)), (pinned, n)
    with pytest.raises(ValueError):
        b.set_field_async("u", np.zeros(3))
    a.close()
    b.close()


def test_fp64_bit_reproducible():
    _need_gpu()
    from chapsim1ww_b200 import TGChannel
    outs = []
    for _ in range(2):
        s = TGChannel(64, 48, 32, ren=3000.0)
        s.random_fl_fld_tg(11, 0.1, project=True)
        s.step(5)
        outs.append([s.get_field(n) for n in ("u", "v", "w", "p")])
        s.close()
    for x, y in zip(*outs):
        assert np.array_equal(x, y)


def test_poisson_piece_parity():
    g, o = pair(32, 24, 16, seed=4)
    rng = np.random.default_rng(5)
    rhs = np.zeros(g.shape)
    rhs[:, 1:-1, :] = rng.standard_normal((16, 24, 32))
    g.set_field("rhsphi", rhs)
    o.set("rhsphi", rhs)
    g.fft99_pois3d()
    o.pois3d()
    e = relerr(g.get_field("phi")[:, 1:-1, :], o.get("phi")[:, 1:-1, :])
    assert e < 1e-12, e


def test_analytic_poisson():
    """TEST_POISSON (src/SOLVERRK3_MOM_IO.f90:171-202): rhs = -4 sin x cos x."""
    _need_gpu()
    from chapsim1ww_b200 import TGChannel
    nx, ny, nz, lx = 64, 16, 8, 4 * math.pi
    g = TGChannel(nx, ny, nz, lx=lx)
    x = (np.arange(nx) + 0.5) * lx / nx
    rhs = np.zeros(g.shape)
    rhs[:, 1:-1, :] = (-4.0 * np.sin(x) * np.cos(x))[None, None, :]
    g.set_field("rhsphi", rhs)
    g.fft99_pois3d()
    phi = g.get_field("phi")[:, 1:-1, :]
    m = round(lx / math.pi)  # sin(2x) is wavenumber index lx/pi
    ak1 = 2.0 * (1.0 - math.cos(2.0 * math.pi * m / nx)) * (nx / lx) ** 2
    exact = 2.0 * np.sin(2.0 * x) / ak1
    assert np.abs(phi - exact[None, None, :]).max() < 1e-12


def test_divg_and_correction_pieces():
    g, o = pair(24, 16, 12, seed=9)
    for s in (g,):
        s.divg_tg(1)
    o.divg(1)
    assert relerr(g.get_field("rhsphi")[:, 1:-1, :], o.get("rhsphi")[:, 1:-1, :]) < 1e-13
    rng = np.random.default_rng(1)
    phi = rng.standard_normal(g.shape)
    g.set_field("phi", phi)
    o.set("phi", phi)
    g.veloupdt_tg(2)
    o.velo_correction(2)
    compare(g, o, tag="correction")


@pytest.mark.parametrize("name", ["tg_16x12x8_seed0", "tg_24x16x12_seed5"])
def test_golden_fixture(name):
    _need_gpu()
    from chapsim1ww_b200 import TGChannel
    z = np.load(os.path.join(GOLDEN, name + ".npz"))
    nx, ny, nz, lx, lz, ren, dt, seed, amp, steps = z["meta"]
    g = TGChannel(int(nx), int(ny), int(nz), lx=lx, lz=lz, ren=ren, dt=dt)
    g.random_fl_fld_tg(int(seed), amp, project=True)
    for n in ("u", "v", "w", "p"):
        assert relerr(g.get_field(n), z["ns0_" + n]) < 1e-10, n
    g.step(int(steps))
    for n in ("u", "v", "w", "p"):
        assert relerr(g.get_field(n), z["end_" + n]) < 1e-10, n


def test_flowdrvtp2_constant_pressure_gradient():
    g, o = pair(24, 16, 12, flowdrvtp=2, cfgv=8.18e-3)
    g.solverrk3_mom_tg(0)
    o.substep(0)
    for ns in (1, 2, 3):
        g.solverrk3_mom_tg(ns)
        o.substep(ns)
    compare(g, o, tag="flowdrvtp2")


def test_uniform_grid_istr2_0():
    g, o = pair(16, 16, 16, istr2=0)
    for ns in (0, 1, 2, 3):
        g.solverrk3_mom_tg(ns)
        o.substep(ns)
    compare(g, o, tag="uniform")


def test_nan_scan_and_divmax():
    _need_gpu()
    from chapsim1ww_b200 import TGChannel
    s = TGChannel(32, 16, 16)
    s.random_fl_fld_tg(2, 0.1, project=True)
    s.step(2)
    assert s.nan_count() == 0
    u = s.get_field("u")
    u[3, 5, 7] = float("nan")
    s.set_field("u", u)
    assert s.nan_count() == 1
    assert math.isinf(s.divgck_tg())


def test_adi_fallback_wide_inverse():
    # Re = 1, dt = 0.05: the x/z inverses are too wide for the banded kernel,
    # so the shared-memory cyclic Thomas kernels run instead
    g, o = pair(32, 24, 16, ren=1.0, dt=0.05)
    for ns in (0, 1):
        g.solverrk3_mom_tg(ns)
        o.substep(ns)
    compare(g, o, tag="fallback")


def test_short_lines_wrap():
    # nx, nz shorter than a 32 x 8 tile plus its halo
    g, o = pair(8, 8, 8, lx=1.0, lz=0.5)
    for ns in (0, 1, 2, 3):
        g.solverrk3_mom_tg(ns)
        o.substep(ns)
    compare(g, o, tag="short")


def test_line_tuning_does_not_change_results():
    """The y-line block width of the Poisson solve (64, 128, 256: one of the
    autotuner's launch shapes) leaves every field bitwise unchanged, TG and
    IO."""
    _need_gpu()
    from chapsim1ww_b200 import IOChannel, TGChannel
    from oracle.pyoracle import synth_table
    out = []
    for bx in (64, 128, 256):
        g = TGChannel(48, 20, 40)
        g.set_line_tuning(bx)
        assert g.get_line_tuning() == bx
        g.random_fl_fld_tg(3, 0.1, project=True)
        g.step(2)
        out.append([g.get_field(n) for n in ("u", "v", "w", "p")])
        g.close()
    for a in out[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(out[0], a))
    table = synth_table(4096)
    res = []
    for bx in (64, 256):
        g = IOChannel(40, 18, 24, table=table)
        g.set_line_tuning(bx)
        g.random_fl_theml_fld_io(2, 0.1)
        g.step(1)
        res.append([g.get_field(n) for n in ("gx", "p", "h")])
        g.close()
    assert all(np.array_equal(x, y) for x, y in zip(*res))


def test_substep_calls_replay_the_same_launches_bitwise():
    """Substep calls (captured from the third call of an NS on) against graph
    steps, bitwise, across a change of DT, of the launch shapes and a field
    written between calls."""
    _need_gpu()
    from chapsim1ww_b200 import TGChannel
    a, b = TGChannel(40, 18, 24), TGChannel(40, 18, 24)
    for x in (a, b):
        x.random_fl_fld_tg(7, 0.1)
    for change in (lambda x: None, lambda x: x.set_dt(5e-4), lambda x: x.set_tuning(8, 4),
                   lambda x: x.set_field("p", 0.5 * x.get_field("p"))):
        for x in (a, b):
            change(x)
        n0 = a.launch_count(), b.launch_count()
        for _ in range(4):
            for ns in (1, 2, 3):
                a.solverrk3_mom_tg(ns)
        b.step(4)
        for f in ("u", "v", "w", "p", "h0u"):
            assert np.array_equal(a.get_field(f), b.get_field(f)), f
        assert a.launch_count() - n0[0] == b.launch_count() - n0[1]


@pytest.mark.parametrize("dims", [(8, 4, 8), (10, 33, 66), (30, 65, 18), (512, 5, 16), (528, 6, 20)])
def test_adi_factor_edges(dims):
    """The x / z and y factors at the ends of their shapes: the shortest and
    longest rows of the row form and the first of the tile form (nx 512, 528),
    one row past a y tile, plane counts that leave short last segments and
    fewer planes than the copies run ahead."""
    g, o = pair(*dims, seed=4)
    for ns in (0, 1, 2, 3):
        g.solverrk3_mom_tg(ns)
        o.substep(ns)
        compare(g, o, tag=f"ns{ns}")


@pytest.mark.parametrize("dt,ren", [(5e-3, 200.0), (1e-2, 100.0), (2e-2, 100.0)])
def test_adi_factor_wider_bands(dt, ren):
    """Wider compiled bands of the factors (larger dt / Re)."""
    g, o = pair(40, 36, 24, ren=ren, dt=dt, seed=4)
    for ns in (0, 1, 2, 3):
        g.solverrk3_mom_tg(ns)
        o.substep(ns)
        compare(g, o, tag=f"ns{ns}")


@pytest.mark.parametrize("nz", [8, 10, 14, 22, 24, 30, 36, 50, 54, 66, 98, 110, 126, 144, 150, 210, 242, 256, 264, 352, 450, 512])
def test_z_transform_lengths(nz):
    """The register-blocked z transforms over their radices (2 to 16, composite
    and prime), two and three stages, and lines per block; 242 = 2 x 11 x 11
    takes three stages."""
    g, o = pair(10, 5, nz, seed=4)
    g.solverrk3_mom_tg(0)
    o.substep(0)
    compare(g, o, tag=f"nz {nz}")


@pytest.mark.parametrize("nx", [8, 10, 14, 22, 24, 36, 50, 54, 66, 98, 126, 144, 150, 210, 242, 256, 264, 352, 450, 512])
def test_x_transform_lengths(nx):
    """The register-blocked x transforms over their radices and stages, with
    an odd row count (the last line holds one row)."""
    g, o = pair(nx, 5, 8, seed=4)
    g.solverrk3_mom_tg(0)
    o.substep(0)
    compare(g, o, tag=f"nx {nx}")


# compiled widths 2, 4, 6 and 12 of the y factors: rows of the ring that
# different warps clear
@pytest.mark.parametrize("dt,ren", [(1e-5, 2800.0), (1e-3, 2800.0), (2e-2, 2800.0), (2e-2, 100.0)])
def test_adi_first_plane_of_a_march(dt, ren):
    """The v rows at the lower wall, which take the u increment of row 1, on
    every plane (the first of each march of the y factors among them), over
    several x tiles and repeated substeps; the same bits on a second run."""
    runs = []
    for _ in range(2):
        g, o = pair(160, 36, 40, ren=ren, dt=dt, seed=6)
        for ns in (0, 1, 2, 3):
            g.solverrk3_mom_tg(ns)
            o.substep(ns)
            v, ref = g.get_field("v"), o.get("v")
            err = np.abs(v - ref)[:, :18, :].max(axis=(1, 2)) / np.abs(ref).max()
            assert (err <= TOL).all(), (ns, np.flatnonzero(err > TOL), err.max())
        runs.append(v)
    assert np.array_equal(*runs)


@pytest.mark.parametrize("mode", ["relaxed", "thread_local", "global"])
def test_substep_calls_beside_a_capture_of_the_caller(mode):
    """Substep calls, those that are captured among them, while the caller
    captures a stream of its own: neither disturbs the other."""
    _need_gpu()
    import torch
    from chapsim1ww_b200 import TGChannel
    g, ref = TGChannel(32, 24, 16), TGChannel(32, 24, 16)
    for x in (g, ref):
        x.random_fl_fld_tg(1, 0.1)
    ref.step(6)
    ref.sync()
    a, b = torch.ones(64, device="cuda"), torch.zeros(64, device="cuda")
    torch.cuda.synchronize()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode=mode):
        b.add_(a)
        for _ in range(6):
            for ns in (1, 2, 3):
                g.solverrk3_mom_tg(ns)
        b.add_(a)
    graph.replay()
    torch.cuda.synchronize()
    assert b.eq(2.0).all()
    for n in ("u", "v", "w", "p"):
        assert np.array_equal(g.get_field(n), ref.get_field(n)), n


@pytest.mark.parametrize("nx", [28, 44, 54, 60, 66, 70, 84, 90, 98, 126, 144, 150, 162, 176, 210, 216, 242, 264, 288, 300, 324, 330, 350,
                                360, 384, 432, 450, 462, 486, 588, 630])
def test_x_transform_lengths_on_more_lines(nx):
    """The x transforms over their radices on more lines than a block holds,
    with an odd row count."""
    g, o = pair(nx, 11, 240, seed=4)
    g.solverrk3_mom_tg(0)
    o.substep(0)
    compare(g, o, tag=f"nx {nx}")


@pytest.mark.parametrize("dims", [(1250, 5, 8), (1458, 6, 8), (10, 5, 750), (10, 6, 924), (16, 9, 1008)])
def test_transform_lengths_without_a_register_plan(dims):
    """FP64 lengths that the staged kernels serve: x without a plan of three
    radices up to 16 (both directions), z with too many threads a line."""
    g, o = pair(*dims, seed=4)
    g.solverrk3_mom_tg(0)
    o.substep(0)
    compare(g, o, tag=str(dims))


@pytest.mark.parametrize("dims", [(10, 5, 360), (10, 5, 504), (66, 100, 360), (66, 100, 504)])
def test_z_transform_forms_by_grid(dims):
    """z lengths whose register lines come two to a block: staged on few
    blocks, register-blocked on many."""
    g, o = pair(*dims, seed=4)
    g.solverrk3_mom_tg(0)
    o.substep(0)
    compare(g, o, tag=str(dims))


@pytest.mark.parametrize("dims", [(48, 217, 250), (96, 113, 240), (100, 105, 252), (240, 61, 176), (360, 40, 180), (640, 20, 200)])
def test_staged_x_transform_of_larger_grids(dims):
    """Lengths that are not powers of two on grids whose inputs exceed half the
    L2: the staged forward x transform, with full and ragged row blocks."""
    g, o = pair(*dims, seed=4)
    g.solverrk3_mom_tg(0)
    o.substep(0)
    compare(g, o, tag=str(dims))
