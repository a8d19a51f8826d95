"""Streaming sweep kernels (stream.cu) at the sizes where their tiles,
segments and copies change: lines of one and of several segments, 16 and 32
lanes per line, tiles with missing lines, odd row lengths and an odd base
address (single-value copies instead of pairs)."""
import os

import numpy as np
import pytest

from conftest import periodic_field, rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-12  # FP64 parity bar of the sweeps against the oracle
THREADS = min(32, os.cpu_count() or 1)


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()


def _grids(oracle, ccfv, nx, ny, K, vp=(0.9, -1.7)):
    return (oracle.grid(nx, ny, bc=1, vel=1, vp=vp, K=K, threads=THREADS, scheme=1),
            ccfv.Solver(ccfv.make_grid(nx, ny, bc=1, velocity=1, vel_params=vp, K=K, scheme=1)))


@pytest.mark.parametrize("nx,ny", [(40, 41), (65, 233), (246, 250), (271, 258), (272, 520),
                                   (500, 44), (42, 1025), (1030, 66)])
@pytest.mark.parametrize("K", [1e-4, 4e-3])
def test_stream_sizes_match_oracle(oracle, ccfv, nx, ny, K):
    dt = 0.8 / max(nx, ny) / 1.7
    C0 = periodic_field(nx, nx + ny, ny=ny)
    g, s = _grids(oracle, ccfv, nx, ny, K)
    assert [v for v, _ in s.sweep_plan(dt)] == ["filter"] * 3
    c = dev(C0)
    s.run(c, 0.0, dt, 2)
    s.check()
    assert rel_l2(c.cpu().numpy(), oracle.run(g, C0, 0.0, dt, 2)) < TOL


@pytest.mark.parametrize("nx,ny", [(96, 80), (300, 260)])
def test_stream_odd_base_address_gives_the_same_values(ccfv, nx, ny):
    import torch
    s = ccfv.Solver(ccfv.make_grid(nx, ny, bc=1, velocity=1, vel_params=(0.9, -1.7), K=1e-3,
                                   scheme=1))
    C0 = dev(periodic_field(nx, 5, ny=ny))
    a = C0.clone()
    b = torch.empty(nx * ny + 1, dtype=torch.float64, device="cuda")[1:].view(nx, ny)
    b.copy_(C0)
    for c in (a, b):
        s.run(c, 0.0, 1e-3, 3)
    s.check()
    assert torch.equal(a, b)


@pytest.mark.parametrize("N,cfl", [(18, 0.7), (34, 2.6), (271, 0.8), (273, 0.8), (290, 12.8),
                                   (545, 1.7), (1100, 3.3)])
@pytest.mark.parametrize("vel,vp", [(0, ()), (1, (3.0, -3.7))], ids=["rot4", "const"])
@pytest.mark.parametrize("scheme", [0, 1])
def test_reference_boundaries_match_oracle(oracle, ccfv, N, cfl, vel, vp, scheme):
    """Line ends of the reference's setting: inflow and outflow, feet several
    cells away, both schemes (the reference's third sweep differentiates the
    remapped field), lines of one lane group, one segment and several."""
    from conftest import seeded_field
    K, dt = 2e-3, cfl * (2.0 / N) / 4.0
    C0 = seeded_field(N, N)
    g = oracle.grid(N, K=K, vel=vel, vp=vp, threads=THREADS, scheme=scheme)
    s = ccfv.Solver(ccfv.make_grid(N, K=K, velocity=vel, vel_params=vp, scheme=scheme))
    assert [v for v, _ in s.sweep_plan(dt)] == ["cell_compat"] * 3
    c = dev(C0)
    s.run(c, 0.0, dt, 2)
    s.check()
    assert rel_l2(c.cpu().numpy(), oracle.run(g, C0, 0.0, dt, 2)) < TOL


def test_reference_boundaries_one_segment_any_diffusion(oracle, ccfv):
    """A y line of one 32-lane segment needs no recurrence warm-up: diffusion
    numbers far above the warm-up limit, on a grid whose x lines fit 16 lanes."""
    from conftest import seeded_field
    nx, ny, K = 200, 500, 0.5
    dt = 0.8 * (2.0 / ny) / 4.0
    C0 = seeded_field(nx, 3, ny=ny)
    g = oracle.grid(nx, ny, K=K, threads=THREADS)
    s = ccfv.Solver(ccfv.make_grid(nx, ny, K=K))
    assert s.sweep_plan(dt)[1] == ("cell_compat", ny)
    c = dev(C0)
    s.run(c, 0.0, dt, 2)
    s.check()
    assert rel_l2(c.cpu().numpy(), oracle.run(g, C0, 0.0, dt, 2)) < TOL


@pytest.mark.parametrize("nx,ny,K", [(60, 52, 1e-3), (272, 300, 5e-3), (1500, 40, 2e-4),
                                     (24, 8400, 1e-6), (70, 64, 0.3)])
@pytest.mark.parametrize("n", [1, 2, 5])
def test_step_sequences_match_oracle(oracle, ccfv, nx, ny, K, n):
    """Sequences of one, an even and an odd number of steps: x sweeps of
    neighbouring steps in one pass, the last y sweep over its own input (lines
    of more segments than a cluster holds: 8400 cells, copied back), strong
    diffusion (cluster form), against the oracle's separate sweeps."""
    dt = 0.8 / max(nx, ny) / 1.7
    C0 = periodic_field(nx, nx + ny, ny=ny)
    g, s = _grids(oracle, ccfv, nx, ny, K)
    c = dev(C0)
    s.run(c, 0.0, dt, n)
    s.check()
    out = c.cpu().numpy()
    assert rel_l2(out, oracle.run(g, C0, 0.0, dt, n)) < TOL
    assert abs(out.sum() - C0.sum()) < 1e-12 * np.abs(C0).sum()


@pytest.mark.parametrize("nx,ny", [(45, 46), (240, 239), (300, 270), (50, 1100)])
@pytest.mark.parametrize("cfl", [0.8, 6.0, 20.0])
def test_swirl_matches_oracle_at_small_and_large_steps(oracle, ccfv, nx, ny, cfl):
    """Corner feet by a short series (fine steps), a longer one and sines of
    their own (coarse steps on small grids); ragged tiles, one and several
    segments, feet several cells from their edge."""
    K, dt = 1e-4, cfl / max(nx, ny)
    C0 = periodic_field(nx, nx + 2, ny=ny)
    g = oracle.grid(nx, ny, bc=1, vel=3, vp=(1.5,), K=K, threads=THREADS, scheme=1)
    s = ccfv.Solver(ccfv.make_grid(nx, ny, bc=1, velocity=3, vel_params=(1.5,), K=K, scheme=1))
    assert "cell" in [v for v, _ in s.sweep_plan(dt)]
    c = dev(C0)
    s.run(c, 0.2, dt, 3)
    s.check()
    out = c.cpu().numpy()
    assert rel_l2(out, oracle.run(g, C0, 0.2, dt, 3)) < TOL
    assert abs(out.sum() - C0.sum()) < 1e-12 * np.abs(C0).sum()


@pytest.mark.parametrize("nx,ny", [(19, 18), (255, 256), (271, 273), (273, 543), (288, 546),
                                   (34, 1089), (1089, 33), (40, 4352)])
@pytest.mark.parametrize("vel,vp", [(1, (0.9, -1.7)), (3, (1.5,))], ids=["const", "swirl"])
@pytest.mark.parametrize("nu", [20.0, 90.0])
def test_strong_diffusion(oracle, ccfv, nx, ny, vel, vp, nu):
    """Strong diffusion: whole lines (no warm-up), long warm-ups with 32 lanes
    per line (uniform field) and lines closed by clusters of up to 16 segments,
    a last segment of one position, whole and ragged lanes, missing lines."""
    N = max(nx, ny)
    dt, K = 0.4 / N, nu / (0.4 * N)
    C0 = periodic_field(nx, nx + ny, ny=ny)
    # K dt / h^2 = nu in the long direction
    g = oracle.grid(nx, ny, bc=1, vel=vel, vp=vp, K=K, threads=THREADS, scheme=1)
    s = ccfv.Solver(ccfv.make_grid(nx, ny, bc=1, velocity=vel, vel_params=vp, K=K, scheme=1))
    assert ("filter_exact" if vel == 1 else "cell_exact") in [v for v, _ in s.sweep_plan(dt)]
    c = dev(C0)
    s.run(c, 0.0, dt, 2)
    s.check()
    assert rel_l2(c.cpu().numpy(), oracle.run(g, C0, 0.0, dt, 2)) < TOL


@pytest.mark.parametrize("nx,ny", [(4, 4), (5, 7), (9, 17)])
@pytest.mark.parametrize("vel,vp,bc,scheme", [(1, (0.9, -1.7), 1, 1), (3, (1.5,), 1, 1),
                                              (1, (0.9, -1.7), 0, 0), (1, (0.9, -1.7), 0, 1)],
                         ids=["const", "swirl", "compat_ref", "compat"])
def test_smallest_grids(oracle, ccfv, nx, ny, vel, vp, bc, scheme):
    """Lines shorter than one lane's positions: periodic (closed exactly) and
    with the reference's boundaries, where every cell is next to a line end."""
    K, dt = 1e-3, 0.8 / max(nx, ny) / 1.7
    C0 = periodic_field(nx, nx + ny, ny=ny)
    g = oracle.grid(nx, ny, bc=bc, vel=vel, vp=vp, K=K, threads=1, scheme=scheme)
    s = ccfv.Solver(ccfv.make_grid(nx, ny, bc=bc, velocity=vel, vel_params=vp, K=K,
                                   scheme=scheme))
    c = dev(C0)
    s.run(c, 0.0, dt, 3)
    s.check()
    assert rel_l2(c.cpu().numpy(), oracle.run(g, C0, 0.0, dt, 3)) < TOL


def test_more_fields_than_a_grid_dimension_holds(ccfv):
    """65,537 slices in one launch: the fields' launch index is flat there."""
    n, N, DT = 65537, 40, 0.02
    s = ccfv.Solver(ccfv.make_grid(N, bc=1, velocity=1, vel_params=(0.9, -1.7), K=1e-3, scheme=1))
    assert [v for v, _ in s.sweep_plan(DT / 2)] == ["filter"] * 3
    C0 = dev(periodic_field(N, 7))
    f = C0.repeat(n, 1, 1).contiguous()
    s.fine_slices(f, 0.0, DT, DT, 2)
    s.run(C0, 0.0, DT / 2, 2)
    s.check()
    # the same sweeps of the same values but for the fused x pass's rounding
    assert float((f - C0).abs().max()) < 1e-13 * float(C0.abs().max())
