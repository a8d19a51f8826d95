"""Sweep kernels at the ends of what they take: last segments shorter than the
recurrence's warm-up, backward steps, the shortest lines in FP32, short tuned
segments, slices in place, what plans and batches prepare."""
import os

import numpy as np
import pytest

from conftest import periodic_field, rel_l2, seeded_field

pytestmark = pytest.mark.gpu
TOL = 1e-12  # FP64 parity bar of the sweeps against the oracle
THREADS = min(32, os.cpu_count() or 1)


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()


def warm_up(nu):
    """Positions after which a start from zero has decayed below FP64 rounding,
    for a sweep of diffusion number nu (half of it on either side)."""
    r = (1 / 12 - 0.5 * nu) / (10 / 12 + nu)
    mu = 2 * r / (1 + np.sqrt(1 - 4 * r * r))
    return int(np.ceil(np.log(2.0 ** -56) / np.log(abs(mu))))


@pytest.mark.parametrize("dir,L,last", [(0, 10225, 1), (0, 10230, 6), (0, 5966, 62),
                                        (1, 86113, 1), (1, 86118, 6)])
@pytest.mark.parametrize("scheme", [0, 1])
def test_reference_boundaries_last_segment_shorter_than_the_warm_up(oracle, ccfv, dir, L, last,
                                                                    scheme):
    """The segment before such a last one reaches the line's end with its
    warm-up: it stops there."""
    nu = 5.4
    J = warm_up(nu)
    h, vel = 2.0 / L, (3.0, -3.7)
    Dt = 0.8 * h / abs(vel[dir])
    dt = 2 * Dt if dir == 0 else Dt
    nx, ny = (L, 24) if dir == 0 else (24, L)
    K = nu * h * h / Dt
    C0 = seeded_field(nx, 5, ny=ny)
    g = oracle.grid(nx, ny, K=K, vel=1, vp=vel, threads=THREADS, scheme=scheme)
    s = ccfv.Solver(ccfv.make_grid(nx, ny, K=K, velocity=1, vel_params=vel, scheme=scheme))
    name, seg = s.sweep_plan(dt)[dir]
    assert name == "cell_compat" and L - (L - 1) // seg * seg == last < J
    c = dev(C0)
    s.run(c, 0.0, dt, 2)
    s.check()
    assert rel_l2(c.cpu().numpy(), oracle.run(g, C0, 0.0, dt, 2)) < TOL


@pytest.mark.parametrize("nx,ny", [(45, 46), (64, 64), (128, 120), (300, 270)])
@pytest.mark.parametrize("cfl", [0.8, 6.0, 20.0])
def test_swirl_backward_steps_match_oracle(oracle, ccfv, nx, ny, cfl):
    """Corner feet of backward steps: the series is chosen by the step's length,
    not its sign."""
    dt = -cfl / max(nx, ny)
    C0 = periodic_field(nx, nx + 2, ny=ny)
    g = oracle.grid(nx, ny, bc=1, vel=3, vp=(1.5,), threads=THREADS, scheme=1)
    s = ccfv.Solver(ccfv.make_grid(nx, ny, bc=1, velocity=3, vel_params=(1.5,), scheme=1))
    c = dev(C0)
    s.run(c, 0.4, dt, 3)
    s.check()
    assert rel_l2(c.cpu().numpy(), oracle.run(g, C0, 0.4, dt, 3)) < TOL


@pytest.mark.parametrize("L", [4, 5, 6])
@pytest.mark.parametrize("dir", [0, 1])
@pytest.mark.parametrize("mu", [2.0 ** -14, -2.0 ** -12, 2.0 ** -11, -2.0 ** -9.5])
@pytest.mark.parametrize("vel,vp", [(1, (0.9, -1.7)), (3, (1.5,))], ids=["const", "swirl"])
def test_fp32_coarse_steps_on_the_shortest_lines(oracle, ccfv, L, dir, mu, vel, vp):
    """Lines of a few cells whose system is next to diagonal (K Dt / h^2 near
    1/6): carries of many orders of magnitude less than one."""
    nx, ny = (L, 8) if dir == 0 else (8, L)
    Dt = 0.3 / 8
    r = mu / (1 + mu * mu)
    nu = (1 / 12 - r * 10 / 12) / (0.5 + r)  # (1/12 - nu/2) / (10/12 + nu) = r
    K = nu / (L * L * Dt)
    dt = 2 * Dt if dir == 0 else Dt
    C0 = periodic_field(nx, L, ny=ny)
    g = oracle.grid(nx, ny, bc=1, vel=vel, vp=vp, K=K, threads=1, scheme=1)
    s = ccfv.Solver(ccfv.make_grid(nx, ny, bc=1, velocity=vel, vel_params=vp, K=K, scheme=1))
    c = dev(C0)
    s.coarse(c, 0.0, dt, 1, precision=ccfv.FP32)
    s.check()
    # three sweeps of at most 20 roundings of 2^-24 each, on values of the
    # field's size
    assert rel_l2(c.cpu().numpy(), oracle.coarse(g, C0, 0.0, dt, 1)) < 60 * 2.0 ** -24


@pytest.mark.parametrize("bc,scheme", [(1, 1), (0, 0)], ids=["periodic", "reference"])
@pytest.mark.parametrize("dir,L", [(0, 3602), (1, 3598)])
def test_slices_in_place_after_short_segments_were_tuned(oracle, ccfv, bc, scheme, dir, L):
    """Lengths are tuned out of place; in place a line's segments form one
    cluster of at most 16, whatever the tuned length."""
    vp = (0.9, -1.7)
    dt = 0.8 / L / 1.7

    def solver(nx, ny):
        return ccfv.Solver(ccfv.make_grid(nx, ny, bc=bc, velocity=1, vel_params=vp, scheme=scheme))

    least = (L + 15) // 16
    for m in (24, 40, 24, 96, 160):  # few x lines: short segments fill more of the GPU
        seg = solver(L, m).autotune(dt)
        if seg < least:
            break
    assert seg < least
    nx, ny = (L, 20) if dir == 0 else (20, L)
    s = solver(nx, ny)
    assert s.sweep_plan(dt)[dir][1] <= seg
    C0 = np.stack([periodic_field(nx, 3 + i, ny=ny) for i in range(2)])
    f = dev(C0)
    s.fine_slices(f, 0.0, 2 * dt, 2 * dt, 2)
    s.check()
    g = oracle.grid(nx, ny, bc=bc, vel=1, vp=vp, threads=THREADS, scheme=scheme)
    for i in range(2):
        assert rel_l2(f[i].cpu().numpy(), oracle.run(g, C0[i], 2 * i * dt, dt, 2)) < TOL


@pytest.mark.parametrize("kw,dt,want", [
    # the reference's boundaries: lines of one segment, of several, the swirl
    (dict(nx=300, ny=270, K=2e-3), 0.8 / 600, [(16, True), (16, False), (16, True)]),
    (dict(nx=64, K=1e-3, velocity=3, vel_params=(1.5,)), 1e-3, "sweep_filter_kernel"),
    (dict(nx=64, K=1e-3), 2.0,  # the third sweep's line ends need more scratch than fits
     "stream_kernel/stream_kernel/sweep_filter_kernel"),
    # periodic: weak diffusion, a long warm-up, closed lines, the swirl
    (dict(nx=300, bc=1, K=1e-4, velocity=1, vel_params=(0.9, -1.7), scheme=1), 1e-3,
     [(16, True), (32, True), (16, True)]),
    (dict(nx=600, bc=1, K=0.1, velocity=1, vel_params=(0.9, -1.7), scheme=1), 5e-4,
     [(32, True)] * 3),
    (dict(nx=600, bc=1, K=1.0, velocity=1, vel_params=(0.9, -1.7), scheme=1), 1e-3,
     [(16, False), (32, False), (16, False)]),
    (dict(nx=64, bc=1, velocity=3, vel_params=(1.5,), scheme=1), 1e-3, "stream_kernel"),
    (dict(nx=64, bc=1, velocity=1, vel_params=(0.9, -1.7)), 1e-3,
     "stream_kernel/stream_kernel/sweep_kernel"),
    (dict(nx=64, bc=1, source=1, source_params=(0.5, 0.5, 1.0, 0.1, 0.0)), 1e-3, "sweep_kernel"),
])
def test_the_plan_names_the_kernels_that_run(ccfv, kw, dt, want):
    """Kernel, lanes per line and whether the recurrences are warmed up."""
    s = ccfv.Solver(ccfv.make_grid(**kw))
    got = s.sweep_kernels(dt)
    if isinstance(want, str):
        names = want.split("/") * (1 if "/" in want else 3)
        assert [k for k, _, _ in got] == names
        assert s.variant_names(dt) == "/".join(names)
    else:
        assert got == [("stream_kernel", n, w) for (n, _), (_, _, w) in zip(want, got)]
        assert [w > 0 for _, _, w in got] == [w for _, w in want]
        assert s.variant_names(dt) == "/".join(["stream_kernel"] * 3)


def test_a_lone_step_prepares_no_pass_that_it_does_not_launch(ccfv):
    """The first step of a new dt fills the tables of its x and y sweeps; the pass
    that joins neighbouring steps gets its own from the first sequence, also a
    captured one."""
    import torch
    N = 200
    s = ccfv.Solver(ccfv.make_grid(N, bc=1, velocity=1, vel_params=(0.9, -1.7), K=1e-3, scheme=1))
    C0 = dev(periodic_field(N, 11))

    def launches(f):
        n = ccfv.kernel_launches()
        f()
        return ccfv.kernel_launches() - n

    a, b = C0.clone(), C0.clone()
    assert launches(lambda: s.step(a, 0.0, 1e-3)) == 2 + 3
    assert launches(lambda: s.step(a, 1e-3, 1e-3)) == 3
    # two steps x y xx y x, captured before any other sequence
    cap = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=cap):
        s.run(b, 0.0, 1e-3, 2)
    graph.replay()
    torch.cuda.synchronize()
    once = b.clone()
    assert float((once - a).abs().max()) < 1e-13 * float(a.abs().max())  # one pass for two
    # eagerly: filled once more, then kept; the same values as replayed
    for n in (5 + 1, 5):
        b.copy_(C0)
        assert launches(lambda: s.run(b, 0.0, 1e-3, 2)) == n
        assert torch.equal(b, once)
    b.copy_(C0)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(b, once)
    # a plan that starts with a sequence serves lone steps as well
    c = C0.clone()
    assert launches(lambda: s.run(c, 0.0, 5e-4, 3)) == 3 + 7
    assert launches(lambda: s.step(c, 0.0, 5e-4)) == 3
    s.check()


def test_a_batch_fills_one_table_per_form_of_pass(ccfv):
    """Problems of one size share every launch but those of their own tables:
    x, y and joined x passes, fine and coarse."""
    import torch
    N = 300  # too large for the coarse propagator that keeps a field in one SM
    grid = ccfv.make_grid(N, bc=1, velocity=1, vel_params=(0.9, -1.7), K=1e-3, scheme=1)
    opts = dict(t0=0.0, t1=0.02, nt_fine=16, n_slices=2, coarse_ratio=2, kmax=1)
    C0 = dev(periodic_field(N, 3))

    def launches(n):
        probs = [dict(grid=grid, C0=C0.clone(), C_T=torch.empty_like(C0), **opts)
                 for _ in range(n)]
        before = ccfv.kernel_launches()
        ccfv.batch_solve(probs)
        assert all(torch.equal(p["C_T"], probs[0]["C_T"]) for p in probs)
        return ccfv.kernel_launches() - before

    one = launches(1)
    assert launches(2) - one == 6 and launches(4) - one == 18


@pytest.mark.parametrize("nx,ny", [(48, 50), (300, 270), (600, 44), (40, 1100)])
@pytest.mark.parametrize("bc,vel,vp,scheme,nu", [
    (0, 0, (), 0, 0.2), (0, 0, (), 1, 0.2), (0, 1, (3.0, -3.7), 0, 3.0), (0, 3, (1.5,), 0, 0.2),
    (1, 3, (1.5,), 1, 0.2), (1, 3, (1.5,), 1, 20.0), (1, 1, (0.9, -1.7), 1, 20.0),
    (1, 1, (0.9, -1.7), 0, 0.2)],
    ids=["ref", "ref_consistent", "ref_const", "ref_swirl", "swirl", "swirl_strong", "strong",
         "third_sweep"])
def test_slices_in_place_by_form(oracle, ccfv, nx, ny, bc, vel, vp, scheme, nu):
    """Slices swept over their input, a line's segments as one cluster: each form
    of sweep, lines of one and of several segments, times from slice to slice."""
    N = max(nx, ny)
    h = (2.0 if bc == 0 else 1.0) / N
    dt = 0.8 * h / 4.0
    K = nu * h * h / dt
    C0 = np.stack([seeded_field(nx, 5 + i, ny=ny) if bc == 0 else periodic_field(nx, 5 + i, ny=ny)
                   for i in range(3)])
    g = oracle.grid(nx, ny, bc=bc, K=K, vel=vel, vp=vp, threads=THREADS, scheme=scheme)
    s = ccfv.Solver(ccfv.make_grid(nx, ny, bc=bc, K=K, velocity=vel, vel_params=vp, scheme=scheme))
    f = dev(C0)
    s.fine_slices(f, 0.1, 0.25, 3 * dt, 3)
    s.check()
    for i in range(3):
        assert rel_l2(f[i].cpu().numpy(), oracle.run(g, C0[i], 0.1 + 0.25 * i, dt, 3)) < TOL


@pytest.mark.parametrize("nx,ny", [(40, 41), (271, 258), (272, 520), (500, 44), (42, 1025),
                                   (1100, 66), (65, 233)])
@pytest.mark.parametrize("vel,vp", [(1, (0.9, -1.7)), (3, (1.5,))], ids=["const", "swirl"])
@pytest.mark.parametrize("nu", [0.1, 20.0, 90.0])
def test_fp32_forms_at_the_sizes_of_their_tiles(oracle, ccfv, nx, ny, vel, vp, nu):
    """FP32 coarse steps: warmed up over one and several segments, long warm-ups
    of 32 lanes, lines closed alone and by clusters, odd rows."""
    N = max(nx, ny)
    dt = 0.4 / N
    K = nu / (0.4 * N)  # K dt / h^2 = nu in the long direction
    C0 = periodic_field(nx, nx + ny, ny=ny)
    g = oracle.grid(nx, ny, bc=1, vel=vel, vp=vp, K=K, threads=THREADS, scheme=1)
    s = ccfv.Solver(ccfv.make_grid(nx, ny, bc=1, velocity=vel, vel_params=vp, K=K, scheme=1))
    c = dev(C0)
    s.coarse(c, 0.2, 2 * dt, 2, precision=ccfv.FP32)
    s.check()
    r = (1 / 12 - 0.5 * nu) / (10 / 12 + nu)
    mu = abs(2 * r / (1 + np.sqrt(1 - 4 * r * r)))
    # six sweeps; in each the right-hand side's ten roundings and those of the two
    # recurrences, which add up over 1 / (1 - |mu|) positions (and the carries')
    tol = 6 * (10 + 3 / (1 - mu)) * 2.0 ** -24
    assert rel_l2(c.cpu().numpy(), oracle.coarse(g, C0, 0.2, 2 * dt, 2)) < tol


@pytest.mark.parametrize("bc,vel,vp,scheme", [(1, 1, (0.9, -1.7), 1), (0, 0, (), 0)],
                         ids=["const", "ref"])
def test_plans_of_several_step_lengths_take_turns(oracle, ccfv, bc, vel, vp, scheme):
    """One solver, three step lengths, lone steps and sequences in turn."""
    nx, ny, K = 300, 130, 1e-3
    C0 = seeded_field(nx, 9, ny=ny) if bc == 0 else periodic_field(nx, 9, ny=ny)
    g = oracle.grid(nx, ny, bc=bc, K=K, vel=vel, vp=vp, threads=THREADS, scheme=scheme)
    s = ccfv.Solver(ccfv.make_grid(nx, ny, bc=bc, K=K, velocity=vel, vel_params=vp, scheme=scheme))
    c, want, t = dev(C0), C0, 0.0
    for dt, n in ((1e-3, 1), (2e-3, 3), (1e-3, 2), (5e-4, 1), (2e-3, 1), (5e-4, 4), (1e-3, 3)):
        s.run(c, t, dt, n)
        want = oracle.run(g, want, t, dt, n)
        t += n * dt
    s.check()
    assert rel_l2(c.cpu().numpy(), want) < TOL


@pytest.mark.parametrize("bc,scheme", [(1, 1), (0, 0)], ids=["periodic", "reference"])
def test_a_run_of_no_steps_makes_the_plan_and_refuses_what_steps_refuse(ccfv, bc, scheme):
    s = ccfv.Solver(ccfv.make_grid(64, bc=bc, K=1e-3, velocity=1, vel_params=(0.9, -1.7),
                                   scheme=scheme))
    C0 = dev(periodic_field(64, 3))
    c = C0.clone()
    before = ccfv.kernel_launches()
    s.run(c, 0.0, 1e-3, 0)
    made = ccfv.kernel_launches()
    assert made > before and bool((c == C0).all())
    s.run(c, 0.0, 1e-3, 2)
    assert ccfv.kernel_launches() - made == (5 if bc == 1 else 6)  # nothing left to prepare
    for n in (0, 1):
        with pytest.raises(ccfv.CcfvError):
            s.run(c, 0.0, 50.0, n)  # feet too far for any kernel's tile


@pytest.mark.parametrize("L", [5, 17, 18, 20, 33, 34, 35, 50])
@pytest.mark.parametrize("dir", [0, 1])
@pytest.mark.parametrize("nu", [0.05, 1 / 6 + 1e-3, 0.5, 2.0, 2.2, 4.0])
def test_closed_lines_of_a_few_lanes(oracle, ccfv, L, dir, nu):
    """Short closed lines on either side of where the carry into the last lane is
    scaled to its end (|q| = 0.35), in FP64 and FP32."""
    nx, ny = (L, 8) if dir == 0 else (8, L)
    Dt = 0.3 / L
    K = nu / (L * L * Dt)
    dt = 2 * Dt if dir == 0 else Dt
    C0 = periodic_field(nx, L, ny=ny)
    g = oracle.grid(nx, ny, bc=1, vel=1, vp=(0.9, -1.7), K=K, threads=1, scheme=1)
    s = ccfv.Solver(ccfv.make_grid(nx, ny, bc=1, velocity=1, vel_params=(0.9, -1.7), K=K, scheme=1))
    want = oracle.coarse(g, C0, 0.0, dt, 1)
    # a sweep's right-hand side has ten roundings, its recurrences add theirs up
    # over 1 / (1 - |mu|) positions; the other direction's sweep has a mu of its own
    other = nu * (8 / L) ** 2 * (2 if dir == 0 else 0.5)

    def roundings(n):
        r = (1 / 12 - 0.5 * n) / (10 / 12 + n)
        return 10 + 3 / (1 - abs(2 * r / (1 + np.sqrt(1 - 4 * r * r))))

    n = 2 * roundings(nu) + 2 * roundings(other)
    for precision, tol in ((ccfv.FP64, TOL), (ccfv.FP32, n * 2.0 ** -24)):
        c = dev(C0)
        s.coarse(c, 0.0, dt, 1, precision=precision)
        s.check()
        assert rel_l2(c.cpu().numpy(), want) < tol
