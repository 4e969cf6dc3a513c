"""Kernel variants at the sizes where their tiling changes: every line length of
the transforms on every axis against the oracle."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def make_sim(cells, extent, **kw):
    import cubismup_3d_b200 as cup
    sd = cup.SimulationData(CFL=kw.pop("CFL", 0.1), cells=cells)
    sd.extent, sd.rampup, sd.DLM, sd.lambda_ = extent, 0, 0.0, 1.0
    for k, v in kw.items():
        setattr(sd, k, v)
    return cup.Simulation(sd)


# each of 16..256 on each axis (the number of threads per line, rows per warp
# and planes per tile all change with the length), the shortest and a long grid
LINES = [(16, 16, 16), (32, 16, 64), (64, 32, 16), (128, 64, 32), (256, 128, 16), (32, 256, 128), (64, 16, 256)]


@pytest.mark.parametrize("cells", LINES)
@pytest.mark.parametrize("precision", ["fp64", "fp32_dc"])
def test_packed_transforms_every_line_length(oracle, cells, precision):
    if precision == "fp32_dc" and cells[0] < 32:
        pytest.skip("FP32 storage needs nx >= 32")
    nx, ny, nz = cells
    sim = make_sim(cells, 1.7, precision=precision)
    rhs = np.random.default_rng(sum(cells)).standard_normal((nz, ny, nx))
    p = sim.pressureSolver.solve_field(rhs)
    # FP64: rounding. FP32 with defect correction: the residual meets dc_tol =
    # 1e-10, so p is off by at most dc_tol times the condition number of the
    # wide Laplacian off its null modes
    kappa = 12.0 / (2.0 - 2.0 * np.cos(4 * np.pi / max(cells)))
    tol = 1e-12 if precision == "fp64" else 1e-10 * kappa
    assert rel_l2(p, oracle.poisson_solve(rhs, sim.h)) < tol
    sim.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32_dc"])
def test_graph_replay_on_the_default_stream(precision):
    """A handle bound to torch's default stream (which cannot be captured)
    replays graphs, with the results of launching every step; inside a capture
    of the caller's it launches."""
    import torch
    from cubismup_3d_b200 import initial_conditions as ic
    cells = (64, 32, 32)
    u = ic.random_solenoidal(cells, 3, lambda k: k ** 4 * np.exp(-2 * (k / 4) ** 2), rms=1.0)
    out = []
    for graphs in (True, False):
        sim = make_sim(cells, 2 * np.pi, nu=1e-3, precision=precision, scheme="upwind3_rk2")
        sim.use_graphs(graphs)
        sim.set_velocity(*u)
        sim.bind_torch_stream()
        sim.run_steps(26)
        assert (sim.prepare_run(13) > 0) == graphs
        sim.run_steps(13)
        sim.timestep(sim.calcMaxTimestep())
        out.append(sim.velocity_raw())
        sim.close()
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("cells", [(16, 16, 16), (64, 32, 16), (256, 16, 32), (32, 64, 128)])
@pytest.mark.parametrize("where", ["aligned", "offset", "in_place"])
def test_poisson_solve_of_device_arrays(oracle, cells, where):
    """cup_poisson_solve_field on device arrays: 16-byte aligned ones (read and
    written by the passes themselves), 8-byte aligned ones and the handle's own
    buffer (copied) give the same solution, which is also the handle's pressure."""
    import ctypes as C
    import torch
    from cubismup_3d_b200 import _lib as L
    nx, ny, nz = cells
    sim = make_sim(cells, 1.3)
    sim.bind_torch_stream()
    rhs = np.random.default_rng(5).standard_normal((nz, ny, nx))
    n = rhs.size
    a = torch.zeros(n + 1, dtype=torch.float64, device="cuda")
    b = torch.zeros(n + 1, dtype=torch.float64, device="cuda")
    k = 1 if where == "offset" else 0
    src = a[k:k + n]
    src.copy_(torch.from_numpy(rhs.ravel()))
    dst = sim.pressureSolver.data.view(-1) if where == "in_place" else b[k:k + n]
    L.check(L.lib().cup_poisson_solve_field(sim._h, C.c_void_p(src.data_ptr()), C.c_void_p(dst.data_ptr()),
                                            L.CUP_WHERE_DEVICE), sim._h, "poisson")
    p = dst.cpu().numpy().reshape(rhs.shape)
    assert rel_l2(p, oracle.poisson_solve(rhs, sim.h)) < 1e-12
    assert np.array_equal(sim.pressure(), p)
    assert np.array_equal(src.cpu().numpy(), rhs.ravel())
    sim.close()


@pytest.mark.parametrize("cells", [(16, 16, 16), (32, 16, 64), (64, 128, 32), (256, 32, 16), (32, 16, 256)])
@pytest.mark.parametrize("extent", [2 * np.pi, 5 * np.pi])
def test_spectral_sums_and_forcing_band(oracle, cells, extent):
    """Every line length of the mode-summing z pass, and the forcing of a band
    summed mode by mode (side 2 pi) and through the transforms (side 5 pi)."""
    nx, ny, nz = cells
    nu, dt = 1e-2, 1e-2
    u, v, w = (np.random.default_rng(k).standard_normal((nz, ny, nx)) for k in range(3))
    tke0 = 0.5 * np.mean(u * u + v * v + w * w)
    sim = make_sim(cells, extent, nu=nu, turbKinEn_target=1.3 * tke0)
    sim.set_velocity(u, v, w)
    got = sim.spectral_analysis()
    ref, E, _ = oracle.spectral(u, v, w, sim.h, nu)
    for k in ("tke", "eps", "uprime", "lambda", "Re_lambda", "l_integral", "tau_integral"):
        assert got[k] == pytest.approx(ref[k], rel=1e-10), k
    assert np.allclose(got["spectrum"], E, rtol=1e-9, atol=1e-13 * E.max())
    op = sim.pipeline[2]
    op(dt)
    forced, st = oracle.spectral_forcing(u, v, w, sim.h, nu, dt, target_tke=1.3 * tke0)
    for a, b in zip(sim.velocity(), forced):
        assert rel_l2(a, b) < 1e-12
    assert op.stats["largeModesKinEn"] == pytest.approx(st[1], rel=1e-10)
    sim.close()


@pytest.mark.parametrize("cells", [(16, 16, 16), (32, 64, 128), (256, 16, 32), (16, 256, 16)])
def test_marching_diagnostics(oracle, cells):
    """ComputeDissipation's sums and the divergence norms at several grids of the z march."""
    nx, ny, nz = cells
    sim = make_sim(cells, 2.0, nu=1e-3)
    orc = oracle.OracleSim(*cells, 2.0, nu=1e-3, CFL=0.1, rampup=0, DLM=0.0, lambda_=1.0)
    u = [0.5 * np.random.default_rng(k).standard_normal((nz, ny, nx)) for k in range(3)]
    sim.set_velocity(*u)
    orc.set_velocity(*u)
    got, ref = np.array(list(sim.compute_dissipation().values())), orc.dissipation()
    assert np.all(np.abs(got - ref) <= 1e-10 * np.abs(ref) + 1e-13 * np.abs(ref).max())
    d, od = sim.diagnostics(), orc.diagnostics()
    for k in ("ke", "div_l2", "div_max"):
        assert d[k] == pytest.approx(od[k], rel=1e-12), k
    sim.close()


@pytest.mark.parametrize("cells,position,radius", [((64, 32, 32), (0.02, 0.49, 0.25), 0.1),  # box over the edges of x and y
                                                   ((32, 16, 64), (0.3, 0.12, 0.99), 0.1),   # all of y, over the edge of z
                                                   ((16, 16, 16), (0.5, 0.5, 0.9), 0.4)])    # all of every axis
def test_sphere_rhs_terms_in_the_x_pass(cells, position, radius):
    """The step adds the obstacle's RHS terms to the RHS that it forms inside
    the first x pass; PressureRHS and PressureProjection go through an RHS
    array. The two differ by the rounding of b: a few 1e-16 of u per step."""
    from cubismup_3d_b200 import Sphere
    u = [0.3 * c for c in np.random.default_rng(4).standard_normal((3, cells[2], cells[1], cells[0]))]
    out = []
    for fused in (True, False):
        sim = make_sim(cells, 1.0, nu=1e-3, lambda_=1e6, bImplicitPenalization=True)
        sim.add_obstacle(Sphere(radius=radius, position=position, enforcedVelocity=(1.0, 0.2, 0.0),
                                bForcedInSimFrame=(True, True, True), bFixFrameOfRef=(True, True, True)))
        sim.set_velocity(*u)
        if fused:
            sim.timestep(1e-3)
        else:
            for op in sim.pipeline[:6]:
                op(1e-3)
        out.append(sim.velocity())
        sim.close()
    for a, b in zip(*out):
        assert np.isfinite(a).all() and rel_l2(a, b) < 1e-13


@pytest.mark.parametrize("cells", [(256, 16, 16), (16, 16, 256), (64, 256, 32)])
def test_run_beyond_the_stability_limit_keeps_its_rounding(cells):
    """38 FP64 upwind3 steps at CFL 0.5 with 12 nu dt / h^2 above 2: the run
    amplifies the rounding of its steps more than 1e9 times, so its results are
    those of one order of arithmetic only. The golden file holds the 1D factors
    of the initial velocity (the products below are exact in their order) and
    512 velocity values of the library before it had a second form of the FP64
    upwind3 stages and of the pressure solve; the second form is 1e-7 to 1e-3
    away. Equal arithmetic gives equal bits; 1e-9 is what FP64 results are held to."""
    import os
    g = np.load(os.path.join(os.path.dirname(__file__), "golden", "amplified_rounding_fp64.npz"))
    sx, sy, sz = (g[f"sin{n}"] for n in cells)
    cx, cy, cz = (g[f"cos{n}"] for n in cells)

    def p(a, b, c):
        return c[:, None, None] * b[None, :, None] * a[None, None, :]

    u0 = (p(sx, cy, cz) + 0.0625 * p(cx, sy, sz), -p(cx, sy, cz) + 0.0625 * p(sx, sy, cz), 0.0625 * p(sx, cy, sz))
    sim = make_sim(cells, 2 * np.pi, nu=0.01, CFL=0.5, scheme="upwind3_rk2")
    sim.set_velocity(*u0)
    sim.run_steps(38)
    key = "x".join(map(str, cells))
    got = np.stack(sim.velocity()).ravel()[g["at" + key]]
    assert rel_l2(got, g["u" + key]) < 1e-9
    sim.close()


@pytest.mark.parametrize("cells", LINES)
@pytest.mark.parametrize("scheme", ["upwind3_rk2", "ref"])
def test_step_of_both_stability_ranges_every_line_length(oracle, cells, scheme):
    """One FP64 step of a CFL number above 1/8 (Hartley passes, RHS formed in
    the x pass, one-sided stencils of both signs) and of one below, with the
    same dt, against the oracle: a few hundred roundings of u and p each."""
    nx, ny, nz = cells
    u = np.random.default_rng(sum(cells)).standard_normal((3, nz, ny, nx))
    for CFL in (0.125, 0.13):
        sim = make_sim(cells, 2.0, nu=1e-3, CFL=CFL, scheme=scheme)
        orc = oracle.OracleSim(*cells, 2.0, nu=1e-3, CFL=CFL, rampup=0, DLM=0.0, lambda_=1.0, scheme=scheme)
        sim.set_velocity(*u)
        orc.set_velocity(*u)
        sim.timestep(1e-3)
        orc.timestep(1e-3)
        for a, b in zip(sim.velocity(), orc.velocity()):
            assert rel_l2(a, b) < 1e-12, CFL
        sim.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32_dc"])
@pytest.mark.parametrize("scheme", ["upwind3_rk2", "ref"])
@pytest.mark.parametrize("sphere", [False, True])
def test_adjoint_step_of_unaligned_fields(precision, scheme, sphere):
    """Adjoint fields between 16-byte boundaries: the central scheme takes them
    (as it takes any address of their type) with the bits of aligned ones, the
    upwind3 scheme refuses them, and both refuse such a state, before anything
    is launched."""
    import torch
    from cubismup_3d_b200 import Sphere
    cells = (64, 32, 32)
    sim = make_sim(cells, 1.0, nu=1e-3, lambda_=1e6, bImplicitPenalization=True, precision=precision, scheme=scheme)
    if sphere:
        sim.add_obstacle(Sphere(radius=0.1, position=(0.5, 0.25, 0.25), enforcedVelocity=(1.0, 0.0, 0.0),
                                bForcedInSimFrame=(True, True, True), bFixFrameOfRef=(True, True, True)))
    t = sim.storage_dtype
    g = torch.Generator(device="cuda").manual_seed(2)
    shape, n = (3,) + cells[::-1], 3 * 64 * 32 * 32
    a, lam0 = (torch.randn(shape, generator=g, device="cuda", dtype=t) for _ in range(2))

    def at(x, k):  # a copy of x that starts k elements after a 256-byte boundary
        return torch.empty(n + 4, dtype=t, device="cuda")[k:k + n].view(shape).copy_(x)

    def step(state, lam):
        if not sphere:
            sim.adjoint_step(state, 1e-3, lam)
            return [lam]
        g_chi = torch.zeros(sim.shape, dtype=torch.float64, device="cuda")
        g_vel = torch.zeros(3, dtype=torch.float64, device="cuda")
        sim.adjoint_step_obstacle(state, 1e-3, lam, (1.0, 0.0, 0.0), g_chi, g_vel)
        return [lam, g_chi, g_vel]

    want = step(a, at(lam0, 0))
    for k in (1, 2, 3):
        lam = at(lam0, k)
        if lam.data_ptr() % 16 == 0:
            continue
        if scheme == "ref":
            for x, y in zip(step(a, lam), want):
                assert torch.equal(x, y)
        else:
            with pytest.raises(ValueError):
                step(a, lam)
            assert torch.equal(lam, lam0)
    lam = at(lam0, 0)
    with pytest.raises(ValueError):
        step(at(a, 1), lam)
    assert torch.equal(lam, lam0)
    sim.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32_dc"])
@pytest.mark.parametrize("kind", ["free", "forced", "moving"])
def test_run_steps_like_single_steps(precision, kind, tmp_path, monkeypatch):
    """run_steps chains dt on the device (forced runs read it back with the mode
    sums, runs with a moving sphere before each step): the same launches with
    the same dt as calcMaxTimestep + timestep, so the same bits, clock and
    statistics, dt being the last step's."""
    import ctypes as C
    from cubismup_3d_b200 import Sphere, _lib as L
    monkeypatch.chdir(tmp_path)  # timestep of a forced run writes forcingData.dat
    cells, n = (64, 32, 32), 5
    u = [0.2 * c for c in np.random.default_rng(8).standard_normal((3,) + cells[::-1])]
    out = []
    for chained in (True, False):
        kw = {"forced": dict(turbKinEn_target=0.1), "moving": dict(lambda_=1e6, bImplicitPenalization=True)}.get(kind, {})
        sim = make_sim(cells, 2 * np.pi if kind == "forced" else 1.0, nu=1e-3, precision=precision,
                       scheme="upwind3_rk2", **kw)
        if kind == "moving":
            sim.add_obstacle(Sphere(radius=0.1, position=(0.5, 0.25, 0.25), enforcedVelocity=(1.0, 0.0, 0.0),
                                    bForcedInSimFrame=(True, True, True)))
        sim.set_velocity(*u)
        if chained:
            st = sim.run_steps(n)
        else:
            for _ in range(n):
                st = sim.timestep(sim.calcMaxTimestep())
        assert sim.dt == st.dt and sim.step == st.step == n and sim.time == st.time
        forcing = (C.c_double * 6)()
        L.check(L.lib().cup_get_forcing_stats(sim._h, forcing), sim._h, "forcing stats")
        assert (forcing[0] > 0) == (kind == "forced")  # totalKinEn of the last step's forcing
        out.append((st.dt, st.time, st.umax, st.kinetic_energy, list(st.force) + forcing[:], sim.velocity(), sim.calcMaxTimestep()))
        sim.close()
    a, b = out
    assert a[:5] == b[:5] and a[6] == b[6]
    for x, y in zip(a[5], b[5]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("precision", ["fp64", "fp32_dc"])
def test_whole_solves_refuse_a_spectral_window(precision):
    """A handle whose z pass is that of a pencil of a larger grid refuses whole
    solves and steps before it changes anything; its single passes run, and a
    window of its own grid gives the solves back."""
    import ctypes as C
    import torch
    from cubismup_3d_b200 import _lib as L
    cells = (32, 16, 16)
    sim = make_sim(cells, 1.0, nu=1e-3, precision=precision)
    sim.bind_torch_stream()
    u = np.random.default_rng(1).standard_normal((3,) + cells[::-1])
    sim.set_velocity(*u)
    before = sim.velocity_raw()
    H, lib = sim._h, L.lib()
    L.check(lib.cup_set_spectral_window(H, 16, 32), H, "window")
    rhs, p = (torch.ones(sim.shape, dtype=torch.float64, device="cuda") for _ in range(2))
    lam, count = torch.zeros_like(before), C.c_int()
    for call in (lambda: lib.cup_step(H, 1e-3, None), lambda: lib.cup_run(H, 1, None),
                 lambda: lib.cup_prepare_run(H, 1, C.byref(count)), lambda: lib.cup_poisson_solve(H, None),
                 lambda: lib.cup_pressure_projection(H, 1e-3, None),
                 lambda: lib.cup_poisson_solve_field(H, C.c_void_p(rhs.data_ptr()), C.c_void_p(p.data_ptr()),
                                                     L.CUP_WHERE_DEVICE),
                 lambda: lib.cup_adjoint_step(H, *[C.c_void_p(before[i].data_ptr()) for i in range(3)], 1e-3,
                                              *[C.c_void_p(lam[i].data_ptr()) for i in range(3)])):
        assert call() == L.CUP_ERR_STATE
    assert torch.equal(sim.velocity_raw(), before) and torch.equal(p, torch.ones_like(p))
    L.check(lib.cup_poisson_pass(H, C.c_void_p(rhs.data_ptr()), 2), H, "pass")
    L.check(lib.cup_set_spectral_window(H, 0, 16), H, "window")
    sim.timestep(1e-3)
    assert np.isfinite(sim.velocity_raw().cpu().numpy()).all()
    sim.close()


def graph_pair(cells, precision, sphere):
    """(graphs on or off, simulation on a stream of torch's, its stream) after the four steps that make FP32-DC's history."""
    import torch
    from cubismup_3d_b200 import Sphere
    u = [0.3 * c for c in np.random.default_rng(6).standard_normal((3,) + cells[::-1])]
    for graphs in (True, False):
        sim = make_sim(cells, 1.0, nu=1e-3, precision=precision, scheme="upwind3_rk2", lambda_=1e6,
                       bImplicitPenalization=True)
        if sphere:
            sim.add_obstacle(Sphere(radius=0.1, position=(0.5, 0.25, 0.25), enforcedVelocity=(1.0, 0.0, 0.0),
                                    bForcedInSimFrame=(True, True, True), bFixFrameOfRef=(True, True, True)))
        sim.use_graphs(graphs)
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            sim.bind_torch_stream()
        sim.set_velocity(*u)
        sim.run_steps(4)
        yield graphs, sim, stream


@pytest.mark.parametrize("precision", ["fp64", "fp32_dc"])
@pytest.mark.parametrize("sphere", [False, True])
def test_replayed_runs_match_launched_ones(precision, sphere):
    """Runs of 20 and 9 steps whose graphs prepare_run has captured (the 6-step
    one is replayed three times and once, the tails one step at a time), then
    single steps on cached graphs: the same bits, clock, statistics and launch
    count as launching every step."""
    out = []
    for graphs, sim, _ in graph_pair((64, 32, 32), precision, sphere):
        got = []
        for n, captured in ((20, 3), (9, 4)):  # one 6-step graph and the tail's 2 or 3 steps
            assert sim.prepare_run(n) == (captured if graphs else 0)
            n0 = sim.launch_count()
            st = sim.run_steps(n)
            got += [st.step, st.time, st.dt, st.umax, st.kinetic_energy, list(st.force), sim.launch_count() - n0,
                    np.stack(sim.velocity()), sim.pressure()]
        for _ in range(8):
            st = sim.timestep(sim.calcMaxTimestep())
            got += [st.time, st.dt, st.kinetic_energy, list(st.force)]
        out.append(got + [np.stack(sim.velocity())])
        sim.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("precision", ["fp64", "fp32_dc"])
def test_step_inside_a_capture_of_the_callers(precision):
    """A step inside a capture of the caller's is launched into it, although the
    handle has a graph of its own for that step; replaying the caller's graph
    takes the step."""
    import torch
    out = []
    for graphs, sim, stream in graph_pair((64, 32, 32), precision, False):
        assert (sim.prepare_run(1) > 0) == graphs
        if graphs:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream):
                sim.timestep(1e-3, stats=False)
            with torch.cuda.stream(stream):
                g.replay()
        else:
            sim.timestep(1e-3, stats=False)
        sim.sync()
        first = sim.velocity()
        st = sim.run_steps(3)
        out.append((*first, *sim.velocity(), st.time, st.dt))
        if graphs:
            g.reset()
        sim.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)
