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
