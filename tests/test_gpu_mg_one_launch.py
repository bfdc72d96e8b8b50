"""The multigrid cycle's coarse levels in one cooperative launch and as one launch a step (option
p.mg_persistent) give the same bits, on hierarchies whose first coarse level is below and above the
65,536 rows from which the prolongation is a step of its own."""
import numpy as np
import pytest

from sysu_cfd_heat_gb300 import meshgen as mg
from sysu_cfd_heat_gb300._lib import lib
from sysu_cfd_heat_gb300.solver import NavierStokesSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", ["hex 7x6x5", "tet 9x8x7", "hex 33x32x31", "hex 91x90x89"])
def test_same_bits(tmp_path, mesh):
    kind, size = mesh.split()
    nx, ny, nz = map(int, size.split("x"))
    m = mg.lid_cavity_tet(nx, ny, nz, jitter=0.2) if kind == "tet" else mg.box_hex(nx, ny, nz, side_ids={"y1": mg.INLET_ID})
    p = mg.write_case(str(tmp_path), m, mg.cavity_param("x", 20, mu=0.0025))
    fields, launches, iters = {}, {}, {}
    for form in (None, 0, 1):
        opts = {"rtc": 1e-8, "p.precond": 4, "p.maxit": 5000, "mom.mixed": 1}
        if form is not None:
            opts["p.mg_persistent"] = form
        with NavierStokesSolver(p, opts) as s:
            assert s.iterate(1) == 1  # sets the hierarchy up
            before = lib().sysu_kernel_launches()
            assert s.iterate(2) == 2
            launches[form] = lib().sysu_kernel_launches() - before
            iters[form] = s.solve_stats()["p"]["iters"][0]
            fields[form] = {f: s.get(f) for f in ("U", "V", "W", "P")}
    for f in ("U", "V", "W", "P"):
        assert np.array_equal(fields[0][f], fields[1][f]) and np.array_equal(fields[0][f], fields[None][f]), f
    assert iters[0] == iters[1] == iters[None]
    assert launches[None] == launches[1] < launches[0]  # a chosen form is the one that runs
