"""The line sweeps of the advection stage against the CPU oracle where they can
go wrong: an upwind side that flips from cell to cell (white noise), lines
with no variation at all (every smoothness indicator at its floor), the frame
velocity alone deciding the side, walls, coarse-fine faces, and meshes of one
block and of fewer blocks than the launch has CTAs.

Tolerance: 1e-12 of max|u|, as the other operator tests; both sides are FP64
and differ in summation order only (a stage is some 200 operations a cell, so
rounding stays below 1e-13).
"""
import numpy as np
import pytest

import cup3d_b200 as cup
import oracle
from tests.meshes import cell_centres, make_ctx, oracle_mesh

pytestmark = pytest.mark.gpu


def _box(bpd, bc):
    flags = f"-bpdx {bpd[0]} -bpdy {bpd[1]} -bpdz {bpd[2]} -levelMax 1 -extent 1 -nu 0.01"
    flags += f" -BC_x {bc[0]} -BC_y {bc[1]} -BC_z {bc[2]} -uinfx 0.1 -uinfy -0.05 -advection "
    return flags


CASES = {
    "one_block": ((1, 1, 1), ("periodic", "periodic", "periodic")),
    "thin_walls": ((3, 1, 2), ("wall", "freespace", "periodic")),
}


@pytest.mark.parametrize("field", ["noise", "constant", "shear"])
@pytest.mark.parametrize("scheme", ["upwind5", "weno5"])
@pytest.mark.parametrize("name", ["one_block", "thin_walls", "amr2_free", "amr3_mixed", "amr3_periodic"])
def test_line_sweeps_match_oracle(name, scheme, field):
    if name in CASES:
        cfg = cup.config(_box(*CASES[name]) + scheme, device=0)
        ctx = cup.Context(cfg)
        ctx.set_mesh_uniform()
        level, index, _ = ctx.blocks()
        m = oracle.Mesh(level, index, list(cfg.bpd), cfg.level_max, list(cfg.bc), cfg.extent)
    else:
        ctx = make_ctx(name, device=0, extra="-nu 0.01 -uinfx 0.1 -uinfy -0.05 -advection " + scheme)
        m = oracle_mesh(ctx)
    n = ctx.nb * 512
    rng = np.random.default_rng(7)
    if field == "noise":
        vel = rng.standard_normal(3 * n)
    elif field == "constant":  # u + uinf is zero in y: the side is the lower one's
        vel = np.concatenate([np.full(n, 0.3), np.full(n, 0.05), np.zeros(n)])
    else:
        z = cell_centres(ctx)[0][:, 2]
        vel = np.concatenate([np.where(z > z.mean(), 1.0, -1.0), 0 * z, 1e-9 * rng.standard_normal(n)])
    dt = 0.2 * m.hmin / np.abs(vel).max()
    ctx.upload("vel", vel)
    ctx.advect_diffuse(dt)
    got = ctx.download("vel")
    ref = m.advect_diffuse(vel, dt, 0.01, uinf=(0.1, -0.05, 0.0), scheme=1 if scheme == "weno5" else 0)
    assert np.abs(got - ref).max() < 1e-12 * np.abs(vel).max()
