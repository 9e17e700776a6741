"""The k-space pass and the x-y passes on 16-byte elements (two FP32
transforms or one FP64 transform per element) against the oracle, at the
shapes where their tiles can go wrong: 4- and 2-element tiles, Nyquist tiles
that end inside a tile (Ly no multiple of the tile, odd Ly), every
compile-time Lz and x-y plane, a plane with compile-time transforms next to a
runtime Lz and the other way round, and the acoustic field.

Tolerances as for the other sizes: the FP64 path's rounding, and the mixed
path's FP32 transforms, relative to the rms force (worst site) and to the
summed energy terms."""
import numpy as np
import pytest

import helpers
import oracle_lib
from feram_b200 import _capi as A

pytestmark = pytest.mark.gpu

FORCE = {A.FG_PREC_FP64: 1e-12, A.FG_PREC_MIXED: 1e-6}
ENERGY = {A.FG_PREC_FP64: 1e-12, A.FG_PREC_MIXED: 1e-5}


@pytest.mark.parametrize("prec", [A.FG_PREC_FP64, A.FG_PREC_MIXED])
@pytest.mark.parametrize("L", ["16 10 16", "8 5 32", "24 6 48", "12 5 64", "20 9 64", "8 3 128", "16 6 128", "24 5 24",
                               "10 6 24", "16 16 9", "48 48 10", "32 32 24", "64 64 6", "30 4 16"])
def test_force_matches_oracle(fg, prec, L):
    p = helpers.params(L=L, kelvin="300")
    u = helpers.fp32_config(helpers.seeded_u(p, 7, sigma=0.1))
    o = oracle_lib.Oracle(p)
    o.set_state(u)
    eo = o.force()
    so = o.get_state()
    for zcw in (0, 4, 2):
        with fg.Context(p, prec) as ctx:
            ctx.build_tables()
            if zcw:
                ctx.set_plan(zcw)
            ctx.set_state(u)
            eg = ctx.mirror_force_mirror()
            worst, rms = helpers.force_error(ctx.get_state()["dVddi"], so["dVddi"], p)
            assert max(worst, rms) <= FORCE[prec], (zcw, worst, rms)
            ee = helpers.energy_errors(eg, eo)
            assert max(ee.values()) <= ENERGY[prec], (zcw, ee)


@pytest.mark.parametrize("prec", [A.FG_PREC_FP64, A.FG_PREC_MIXED])
@pytest.mark.parametrize("L", ["16 6 24", "8 5 64", "16 4 128"])
def test_acoustic_step_matches_oracle(fg, prec, L):
    p = helpers.params("zzzlf.feram", L=L, kelvin="200")
    f = [helpers.fp32_config(helpers.seeded_u(p, 20 + i, sigma=s)) for i, s in enumerate((0.06, 0.01, 0.003, 0.004))]
    o = oracle_lib.Oracle(p)
    o.set_state(f[0], f[1])
    o.set_acou(f[2], f[3])
    eo, eg = A.fg_energy(), A.fg_energy()
    with fg.Context(p, prec) as ctx:
        ctx.build_tables()
        ctx.set_state(f[0], f[1])
        ctx.set_acou(f[2], f[3])
        for step in range(3):
            o.leapfrog(eo, step)
            ctx.leapfrog(eg, step)
        g, r = ctx.get_acou(), o.get_acou()
    tol = 1e-11 if prec == A.FG_PREC_FP64 else 1e-5
    for k in ("acouR", "acouP", "dVdacR"):
        a, b = A.physical(g[k], p), A.physical(r[k], p)
        assert np.abs(a - b).max() <= tol * np.abs(b).max(), k
