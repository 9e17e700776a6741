"""Nose-Poincare steps of films, whose mirror runs inside the drift and the
assembly, against the oracle's: every gap_id with its parity of Lz (layers
without a partner at z = 0 and Lz / 2), layers that are and are not multiples
of a 16-byte vector (the vector and the scalar loop), an epitaxial cell, and a
field with components along x and y, whose energy is not the same on a layer
and its image.  Tolerances as for the bulk steps."""
import ctypes as C

import numpy as np
import pytest

import helpers
import oracle_lib
from feram_b200 import _capi as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [A.FG_PREC_FP64, A.FG_PREC_MIXED])
@pytest.mark.parametrize("kind,L,gap", [("film", "12 10 8", 0), ("film", "16 16 9", 1), ("film", "10 9 15", 1),
                                        ("film", "8 12 10", 2), ("film", "10 9 6", 2), ("epit", "10 9 4", 0),
                                        ("epit", "32 32 16", 2)])
def test_film_steps_match_oracle(fg, prec, kind, L, gap):
    extra = {"epi_strain": "0.01"} if kind == "epit" else {}
    p = helpers.params(L=L, kelvin="250", bulk_or_film=f"'{kind}'", gap_id=str(gap),
                       external_E_field="0.001 -0.0005 0.002", **extra)
    u, q = helpers.seeded_u(p, 21, sigma=0.08), helpers.seeded_p(p, 21, sigma=0.01)
    o = oracle_lib.Oracle(p)
    o.set_state(u, q)
    eo = o.force()
    eo.dipo_kinetic = o.kinetic_energy_dipo()
    with fg.Context(p, prec) as ctx:
        ctx.build_tables()
        ctx.set_state(u, q)
        eg = ctx.mirror_force_mirror()
        o.set_state(None, None, 1.0, 0.0, 0.0)
        h = o.L.oracle_nose_poincare_hamiltonian(o.h, C.byref(eo))
        o.set_state(None, None, 1.0, 0.0, h)
        ctx.set_thermostat(1.0, 0.0, h)
        for _ in range(10):
            o.nose_poincare(eo)
            ctx.nose_poincare(eg)
        so, sg = o.get_state(), ctx.get_state()
    tol = 1e-9 if prec == A.FG_PREC_FP64 else 2e-5
    for k in ("dipoR", "dipoP", "dVddi"):  # the images too
        a, b = A.physical(sg[k], p), A.physical(so[k], p)
        assert np.abs(a - b).max() <= tol * np.abs(b).max(), k
    assert abs(sg["s"] - so["s"]) <= tol
    ee = helpers.energy_errors(eg, eo, A.POTENTIAL_FIELDS + ["dipo_kinetic"])
    assert max(ee.values()) <= tol, ee
