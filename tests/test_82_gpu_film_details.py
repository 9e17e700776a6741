"""Films whose mirror runs inside the step's kernels, where the inputs are out
of the ordinary: a negative gap_id (every gap_id but 0 mirrors layer z to
Lz - z, mirror.F:9-36; only positive ones freeze layers), against the oracle,
and planes that are no multiple of a 16-byte vector."""
import ctypes as C

import numpy as np
import pytest

import helpers
import oracle_lib
from feram_b200 import _capi as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [A.FG_PREC_FP64, A.FG_PREC_MIXED])
@pytest.mark.parametrize("L", ["8 12 10", "10 9 6"])
def test_negative_gap_id_steps_match_oracle(fg, prec, L):
    p = helpers.params(L=L, kelvin="250", bulk_or_film="'film'", gap_id="-2", external_E_field="0.001 -0.0005 0.002")
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
    tol = 1e-9 if prec == A.FG_PREC_FP64 else 2e-5  # as the films of the other gap_ids
    for k in ("dipoR", "dipoP", "dVddi"):
        a, b = A.physical(sg[k], p), A.physical(so[k], p)
        assert np.abs(a - b).max() <= tol * np.abs(b).max(), k
    assert abs(sg["s"] - so["s"]) <= tol


@pytest.mark.parametrize("kind,L,gap", [("film", "10 9 15", 1), ("film", "10 9 6", 2), ("epit", "6 5 4", 0)])
def test_mixed_kinetic_energy_of_planes_cut_off_a_vector(fg, kind, L, gap):
    """Planes that are no multiple of four sites take the site loop, which forms
    p^2/m of the FP32 momenta in FP64: the kinetic energy that a step reports
    is that of the momenta it leaves, to the rounding of an FP64 sum of 3 N
    positive terms in any order (3 N 2^-53); FP32 products are off by 1e-9."""
    extra = {"epi_strain": "0.01"} if kind == "epit" else {}
    p = helpers.params(L=L, kelvin="250", bulk_or_film=f"'{kind}'", gap_id=str(gap), **extra)
    e = A.fg_energy()
    with fg.Context(p, A.FG_PREC_MIXED) as ctx:
        ctx.build_tables()
        ctx.set_state(helpers.seeded_u(p, 5, sigma=0.08), helpers.seeded_p(p, 5, sigma=0.01))
        ctx.mirror_force_mirror()
        for _ in range(3):
            ctx.nose_poincare(e)
            step = e.dipo_kinetic
            ke = ctx.kinetic_energy_dipo()
            assert abs(step - ke) <= 3 * p.N * 2.0**-53 * ke, (step, ke)


@pytest.mark.parametrize("prec", [A.FG_PREC_FP64, A.FG_PREC_MIXED])
@pytest.mark.parametrize("kind,L,gap", [("film", "12 10 8", 0), ("epit", "8 12 10", 2)])
def test_device_field_wave_through_run_steps(fg, prec, kind, L, gap):
    """The field wave set in the mirrored drift's launch, over two graphs of
    eight steps and three single ones (molecular-dynamics.F:66-76), against
    the oracle's molecular_dynamics.  Tolerances as for the films' steps."""
    extra = {"epi_strain": "-0.01"} if kind == "epit" else {}
    p = helpers.params(L=L, kelvin="280", bulk_or_film=f"'{kind}'", gap_id=str(gap), E_wave_type="'triangular_sin'",
                       external_E_field="0.001 -0.0005 0.002", n_E_wave_period="12", n_thermalize="2", n_average="17",
                       **extra)
    u, q = helpers.seeded_u(p, 31, sigma=0.05), helpers.seeded_p(p, 31, sigma=0.01)
    n = 19
    w0 = (C.c_double * 3)()
    amp = (C.c_double * 3)(*p.external_E_field)
    assert A.lib().fg_wave(p.E_wave_type, 0, p.n_thermalize, p.n_E_wave_period, amp, w0) == 0
    o = oracle_lib.Oracle(p)
    o.set_state(u, q)
    o.set_uniform_E(list(w0))
    eo = o.force()
    eo.dipo_kinetic = o.kinetic_energy_dipo()
    o.md(1, n, 1, eo)
    so = o.get_state()
    with fg.Context(p, prec) as ctx:
        ctx.build_tables()
        ctx.set_state(u, q)
        ctx.set_uniform_E(list(w0))
        e = ctx.mirror_force_mirror()
        e.dipo_kinetic = ctx.kinetic_energy_dipo()
        ctx.nose_poincare_hamiltonian(e)
        ctx.set_thermostat(1.0, 0.0, e.H_Nose_Poincare)
        ctx.set_wave(True, 0)
        eg = ctx.run_steps(n)
        sg = ctx.get_state()
    tol = 1e-9 if prec == A.FG_PREC_FP64 else 2e-5
    for k in ("dipoR", "dipoP"):
        a, b = A.physical(sg[k], p), A.physical(so[k], p)
        assert np.abs(a - b).max() <= tol * np.abs(b).max(), k
    assert abs(sg["s"] - so["s"]) <= tol
    ee = helpers.energy_errors(eg, eo, A.POTENTIAL_FIELDS + ["dipo_kinetic"])
    assert max(ee.values()) <= tol, ee
