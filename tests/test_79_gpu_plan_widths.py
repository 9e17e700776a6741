"""Plan widths that are no power of two (fg_set_plan and fg_wisdom_import take
any number): every k-space tile is processed, whatever the width.  A plan
changes the order of the energies' partial sums only, so the forces are those
of the default plan bit for bit and the energies agree to the rounding of FP64
sums (at most 1e5 terms here: 1e5 * 2^-53 of the summed energy terms).
Compile-time and runtime lengths, Lx/2 odd and divisible by 3, and the
per-site Z* pass."""
import numpy as np
import pytest

import feram_b200 as fb
import helpers
from feram_b200 import _capi as A

pytestmark = pytest.mark.gpu

WIDTHS = (1, 3, 5, 6, 7, 9, 12)


@pytest.fixture(autouse=True)
def _no_wisdom(fg):
    fb.wisdom_forget()
    yield
    fb.wisdom_forget()


def _force(ctx, u):
    ctx.set_state(u)
    e = ctx.mirror_force_mirror()
    return ctx.get_state()["dVddi"].copy(), e


def _check(got, want):
    assert np.array_equal(got[0], want[0])
    assert max(helpers.energy_errors(got[1], want[1]).values()) <= 1e5 * 2.0**-53 * 1e3  # energy_errors' 1e-3 floor


@pytest.mark.parametrize("prec", [A.FG_PREC_FP64, A.FG_PREC_MIXED])
@pytest.mark.parametrize("L", ["16 10 16", "18 5 9", "20 6 24", "48 4 12", "24 5 128"])
def test_any_width_gives_the_default_plans_force(fg, prec, L):
    p = helpers.params(L=L, kelvin="300")
    u = helpers.seeded_u(p, 3, sigma=0.1)
    with fb.Context(p, prec) as ctx:
        ctx.build_tables()
        want = _force(ctx, u)
        for z in WIDTHS:
            ctx.set_plan(z)
            _check(_force(ctx, u), want)
    name = "mixed" if prec == A.FG_PREC_MIXED else "fp64"
    assert fb.wisdom_import("feram_b200 wisdom 1\nsolo %s %s 9 3 1\n" % (name, L)) == 1
    with fb.Context(p, prec) as ctx:
        ctx.build_tables()
        _check(_force(ctx, u), want)


@pytest.mark.parametrize("prec", [A.FG_PREC_FP64, A.FG_PREC_MIXED])
def test_any_width_with_a_zstar_per_site(fg, prec):
    p = helpers.params(L="24 6 8", kelvin="300", P_kappa2="5.502 4.61 4.61", P_alpha="110.4 98.2 98.2",
                       P_gamma="-163.1 -151.0 -151.0", mass_amu="39.0 47.5 47.5", Z_star="9.956 7.2 7.2")
    rng = np.random.default_rng(4)
    relaxor = np.ones((p.Lz, p.Ly + p.padding_y, 2 * (p.Lx // 2 + 1)), dtype=np.int32)
    relaxor[:, :p.Ly, :p.Lx] = rng.integers(1, 3, size=(p.Lz, p.Ly, p.Lx))
    u = helpers.seeded_u(p, 5, sigma=0.1)
    with fb.Context(p, prec) as ctx:
        ctx.build_tables()
        ctx.upload_site_arrays(relaxor=relaxor)
        want = _force(ctx, u)
        for z in WIDTHS:
            ctx.set_plan(z)
            _check(_force(ctx, u), want)


@pytest.mark.parametrize("prec", [A.FG_PREC_FP64, A.FG_PREC_MIXED])
@pytest.mark.parametrize("L", ["16 16 16", "32 32 32", "24 24 24", "20 18 20", "18 5 9"])
def test_fft_entry_points_at_any_width(fg, prec, L):
    """The 3-component transforms, whose z tiles follow the plan but not the
    k-space pass's default, against numpy: relative to the largest bin, 5
    roundings per radix-2 level of the forward transform and as many again
    for the way back."""
    p = helpers.params(L=L)
    f = helpers.fp32_config(helpers.seeded_u(p, 8, sigma=1.0))
    x = A.physical(f, p)
    want = np.fft.rfftn(x, axes=(0, 1, 2))
    tol = 5 * np.log2(p.N) * (2.0**-53 if prec == A.FG_PREC_FP64 else 2.0**-24)
    with fb.Context(p, prec) as ctx:
        for z in (0,) + WIDTHS:
            ctx.set_plan(z)
            X = ctx.fft_r2c3(f)[:p.Lz, :p.Ly, :p.Lx // 2 + 1]
            assert np.abs(X - want).max() <= tol * np.abs(want).max(), z
            back = A.physical(ctx.fft_c2r3(ctx.fft_r2c3(f)), p) / p.N
            assert np.abs(back - x).max() <= 2 * tol * np.abs(x).max(), z
