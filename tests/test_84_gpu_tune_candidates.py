"""fg_tune and fg_batch_tune time every distinct k-space tile, also where the
widths do not divide Lx/2 (their tiles then end short).  Lx/2 = 5 with few and
long pencils: the widest tile leaves most SMs without one (a step takes 43.3 us
at the widest and 32.5 at the narrowest in FP64, 54.5 and 43.9 mixed), so that a
tuner that sees the narrower ones does not keep the widest."""
import pytest

import feram_b200 as fb
import helpers
from feram_b200 import _capi as A

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _no_wisdom(fg):
    fb.wisdom_forget()
    yield
    fb.wisdom_forget()


@pytest.mark.parametrize("prec", [A.FG_PREC_FP64, A.FG_PREC_MIXED])
@pytest.mark.parametrize("mode", ["solo", "batch"])
def test_tuner_times_tiles_that_do_not_divide_the_row(fg, prec, mode):
    p = helpers.params(L="10 8 160", kelvin="300")
    u, q = helpers.seeded_u(p, 5, sigma=0.05), helpers.seeded_p(p, 5, sigma=0.01)
    with fb.Context(p, prec) if mode == "solo" else fb.Batch([p], prec) as c:
        ctx = c if mode == "solo" else c[0]
        ctx.build_tables()
        ctx.set_state(u, q)
        ctx.mirror_force_mirror()
        c.tune(steps=16)
    line = next(v for v in fb.wisdom_export().splitlines() if v.startswith(mode + " "))
    zcw = int(line.split()[6])
    assert 0 < zcw < (8 if prec == A.FG_PREC_MIXED else 4), line
