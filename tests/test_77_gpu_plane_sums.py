"""The mixed path's homogeneous strain, which follows the FP64 plane sums of
u_i u_j instead of the FP32 spectrum's k = 0 values, against the FP64 path's
for the same (FP32-representable) u: one size for each forward x-y kernel that
writes the sums (compile-time planes, two runtime stages, general plans) and
the films' mirrored planes.

Tolerance: a product is rounded once and a thread's partial sum over at most
16 products about 5 times, by 2^-24 / sqrt(3) each in rms; N / 16 such sums
average it, and the strain is a well-conditioned 6 x 6 map of the result (3).
Five rms: 5 * 3 * sqrt(6 / 3) * 2^-24 / sqrt(N / 16)."""
import numpy as np
import pytest

import helpers
from feram_b200 import _capi as A

pytestmark = pytest.mark.gpu


def _tol(n):
    return 15 * np.sqrt(2.0) * 2.0**-24 / np.sqrt(n / 16)


@pytest.mark.parametrize("L,kw", [("8 5 32", {}), ("16 16 16", {}), ("24 24 24", {}), ("40 18 20", {}), ("64 64 64", {}),
                                  ("200 8 6", {}), ("256 64 4", {}), ("128 128 8", {}),
                                  ("32 32 15", {"bulk_or_film": "'film'", "gap_id": "1"}),
                                  ("32 32 16", {"bulk_or_film": "'epit'", "epi_strain": "-0.01"})])
def test_strain_of_the_mixed_path(fg, L, kw):
    p = helpers.params(L=L, kelvin="300", **kw)
    u = helpers.fp32_config(helpers.seeded_u(p, 11, sigma=0.1) + 0.05)
    st = {}
    for prec in (A.FG_PREC_FP64, A.FG_PREC_MIXED):
        with fg.Context(p, prec) as ctx:
            ctx.build_tables()
            ctx.set_state(u)
            e = ctx.mirror_force_mirror()
            st[prec] = np.array(ctx.get_state()["strain"]), e
    (a, ea), (b, eb) = st[A.FG_PREC_FP64], st[A.FG_PREC_MIXED]
    n = np.prod([int(v) for v in L.split()])
    assert np.abs(b - a).max() <= _tol(n) * np.abs(a).max()
    for k in ("homo_strain", "homo_coupling"):
        x, y = getattr(ea, k), getattr(eb, k)
        assert abs(y - x) <= 2 * _tol(n) * abs(x), k  # quadratic and bilinear in the strain
