"""The calls of the stepping loop from a thread whose current device is not the
context's (a program with a context per GPU and worker threads): the field and
the thermostat set between steps take effect as on the context's own device."""
import threading

import numpy as np
import pytest
import torch

import helpers
from feram_b200 import _capi as A

pytestmark = pytest.mark.gpu


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_field_and_thermostat_from_a_thread_on_another_device(fg):
    p = helpers.params(L="8 8 8", kelvin="300")
    u = helpers.seeded_u(p, 3, sigma=0.08)

    def loop(ctx, out):
        e = A.fg_energy()
        for k in range(3):
            ctx.set_uniform_E([0.0, 0.0, 1e-3 * k])
            ctx.nose_poincare(e)
        out.append(e.total)

    got = []
    with torch.cuda.device(1):
        for threaded in (False, True):
            with fg.Context(p, A.FG_PREC_FP64) as ctx:
                ctx.build_tables()
                ctx.set_state(u)
                ctx.nose_poincare(A.fg_energy())
                if threaded:
                    t = threading.Thread(target=loop, args=(ctx, got))  # starts on device 0
                    t.start()
                    t.join()
                else:
                    loop(ctx, got)
    assert len(got) == 2 and np.isfinite(got[0]) and got[0] == got[1]
