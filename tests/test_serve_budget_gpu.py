"""What a served set takes on the device against what its admission was charged."""
import pytest

from cosmosphere_b200 import capi, inputs
from test_serve_gpu import thermo_for

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300, method="thread")]


@pytest.mark.parametrize("quintic,mixed", [(False, False), (False, True), (True, False), (True, True)])
def test_a_solved_set_holds_no_more_than_it_was_charged(quintic, mixed):
    """The admission estimate covers what a set takes, so that concurrent admissions stay inside
    the budget.  (Where h scatters by more, the lists of a mixed solve may take a tenth more.)"""
    hf = 1.0 if quintic else 1.2
    L = capi.load(quintic)
    L.cosmo_set_precision(1 if mixed else 0)
    try:
        for make in (lambda n: inputs.uniform_box(n, hfac=hf, seed=50),
                     lambda n: inputs.plummer(n, hfact=hf, lnsigma=0.3, seed=51)):
            for n in (700, 8000, 60000):
                S = capi.Server(slots=1, quintic=quintic)
                try:
                    base = S.server_stat("device_bytes")
                    p = make(n)
                    assert S.wait(S.submit(p, thermo_for(p, hf), hfact=hf, keep=True))[0] == 1
                    held = S.server_stat("device_bytes") - base
                    est = S.server_stat("bytes_fixed") + S.server_stat("bytes_per_particle") * p.n
                    assert 0.4 * (est - S.server_stat("bytes_fixed")) <= held <= est
                finally:
                    S.stop()
    finally:
        L.cosmo_set_precision(0)
