"""The rounding of the single-run stepper's exponents: one prescribed step from a
state variable of almost zero, so that its new value is the rate b/dc V0 e^{(f0 - psi)/b}
with (f0 - psi)/b of 55 to 60, whose rounding is the larger part of the rate's error.
The rms error over the cells against long double is that of the reference formula
(the exponent a rounded quotient: half a unit in its last place) within 10 %; a
product with 1/b has 1.3 times it.  Four lanes per cell, and a thread per cell."""
import numpy as np
import pytest
import torch

from pyquake3d_gb300.QDsim_gpu import DenseDeviceSim

pytestmark = pytest.mark.gpu
# the reference's tableau (src/QDsim_gpu.py:1266-1397)
ROWS = ((1 / 5,), (3 / 40, 9 / 40), (44 / 45, -56 / 15, 32 / 9), (19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729),
        (9017 / 3168, -355 / 33, -46732 / 5247, 49 / 176, -5103 / 18656),
        (35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84))


def _psi(s, v0, h, T, product=False):
    """The state variable after one step in the type T, by the reference formula (with
    product: (f0 - psi) * (1/b) for the quotient)."""
    b, dc, f0, y = (s[k].astype(T) for k in ("b", "dc", "f0", "state"))
    k = []
    for row in ((),) + ROWS[:-1]:
        d = f0 - (y + T(h) * sum(T(w) * q for w, q in zip(row, k)))
        k.append(b / dc * (T(v0) * np.exp(d * (1 / b) if product else d / b)))
    return y + T(h) * sum(T(w) * q for w, q in zip(ROWS[-1], k))


@pytest.mark.parametrize("N", [4000, 6000])
def test_exponents_are_rounded_quotients(cuda, N):
    rng = np.random.default_rng(N)
    b = rng.uniform(0.005, 0.01, N)
    s = {k: np.zeros(N) for k in ("slip1", "slip2", "slip", "Tt", "fric", "slipv", "slipv1", "slipv2", "rake", "rake0",
                                  "shear_loading", "normal_loading", "Tt2o")}
    s.update(a=np.full(N, 0.02), b=b, dc=10 ** rng.uniform(-2, -1, N), f0=b * rng.uniform(55.0, 60.0, N),
             Tno=np.full(N, 50.0), Tt1o=np.full(N, 1.0), state=np.full(N, 1e-30))
    v0, h = 1e-30, 1e-4
    sim = DenseDeviceSim(torch.zeros((3 * N, 2 * N), dtype=torch.float64, device=cuda), s, mu=32038120320.0, Cs=3464.0,
                         V0=v0, Vpl=0.0)
    sim.step(1, h_force=[h])
    got = sim.t["state"].cpu().numpy()
    exact = _psi(s, v0, h, np.longdouble)
    rms = [float(np.sqrt(np.mean(np.square((v / exact - 1).astype(np.float64))))) for v in
           (_psi(s, v0, h, np.float64), _psi(s, v0, h, np.float64, True), got)]
    assert rms[1] > 1.2 * rms[0]   # the cells tell the two apart
    assert rms[2] <= 1.1 * rms[0], rms
