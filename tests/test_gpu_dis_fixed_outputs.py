"""The mixed fixed-Sobol path keeps its outputs: values and errors of I1, I2, I3 and their sum.

The error is the spread of replicates, and FP32 rounding of I1's cancelling parts sets its leading
digits, so another order of operations in the integrand is another error (by 1e-4 of it).  The
numbers are those of the lane-per-sample evaluation on a B200, 13 digits of them; the same operations
in the same order give the same bits, and 1e-9 leaves room for the digits alone."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

# (Q^2, quark mass, Qs0^2, polarisation, seed): values, errors
OUTPUTS = {
    (9.0, 1.4, 1.0, "T", 0):
        ((3.996703938368e-01, -8.676860657179e-02, 4.839939878743e-02, 3.613011860524e-01),
         (3.732914530763e-03, 2.164535964830e-04, 9.715109132320e-05, 3.717856607702e-03)),
    (9.0, 1.4, 1.0, "L", 0):
        ((1.020262145287e-01, -2.441794045934e-02, 9.426589283545e-03, 8.703486335288e-02),
         (5.268995339635e-04, 2.142249474616e-05, 9.550924034379e-06, 5.318657851539e-04)),
    (9.0, 1.4, 0.7, "L", 3):
        ((9.435864776710e-02, -2.238992816973e-02, 8.577771985516e-03, 8.054649158288e-02),
         (4.070182525623e-04, 2.390192032056e-05, 1.124631784755e-05, 4.091054962987e-04)),
    (4.0, 0.14, 0.9, "T", 5):
        ((-2.506183191838e-01, 3.542836501653e-03, 8.109925600072e-03, -2.389655570821e-01),
         (6.575207236098e-03, 1.891340427321e-05, 1.241557952067e-05, 6.581064136794e-03)),
    (4.0, 0.14, 1.3, "L", 5):
        ((1.067699395378e-01, -5.478803953597e-03, 3.681061725277e-03, 1.049721973095e-01),
         (3.567322218936e-03, 3.329471327613e-06, 2.770232054871e-06, 3.566872657165e-03)),
    (25.0, 1.4, 1.2, "T", 8):
        ((3.599995542107e-01, -4.692018221376e-02, 2.969758876753e-02, 3.427769607644e-01),
         (4.084388742137e-03, 1.464773957032e-04, 6.381268114905e-05, 4.034714442579e-03)),
}


@pytest.mark.parametrize("case", list(OUTPUTS))
def test_outputs(case):
    from nlo_bk_optimized_b200.dipole import GBW
    from nlo_bk_optimized_b200.dis import DISConfig, Polarization, Quark, QuarkType
    from nlo_bk_optimized_b200.dis.fixed_sobol import gbw_qg_fixed_sobol

    q2, mass, qs0sqr, pol, seed = case
    quark = Quark(QuarkType.C, mass)
    config = DISConfig(maxr=5.0, nf_alphas=1, quarks=(quark,))
    dipole = GBW(Qs0sqr=qs0sqr, lambda_=0.3, gamma=1.0, x0=1.0)
    q2, xbj = torch.tensor(q2, dtype=torch.float32), torch.tensor(1e-3, dtype=torch.float32)
    got = gbw_qg_fixed_sobol(q2, xbj, Polarization[pol], quark, dipole, config, seed=seed)
    parts = (*got.contributions, got.total)
    values, errors = OUTPUTS[case]
    assert [float(p.value) for p in parts] == pytest.approx(values, rel=1e-9)
    assert [float(p.error) for p in parts] == pytest.approx(errors, rel=1e-9)
