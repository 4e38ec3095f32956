"""The third-order vertical fluxes divide by 12 in two operations
(dycore_kernels.cuh: div12_wide, div12_any): the same words as IEEE division.

The two operations are restated in NumPy here, and swept over every mantissa of
both signs at the exponents that can differ: while x RL, x RH and the quotient
are normal numbers (biased exponent 29 and up) every operation scales with the
power of two, so one exponent stands for all; below, the rounding of x RL is at
most 2^-150, which is the largest part of a step of the quotient, 1/32, at the
smallest exponent that the form serves (9), and half of that at each above.
Both ends of that range and exponents between are swept, and the top.  The
64-bit form is swept where it is used, over the subnormal and smallest normal
numbers.  On the GPU the step itself is compared with the oracle, with tracers
in the range where the two-operation form does not hold.
"""

import numpy as np
import pytest

F32 = np.float32
RH = np.array(0x3DAAAAAA, dtype=np.uint32).view(F32)[()]
RL = np.array(0x31AAAAAB, dtype=np.uint32).view(F32)[()]
SMALL = np.array(0x04800000, dtype=np.uint32).view(F32)[()]


def wide(x):
    """fma(x, RH, x RL).  x RH is exact in 64 bits (48 bits) and so nearly is
    the sum: its rounding boundaries in 32 bits lie 1/6 ulp away."""
    with np.errstate(over="ignore", invalid="ignore", under="ignore"):
        low = (x * RL).astype(F32)
        return (x.astype(np.float64) * np.float64(RH) + low.astype(np.float64)).astype(F32)


def any_range(x):
    with np.errstate(over="ignore", invalid="ignore", under="ignore"):
        return (x.astype(np.float64) * (1.0 / 12.0)).astype(F32)


def quotient(x):
    with np.errstate(over="ignore", invalid="ignore", under="ignore"):
        return (x / F32(12.0)).astype(F32)


def same(a, b):
    nan = np.isnan(a) & np.isnan(b)
    return np.array_equal(a.view(np.uint32)[~nan], b.view(np.uint32)[~nan])


@pytest.mark.parametrize("sign", [0, 1])
@pytest.mark.parametrize("exponent", [9, 10, 11, 13, 17, 29, 30, 64, 127, 250, 254])
def test_two_operations_divide_every_mantissa(exponent, sign):
    mantissa = np.arange(1 << 23, dtype=np.uint32)
    x = (np.uint32(sign << 31 | exponent << 23) | mantissa).view(F32)
    assert np.abs(x[0]) >= SMALL
    assert same(wide(x), quotient(x))


@pytest.mark.parametrize("sign", [0, 1])
@pytest.mark.parametrize("exponent", range(9))
def test_64_bit_form_divides_every_small_mantissa(exponent, sign):
    mantissa = np.arange(1 << 23, dtype=np.uint32)
    x = (np.uint32(sign << 31 | exponent << 23) | mantissa).view(F32)
    assert np.abs(x[-1]) < SMALL
    assert same(any_range(x), quotient(x))


def test_zeros_infinities_and_nan():
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan], dtype=F32)
    for f in (wide, any_range):
        assert same(f(x), quotient(x))


@pytest.mark.gpu
@pytest.mark.parametrize("levels", [4, 9, 12])
@pytest.mark.parametrize("scale", [1e-30, 1e-36, 1e-41])
def test_step_with_tiny_tracers_equals_the_oracle(levels, scale):
    import hexdyn
    from fixtures import differing_words
    from hexdyn.case import build_case, case_arrays
    from hexdyn.config import DycoreConfig
    from hexdyn.mesh import build_mesh
    from oracle.dycore import OracleConfig, OracleDycore, State

    mesh = build_mesh(2, lloyd=2, seed=0)
    case = build_case(mesh, n_levels=levels, seed=0, n_condensates=1)
    case.scalars[:] = (case.scalars.astype(np.float64) * (scale / case.scalars.max())).astype(F32)
    case.scalars[1, :, ::3] = 0.0
    oracle = OracleDycore(case_arrays(case), OracleConfig(dt=600.0, n_sub_steps=2, moist="native"))
    drv = hexdyn.from_case(case, DycoreConfig(config_dt=600.0, config_number_of_sub_steps=2,
                                              moist_coefficients="native"))
    state, side = State(case.rho, case.rho_theta, case.rho_u, case.rho_w, case.scalars), None
    for _ in range(2):
        state, side = oracle.step(state, side)
        got = drv.step().state
        for name in ("rho", "rho_u", "rho_w", "scalars"):
            assert differing_words(getattr(got, name), getattr(state, name)) == 0, (levels, scale, name)
    drv.close()
