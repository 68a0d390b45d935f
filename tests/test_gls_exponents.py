"""The GLS corrector's powers: exponents that are multiples of 1/2 (products and a square root, up to
8), others (pow), either sign of n, and the shortest and longest columns, against the oracle within the
tolerance of the other FP64 comparisons (1e-9)."""
import numpy as np
import pytest

import gls_oracle as go
from gls_case import make
from test_gls import FIELDS, gpu_run, run_oracle

CASES = [(3.0, 1.5, -1.0, 5), (-1.0, 0.5, -1.0, 6), (2.0, 1.0, -0.67, 64), (2.0, 1.3, -0.7, 7), (1.0, 2.0, 0.5, 9),
         (0.0, 1.25, 0.75, 10), (1.5, 8.5, -2.0, 12), (3.0, 8.0, -0.5, 11)]


@pytest.mark.gpu
@pytest.mark.parametrize("p,m,n,N", CASES)
def test_exponents_match_oracle(p, m, n, N):
    P = dict(go.DEFAULT, p=p, m=m, n=n, Pmin=1e-60)
    c = make(N=N, seed=N)
    c["gls"] = P["cmu0"] ** p * c["tke"] ** m * c["Lscale"] ** n
    ref = dict(zip(FIELDS, run_oracle(c, P=P)))
    got = gpu_run(c, "fp64", preset=P)
    for k in FIELDS:
        np.testing.assert_allclose(got[k], ref[k], rtol=1e-9, atol=0, err_msg=k)


@pytest.mark.gpu
@pytest.mark.parametrize("N", [5, 8, 9, 64])
def test_k_epsilon_constants_match_oracle(N):
    """The default model's own variant: remainders of the level chunks, the shortest and longest column."""
    c = make(N=N, seed=20 + N)
    ref = dict(zip(FIELDS, run_oracle(c)))
    got = gpu_run(c, "fp64")
    for k in FIELDS:
        np.testing.assert_allclose(got[k], ref[k], rtol=1e-9, atol=0, err_msg=k)
