"""3-D right-hand sides at the long padded lengths, each with its own plans, tiles and shared memory.

A right-hand side does not depend on the padded length once every product of two retained modes fits
(M >= 2 N + 2), so the oracle runs on a small padded grid and the solver on the long one.  Tolerances:
FP64 the parity tolerance, FP32 ten roundings (6e-8) for each of the log2(M) levels of both transforms.
"""

import math

import numpy as np
import pytest
import torch

import azeban_b200 as az
from oracle import euler_oracle as ora
from tests.gpu_helpers import VISC_CFGS, random_field_hat, rel_l2, to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("N,M,batch,M_oracle", [(8, 192, 2, 18), (10, 256, 1, 24), (100, 256, 1, 216), (8, 384, 1, 18),
                                                (8, 512, 2, 18), (100, 512, 1, 216), (8, 768, 1, 18), (40, 768, 1, 96),
                                                (8, 1024, 1, 18), (24, 1024, 1, 54), (8, 1536, 1, 18)])
def test_3d_long_lengths(N, M, batch, M_oracle, prec):
    og, g = ora.Grid(3, N, M_oracle), az.Grid(3, N, M)
    fields = [random_field_hat(3, N, seed=70 + N + b) for b in range(batch)]
    eq = az.IncompressibleEuler(g, az.make_viscosity(VISC_CFGS["smooth"], g), prec, batch)
    u = to_dev(np.stack(fields), prec)
    out = torch.empty_like(u)
    eq.dudt(out, u)
    got = to_host(out)
    tol = 1e-12 if prec == "f64" else 10 * 6e-8 * 2 * math.log2(M)
    for b in range(batch):
        oeq = ora.IncompressibleEuler(og, ora.make_viscosity(VISC_CFGS["smooth"], og))
        assert rel_l2(got[b], oeq.dudt(fields[b])) <= tol, b
