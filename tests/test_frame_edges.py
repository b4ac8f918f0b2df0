"""Edges of the frame and Pauli plans (csrc/frame.h): inputs and sizes at which
they branch, against the general passes (an explicit |0..0> start or
``expval_only = 1``), against single calls, or against the oracle.

Tolerances, set before the first run, are those of the other parity tests:
1e-10 (complex128) and 1e-5 (complex64), absolute, times the weight of the
cotangents.
"""
import numpy as np
import pytest
import torch

import jaqsi_b200 as jq
from jaqsi_b200 import _lib as L
from jaqsi_b200 import simulation as sim

pytestmark = pytest.mark.gpu
TOL = {torch.complex64: 1e-5, torch.complex128: 1e-10}


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n", [5, 6])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("gate", [jq.RZ, jq.RY])
def test_noisy_values_of_an_angle_that_is_not_finite(n, bad, gate, dtype):
    """One such angle leaves the density matrix without a finite entry: every
    value and every gradient of its sample is NaN, those of the others are not."""

    def circuit(p):
        gate(p[0], wires=0)
        for w in range(1, n):
            jq.RY(p[w], wires=w)
        jq.DepolarizingChannel(0.1, wires=1)

    params = torch.full((3, n), 0.3, dtype=torch.float64)
    params[1, 0] = bad
    params.requires_grad_(True)
    script = jq.Script(circuit, n_qubits=n)
    ev = script.execute("expval", [jq.PauliZ(w) for w in range(n)], args=(params,), in_axes=(0,), dtype=dtype)
    ev.sum().backward()
    assert torch.isnan(ev[1]).all() and torch.isnan(params.grad[1]).all()
    assert torch.isfinite(ev[[0, 2]]).all() and torch.isfinite(params.grad[[0, 2]]).all()
    assert torch.equal(ev[0], ev[2])
