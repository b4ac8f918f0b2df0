"""Which plans run in the moving frame or on Pauli coefficients, from the plan's
summary: it differs from that of the general passes (``expval_only = 1``), which
also count permutations as operations."""
import numpy as np
import pytest
import torch

import jaqsi_b200 as jq
from jaqsi_b200 import _lib as L
from jaqsi_b200 import simulation as sim
from jaqsi_b200 import workloads as wl


def _infos(circuit, n, obs, dtype=torch.complex64, tune=None):
    with jq.recording() as tape:
        circuit()
    lw = sim.lower_tape(tape, n)
    specs, _ = sim._lower_obs(obs, n)
    mode = L.JQ_DENSITY if sim.has_noise(tape) else L.JQ_STATEVECTOR
    return [sim.Plan(lw.statics, specs, n, mode, dtype, dict(tune or {}, expval_only=e)).info for e in (1, 2)]


def _own(circuit, n, obs, dtype=torch.complex64, tune=None):
    general, chosen = _infos(circuit, n, obs, dtype, tune)
    return general != chosen


def _wires(n, layers, count, control=True):
    """Layers of rotations and a CX ring on `count` wires out of n."""

    def circuit():
        ws = [int(x) for x in np.linspace(0, n - 1, count).round()]
        for l in range(layers):
            for w in ws:
                jq.Rot(0.1, 0.2 + l, 0.3, wires=w)
            for i in range(count):
                jq.CX(wires=[ws[i], ws[(i + 1) % count]])

    return circuit


def _serial(n, layers):
    """Gates that each wait for the one before."""

    def circuit():
        for l in range(layers):
            for w, v in ((0, n - 1), (n - 1, 0)):
                jq.Rot(0.1, 0.2 + l, 0.3, wires=w)
                jq.CX(wires=[w, v])

    return circuit


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_deep_circuits_on_few_wires_keep_the_specialised_passes(dtype):
    z = [jq.PauliZ(0)]
    for n in (20, 22, 24):
        assert not _own(_wires(n, 50, 2), n, z, dtype)
        assert not _own(_serial(n, 8), n, z, dtype)
        assert _own(_wires(n, 2, 2), n, z, dtype)
        assert _own(_wires(n, 50, 3), n, z, dtype)
    assert not _own(_serial(17, 50), 17, z, dtype)
    assert _own(_wires(17, 50, 2), 17, z, dtype)
    # below 2^16 amplitudes the general passes are interpreted
    assert _own(_serial(12, 50), 12, z, dtype) and _own(_wires(15, 50, 2), 15, z, dtype)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("family", [wl.sweep_ansatz, wl.strongly_entangling, wl.rot_ring])
def test_circuits_on_every_wire_run_in_the_frame(family, dtype):
    for n in list(range(9, 25, 3)) + [16, 17, 19, 20, 22, 23]:
        for layers in (2, 5, 20):
            a = np.full((layers, n, 3), 0.1)
            assert _own(lambda: family(n, layers, a), n, [jq.PauliZ(w) for w in range(n)], dtype), (n, layers)


def _noisy(n, layers):
    return lambda: wl.noisy_ansatz(n, layers, np.full((layers, n, 3), 0.1), 0.01, 0.005)


def _workspaces(circuit, n, dtype, batch, with_grad):
    with jq.recording() as tape:
        circuit()
    lw = sim.lower_tape(tape, n)
    specs, _ = sim._lower_obs([jq.PauliZ(0)], n)
    return [sim.Plan(lw.statics, specs, n, L.JQ_DENSITY, dtype, {"expval_only": e}).workspace_bytes(batch, with_grad)
            for e in (1, 2)]


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n,layers,batch", [(7, 40, 1), (9, 20, 3), (12, 8, 1), (15, 2, 1), (15, 8, 1)])
def test_reverse_call_on_pauli_coefficients_needs_no_more_than_the_general_one(n, layers, batch, dtype):
    """The least jq_backward takes is what the general passes take: 15 qubits with 8
    layers fit one GPU in complex64 (17 states of 8.6 GB) as they did without the
    coefficients.  With room for more it is half as much again at most."""
    general, own = _workspaces(_noisy(n, layers), n, dtype, batch, 2)
    assert own == general
    roomy = _workspaces(_noisy(n, layers), n, dtype, batch, 3)
    assert roomy[0] == general
    assert general <= roomy[1] <= max(1.5 * general, general + (256 << 20))
