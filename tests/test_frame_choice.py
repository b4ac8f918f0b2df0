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


def _staircase(n, layers):
    """A CX after every rotation: each gate waits for the one on the wire before."""

    def circuit():
        for l in range(layers):
            for w in range(n):
                jq.Rot(0.1, 0.2 + l, 0.3, wires=w)
                if w + 1 < n:
                    jq.CX(wires=[w, w + 1])

    return circuit


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_staircases_run_in_the_frame_up_to_18_qubits(dtype):
    z = [jq.PauliZ(0)]
    for n in (9, 12, 14, 16, 17):
        assert _own(_staircase(n, 4), n, z, dtype), n
    assert _own(_staircase(18, 12), 18, z, torch.complex64)
    for n in (19, 20, 22, 24):
        assert not _own(_staircase(n, 12), n, z, dtype), n
        assert not _own(_staircase(n, 4), n, z, dtype), n


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


@pytest.mark.parametrize("off", [4e-16, 1e-13, 1e-9])
def test_constants_that_are_not_exact_keep_their_modulus(off):
    """The frame divides by a gate's modulus and the Pauli basis keeps the trace: a
    constant that is further off than rounding runs the general passes, which
    apply it as it is (complex64: than 1e-12)."""
    scale = 1.0 + off

    class Scaled(jq.Operation):
        _matrix = scale * np.array([[1, 1], [1, -1]], dtype=np.complex128) / np.sqrt(2)
        _num_wires = 1
        is_unitary = True

    def pure():
        for l in range(3):
            for w in range(9):
                jq.RX(0.1, wires=w)
                Scaled(wires=w)
                jq.CX(wires=[w, (w + 1) % 9])

    def noisy():
        for l in range(3):
            for w in range(6):
                jq.RX(0.1, wires=w)
                jq.QubitChannel([scale * np.sqrt(0.9) * np.eye(2), scale * np.sqrt(0.1) * np.diag([1.0, -1.0])], wires=w)
                jq.CX(wires=[w, (w + 1) % 6])

    z = [jq.PauliZ(0)]
    for circuit, n in ((pure, 9), (noisy, 6)):
        assert _own(circuit, n, z, torch.complex128) == (off < 1e-15)
        assert _own(circuit, n, z, torch.complex64) == (off < 1e-12)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_computed_constants_count_as_exact(dtype):
    """Random channels of the library and Kraus sets from QR factors."""
    rng = np.random.default_rng(7)

    def noisy():
        for _ in range(40):
            for w in range(6):
                jq.RX(0.1, wires=w)
                p = rng.uniform(0, 0.3)
                jq.DepolarizingChannel(p, wires=w)
                jq.AmplitudeDamping(p, wires=w)
                jq.ThermalRelaxationError(rng.uniform(0, 0.5), rng.uniform(1, 5), rng.uniform(0.5, 2), rng.uniform(0, 2), wires=w)
                q, _ = np.linalg.qr(rng.normal(size=(4, 2)) + 1j * rng.normal(size=(4, 2)))
                jq.QubitChannel([q[:2], q[2:]], wires=w)
                jq.CX(wires=[w, (w + 1) % 6])

    assert _own(noisy, 6, [jq.PauliZ(0)], dtype)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_circuits_and_sizes_outside_the_rules(dtype):
    def ring(n, extra=None, noise=False):
        def circuit():
            for l in range(3):
                for w in range(n):
                    jq.Rot(0.1, 0.2, 0.3 + l, wires=w)
                    if noise:
                        jq.DepolarizingChannel(0.1, wires=w)
                for w in range(n):
                    jq.CX(wires=[w, (w + 1) % n])
                if extra:
                    extra()
                    jq.RX(0.2, wires=0)

        return circuit

    z = [jq.PauliZ(0), jq.build_parity_observable([1, 3])]
    assert _own(ring(9), 9, z, dtype) and not _own(ring(8), 8, z, dtype)
    assert _own(ring(5, noise=True), 5, z, dtype) and not _own(ring(4, noise=True), 4, z, dtype)
    for extra in (lambda: jq.CRX(0.3, wires=[0, 2]), lambda: jq.CZ(wires=[0, 1]), lambda: jq.RZZ(0.3, wires=[1, 2]),
                  lambda: jq.CCX(wires=[0, 1, 2])):
        assert not _own(ring(9, extra), 9, z, dtype)
        assert not _own(ring(5, extra, True), 5, z, dtype)
    assert not _own(ring(9), 9, [jq.PauliX(0)], dtype)
    dense = jq.Hermitian(np.array([[1, 0.5], [0.5, 2.0]]), wires=[1], record=False)
    assert not _own(ring(9), 9, [dense], dtype) and not _own(ring(5, noise=True), 5, [dense], dtype)
    assert _own(ring(5, noise=True), 5, [jq.PauliX(0), jq.PauliY(3)], dtype)
    for tune in ({"jit": -1}, {"tile_bits": 10}, {"threads": 256}):
        assert not _own(ring(9), 9, z, dtype, tune) and not _own(ring(5, noise=True), 5, z, dtype, tune)
