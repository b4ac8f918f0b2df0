"""Expectation-value plans of one-wire unitaries and affine permutations run in
a moving frame (csrc/frame.h).  Values and gradients against the CPU oracle,
which runs every gate: states of one tile (9 to 12 bits), the first sizes with
several tiles, odd and batched ones.

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
from oracle import sim_np as O
from tests.helpers import obs_records, to_records

pytestmark = pytest.mark.gpu
TOL = {torch.complex64: 1e-5, torch.complex128: 1e-10}


def _circuit(n, seed, n_gates):
    """Random rotations, fused constants, X, CX, SWAP; the last gates rotate."""

    def f(p):
        rng = np.random.default_rng(seed)
        k = 0
        for i in range(n_gates):
            w, v = (int(x) for x in rng.choice(n, 2, replace=False))
            kind = int(rng.integers(10)) if i < n_gates - n else 3
            if kind == 0:
                jq.PauliX(wires=w)
            elif kind == 1:
                jq.SWAP(wires=[w, v])
            elif kind == 2:
                jq.H(wires=w)
                jq.S(wires=w)
            elif kind == 3:
                jq.Rot(p[k], p[k + 1], p[k + 2], wires=w)
                k += 3
            elif kind == 4:
                jq.RZ(p[k], wires=w)  # a diagonal block
                k += 1
            elif kind == 5:
                jq.RX(p[k], wires=w)
                jq.PauliRot(p[k + 1], "Y", wires=[w])
                k += 2
            else:
                jq.CX(wires=[w, v])
        return k

    return f


def _plan(script, args, obs, n, dtype):
    lw = sim.lower_tape(script.record(*args), n)
    specs, okey = sim._lower_obs(obs, n)
    return sim.get_plan(lw, specs, okey, n, L.JQ_STATEVECTOR, dtype)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n,gates", [(9, 60), (10, 1), (11, 120), (12, 90), (13, 70), (14, 60), (17, 60)])
def test_frame_values_and_gradients(n, gates, dtype):
    body = _circuit(n, 10 * n + gates, gates)
    rng = np.random.default_rng(n)
    base = rng.uniform(0, 2 * np.pi, 3 * gates + 3)
    # exact quarter turns: the rotation's pivot and zero entries
    base[::5] = rng.integers(0, 5, base[::5].size) * (np.pi / 2)
    obs = [jq.PauliZ(0), jq.PauliZ(n - 1), jq.build_parity_observable([1, 4]),
           jq.build_parity_observable([0, 2, 5, 7, n - 1])]
    ct = rng.normal(size=len(obs))
    script = jq.Script(lambda p: body(p) and None, n_qubits=n)
    params = torch.tensor(base, requires_grad=True)
    ev = script.execute("expval", obs, args=(params,), dtype=dtype)
    (ev.to(torch.float64) @ torch.tensor(ct, device=ev.device)).backward()
    recs = to_records(script.record(torch.tensor(base)))
    ev_ref, g_ref = O.adjoint_grad(recs, n, obs_records(obs), ct=ct)
    np.testing.assert_allclose(ev.detach().cpu().numpy(), ev_ref, atol=TOL[dtype], rtol=0)
    np.testing.assert_allclose(params.grad.numpy()[: len(g_ref)], g_ref, atol=TOL[dtype] * max(1.0, np.abs(ct).sum()),
                               rtol=0)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n,batch", [(9, 3), (12, 5), (13, 2)])
def test_frame_batches_and_initial_states(n, batch, dtype):
    """Per-instance parameters (in_axes) and initial states, and the cotangent
    of the initial state, against the oracle instance by instance."""
    body = _circuit(n, n, 40)
    rng = np.random.default_rng(5 + n)
    base = rng.uniform(0, 2 * np.pi, (batch, 123))
    init = rng.normal(size=(batch, 2**n)) + 1j * rng.normal(size=(batch, 2**n))
    init /= np.linalg.norm(init, axis=1, keepdims=True)
    obs = [jq.PauliZ(w) for w in range(n)]
    script = jq.Script(lambda p: body(p) and None, n_qubits=n)
    params = torch.tensor(base, requires_grad=True)
    start = torch.tensor(init, requires_grad=True)
    ev = script.execute("expval", obs, args=(params,), in_axes=(0,), initial_state=start, dtype=dtype)
    for b in range(batch):
        recs = to_records(script.record(torch.tensor(base[b])))
        want = O.expval_state(O.simulate_pure(recs, n, init[b]), n, obs_records(obs))
        np.testing.assert_allclose(ev[b].detach().cpu().numpy(), want, atol=TOL[dtype], rtol=0)
    ev.sum().backward()
    # one parameter and one amplitude of the last instance by central differences
    h, b = 1e-5, batch - 1

    def total(p, s):
        return O.expval_state(O.simulate_pure(to_records(script.record(torch.tensor(p))), n, s), n,
                              obs_records(obs)).sum()

    for k in (0, 7):
        lo, hi = base[b].copy(), base[b].copy()
        lo[k] -= h
        hi[k] += h
        fd = (total(hi, init[b]) - total(lo, init[b])) / (2 * h)
        # the difference quotient is good to h^2 n and rounding / h
        np.testing.assert_allclose(params.grad[b, k].item(), fd, atol=TOL[dtype] * n + 1e-8)
    lo, hi = init[b].copy(), init[b].copy()
    lo[3] -= h
    hi[3] += h
    fd = (total(base[b], hi) - total(base[b], lo)) / (2 * h)
    np.testing.assert_allclose(start.grad[b, 3].real.item(), fd, atol=TOL[dtype] * n + 1e-8)


def test_frame_plans_run_fewer_passes():
    """CX rings cost no pass: the 16-qubit ring of 6 layers (96 gates in tiles of
    11 bits) takes fewer passes than layers x ceil(16 / 8)."""
    n, layers = 16, 6

    def circuit(p):
        for l in range(layers):
            for w in range(n):
                jq.Rot(p[l, w, 0], p[l, w, 1], p[l, w, 2], wires=w)
            for w in range(n):
                jq.CX(wires=[w, (w + 1) % n])

    script = jq.Script(circuit, n_qubits=n)
    plan = _plan(script, (torch.zeros(layers, n, 3),), [jq.PauliZ(0)], n, torch.complex64)
    assert plan.info["n_passes_fwd"] < 2 * layers
    assert plan.info["n_tile_ops_fwd"] == n * layers


# ---- noisy circuits on Pauli coefficients (csrc/pauli.cu) --------------------
def _noisy(n, seed, layers, p):
    """Rotations, constants and every one-qubit channel on each wire, X, CX and
    SWAP between them; returns the number of parameters used."""
    rng = np.random.default_rng(seed)
    k = 0
    for _ in range(layers):
        for w in range(n):
            kind = int(rng.integers(7))
            jq.Rot(p[k], p[k + 1], p[k + 2], wires=w)
            k += 3
            if kind == 0:
                jq.DepolarizingChannel(0.03, wires=w)
            elif kind == 1:
                jq.AmplitudeDamping(0.05, wires=w)
            elif kind == 2:
                jq.RX(p[k], wires=w)
                k += 1
                jq.ThermalRelaxationError(0.1, 3.0, 2.0, 0.4, wires=w)
            elif kind == 3:
                jq.H(wires=w)
                jq.BitFlip(0.04, wires=w)
            elif kind == 4:
                jq.RZ(p[k], wires=w)
                k += 1
                jq.PhaseDamping(0.06, wires=w)
        for _ in range(n):
            w, v = (int(x) for x in rng.choice(n, 2, replace=False))
            kind = int(rng.integers(6))
            if kind == 0:
                jq.SWAP(wires=[w, v])
            elif kind == 1:
                jq.PauliX(wires=w)
            else:
                jq.CX(wires=[w, v])
            if kind == 2:
                jq.RZ(p[k], wires=v)  # a diagonal block of its own
                k += 1
            elif kind == 3:
                jq.PhaseFlip(0.05, wires=w)
    return k


def _words(n):
    y = np.array([[0, -1j], [1j, 0]])
    z = np.diag([1.0, -1.0])
    x = np.array([[0, 1.0], [1.0, 0]])
    return [jq.PauliZ(0), jq.PauliX(n - 1), jq.PauliY(1), jq.build_parity_observable([0, n - 1]),
            jq.Hermitian(np.kron(y, np.kron(x, y)), wires=[0, 2, 3], record=False),
            jq.Hermitian(0.5 * np.kron(y, z), wires=[1, n - 1], record=False)]


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n,layers", [(5, 1), (5, 6), (6, 3)])
def test_pauli_basis_values_and_gradients(n, layers, dtype):
    """Values of X, Y, Z and mixed words against the oracle, angle gradients
    against its central differences."""
    rng = np.random.default_rng(n + layers)
    base = rng.uniform(0, 2 * np.pi, 8 * n * layers)
    base[::4] = rng.integers(0, 5, base[::4].size) * (np.pi / 2)
    script = jq.Script(lambda p: _noisy(n, 7 * n + layers, layers, p) and None, n_qubits=n)
    obs = _words(n)
    ct = rng.normal(size=len(obs))
    params = torch.tensor(base, requires_grad=True)
    ev = script.execute("expval", obs, args=(params,), dtype=dtype)

    def reference(b):
        recs = to_records(script.record(torch.tensor(b)))
        return O.expval_density(O.simulate_mixed(recs, n), n, obs_records(obs))

    np.testing.assert_allclose(ev.detach().cpu().numpy(), reference(base), atol=TOL[dtype], rtol=0)
    (ev.to(torch.float64) @ torch.tensor(ct, device=ev.device)).backward()
    h = 1e-5
    used = np.flatnonzero(params.grad.numpy())
    for k in rng.choice(used, 6, replace=False):
        lo, hi = base.copy(), base.copy()
        lo[k] -= h
        hi[k] += h
        fd = ((reference(hi) - reference(lo)) / (2 * h)) @ ct
        np.testing.assert_allclose(params.grad[k].item(), fd, atol=TOL[dtype] * n + 1e-8)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n,layers,batch", [(6, 2, 5), (7, 3, 3), (9, 2, 1)])
def test_pauli_basis_against_the_general_passes(n, layers, batch, dtype):
    """The same circuit with an explicit |0..0> start runs the general passes:
    values and every gradient, batched; coarse and fine checkpoints alike."""
    rng = np.random.default_rng(n)
    base = torch.tensor(rng.uniform(0, 2 * np.pi, (batch, 8 * n * layers)))
    script = jq.Script(lambda p: _noisy(n, n, layers, p) and None, n_qubits=n)
    obs = [jq.PauliZ(w) for w in range(n)] + [jq.PauliY(1)]
    zero = torch.zeros(2**n, dtype=dtype)
    zero[0] = 1
    got = []
    for init in (None, zero):
        params = base.clone().requires_grad_(True)
        ev = script.execute("expval", obs, args=(params,), in_axes=(0,), initial_state=init, dtype=dtype)
        ev.sum().backward()
        got.append((ev.detach().cpu().numpy(), params.grad.numpy()))
    np.testing.assert_allclose(got[0][0], got[1][0], atol=TOL[dtype], rtol=0)
    np.testing.assert_allclose(got[0][1], got[1][1], atol=TOL[dtype] * n, rtol=0)


def test_pauli_basis_checkpoint_levels():
    """A long circuit in a workspace that cannot keep every pass input: the
    segments recomputed from checkpoints give the gradient of the short form."""
    from jaqsi_b200 import _lib as lib

    n, layers = 11, 4
    rng = np.random.default_rng(1)
    base = torch.tensor(rng.uniform(0, 2 * np.pi, 8 * n * layers))
    script = jq.Script(lambda p: _noisy(n, 3, layers, p) and None, n_qubits=n)
    obs = [jq.PauliZ(0), jq.PauliX(4)]
    params = base.clone().requires_grad_(True)
    ev = script.execute("expval", obs, args=(params,), dtype=torch.complex64)
    ev.sum().backward()
    again = base.clone().requires_grad_(True)
    zero = torch.zeros(2**n, dtype=torch.complex64)
    zero[0] = 1
    ev2 = script.execute("expval", obs, args=(again,), initial_state=zero, dtype=torch.complex64)
    ev2.sum().backward()
    assert lib is not None
    np.testing.assert_allclose(ev.detach().cpu().numpy(), ev2.detach().cpu().numpy(), atol=1e-5, rtol=0)
    np.testing.assert_allclose(params.grad.numpy(), again.grad.numpy(), atol=1e-5 * n, rtol=0)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n", [9, 10, 11, 12, 13])
@pytest.mark.parametrize("frame", [True, False])
def test_seed_of_many_z_strings(n, frame, dtype):
    """The reverse pass's seed over Z strings: the smallest sizes of both thread
    widths, more words than one load holds, zero cotangents, and an instance
    whose cotangents are all zero."""
    gates, rng = 30, np.random.default_rng(100 + n)
    inner = _circuit(n, 7 * n, gates)

    def body(p):
        if not frame:
            jq.CRX(p[-1], wires=[0, n - 1])
        inner(p)

    base = rng.uniform(0, 2 * np.pi, (2, 3 * gates + 4))
    obs = [jq.PauliZ(w) for w in range(n)]
    obs += [jq.build_parity_observable([a, b]) for a in range(n) for b in range(a + 1, n)]
    ct = rng.normal(size=(2, len(obs)))
    ct[0, ::3] = 0.0
    ct[1] = 0.0
    script = jq.Script(lambda p: body(p) and None, n_qubits=n)
    params = torch.tensor(base, requires_grad=True)
    ev = script.execute("expval", obs, args=(params,), in_axes=(0,), dtype=dtype)
    (ev.to(torch.float64) * torch.tensor(ct, device=ev.device)).sum().backward()
    _, ref = O.adjoint_grad(to_records(script.record(torch.tensor(base[0]))), n, obs_records(obs), ct=ct[0])
    got = params.grad[0].numpy()
    if not frame:  # recorded first, held last
        got = np.concatenate([got[-1:], got[:-1]])
    np.testing.assert_allclose(got[: len(ref)], ref, atol=TOL[dtype] * np.abs(ct[0]).sum(), rtol=0)
    assert not params.grad[1].any()


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n", [9, 13])
def test_other_calls_of_a_frame_plan_run_the_circuit(n, dtype):
    """A plan that absorbed nothing also answers for states and probabilities and
    takes jq_backward: these run the circuit itself.  With expval_only = 1 the
    state buffer of an expectation value is the final state."""
    body = _circuit(n, 3 * n, 50)
    base = np.random.default_rng(n).uniform(0, 2 * np.pi, 153)
    obs = [jq.PauliZ(w) for w in range(n)]
    script = jq.Script(lambda p: body(p) and None, n_qubits=n)
    recs = to_records(script.record(torch.tensor(base)))
    lw = sim.lower_tape(script.record(torch.tensor(base)), n)
    specs, okey = sim._lower_obs(obs, n)
    angles = torch.tensor([float(a) for a in lw.angles], dtype=torch.float64, device="cuda")
    statics = [st[:10] + (1,) + st[11:] if st[3] >= 0 else st for st in lw.statics]  # every angle trainable
    psi = O.simulate_pure(recs, n)
    ev_ref, g_ref = O.adjoint_grad(recs, n, obs_records(obs), ct=np.ones(n))

    def call(plan, out_type):
        state, out = sim._forward_launch(plan, out_type, 1, 0, angles, None, None)
        return state[0].cpu().numpy(), None if out is None else out[0].cpu().numpy()

    plain = sim.Plan(statics, specs, n, L.JQ_STATEVECTOR, dtype, {"expval_only": 1})
    state, ev = call(plain, L.JQ_OUT_EXPVAL)
    np.testing.assert_allclose(state, psi, atol=TOL[dtype], rtol=0)
    np.testing.assert_allclose(ev, ev_ref, atol=TOL[dtype], rtol=0)
    plan = sim.Plan(statics, specs, n, L.JQ_STATEVECTOR, dtype, {"expval_only": 2})
    np.testing.assert_allclose(call(plan, L.JQ_OUT_EXPVAL)[1], ev_ref, atol=TOL[dtype], rtol=0)
    np.testing.assert_allclose(call(plan, L.JQ_OUT_STATE)[0], psi, atol=TOL[dtype], rtol=0)
    np.testing.assert_allclose(call(plan, L.JQ_OUT_PROBS)[1], np.abs(psi) ** 2, atol=TOL[dtype], rtol=0)
    grad = torch.empty((1, len(lw.angles)), dtype=torch.float64, device="cuda")
    ct = torch.ones((1, n), dtype=torch.float64, device="cuda")
    wsb = plan.workspace_bytes(1, 2)
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    L.check(plan._lib.jq_backward(plan.handle, 1, sim._ptr(angles), None, None, 0, L.JQ_OUT_EXPVAL, sim._ptr(ct), None,
                                  sim._ptr(grad), None, None, sim._ptr(ws), wsb, sim._stream()))
    np.testing.assert_allclose(grad[0].cpu().numpy(), g_ref, atol=TOL[dtype] * n, rtol=0)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n", [9, 12, 13])
@pytest.mark.parametrize("gates", [0, 1])
def test_frame_runs_that_start_at_zero(n, gates, dtype):
    """The first pass writes the start state: of no gate (no pass), of one, and
    over memory that holds something else."""
    torch.full((1 << 22,), float("nan"), device="cuda")  # freed at once: the call's buffers land on it

    def body(p):
        jq.PauliX(wires=n - 1)
        jq.CX(wires=[n - 1, 0])
        if gates:
            jq.RX(p[0], wires=0)
            jq.CX(wires=[0, 3])

    base = np.array([0.7])
    obs = [jq.PauliZ(w) for w in range(n)]
    script = jq.Script(lambda p: body(p) and None, n_qubits=n)
    params = torch.tensor(base, requires_grad=True)
    ev = script.execute("expval", obs, args=(params,), dtype=dtype)
    want = O.expval_state(O.simulate_pure(to_records(script.record(torch.tensor(base))), n), n, obs_records(obs))
    np.testing.assert_allclose(ev.detach().cpu().numpy(), want, atol=TOL[dtype], rtol=0)
    if gates:
        ev.sum().backward()
        _, g = O.adjoint_grad(to_records(script.record(torch.tensor(base))), n, obs_records(obs), ct=np.ones(n))
        np.testing.assert_allclose(params.grad.numpy(), g, atol=TOL[dtype] * n, rtol=0)
